"""GPU: the fused decode-batch forward (products of x in one launch, cluster routing, combined down products) and the
one-call block against the same layer run stage by stage and plain fp32 products."""
import pytest
import torch

from bitsmoe_b200 import capi, synth
from bitsmoe_b200.layer import route_build, route_topk
from tests import helpers

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(E, k, H=256, I=128, r=64, shared=0, seed=5):
    cfg = synth.tiny(hidden=H, num_experts=E, intermediate=I, top_k=k, rank=r, shared_intermediate=shared, shared_gated=shared > 0)
    s = synth.make_layer(cfg, seed=seed, device=DEV)
    return cfg, s, synth.to_packed_layer(s)


def _staged(layer, x, logits, k, dtype, E):
    idx, w = route_topk(logits, k, True, dtype)
    tok, off, rw, _, _ = route_build(idx, w, E)
    hg, hu = layer.basis_project(x)
    return layer.combine_down_basis(layer.experts_forward(hg, hu, tok, off, rw), torch.float32)


# token counts around the 8-token MMA block, the 64-token chunk, the 32-bit mask word and the largest decode batch;
# expert counts around the register classes of the top-k
@pytest.mark.parametrize("T", [1, 7, 9, 32, 33, 64, 65, 255, 256])
@pytest.mark.parametrize("E,k", [(5, 5), (64, 6), (65, 8), (300, 10), (512, 10)])
def test_fused_forward_matches_stages(T, E, k):
    cfg, s, layer = _layer(E, k)
    x = synth.activations(cfg, T, seed=T, device=DEV, dtype=torch.bfloat16)
    logits = synth.router_logits(cfg, T, seed=T + 1, device=DEV)
    y = layer.forward(x, logits, k, True, torch.bfloat16)
    helpers.assert_close(y.cpu(), _staged(layer, x, logits, k, torch.bfloat16, E).cpu(), what=f"T={T} E={E}")


# passes of 16: assignments per expert around one and two passes and none at all, on average more than eight; few units, cut along
# the tiles, and more than one per CTA; ranks whose row slots are an odd number of pairs, are not whole octets, or pass 256
@pytest.mark.parametrize("rank,inter", [(64, 256), (80, 128), (256, 384), (328, 128)])
@pytest.mark.parametrize("E", [5, 400])
def test_passes_of_sixteen_match_generic_kernel(rank, inter, E):
    counts = [(15, 0, 16, 17, 33, 1, 32, 8)[e % 8] for e in range(E)]
    T = 64
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=inter, top_k=1, rank=rank)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=rank, device=DEV))
    gen = torch.Generator(device=DEV).manual_seed(E)
    tok = torch.cat([torch.sort(torch.randperm(T, generator=gen, device=DEV)[:c]).values for c in counts]).to(torch.int32)
    off = torch.zeros(E + 1, dtype=torch.int32, device=DEV)
    off[1:] = torch.tensor(counts, device=DEV).cumsum(0)
    rw = torch.rand(tok.numel(), generator=gen, device=DEV)
    hg, hu = layer.basis_project(synth.activations(cfg, T, seed=2, device=DEV, dtype=torch.bfloat16))
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    nan = torch.full_like(hg, float("nan"))
    layer.experts_forward(nan, nan, tok, off, rw)      # what a kernel does not write still holds these
    for path in (capi.PATH_AUTO, capi.PATH_BATCH):
        got = layer.experts_forward(hg, hu, tok, off, rw, path=path)
        layer.check_status()
        helpers.assert_close(got.cpu(), want.cpu(), what=f"path {path} rank {rank} E {E}")
    capi.check(capi.lib().bm_layer_set_option(layer._handle, 2, 0))
    layer.experts_forward(hg, hu, tok, off, rw)
    with pytest.raises(capi.BitsMoEError, match="bounded wait"):
        layer.check_status()
    capi.check(capi.lib().bm_layer_set_option(layer._handle, 2, 2000000))
    helpers.assert_close(layer.experts_forward(hg, hu, tok, off, rw).cpu(), want.cpu(), what=f"rank {rank} E {E} after a time-out")


@pytest.mark.parametrize("T,wdtype,shared", [(1, torch.bfloat16, 0), (5, torch.float16, 48), (64, torch.bfloat16, 200), (70, torch.bfloat16, 48),
                                             (300, torch.bfloat16, 48), (300, torch.float16, 0)])
def test_block_forward_matches_plain_products(T, wdtype, shared):
    E, k = 40, 4
    cfg, s, layer = _layer(E, k, shared=shared)
    gen = torch.Generator(device=DEV).manual_seed(3)
    x = synth.activations(cfg, T, seed=T, device=DEV, dtype=wdtype)
    gate = (torch.randn(E, cfg.hidden, generator=gen, device=DEV) / 16).to(wdtype)
    sh = tuple(s.shared[n].to(wdtype) for n in ("gate", "up", "down", "gate_logit_w")) if shared else None
    y, logits = layer.block_forward(x, gate, k, True, wdtype, sh)
    assert logits.dtype == wdtype
    helpers.assert_close(logits.cpu(), (x.float() @ gate.float().T).cpu(), what="router logits")
    want = _staged(layer, x, logits, k, wdtype, E)
    if shared:
        xf, (g, u, d, t) = x.float(), (w.float() for w in sh)
        want = want + torch.sigmoid(xf @ t.T) * ((torch.nn.functional.silu(xf @ g.T) * (xf @ u.T)) @ d.T)
    helpers.assert_close(y.cpu(), want.cpu(), what=f"block T={T}")


def test_block_forward_declines_weights_of_another_kind():
    cfg, s, layer = _layer(40, 4)
    x = synth.activations(cfg, 3, seed=1, device=DEV, dtype=torch.bfloat16)
    assert layer.block_forward(x, torch.zeros(40, cfg.hidden, device=DEV), 4) is None
