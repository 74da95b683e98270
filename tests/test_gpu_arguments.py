"""GPU: tensors whose shapes, types or devices do not fit are refused on the host, before anything is launched."""
import pytest
import torch

from bitsmoe_b200 import synth
from bitsmoe_b200.algorithms import mlp_forward_cuda
from bitsmoe_b200.layer import PackedLayer, dense_mlp, gate_logits, route_build
from tests import helpers

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
T, E, H, R, I, K = 6, 5, 128, 64, 128, 2


@pytest.fixture(scope="module")
def env():
    s = synth.make_layer(synth.tiny(hidden=H, num_experts=E, intermediate=I, top_k=K, rank=R), seed=4, device=DEV)
    layer = synth.to_packed_layer(s)
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(T, H, generator=gen, device=DEV).half()
    logits = torch.randn(T, E, generator=gen, device=DEV)
    idx, w = layer.route_topk(logits, K, True, None)
    tok, off, rw = route_build(idx, w, E)[:3]
    hg, hu = layer.basis_project(x)
    return dict(s=s, layer=layer, x=x, logits=logits, res=torch.zeros_like(x), routed=(hg, hu, tok, off, rw), want=layer.forward(x, logits, K),
                g2l=torch.arange(E, dtype=torch.int32, device=DEV))


def z(*shape, dtype=torch.float16, device=DEV):
    return torch.zeros(*shape, dtype=dtype, device=device)


LAYER = {  # what a wrong argument replaces
    "narrow rows": dict(x=lambda: z(T, H // 2)),
    "other token count": dict(logits=lambda: z(T - 1, E, dtype=torch.float32)),
    "short residual": dict(residual=lambda: z(T - 1, H)),
    "residual on the host": dict(residual=lambda: z(T, H, device="cpu")),
    "short out": dict(out=lambda: z(T - 1, H)),
    "out of another type": dict(out=lambda: z(T, H, dtype=torch.float32)),
    "strided out": dict(out=lambda: z(H, T).t()),
    "short id map": dict(global_to_local=lambda: z(E - 1, dtype=torch.int32)),
    "id map of another type": dict(global_to_local=lambda: z(E, dtype=torch.int64)),
}


@pytest.mark.parametrize("case", LAYER)
def test_layer_forward_refuses(env, case):
    args = dict(x=env["x"], logits=env["logits"], top_k=K)
    args.update({k: make() for k, make in LAYER[case].items()})
    with pytest.raises(RuntimeError):
        env["layer"].forward(**args)


def test_layer_forward_takes_what_fits(env):
    layer, x, logits, want = env["layer"], env["x"], env["logits"], env["want"]
    out = z(T, H)
    for got in (layer.forward(x, logits, K, residual=env["res"], out=out), layer.forward(x.reshape(T, 1, H), logits, K).reshape(T, H),
                layer.forward(x, logits, K, residual=env["res"].float().reshape(1, T, H), global_to_local=env["g2l"])):
        helpers.assert_close(got.cpu(), want.cpu(), what="forward")
    assert layer.forward(x[:0], logits[:0], K).shape == (0, H)


EXPERTS = {
    "gate rows of another rank": (0, lambda t: z(T, R - 8)),
    "up rows of another rank": (1, lambda t: z(T, R + 8)),
    "fp32 rows": (0, lambda t: t.float()),
    "strided rows": (1, lambda t: z(R, T).t()),
    "64-bit tokens": (2, lambda t: t.long()),
    "offsets of another layer": (3, lambda t: t[:-1]),
    "too few weights": (4, lambda t: t[:-1]),
    "weights on the host": (4, lambda t: t.cpu()),
}


@pytest.mark.parametrize("case", EXPERTS)
def test_experts_and_op_refuse(env, case):
    i, make = EXPERTS[case]
    args = list(env["routed"])
    args[i] = make(args[i]).contiguous() if case != "strided rows" else make(args[i])
    with pytest.raises(RuntimeError):
        env["layer"].experts_forward(*args)
    lists = helpers.ref_args(env["s"], DEV)
    good = mlp_forward_cuda.moe_packed_forward(*env["routed"], *lists, R, I, 0)      # the layer of these lists is known now
    helpers.assert_close(good.cpu(), env["layer"].experts_forward(*env["routed"]).cpu(), what="op")
    with pytest.raises(RuntimeError):
        mlp_forward_cuda.moe_packed_forward(*args, *lists, R, I, 0)


def test_experts_take_fewer_up_rows_than_gate_rows(env):
    """The gathered exchange passes views of one buffer: up rows start T rows later, so their view is shorter."""
    hg, hu, tok, off, rw = env["routed"]
    flat = torch.cat([hg, hu])
    got = env["layer"].experts_forward(flat, flat[T:], tok, off, rw)
    helpers.assert_close(got[:T].cpu(), env["layer"].experts_forward(hg, hu, tok, off, rw).cpu(), what="views of one buffer")


def test_other_entries_refuse(env):
    layer, x, s = env["layer"], env["x"], env["s"]
    gate, sh = z(E, H), (z(32, H), z(32, H), z(H, 32), z(1, H))
    assert layer.block_forward(x, gate, K, shared=sh) is not None
    wrong = [lambda: layer.block_forward(z(T, H // 2), z(E, H // 2), K), lambda: layer.block_forward(x, z(E, H // 2), K),
             lambda: layer.block_forward(x, gate, K, global_to_local=z(E - 1, dtype=torch.int32)),
             lambda: layer.basis_project(z(T, H // 2)), lambda: layer.basis_project(x, out=z(2, T, R // 2)),
             lambda: layer.combine_down_basis(z(T, R // 2, dtype=torch.float32), torch.float16),
             lambda: layer.combine_down_basis(z(T, R, dtype=torch.float32), torch.float16, residual=z(1, H)),
             lambda: gate_logits(x, z(E, H // 2)), lambda: route_build(z(T, K, dtype=torch.int32), z(T, K - 1), E),
             lambda: PackedLayer(s.tables["gate"], s.tables["up"], s.tables["down"], I, R, s.vh_gate, s.vh_up[:-8], s.u_down),
             lambda: PackedLayer(s.tables["gate"], s.tables["up"], s.tables["down"], I, R, s.vh_gate, s.vh_up, s.u_down[:-8])]
    for i in range(4):
        bad = list(sh)
        bad[i] = z(bad[i].shape[0], bad[i].shape[1] - 8)
        wrong += [lambda bad=bad: layer.block_forward(x, gate, K, shared=tuple(bad)), lambda bad=bad: dense_mlp(x, *bad)]
    wrong.append(lambda: dense_mlp(x, *sh, residual=z(T - 1, H)))
    for call in wrong:
        with pytest.raises(RuntimeError):
            call()
    layer.check_status()


def test_dropped_workspace_waits_for_the_streams_that_use_it(env):
    """A workspace made on one stream, used on another and dropped there (a layer keeps the last few shapes) must not be
    handed out again while that use is still to come."""
    layer = synth.to_packed_layer(env["s"])
    xs = {t: env["x"].repeat(50, 1)[:t] for t in range(200, 212)}
    lg = {t: env["logits"].repeat(50, 1)[:t] for t in xs}
    ws = layer.workspace(200, K)
    at, size = ws.data_ptr(), ws.numel()
    del ws
    side, awake = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(side):
        env["layer"].forward(xs[200], lg[200], K)      # kernels loaded, this stream's pool filled
        torch.cuda.synchronize()
        torch.cuda._sleep(1_000_000_000)
        awake.record()
        for t in xs:
            layer.forward(xs[t], lg[t], K)      # the first uses the buffer, a later one drops it
    taken = [torch.empty(size, dtype=torch.uint8, device=DEV) for _ in range(4)]
    assert not awake.query(), "the side stream should still sleep"
    assert at not in [t.data_ptr() for t in taken]
    torch.cuda.synchronize()


def test_captured_call_keeps_its_workspace(env):
    """A graph replays on the buffers that it was captured with; shapes met later must not free one of them."""
    layer = synth.to_packed_layer(env["s"])
    x, lg = env["x"].repeat(50, 1), env["logits"].repeat(50, 1)
    want = layer.forward(x[:200], lg[:200], K)
    size = layer.workspace(200, K).numel()
    y, graph = torch.empty_like(want), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.forward(x[:200], lg[:200], K, out=y)
    for t in range(201, 212):
        layer.forward(x[:t], lg[:t], K)
    torch.cuda.synchronize()
    others = [torch.full((size,), 7, dtype=torch.uint8, device=DEV) for _ in range(12)]
    for _ in range(2):
        y.zero_()
        graph.replay()
    helpers.assert_close(y.cpu(), want.cpu(), what="replay")
    assert all(bool(t.eq(7).all()) for t in others), "the graph wrote into memory of other tensors"


def _shifted(t, by=1):
    """The same values in a contiguous view that starts ``by`` elements off an aligned address."""
    v = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)[by:].view(t.shape)
    assert v.is_contiguous() and v.data_ptr() % 16
    return v.copy_(t)


# contiguous views may start anywhere: x, the basis, the router's and the shared expert's weights, each side of the batch size
# at which the products change kernels
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens", [5, 300])
def test_products_take_views_at_any_address(env, tokens, dtype):
    s, layer, gen = env["s"], env["layer"], torch.Generator(device=DEV).manual_seed(tokens)
    x = torch.randn(tokens, H, generator=gen, device=DEV).to(dtype)
    logits = torch.randn(tokens, E, generator=gen, device=DEV)
    gate = (torch.randn(E, H, generator=gen, device=DEV) / 16).half()
    sh = [(torch.randn(*d, generator=gen, device=DEV) / 16).half() for d in ((32, H), (32, H), (H, 32), (H,))]
    moved = PackedLayer(s.tables["gate"], s.tables["up"], s.tables["down"], I, R, *(_shifted(b) for b in (s.vh_gate, s.vh_up, s.u_down)))
    want = layer.forward(x, logits, K).cpu()
    helpers.assert_close(layer.forward(_shifted(x, 3), logits, K).cpu(), want, what="x")
    helpers.assert_close(moved.forward(x, logits, K).cpu(), want, what="basis")
    res = x * 1e-4      # of the output's size
    helpers.assert_close(moved.forward(x, logits, K, residual=_shifted(res), out=_shifted(x)).cpu(),
                         layer.forward(x, logits, K, residual=res).cpu(), what="residual and out")
    want = gate_logits(x, gate).cpu()
    for a, b in ((_shifted(x), gate), (x, _shifted(gate, 5)), (_shifted(x.float()), gate)):
        helpers.assert_close(gate_logits(a, b).cpu(), want, what="router")
    want = dense_mlp(x, *sh).cpu()
    for i in range(5):
        args = [_shifted(t, 2 * i + 1) if j == i else t for j, t in enumerate([x, *sh])]
        helpers.assert_close(dense_mlp(*args).cpu(), want, what=f"dense {i}")
    y, lg = layer.block_forward(x, gate.to(dtype), K, True, None, tuple(t.to(dtype) for t in sh))
    y2, lg2 = layer.block_forward(_shifted(x), gate.to(dtype), K, True, None, tuple(t.to(dtype) for t in sh))
    helpers.assert_close(lg2.cpu(), lg.cpu(), what="block logits")
    helpers.assert_close(y2.cpu(), y.cpu(), what="block")
