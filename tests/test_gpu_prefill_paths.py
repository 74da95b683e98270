"""GPU: edges of the prefill kernels -- items and units of the packed experts, the routing passes over several blocks, and
the products whose rows, columns and contractions do not fill a tile."""
import pytest
import torch

from bitsmoe_b200 import capi, synth
from bitsmoe_b200.layer import PackedLayer, dense_mlp, route_build, route_topk
from tests import helpers

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _route(counts, k, T, gen):
    """Permutation tables in which expert e has counts[e] assignments of distinct tokens."""
    tok = torch.cat([torch.sort(torch.randperm(T, generator=gen, device=DEV)[:c]).values for c in counts]).to(torch.int32)
    off = torch.zeros(len(counts) + 1, dtype=torch.int32, device=DEV)
    off[1:] = torch.tensor(counts, device=DEV).cumsum(0)
    return tok, off, torch.rand(tok.numel(), generator=gen, device=DEV)


# assignments per expert around an item (128) and a pass (8), none at all, one expert alone; ranks whose row slots are an odd
# number of pairs, are not whole octets of one group, or pass 256; intermediate sizes of one and of several tiles
@pytest.mark.parametrize("rank,inter", [(64, 128), (80, 256), (256, 384), (328, 128), (384, 256)])
@pytest.mark.parametrize("counts", [(1, 0, 127, 128, 129, 7), (9, 8, 300, 0, 255, 257), (512,)])
def test_packed_experts_match_generic_kernel(rank, inter, counts):
    cfg = synth.tiny(hidden=128, num_experts=len(counts), intermediate=inter, top_k=1, rank=rank)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=rank, device=DEV))
    T = 520
    gen = torch.Generator(device=DEV).manual_seed(11)
    tok, off, rw = _route(counts, 1, T, gen)
    hg, hu = layer.basis_project(synth.activations(cfg, T, seed=2, device=DEV, dtype=torch.bfloat16))
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    for path in (capi.PATH_DECODE, capi.PATH_TENSOR, capi.PATH_BATCH):
        try:
            got = layer.experts_forward(hg, hu, tok, off, rw, path=path)
        except capi.BitsMoEError as e:      # a layer whose largest expert does not fit that path
            assert e.status == 2      # BM_ERR_UNSUPPORTED
            continue
        helpers.assert_close(got.cpu(), want.cpu(), what=f"path {path} rank {rank} counts {counts}")


# whole rounds of items, so that a pair of CTAs walks several items of several chunks: both CTAs with tokens, one with none,
# items around 2 x 64 tokens and (many per expert on average) around 2 x 128, ranks of one to three slot tiles and of an odd number
# of pairs
@pytest.mark.parametrize("pattern", [(1, 2, 0, 63, 64, 65, 127, 128, 129), (255, 256, 257, 300, 1, 299, 254, 300, 300)])
@pytest.mark.parametrize("rank,inter", [(64, 384), (96, 128), (256, 256), (328, 256)])
def test_pairs_walk_several_items(rank, inter, pattern):
    counts = tuple(pattern[e % 9] for e in range(210))
    cfg = synth.tiny(hidden=128, num_experts=len(counts), intermediate=inter, top_k=1, rank=rank)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=rank, device=DEV))
    T = 300
    gen = torch.Generator(device=DEV).manual_seed(17)
    tok, off, rw = _route(counts, 1, T, gen)
    hg, hu = layer.basis_project(synth.activations(cfg, T, seed=2, device=DEV, dtype=torch.bfloat16))
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    for _ in range(3):
        got = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_TENSOR)
        layer.check_status()
        helpers.assert_close(got.cpu(), want.cpu(), what=f"rank {rank} inter {inter}")


def _with_output_rank(rank_in, rank_out, inter, E):
    """A layer whose down matrices have ``rank_out`` rows while gate and up have ``rank_in``."""
    a = synth.make_layer(synth.tiny(hidden=128, num_experts=E, intermediate=inter, top_k=1, rank=rank_in), seed=1, device=DEV)
    b = synth.make_layer(synth.tiny(hidden=128, num_experts=E, intermediate=inter, top_k=1, rank=rank_out), seed=2, device=DEV)
    return PackedLayer(a.tables["gate"], a.tables["up"], b.tables["down"], inter, rank_out, a.vh_gate, a.vh_up, b.u_down)


# rank_accum rows that start on a 16-byte boundary for every token, for every second or fourth one only, and (base one float
# off) for none at all
@pytest.mark.parametrize("rank_out,shift", [(256, 0), (256, 1), (252, 0), (250, 0), (250, 1), (241, 0), (72, 0)])
def test_sums_reach_rows_of_any_alignment(rank_out, shift):
    counts, T, lib = (130, 0, 61, 1), 140, capi.lib()
    layer = _with_output_rank(256, rank_out, 256, len(counts))
    gen = torch.Generator(device=DEV).manual_seed(5)
    tok, off, rw = _route(counts, 1, T, gen)
    hg, hu = layer.basis_project(torch.randn(T, 128, generator=gen, device=DEV).half())
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    for path in (capi.PATH_DECODE, capi.PATH_TENSOR, capi.PATH_BATCH):
        buf = torch.full((T * rank_out + 2,), 7.0, device=DEV)
        acc = buf[shift:shift + T * rank_out].view(T, rank_out)
        assert acc.data_ptr() % 16 == 4 * shift
        capi.check(lib.bm_experts_forward(layer._handle, hg.data_ptr(), hu.data_ptr(), tok.data_ptr(), off.data_ptr(), rw.data_ptr(), T,
                                          tok.numel(), acc.data_ptr(), path, None, 0, capi.stream_ptr(torch.device(DEV))))
        layer.check_status()
        helpers.assert_close(acc.cpu(), want.cpu(), what=f"path {path} rank_out {rank_out} shift {shift}")
        assert buf[:shift].eq(7.0).all() and buf[shift + T * rank_out:].eq(7.0).all()


# A kernel that is asked for by name runs whatever the load.  One tile and one assignment a token: in deterministic mode a row's bits then
# depend on the kernel alone, not on how many tokens share its pass, and the two kernels round weights and operand at different places.
def test_named_kernels_run_at_any_load():
    E, counts = 12, [17, 9, 0, 24, 12, 1, 31, 8, 16, 40, 7, 15]
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=128, top_k=1, rank=64)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=4, device=DEV))
    layer.set_deterministic(True)
    T = sum(counts)
    gen = torch.Generator(device=DEV).manual_seed(12)
    hg, hu = layer.basis_project(torch.randn(T, 128, generator=gen, device=DEV).half())
    rw = torch.rand(T, generator=gen, device=DEV)
    start = [sum(counts[:e]) for e in range(E)]

    def run(path, first, last):      # every expert's assignments first .. last - 1
        rows = [range(s + min(first, c), s + min(last, c)) for s, c in zip(start, counts)]
        tok = torch.tensor([i for r in rows for i in r], dtype=torch.int32, device=DEV)
        off = torch.tensor([0] + [len(r) for r in rows], device=DEV).cumsum(0).to(torch.int32)
        return layer.experts_forward(hg, hu, tok, off, rw[tok.long()], path=path)

    whole = {path: run(path, 0, T) for path in (capi.PATH_DECODE, capi.PATH_BATCH)}
    for path in (capi.PATH_DECODE, capi.PATH_BATCH):
        assert torch.equal(whole[path], sum(run(path, i, i + 4) for i in range(0, max(counts), 4))), path
    layer.check_status()
    assert not torch.equal(whole[capi.PATH_DECODE], whole[capi.PATH_BATCH])


# passes of 16 around the numbers at which the last round is handed out in even shares of its tiles (here 6, on 296 CTAs: 149 to 246
# passes), alone and behind a whole round; a share holds the end of one pass and the start of the next
@pytest.mark.parametrize("passes", [148, 149, 150, 197, 198, 246, 247, 296, 297, 296 + 149, 296 + 246])
def test_passes_in_even_shares(passes):
    E, T = 8, 1200
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=768, top_k=1, rank=64)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=11, device=DEV))
    layer.set_deterministic(True)
    gen = torch.Generator(device=DEV).manual_seed(passes)
    parts = [passes // E + (e < passes % E) for e in range(E)]
    tok, off, rw = _route([16 * n - (7 if n > 1 else 0) for n in parts], 1, T, gen)
    hg, hu = layer.basis_project(torch.randn(T, 128, generator=gen, device=DEV).half())
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    got = [layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_BATCH) for _ in range(2)]
    layer.check_status()
    helpers.assert_close(got[0], want, what=f"{passes} passes")
    assert torch.equal(*got)


# The automatic choice, told by its bits in deterministic mode: passes of 8 while one is enough for most experts or where few experts leave
# room to cut them, passes of 16 up to about 24 assignments an expert, products on tcgen05 above
@pytest.mark.parametrize("E,inter,load,path", [(16, 512, 8, capi.PATH_DECODE), (16, 1536, 20, capi.PATH_DECODE), (48, 768, 6, capi.PATH_DECODE),
                                               (128, 768, 4, capi.PATH_DECODE), (128, 768, 8, capi.PATH_BATCH), (128, 768, 12, capi.PATH_BATCH),
                                               (128, 768, 18, capi.PATH_BATCH), (128, 768, 40, capi.PATH_TENSOR), (160, 1536, 4, capi.PATH_DECODE),
                                               (160, 1536, 8, capi.PATH_BATCH), (160, 1536, 26, capi.PATH_TENSOR)])
def test_automatic_choice_of_kernel(E, inter, load, path):
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=inter, top_k=1, rank=256)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=8, device=DEV))
    layer.set_deterministic(True)
    gen = torch.Generator(device=DEV).manual_seed(13)
    tok, off, rw = _route([load] * E, 1, 64, gen)
    hg, hu = layer.basis_project(torch.randn(64, 128, generator=gen, device=DEV).half())
    runs = {p: layer.experts_forward(hg, hu, tok, off, rw, path=p) for p in (capi.PATH_AUTO, capi.PATH_DECODE, capi.PATH_BATCH, capi.PATH_TENSOR)}
    layer.check_status()
    assert [p for p in runs if p and torch.equal(runs[p], runs[capi.PATH_AUTO])] == [path]


# A shard of the experts: the kernel is chosen for its share of the assignments, not for all of them
@pytest.mark.parametrize("T,path", [(96, capi.PATH_DECODE), (128, capi.PATH_DECODE), (256, capi.PATH_BATCH), (512, capi.PATH_TENSOR)])
def test_a_shard_is_chosen_for_by_its_share(T, path):
    E, routed, k = 64, 128, 8
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=768, top_k=k, rank=256)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=9, device=DEV))
    layer.set_deterministic(True)
    gen = torch.Generator(device=DEV).manual_seed(14)
    x = torch.randn(T, 128, generator=gen, device=DEV).half()
    logits = torch.randn(T, routed, generator=gen, device=DEV)
    g2l = torch.full((routed,), -1, dtype=torch.int32, device=DEV)
    g2l[1::2] = torch.arange(E, dtype=torch.int32, device=DEV)
    runs = {p: layer.forward(x, logits, k, True, torch.float16, global_to_local=g2l, path=p).clone()
            for p in (capi.PATH_AUTO, capi.PATH_DECODE, capi.PATH_BATCH, capi.PATH_TENSOR)}
    layer.check_status()
    assert [p for p in runs if p and torch.equal(runs[p], runs[capi.PATH_AUTO])] == [path]


# lists shorter than their bound (a rank of an expert-parallel group): chosen for the expected length, right for any
def test_expected_length_chooses_the_kernel():
    E, bound, load = 48, 48 * 22, [3] * 48
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=768, top_k=1, rank=256)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=10, device=DEV))
    layer.set_deterministic(True)
    lib, gen, T = capi.lib(), torch.Generator(device=DEV).manual_seed(16), 64
    hg, hu = layer.basis_project(torch.randn(T, 128, generator=gen, device=DEV).half())
    tok, off, rw = _route(load, 1, T, gen)
    ws = torch.empty(lib.bm_experts_workspace_bytes(layer._handle, T, bound, capi.PATH_AUTO), dtype=torch.uint8, device=DEV)

    def run(expected, num_assign=bound):
        acc = torch.empty(T, layer.rank_out, device=DEV)
        capi.check(lib.bm_experts_forward_expecting(layer._handle, hg.data_ptr(), hu.data_ptr(), tok.data_ptr(), off.data_ptr(), rw.data_ptr(), T,
                                                    num_assign, expected, acc.data_ptr(), capi.PATH_AUTO, ws.data_ptr(), ws.numel(),
                                                    capi.stream_ptr(acc.device)))
        layer.check_status()
        return acc

    by_path = {p: layer.experts_forward(hg, hu, tok, off, rw, path=p) for p in (capi.PATH_DECODE, capi.PATH_BATCH)}
    for expected, path in ((0, capi.PATH_DECODE), (len(tok), capi.PATH_DECODE), (bound, capi.PATH_BATCH)):
        assert [p for p in by_path if torch.equal(by_path[p], run(expected))] == [path]
    for expected in (-1, bound + 1):
        with pytest.raises(capi.BitsMoEError, match="expected of at most"):
            run(expected)


# matrices in which several rows hold the same rank: single rows (of one width and of two), and a whole aligned octet twice
def test_rows_that_repeat_a_rank():
    E, rank, inter, T = 3, 64, 256, 200
    s = synth.make_layer(synth.tiny(hidden=128, num_experts=E, intermediate=inter, top_k=1, rank=rank), seed=3, device=DEV)
    for tag in ("gate", "up", "down"):
        idx = [t.clone() for t in s.tables[tag]["rank_idx"]]
        idx[0][40] = idx[0][41]
        idx[0][2] = idx[0][60]
        idx[1][8:16] = torch.arange(16, 24)
        idx[1][48:56] = torch.arange(16, 24)
        s.tables[tag]["rank_idx"] = idx
    layer = synth.to_packed_layer(s)
    gen = torch.Generator(device=DEV).manual_seed(6)
    tok, off, rw = _route((150, 131, 20), 1, T, gen)
    hg, hu = layer.basis_project(torch.randn(T, 128, generator=gen, device=DEV).half())
    want = layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC)
    for path in (capi.PATH_DECODE, capi.PATH_TENSOR, capi.PATH_BATCH):
        nan = torch.full_like(hg, float("nan"))
        layer.experts_forward(nan, nan, tok, off, rw, path=path)      # what a kernel does not write still holds these
        got = layer.experts_forward(hg, hu, tok, off, rw, path=path)
        layer.check_status()
        helpers.assert_close(got.cpu(), want.cpu(), what=f"path {path}")


# token counts around the blocks of the counting pass; expert counts around a warp of the scan and the top-k's registers
@pytest.mark.parametrize("T", [129, 205, 1025, 2048, 2049, 4097, 16385])
@pytest.mark.parametrize("E,k", [(2, 2), (33, 5), (128, 8), (512, 10), (1024, 4)])
def test_routing_is_the_stable_permutation(T, E, k):
    logits = torch.randn(T, E, device=DEV).round(decimals=1)      # ties: the lower expert id comes first
    idx, w = route_topk(logits, k, False, torch.float32)
    p = torch.softmax(logits, -1)
    order = torch.argsort(p, dim=-1, descending=True, stable=True)[:, :k]
    assert torch.equal(idx.long(), order)
    helpers.assert_close(w.cpu(), torch.gather(p, 1, order).cpu(), what="weights")
    tok, off, rw, _, counts = route_build(idx, w, E)
    flat, by = torch.sort(idx.reshape(-1), stable=True)
    assert torch.equal(off[1:].long(), torch.bincount(flat.long(), minlength=E).cumsum(0))
    assert int(counts[0]) == T * k
    assert torch.equal(tok.long(), by // k) and torch.equal(rw, w.reshape(-1)[by])


# rows around a tile of 128 and the decode kernel's 8, 64 and 256; inner sizes that are no multiple of a tile, or so many
# that the decode products take several row tiles per block
@pytest.mark.parametrize("T", [1, 9, 65, 256, 257, 385, 1000])
@pytest.mark.parametrize("H,I", [(128, 48), (256, 200), (512, 2824), (1024, 4104)])
def test_dense_mlp_matches_plain_products(T, H, I):
    gen = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, H, generator=gen, device=DEV).to(torch.bfloat16)
    g, u = ((torch.randn(I, H, generator=gen, device=DEV) / H ** 0.5).half() for _ in range(2))
    d = (torch.randn(H, I, generator=gen, device=DEV) / I ** 0.5).half()
    t = (torch.randn(H, generator=gen, device=DEV) / H ** 0.5).half()
    xf = x.float()
    want = torch.sigmoid(xf @ t.float())[:, None] * ((torch.nn.functional.silu(xf @ g.float().T) * (xf @ u.float().T)) @ d.float().T)
    helpers.assert_close(dense_mlp(x, g, u, d, t).float().cpu(), want.cpu(), what=f"T={T} H={H} I={I}")


# prefill blocks: tiles of 128 rows that are full, ragged or hold one row; router and shared widths that are ragged
@pytest.mark.parametrize("T", [257, 384, 513])
@pytest.mark.parametrize("E,shared,wdtype", [(5, 48, torch.bfloat16), (40, 200, torch.float16), (300, 0, torch.bfloat16)])
def test_prefill_block_matches_stages(T, E, shared, wdtype):
    cfg = synth.tiny(hidden=256, num_experts=E, intermediate=128, top_k=4, rank=64, shared_intermediate=shared, shared_gated=shared > 0)
    s = synth.make_layer(cfg, seed=7, device=DEV)
    layer = synth.to_packed_layer(s)
    gen = torch.Generator(device=DEV).manual_seed(3)
    x = synth.activations(cfg, T, seed=T, device=DEV, dtype=wdtype)
    gate = (torch.randn(E, cfg.hidden, generator=gen, device=DEV) / 16).to(wdtype)
    sh = tuple(s.shared[n].to(wdtype) for n in ("gate", "up", "down", "gate_logit_w")) if shared else None
    y, logits = layer.block_forward(x, gate, 4, True, wdtype, sh)
    xf = x.float()
    helpers.assert_close(logits.cpu(), (xf @ gate.float().T).cpu(), what="router logits")
    idx, w = route_topk(logits, 4, True, wdtype)
    tok, off, rw, _, _ = route_build(idx, w, E)
    hg, hu = layer.basis_project(x)
    want = layer.combine_down_basis(layer.experts_forward(hg, hu, tok, off, rw, path=capi.PATH_GENERIC), torch.float32)
    if shared:
        g, u, d, t = (v.float() for v in sh)
        want = want + torch.sigmoid(xf @ t.T) * ((torch.nn.functional.silu(xf @ g.T) * (xf @ u.T)) @ d.T)
    helpers.assert_close(y.cpu(), want.cpu(), what=f"block T={T} E={E}")


# contractions split over two and four CTAs: uneven shares (17 slices), stacks that fill part of a tile, ragged token counts; the
# last pair of sizes has the down basis split as well
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hidden,rank", [(512, 72), (1024, 40), (1088, 104), (1024, 512)])
@pytest.mark.parametrize("T", [257, 300, 513])
def test_split_contractions_vs_double(hidden, rank, T, dtype):
    cfg = synth.tiny(hidden=hidden, num_experts=2, intermediate=128, rank=rank)
    raw = synth.make_layer(cfg, seed=rank, device=DEV)
    layer = synth.to_packed_layer(raw)
    gen = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, hidden, generator=gen, device=DEV).to(dtype)

    def check(got, a, w, extra, eps):
        # operands are fp16; fp32 sums of n products err by n * 2^-24 of the sum of magnitudes, the result by its own rounding
        a, w = a.half().double(), w.half().double()
        want = a @ w.t() + extra.double()
        bound = eps * want.abs() + a.shape[1] * 2.0 ** -24 * (a.abs() @ w.abs().t() + extra.double().abs()) + 2.0 ** -24
        worst = float(((got.double() - want).abs() / bound).max())
        assert worst <= 1.0, worst

    eps = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 0.0}
    zero = torch.zeros((), device=DEV)
    for got, w in zip(layer.basis_project(x), (raw.vh_gate, raw.vh_up)):
        check(got, x, w.to(DEV), zero, eps[torch.float16])
    acc = torch.randn(T, rank, generator=gen, device=DEV) * 0.05
    res = torch.randn(T, hidden, generator=gen, device=DEV).to(dtype)
    check(layer.combine_down_basis(acc, dtype, residual=res), acc, raw.u_down.to(DEV), res, eps[dtype])
    layer.check_status()


@pytest.mark.parametrize("T,inter", [(257, 64), (400, 192)])
def test_split_gated_pair(T, inter):
    gen = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, 1024, generator=gen, device=DEV).half()
    wg, wu = (torch.randn(inter, 1024, generator=gen, device=DEV).half() / 32 for _ in range(2))
    wd = (torch.randn(1024, inter, generator=gen, device=DEV) / inter ** 0.5).half()
    g, u = x.double() @ wg.double().t(), x.double() @ wu.double().t()
    z = torch.nn.functional.silu(g) * u
    want = z @ wd.double().t()
    # z is rounded to fp16 (one rounding, and what the fp32 sums and __expf add: a few 2^-20), y as well
    bound = 2.0 ** -10 * (z.abs() @ wd.double().abs().t()) + 2.0 ** -11 * want.abs() + 2.0 ** -24
    assert float(((dense_mlp(x, wg, wu, wd).double() - want).abs() / bound).max()) <= 1.0


# the layer's one call against its stages: assignments that one, two, four and eight rounds of the routing's cluster take and more than it
# takes, tokens around the launch chains' limits, a rank that is no multiple of a slice
@pytest.mark.parametrize("T,E,k,rank", [(49, 8, 2, 64), (65, 8, 2, 64), (129, 8, 2, 64), (129, 8, 2, 72), (300, 40, 8, 64), (2049, 16, 4, 64),
                                        (4097, 16, 4, 64), (8193, 8, 4, 64), (16385, 8, 4, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_layer_call_is_its_stages(T, E, k, rank, dtype):
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=128, top_k=k, rank=rank)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=T, device=DEV))
    layer.set_deterministic(True)
    gen = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, 128, generator=gen, device=DEV).to(dtype)
    logits = torch.randn(T, E, generator=gen, device=DEV)
    idx, w = route_topk(logits, k, True, dtype)
    tok, off, rw, _, _ = route_build(idx, w, E)
    hg, hu = layer.basis_project(x)
    acc = layer.experts_forward(hg, hu, tok, off, rw)
    # alone, and on a residual of the experts' own size: beside a larger one a wrong or missing result would pass
    alone = layer.combine_down_basis(acc, dtype)
    res = (torch.randn(T, 128, generator=gen, device=DEV) * alone.float().std()).to(dtype)
    for residual, want in ((None, alone), (res, layer.combine_down_basis(acc, dtype, residual=res))):
        for _ in range(2):
            got = layer.forward(x, logits, k, True, dtype, residual=residual)
            layer.check_status()
            # (products of another kernel may differ in the last place of h, and so of y: the bounds on peak and norm are what counts)
            helpers.assert_close(got, want, rtol=2.0 ** -7, atol=2e-3, what="layer call")
        with pytest.raises(AssertionError):
            helpers.assert_close(torch.zeros_like(got) if residual is None else residual, want, rtol=2.0 ** -7, atol=2e-3, what="nothing from the experts")


# placement of a layer call's assignments by one cluster: the edges of four and of eight rounds and the first size beyond, tables of
# many experts, choices spread out, gathered on few experts, and (top 1) all on one, whose prefixes are the largest
@pytest.mark.parametrize("E,k", [(128, 8), (512, 10), (1024, 4), (128, 1)])
def test_placement_of_many_assignments(E, k):
    cfg = synth.tiny(hidden=128, num_experts=E, intermediate=128, top_k=k, rank=64)
    layer = synth.to_packed_layer(synth.make_layer(cfg, seed=E + k, device=DEV))
    layer.set_deterministic(True)
    gen = torch.Generator(device=DEV).manual_seed(15)
    for T in (16384 // k + 1, 32768 // k, 32768 // k + 1, 65536 // k, 65536 // k + 1):
        x = torch.randn(T, 128, generator=gen, device=DEV).half()
        for skew in (0.0, 3.0, 100.0):
            logits = torch.randn(T, E, generator=gen, device=DEV) - skew * torch.log(torch.arange(1.0, E + 1, device=DEV)).flip(0)
            idx, w = route_topk(logits, k, True, torch.float16)
            flat, by = torch.sort(idx.reshape(-1), stable=True)
            off = torch.zeros(E + 1, dtype=torch.int32, device=DEV)
            off[1:] = torch.bincount(flat.long(), minlength=E).cumsum(0)
            acc = layer.experts_forward(*layer.basis_project(x), (by // k).to(torch.int32), off, w.reshape(-1)[by])
            # sums do not depend on their order here, and the products are the same launches: every bit agrees
            assert torch.equal(layer.forward(x, logits, k, True, torch.float16), layer.combine_down_basis(acc, torch.float16)), (T, skew)
    layer.check_status()
