"""GPU tests of the kernels at the sizes where they can go wrong: edges of tiles, remainders of K, the lines
between two kernels, the smallest and largest of a kernel's range.  Against the CPU oracle on the same seeded bytes.

Tolerance: every product of an E4M3 (FP4) weight, an E4M3 activation and their scales is exact, so what differs is
the order of K additions in fp32.  Each is off by at most 2^-24 of a running sum of random signs that is no larger
than the result's scale: relative L2 <= K * 2^-24, and never above the 5e-5 of the other parity tests.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    torch.cuda.set_device(0)
    return torch.device("cuda:0")


def check(got, want, k):
    got, want = got.cpu().numpy().astype(np.float64), want.astype(np.float64)
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= min(5e-5, k * 2.0 ** -24), err


FP8 = [
    # n, k, k0, K of the whole matrix, scale, rows
    (1040, 640, 0, 640, "f32", (1, 2)),              # CUDA cores: K not a multiple of 512, rows not of 4
    (1040, 512, 128, 1024, "f32", (1, 2)),           # a column window of a wider matrix, its rows not contiguous
    (2064, 544, 32, 1280, "ue8m0", (1, 2)),          # K not a multiple of 128, 32-row scale blocks inside a group of rows
    (4096, 6400, 0, 6400, "f32", (2,)),              # two rows, above the line to the tensor cores
    (1040, 1024, 0, 1024, "f32", (3, 16, 17, 32, 33)),    # 8192 values per CTA: quantised there up to 16 rows
    (1040, 1056, 0, 1056, "ue8m0", (3, 12, 13, 64, 65)),  # 33 scale columns: exponents collected byte by byte
    (1040, 1056, 128, 1280, "ue8m0", (4, 40)),       # word loads with a K tail
    (5120, 2304, 0, 2304, "ue8m0", (6, 19, 128)),    # two CTAs per SM, word loads, K halves of nine slabs
    # CTA pairs swap groups of four tokens: a group or a half alone, ragged last groups, every accumulator width
    (2064, 1024, 0, 1024, "f32", (4, 5, 8, 9, 15, 20, 31, 36, 63, 66, 97, 127)),
    (2064, 1056, 0, 1056, "ue8m0", (4, 5, 9, 20, 36, 66, 127)),
    # the partner's sums arrive behind the activations: half an SM, and the third stage of UE8M0 scales
    (608, 7040, 0, 7040, "f32", (11, 12)),
    (8432, 1408, 0, 1408, "f32", (14,)),
    (8528, 1408, 0, 1408, "ue8m0", (3, 4)),
    (8208, 1664, 0, 1664, "ue8m0", (61, 124)),
    (1040, 768, 0, 768, "f32", (129, 225, 449)),     # prefill tiles: last row tile of 16, token tiles of 1 and up
    (1040, 1056, 0, 1056, "ue8m0", (129, 449)),
    (1040, 1056, 128, 1280, "ue8m0", (200,)),
    (272, 512, 0, 512, "f32", (4096, 4097)),         # prefill in one launch, and in two
]


@pytest.mark.parametrize("n,k,k0,kfull,scale,ms", FP8)
def test_fp8_edges(dev, oracle, n, k, k0, kfull, scale, ms):
    from weightstream_b200 import formats as F, synth, tp
    b = 128 if scale == "f32" else 32
    rng = np.random.default_rng(synth.config_seed(f"fp8-edges-{n}-{k}-{k0}", 0, 1))
    w, sc = synth.fp8_weight(rng, n, kfull, scale=scale, bn=b, bk=b)
    wd, sd = torch.from_numpy(w).to(dev), torch.from_numpy(np.ascontiguousarray(sc)).to(dev)
    ep = tp.Endpoint(max_m=max(16, max(ms)), max_n=n)
    try:
        for m in ms:
            x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, k))
            want = oracle.fp8_gemv(w[:, k0:k0 + k], sc, x, bn=b, bk=b, k0=k0, threads=oracle.max_threads())
            for act in (torch.bfloat16, torch.float32):  # (the values are bf16's: the same result)
                out = ep.fp8_rowpar_gemm_allreduce(torch.from_numpy(x).to(dev).to(act), wd[:, k0:k0 + k], sd, block=(b, b), k0=k0)
                ep.check()
                check(out, want, k)
    finally:
        ep.close()


@pytest.mark.parametrize("k,ms", [
    (512, (1, 2, 3, 40, 65, 128, 200)),  # all of a 64-row launch fits; two launches, three, four
    (8192, (24, 70)),                    # only eight rows' copies fit
])
def test_scale_columns_that_slabs_straddle(dev, oracle, k, ms):
    """fp32 scales on a K slice that starts inside a scale block: a 128-wide slab has two scale columns, which the
    tensor-memory kernels cannot take, at any row count.  The device call, the host call and two virtual ranks."""
    from weightstream_b200 import formats as F, synth, tp
    n, k0 = 1040, 64
    rng = np.random.default_rng(synth.config_seed("straddle", k, 1))
    w, sc = synth.fp8_weight(rng, n, k0 + 2 * k + 64)  # whole blocks; the slice behind this one starts the same way
    wd, sd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev)
    ep, grp = tp.Endpoint(max_m=max(ms), max_n=n), tp.LocalGroup(2, max_m=max(ms), max_n=n)
    cuts = [slice(k0, k0 + k), slice(k0 + k, k0 + 2 * k)]
    try:
        for m in ms:
            bits = synth.activations_bf16(rng, m, 2 * k)
            x = F.bf16_bits_to_f32(bits)
            xd = torch.from_numpy(x).to(dev).to(torch.bfloat16)
            parts = [oracle.fp8_gemv(w[:, c], sc, np.ascontiguousarray(x[:, i * k:(i + 1) * k]), bn=128, bk=128, k0=c.start,
                                     threads=oracle.max_threads()) for i, c in enumerate(cuts)]
            out = ep.fp8_rowpar_gemm_allreduce(xd[:, :k], wd[:, cuts[0]], sd, k0=k0)
            ep.check()
            check(out, parts[0], k)
            host = ep.fp8_rowpar_gemm_allreduce_host(bits[:, :k], wd[:, cuts[0]], sd, k0=k0)
            assert np.array_equal(host.view(np.uint32), out.cpu().numpy().view(np.uint32))
            outs = grp.fp8_rowpar_gemm_allreduce([xd[:, :k], xd[:, k:]], [wd[:, c] for c in cuts], [sd, sd], k0s=[c.start for c in cuts])
            grp.check()
            assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))
            check(outs[0], oracle.allreduce_fold(np.stack(parts)), 2 * k)
    finally:
        ep.close()
        grp.close()


@pytest.mark.parametrize("m", [3, 40, 100, 200])
def test_ue8m0_sums_against_64_bits(dev, m):
    """UE8M0 scales spread over 2^24, so that a few blocks carry a sum and every later addition is truncated where the
    tensor cores make it.  Bound: they make eight of an accumulator's additions (two slabs), each off by less than
    2^-23 of it; the rest (at most 32 of K 8192) are rounded, errors of random sign: 8 * 2^-23 + sqrt(32) * 2^-24."""
    from weightstream_b200 import synth, tp
    n, k = 1040, 8192
    rng = np.random.default_rng(m)
    w, sc = synth.fp8_weight(rng, n, k, scale="ue8m0", bn=32, bk=32)
    sc = rng.integers(103, 128, sc.shape, dtype=np.uint8)
    wd, sd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev)
    x = torch.randn((m, k), device=dev)
    q, e = tp.act_quant_fp8(x)
    xq = q.view(torch.float8_e4m3fn).double().view(m, -1, 32) * torch.exp2(e.double() - 127).unsqueeze(2)
    ws = torch.exp2(sd.double() - 127).repeat_interleave(32, 0)[:n].repeat_interleave(32, 1)
    want = xq.view(m, k) @ (wd.view(torch.float8_e4m3fn).double() * ws).T
    ep = tp.Endpoint(max_m=m, max_n=n)
    try:
        out = ep.fp8_rowpar_gemm_allreduce(x, wd, sd, block=(32, 32))
        ep.check()
        err = float((out.double() - want).norm() / want.norm())
        assert err <= 8 * 2.0 ** -23 + 32 ** 0.5 * 2.0 ** -24, err
    finally:
        ep.close()


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("m", [1, 3, 40])  # tokens in pairs, one left over; sums by owners from 17 rows on four ranks
def test_fold_of_virtual_ranks(dev, oracle, world, m):
    from weightstream_b200 import formats as F, synth, tp
    n, k = 1040, 256  # K per rank; the last tile of rows is short
    rng = np.random.default_rng(synth.config_seed("fold-edges", m, world))
    w, sc = synth.fp8_weight(rng, n, world * k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, world * k))
    wd, sd, xd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev), torch.from_numpy(x).to(dev)
    cut = [slice(r * k, (r + 1) * k) for r in range(world)]
    parts = [oracle.fp8_gemv(w[:, c], sc, np.ascontiguousarray(x[:, c]), bn=128, bk=128, k0=c.start) for c in cut]
    grp = tp.LocalGroup(world, max_m=64, max_n=n)
    try:
        for _ in range(3):  # both banks of the exchange, and the first again
            outs = grp.fp8_rowpar_gemm_allreduce([xd[:, c].contiguous() for c in cut], [wd[:, c] for c in cut], [sd] * world,
                                                 k0s=[c.start for c in cut])
            grp.check()
            for o in outs:
                assert torch.equal(o.view(torch.int32), outs[0].view(torch.int32))
            check(outs[0], oracle.allreduce_fold(np.stack(parts)), world * k)
    finally:
        grp.close()


def _ranks_one_after_another(grp, order, xs, ws, sd, k0s):
    """One step of every rank, each on its own and after the one before has ended: all but the last give up on the words
    that are not there yet (their own have been sent).  The last one's endpoint and output."""
    from weightstream_b200 import tp
    for r in order[:-1]:
        grp.eps[r].fp8_rowpar_gemm_allreduce(xs[r], ws[r], sd, k0=k0s[r])
        with pytest.raises(tp.WsError) as ei:
            grp.eps[r].check()
        assert ei.value.status == tp._lib.WS_ERR_TIMEOUT
    r = order[-1]
    return grp.eps[r], grp.eps[r].fp8_rowpar_gemm_allreduce(xs[r], ws[r], sd, k0=k0s[r])


def _shards(dev, oracle, n, k, m, world):
    """K slices of a step, and the fold of the oracle's partial sums."""
    from weightstream_b200 import formats as F, synth
    rng = np.random.default_rng(synth.config_seed("pair-fold", m, world))
    w, sc = synth.fp8_weight(rng, n, world * k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, world * k))
    wd, sd, xd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev), torch.from_numpy(x).to(dev)
    cut = [slice(r * k, (r + 1) * k) for r in range(world)]
    parts = [oracle.fp8_gemv(w[:, c], sc, np.ascontiguousarray(x[:, c]), bn=128, bk=128, k0=c.start, threads=oracle.max_threads()) for c in cut]
    return [xd[:, c].contiguous() for c in cut], [wd[:, c] for c in cut], sd, [c.start for c in cut], oracle.allreduce_fold(np.stack(parts))


@pytest.mark.parametrize("m", [3, 4, 5, 8, 11, 12, 16, 33, 63, 128])
def test_fold_of_cta_pairs(dev, oracle, m):
    """The exchange as one rank per launch runs it, on CTA pairs (virtual ranks have none): ragged and lone groups of four
    tokens, quantised in the main kernel and ahead of it.  The last rank finds the other's words and folds them."""
    from weightstream_b200 import tp
    n, k = 2064, 512
    xs, ws, sd, k0s, want = _shards(dev, oracle, n, k, m, 2)
    grp = tp.LocalGroup(2, max_m=m, max_n=n, wait_ms=20)
    try:
        outs = []
        for order in ((1, 0), (0, 1), (1, 0)):  # both banks, and the first again
            ep, out = _ranks_one_after_another(grp, order, xs, ws, sd, k0s)
            ep.check()
            check(out, want, 2 * k)
            outs.append(out)
        assert all(torch.equal(o.view(torch.int32), outs[0].view(torch.int32)) for o in outs)
    finally:
        grp.close()


@pytest.mark.parametrize("world,m", [(4, 17), (4, 21), (4, 40), (4, 63), (8, 100), (8, 128)])
def test_owners_of_void_sums_keep_them(dev, oracle, world, m):
    """Sums by owners: the last rank folds the tiles it owns, but those of an owner that gave up on a rank never reach
    it, so that its step fails, too, instead of returning what was folded without that rank."""
    from weightstream_b200 import tp
    n, k = 2064, 256
    xs, ws, sd, k0s, want = _shards(dev, oracle, n, k, m, world)
    grp = tp.LocalGroup(world, max_m=m, max_n=n, wait_ms=20)
    try:
        for last in (0, world - 1):
            ep, out = _ranks_one_after_another(grp, [r for r in range(world) if r != last] + [last], xs, ws, sd, k0s)
            with pytest.raises(tp.WsError) as ei:
                ep.check()
            assert ei.value.status == tp._lib.WS_ERR_TIMEOUT
            tile_rows = -(-n // (ep.num_ctas // 2))  # a tile for every CTA pair
            mine = np.arange(n) // tile_rows % world == last
            check(out[:, torch.from_numpy(mine).to(dev)], want[:, mine], world * k)
    finally:
        grp.close()


def test_step_behind_one_that_waits_longer_than_two_seconds(dev):
    """A step that starts early (programmatic dependent launch) behind one whose peer stays away: the time its
    predecessor spends waiting (wait_ms) is not its own.  Both take half an SM and the second has more stages to
    fill than its ring holds, so its producer is at a stage that only the end of the first step can free."""
    from weightstream_b200 import synth, tp
    n, k = 7168, 4096
    w, sc = synth.torch_fp8_weight(n, k, seed=3, device=dev)
    x = torch.randn((1, k), device=dev)
    ep, grp = tp.Endpoint(max_m=1, max_n=n), tp.LocalGroup(2, max_m=1, max_n=n, wait_ms=3000)
    try:
        want = ep.fp8_rowpar_gemm_allreduce(x, w, sc)
        ep.check()
        grp.eps[0].fp8_rowpar_gemm_allreduce(x, w, sc)  # rank 1 takes no step
        got = ep.fp8_rowpar_gemm_allreduce(x, w, sc)
        ep.check()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
        with pytest.raises(tp.WsError) as ei:
            grp.eps[0].check()
        assert ei.value.status == tp._lib.WS_ERR_TIMEOUT
    finally:
        ep.close()
        grp.close()


def test_first_steps_on_a_side_stream_behind_a_busy_default_stream(dev):
    """What an endpoint allocates on its first step is not touched later by work on another stream than the step's."""
    from weightstream_b200 import synth, tp
    n, k, m = 1040, 8192, 40
    w, sc = synth.torch_fp8_weight(n, k, seed=5, device=dev)
    x = torch.randn((m, k), device=dev).to(torch.bfloat16)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(8):
        ep = tp.Endpoint(max_m=m, max_n=n)
        try:
            torch.cuda._sleep(3_000_000)  # ~1.5 ms on the default stream
            with torch.cuda.stream(side):
                outs = [ep.fp8_rowpar_gemm_allreduce(x, w, sc) for _ in range(200)]
            torch.cuda.synchronize()
            ep.check()
            assert all(torch.equal(o.view(torch.int32), outs[-1].view(torch.int32)) for o in outs)
        finally:
            ep.close()


@pytest.mark.parametrize("scale", ["f32", "ue8m0"])
def test_captured_steps_outlive_the_growth_of_the_scratch(dev, scale):
    """A caller's graphs of a decode step, a prefill and a MoE step, captured on an endpoint that has run nothing yet,
    replay the same bits after a longer prefill and a larger K have made the endpoint's scratch grow."""
    from weightstream_b200 import synth, tp
    n, k, kw, top_k = 1040, 1024, 4096, 4
    b = 128 if scale == "f32" else 32
    rng = np.random.default_rng(11)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    w, sc = map(to, synth.fp8_weight(rng, n, k, scale=scale, bn=b, bk=b))
    wide, wsc = map(to, synth.fp8_weight(rng, n, kw, scale=scale, bn=b, bk=b))
    w2, s2 = map(to, synth.fp4_experts(rng, 16, n, k))
    ids, rw = map(to, synth.routes(rng, 20, 16, top_k))
    h = torch.randn((20 * top_k, k), device=dev)
    x = torch.randn((3000, kw), device=dev)
    steps = [lambda ep: ep.fp8_rowpar_gemm_allreduce(x[:40, :k], w, sc, block=(b, b)),
             lambda ep: ep.fp8_rowpar_gemm_allreduce(x[:300, :k], w, sc, block=(b, b)),
             lambda ep: ep.moe_down_combine_allreduce(h, ids, rw, w2, s2, 0)]
    ep, other = (tp.Endpoint(max_m=3000, max_n=n) for _ in range(2))
    graphs = []
    try:
        want = [f(other) for f in steps]
        other.check()
        for f in steps:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                out = f(ep)
            graphs.append((g, out))
        ep.fp8_rowpar_gemm_allreduce(x[:, :k], w, sc, block=(b, b))
        ep.fp8_rowpar_gemm_allreduce(x[:100], wide, wsc, block=(b, b))
        ep.check()
        fill = torch.full((64 << 20,), 0x55, dtype=torch.uint8, device=dev)  # what was given back is written by others
        for _ in range(2):
            for (g, out), ref in zip(graphs, want):
                out.zero_()
                g.replay()
                ep.check()
                assert torch.equal(out.view(torch.int32), ref.view(torch.int32))
        assert bool((fill == 0x55).all())
    finally:
        ep.close()
        other.close()


@pytest.mark.parametrize("m", [1, 2, 3])
def test_infinite_weight_scale(dev, oracle, m):
    """Rows whose first scale is infinite are infinite, the others untouched; K leaves lanes without a chunk."""
    from weightstream_b200 import tp
    n, k = 1040, 544
    rng = np.random.default_rng(9)
    w = rng.integers(0x30, 0x48, (n, k), dtype=np.uint8)  # positive, 0.5 to 3.75
    sc = rng.uniform(0.5, 1.0, (9, 5)).astype(np.float32)
    sc[2, 0] = np.inf
    x = rng.uniform(1.0, 2.0, (m, k)).astype(np.float32)
    want = oracle.fp8_gemv(w, sc, x, bn=128, bk=128)
    ep = tp.Endpoint(max_m=m, max_n=n)
    try:
        out = ep.fp8_rowpar_gemm_allreduce(*(torch.from_numpy(a).to(dev) for a in (x, w, sc)))
        ep.check()
        hit = np.zeros(n, bool)
        hit[256:384] = True
        assert (want[:, hit] == np.inf).all() and (out.cpu().numpy()[:, hit] == np.inf).all()
        check(out[:, torch.from_numpy(~hit).to(dev)], want[:, ~hit], k)
    finally:
        ep.close()


MOE = [
    # tokens, experts, top_k, n, k, first local expert, local experts
    (8, 16, 2, 1040, 512, 0, 16),      # 16 routes: sorted and quantised in the main kernel; a whole pass per stage
    (17, 16, 1, 1040, 512, 0, 16),     # 17: by the prep kernel
    (2, 32, 6, 2048, 1280, 8, 8),      # few routes, most of them other ranks'
    (21, 16, 6, 5120, 2304, 4, 8),     # K halves of nine slabs
    (9, 8, 8, 1040, 2560, 0, 8),       # ten slabs; every expert takes every token
    (85, 12, 6, 2048, 768, 0, 12),     # the most tokens the form takes; several passes an expert, the last not full
]


@pytest.mark.parametrize("m,experts,top_k,n,k,e0,local", MOE)
def test_moe_edges(dev, oracle, m, experts, top_k, n, k, e0, local):
    from weightstream_b200 import synth, tp
    rng = np.random.default_rng(synth.config_seed(f"moe-edges-{m}-{n}-{k}", 0, 1))
    w2, s2 = synth.fp4_experts(rng, experts, n, k)
    ids, rw = synth.routes(rng, m, experts, top_k)
    h = rng.standard_normal((m * top_k, k)).astype(np.float32)
    w2, s2 = np.ascontiguousarray(w2[e0:e0 + local]), np.ascontiguousarray(s2[e0:e0 + local])
    want = oracle.moe_down_combine(w2, s2, e0, h, ids, rw, threads=oracle.max_threads())
    ep = tp.Endpoint(max_m=85, max_n=n)
    try:
        to = lambda a: torch.from_numpy(a).to(dev)
        out = ep.moe_down_combine_allreduce(to(h), to(ids), to(rw), to(w2), to(s2), e0)
        ep.check()
        check(out, want, k * top_k)
    finally:
        ep.close()


@pytest.mark.parametrize("vocab,k,m", [(16160, 2176, 12), (16160, 2176, 65)])
def test_lm_head_logits_of_a_lone_rank(dev, oracle, vocab, k, m):
    """Logits written by the tensor-core kernel itself, rows past the last whole tile, and their argmax."""
    from weightstream_b200 import formats as F, synth, tp
    rng = np.random.default_rng(synth.config_seed("head-edges", m, 1))
    w, sc = synth.fp8_weight(rng, vocab, k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, k))
    want = oracle.fp8_gemv(w, sc, x, bn=128, bk=128, threads=oracle.max_threads())
    grp = tp.LocalGroup(1, max_m=128, max_n=16, max_vocab=vocab)
    try:
        logits, amax = grp.lm_head_allgather_argmax([torch.from_numpy(x).to(dev)], [torch.from_numpy(w).to(dev)],
                                                    [torch.from_numpy(sc).to(dev)], vocab=vocab, vocab_row0s=[0], row0s=[0])
        grp.check()
        check(logits[0], want, k)
        assert torch.equal(amax[0].cpu().long(), logits[0].argmax(dim=1).cpu())
    finally:
        grp.close()


@pytest.mark.parametrize("vocab,k,m", [(vocab, 1024, m) for vocab in (2064, 8192) for m in (4, 5, 9, 20, 36, 66, 127)] +
                         [(9472, 2176, 12), (9488, 2176, 12)])  # the largest shard of CTA pairs on 148 SMs, and the first without
def test_lm_head_of_cta_pairs(dev, oracle, vocab, k, m):
    """Small shards run on CTA pairs, each finishing every other group of four tokens: logits, their argmax, and the
    argmax by itself (ragged and lone groups, every accumulator width)."""
    from weightstream_b200 import formats as F, synth, tp
    rng = np.random.default_rng(synth.config_seed("head-pairs", m, 1))
    w, sc = synth.fp8_weight(rng, vocab, k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, k))
    want = oracle.fp8_gemv(w, sc, x, bn=128, bk=128, threads=oracle.max_threads())
    wd, sd, xd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev), torch.from_numpy(x).to(dev)
    ep = tp.Endpoint(max_m=128, max_n=16, max_vocab=vocab)
    try:
        for _ in range(2):  # both banks of the candidate table
            logits, amax = ep.lm_head_allgather_argmax(xd, wd, sd, vocab_row0=0, vocab=vocab)
            _, only = ep.lm_head_allgather_argmax(xd, wd, sd, vocab_row0=0, vocab=vocab, want_logits=False)
            ep.check()
            check(logits, want, k)
            first = np.argmax(logits.cpu().numpy(), axis=1)  # the first of equals
            assert np.array_equal(amax.cpu().numpy(), first) and np.array_equal(only.cpu().numpy(), first)
    finally:
        ep.close()


@pytest.mark.parametrize("want_logits", [True, False])
@pytest.mark.parametrize("m", [3, 5, 12, 40])
def test_lm_head_of_cta_pairs_and_a_peer(dev, oracle, m, want_logits):
    """The head as one rank per launch runs it: two ranks one after the other, each alone.  The first gives up on the flags of
    the second, which finds the first's logits and candidates."""
    from weightstream_b200 import formats as F, synth, tp
    rows, k = 2064, 1024  # (not a multiple of the scale block)
    rng = np.random.default_rng(synth.config_seed("head-pairs-peer", m, 2))
    w, sc = synth.fp8_weight(rng, 2 * rows, k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, k))
    want = oracle.fp8_gemv(w, sc, x, bn=128, bk=128, threads=oracle.max_threads())
    wd, sd, xd = torch.from_numpy(w).to(dev), torch.from_numpy(sc).to(dev), torch.from_numpy(x).to(dev)
    grp = tp.LocalGroup(2, max_m=64, max_n=16, max_vocab=2 * rows, wait_ms=20)
    step = lambda r: grp.eps[r].lm_head_allgather_argmax(xd, wd[r * rows:(r + 1) * rows], sd, vocab_row0=r * rows, vocab=2 * rows,
                                                         row0=r * rows, want_logits=want_logits)
    try:
        for first in (1, 0, 1):
            step(first)
            with pytest.raises(tp.WsError) as ei:
                grp.eps[first].check()
            assert ei.value.status == tp._lib.WS_ERR_TIMEOUT
            logits, amax = step(1 - first)
            grp.eps[1 - first].check()
            if want_logits:
                check(logits, want, k)
            assert np.array_equal(amax.cpu().numpy(), np.argmax(want, axis=1))
    finally:
        grp.close()


@pytest.mark.parametrize("world,m", [(1, 1), (1, 4), (1, 5), (1, 33), (1, 128), (2, 5), (2, 65)])
def test_lm_head_equal_candidates_of_many_ctas(dev, oracle, world, m):
    """Every row of the vocabulary returns in each 1024 rows, so that every token's largest logit is there in many tiles,
    CTAs and ranks (equal rows have equal sums, bit for bit): the answer is the first of them, also by the oracle's logits."""
    from weightstream_b200 import formats as F, synth, tp
    rng = np.random.default_rng(synth.config_seed("head-ties", m, world))
    vocab, k = 17 * 1024 * world, 2048
    w, sc = synth.fp8_weight(rng, 1024, k)
    x = F.bf16_bits_to_f32(synth.activations_bf16(rng, m, k))
    ref = oracle.fp8_gemv(w, sc, x, bn=128, bk=128, threads=oracle.max_threads())
    x = torch.from_numpy(x).to(dev)
    wd, sd = torch.from_numpy(np.tile(w, (17, 1))).to(dev), torch.from_numpy(np.tile(sc, (17, 1))).to(dev)
    grp = tp.LocalGroup(world, max_m=128, max_n=16, max_vocab=vocab)
    try:
        logits, amax = grp.lm_head_allgather_argmax([x] * world, [wd] * world, [sd] * world, vocab=vocab,
                                                    vocab_row0s=[r * 17 * 1024 for r in range(world)], row0s=[0] * world)
        grp.check()
        check(logits[0], np.tile(ref, (1, 17 * world)), k)
        want = np.argmax(logits[0].cpu().numpy(), axis=1)  # the first of equals
        assert want.max() < 1024 and np.array_equal(want, np.argmax(ref, axis=1))
        for r in range(world):
            assert np.array_equal(amax[r].cpu().numpy().astype(np.int64), want)
    finally:
        grp.close()
