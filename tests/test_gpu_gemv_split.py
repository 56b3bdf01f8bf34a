"""The fp16-split decode kernels (cmlb200_gemv for NF4, Q4_1, Q4_K, Q6_K, larger batches of the others) where their tiles, units
of columns, warps and batches end, against the dequantised weight in 64 bits.

Bound of an output's error: x enters as two fp16 numbers (2^-23 of every value, once more for what fp16's smallest steps
cut off of a 256-column unit), sums of a block and of the blocks are fp32 (2^-24 for each of K / 32 + 32 additions, twice that in the tensor core,
which truncates), all of it relative to the sum of the products' magnitudes."""
import numpy as np
import pytest
import torch

from gpu_util import DevQMat, make_block_stream, make_weight, stream_ptr, to_dev

pytestmark = pytest.mark.gpu
STREAM_TYPES = {"q4_1": 3, "q4_k": 12, "q5_k": 13, "q6_k": 14}


def _weight(pkg, synth, ob, orc, dev, rng, kind, N, K, block=64):
    if kind in STREAM_TYPES:
        return make_block_stream(pkg, synth, ob, orc, dev, rng, STREAM_TYPES[kind], N, K)
    return make_weight(pkg, synth, ob, orc, dev, rng, kind, N, K, block)


def _check(pkg, W, Wf, x, dev, y0=None):
    M, K = x.shape
    N = Wf.shape[0]
    d_x = to_dev(x, dev)
    d_y = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev) if y0 is None else to_dev(y0, dev)
    fn = pkg.lib.cmlb200_gemv if y0 is None else pkg.lib.cmlb200_gemv_accum
    pkg.check(fn(W.q, d_x.data_ptr(), d_y.data_ptr(), M, stream_ptr()), "gemv")
    got = d_y.cpu().numpy().astype(np.float64)
    X, F = x.astype(np.float64), Wf.astype(np.float64)
    want = X @ F.T + (0 if y0 is None else y0)
    bound = (2.0 ** -21 + (K / 32 + 32) * 2.0 ** -23) * (np.abs(X) @ np.abs(F).T) + (0 if y0 is None else 2.0 ** -23 * np.abs(want))
    assert (np.abs(got - want) <= bound + 1e-37).all(), np.max(np.abs(got - want) / (bound + 1e-37))


@pytest.mark.parametrize("kind", ["q4_0", "q8_0", "nf4", "q4_1", "q4_k", "q5_k", "q6_k"])
@pytest.mark.parametrize("N,K", [(1, 256), (16, 512), (17, 4352), (161, 1024), (2400, 768)])
def test_rows_columns_and_batches_at_their_edges(pkg, synth, ob, orc, torch_dev, kind, N, K):
    rng = np.random.default_rng(N + K)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32):
        _check(pkg, W, Wf, rng.standard_normal((M, K)).astype(np.float32), torch_dev)
    _check(pkg, W, Wf, rng.standard_normal((16, K)).astype(np.float32), torch_dev, rng.standard_normal((16, N)).astype(np.float32))


@pytest.mark.parametrize("block,K", [(32, 32), (32, 800), (64, 1088), (128, 384), (256, 768), (512, 1024)])
@pytest.mark.parametrize("M", [1, 4, 8, 32])
def test_nf4_blocks_and_partial_units(pkg, synth, ob, orc, torch_dev, block, K, M):
    rng = np.random.default_rng(block + K + M)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", 83, K, block)
    _check(pkg, W, Wf, rng.standard_normal((M, K)).astype(np.float32), torch_dev)


@pytest.mark.parametrize("M", [3, 4, 5, 32])
@pytest.mark.parametrize("N,K,block", [(13824, 5120, 64), (28352, 3904, 64), (11904, 3872, 32)])
def test_nf4_six_row_tiles_a_cta(pkg, synth, ob, orc, torch_dev, N, K, block, M):
    """What needs most shared memory: six row tiles for each of sixteen warps, the table of codes beside them."""
    rng = np.random.default_rng(N + M)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K, block)
    X, F = to_dev(rng.standard_normal((M, K)).astype(np.float32), torch_dev), to_dev(Wf, torch_dev).double()
    y = torch.empty(M, N, device=torch_dev)
    pkg.check(pkg.lib.cmlb200_gemv(W.q, X.data_ptr(), y.data_ptr(), M, stream_ptr()), "gemv")
    want, size = X.double() @ F.T, X.double().abs() @ F.abs().T
    assert ((y.double() - want).abs() <= (2.0 ** -21 + (K / 32 + 32) * 2.0 ** -23) * size).all()


@pytest.mark.parametrize("M", [4, 8])
@pytest.mark.parametrize("N,K", [(4800, 3904), (11008, 4096)])
def test_nf4_swiglu_of_large_pairs(pkg, synth, ob, orc, torch_dev, N, K, M):
    """Six row tiles a CTA of the two weights in turn. The error of silu(g) u is at most 1.1 |u| of g's and |silu(g)| of u's, and 2^-20 of
    the value for the exponential, the division and the product."""
    rng = np.random.default_rng(N + M)
    (G, Gf), (U, Uf) = (_weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K) for _ in range(2))
    X = to_dev(rng.standard_normal((M, K)).astype(np.float32), torch_dev)
    y = torch.empty(M, N, device=torch_dev)
    pkg.check(pkg.lib.cmlb200_gemv_swiglu(G.q, U.q, X.data_ptr(), y.data_ptr(), M, stream_ptr()), "swiglu")
    off, of = 2.0 ** -21 + (K / 32 + 32) * 2.0 ** -23, []
    for f in (Gf, Uf):
        F = to_dev(f, torch_dev).double()
        of.append((X.double() @ F.T, off * (X.double().abs() @ F.abs().T)))
    (g, dg), (u, du) = of
    silu = g / (1 + torch.exp(-g))
    assert ((y.double() - silu * u).abs() <= 1.1 * dg * (u.abs() + du) + silu.abs() * du + 2.0 ** -20 * (silu * u).abs()).all()


@pytest.mark.parametrize("kind,block", [("q8_0", 32), ("q4_1", 32), ("q6_k", 32), ("nf4", 64), ("nf4", 32)])
@pytest.mark.parametrize("N,K", [(24, 256), (2400, 512), (80, 768), (4752, 1280), (33, 1536), (49, 1792)])
def test_short_rows_of_large_batches(pkg, synth, ob, orc, torch_dev, kind, block, N, K):
    """17 to 32 rows of x where a row's units of columns are fewer than the warps that share them: on both sides of the line."""
    rng = np.random.default_rng(N + K)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K, block)
    for M in (17, 24, 32):
        _check(pkg, W, Wf, rng.standard_normal((M, K)).astype(np.float32), torch_dev)


@pytest.mark.parametrize("N,K,block,M,pair", [(700, 512, 64, 6, False), (4100, 768, 32, 5, False), (20000, 2048, 64, 4, False), (14300, 2048, 32, 8, False),
                                              (28660, 256, 64, 5, True), (20000, 1024, 32, 7, True), (20000, 1024, 64, 4, True), (9000, 1024, 64, 13, True),
                                              (5000, 768, 32, 30, True), (10000, 320, 32, 12, False), (10000, 8512, 32, 16, False), (400, 512, 64, 32, False)])
def test_nf4_codes_with_and_without_the_table(pkg, synth, ob, orc, torch_dev, N, K, block, M, pair):
    """Where NF4 codes come by byte permutes: a few items a CTA, several CTAs an SM, short pairs, five row tiles of blocks of 32. The bounds are
    those of test_nf4_swiglu_of_large_pairs."""
    rng = np.random.default_rng(N + K + M)
    X = to_dev(rng.standard_normal((M, K)).astype(np.float32), torch_dev)
    off, of, weights = 2.0 ** -21 + (K / 32 + 32) * 2.0 ** -23, [], []
    for _ in range(1 + pair):
        W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K, block)
        F = to_dev(Wf, torch_dev).double()
        weights.append(W)
        of.append((X.double() @ F.T, off * (X.double().abs() @ F.abs().T)))
    y = torch.full((M, N), float("nan"), device=torch_dev)
    if pair:
        pkg.check(pkg.lib.cmlb200_gemv_swiglu(weights[0].q, weights[1].q, X.data_ptr(), y.data_ptr(), M, stream_ptr()), "swiglu")
        (g, dg), (u, du) = of
        silu = g / (1 + torch.exp(-g))
        assert ((y.double() - silu * u).abs() <= 1.1 * dg * (u.abs() + du) + silu.abs() * du + 2.0 ** -20 * (silu * u).abs()).all()
    else:
        pkg.check(pkg.lib.cmlb200_gemv(weights[0].q, X.data_ptr(), y.data_ptr(), M, stream_ptr()), "gemv")
        assert ((y.double() - of[0][0]).abs() <= of[0][1]).all()


@pytest.mark.parametrize("scale", [1e-30, 1e-6, 1e6, 1e30])
@pytest.mark.parametrize("M", [3, 7, 20])
def test_any_range_of_x(pkg, synth, ob, orc, torch_dev, scale, M):
    rng = np.random.default_rng(M)
    for kind in ("nf4", "q4_k", "q8_0"):
        W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, kind, 40, 1024)
        x = (rng.standard_normal((M, 1024)) * scale).astype(np.float32)
        x[1] = 0.0                                             # a row without a largest value
        x[2, ::7] *= 1e-4                                      # values of very different sizes in one row
        _check(pkg, W, Wf, x, torch_dev)


def _with_zeros(pkg, synth, ob, orc, dev, rng, kind, N, K):
    """A weight whose first 256 columns are zero."""
    if kind == "nf4":
        packed, scales = synth.nf4_weight(rng, N, K, 64)
        packed = packed.reshape(N, K // 2)
        packed[:, :128] = 0x77
        packed = packed.reshape(-1)
        return DevQMat.from_nf4(pkg, dev, packed, scales, N, K, 64), ob.dequant_nf4(orc, packed, scales, 64, N * K).reshape(N, K)
    blocks = synth.q8_0_blocks(rng, N, K)
    b = blocks.reshape(N, K // 32, 34)
    b[:, :8, 2:] = 0
    return DevQMat.from_gguf(pkg, dev, pkg.Q8_0, blocks, N, K), ob.dequant_blocks(orc, pkg.Q8_0, blocks, N * K).reshape(N, K)


@pytest.mark.parametrize("kind", ["nf4", "q8_0"])
@pytest.mark.parametrize("K", [2048, 8192, 9216])
def test_units_of_very_different_sizes(pkg, synth, ob, orc, torch_dev, kind, K):
    """Large values that meet zero weights take no bits from those in other units of 256 columns."""
    rng = np.random.default_rng(K)
    W, Wf = _with_zeros(pkg, synth, ob, orc, torch_dev, rng, kind, 70, K)
    for M in (3, 7, 12, 30):
        x = rng.standard_normal((M, K)).astype(np.float32)
        for m in range(M):
            x[m, :256] *= 10.0 ** (m % 8)                     # (2^40 lie between the scalings of a row's units at most)
            x[m, 512:1024] *= 10.0 ** -(m % 5)
        _check(pkg, W, Wf, x, torch_dev)


@pytest.mark.parametrize("K", [1024, 4096, 11008])
@pytest.mark.parametrize("kind,most", [("nf4", 1.42e-7), ("q6_k", 1.45e-7)])
def test_error_against_64_bits(pkg, synth, ob, orc, torch_dev, kind, most, K):
    """What plain fp32 multiply-adds (NF4: 1.17 to 1.34e-7) and 24-bit digits (Q6_K: 1.28 to 1.41e-7) of these inputs give, relative to
    the norm of the results. 512 x M results: their norm spreads by less than 2 %."""
    rng = np.random.default_rng(K)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, kind, 512, K)
    for M in (1, 4, 5, 8, 9, 16, 17, 32):
        x = rng.standard_normal((4, M, K)).astype(np.float32)
        off = []
        for part in x:
            d_x, d_y = to_dev(part, torch_dev), torch.empty(M, 512, device=torch_dev)
            pkg.check(pkg.lib.cmlb200_gemv(W.q, d_x.data_ptr(), d_y.data_ptr(), M, stream_ptr()), "gemv")
            want = part.astype(np.float64) @ Wf.T.astype(np.float64)
            off.append(np.linalg.norm(d_y.cpu().numpy() - want) / np.linalg.norm(want))
        assert np.sqrt(np.mean(np.square(off))) <= most, (M, off)


@pytest.mark.parametrize("M", [12, 32])
def test_long_rows_of_nf4_blocks_of_32(pkg, synth, ob, orc, torch_dev, M):
    """More units of 256 columns than two a warp: no further off 64 bits than blocks of 64 (the bound above), and sums of large units
    are kept where zero units follow them (scalings of a row then lie further apart than an fp32 factor reaches)."""
    rng = np.random.default_rng(M)
    N, K, shares = 512, 11008, 16 if M <= 16 else 8
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K, 32)
    off = []
    for _ in range(4):
        x = rng.standard_normal((M, K)).astype(np.float32)
        d_x, d_y = to_dev(x, torch_dev), torch.empty(M, N, device=torch_dev)
        pkg.check(pkg.lib.cmlb200_gemv(W.q, d_x.data_ptr(), d_y.data_ptr(), M, stream_ptr()), "gemv")
        want = x.astype(np.float64) @ Wf.T.astype(np.float64)
        off.append(np.linalg.norm(d_y.cpu().numpy() - want) / np.linalg.norm(want))
    for scale in (1.0, 1e6):
        x = rng.standard_normal((M, K)).astype(np.float32)
        x[:, :256 * shares] *= scale
        x[:, 256 * shares:512 * shares] = 0.0
        _check(pkg, W, Wf, x, torch_dev)
    assert np.sqrt(np.mean(np.square(off))) <= 1.42e-7, off


@pytest.mark.parametrize("kind,batches", [("nf4", (1, 4, 5, 8, 9, 16, 17, 32)), ("q8_0", (9, 32))])
def test_infinities_and_nan(pkg, synth, ob, orc, torch_dev, kind, batches):
    """Rows of x that are not finite give what fp32 multiply-adds give: infinities with their signs, NaN where an infinity meets a zero
    weight or one of the other sign; the rows beside them stay as they are."""
    rng = np.random.default_rng(9)
    N, K = 130, 2304
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    for M in batches:
        x = rng.standard_normal((M, K)).astype(np.float32)
        clean = x.copy()
        bad = sorted({0, M - 1})
        x[0, 300] = np.inf
        x[M - 1, 7] = -np.inf
        if M > 4:
            x[2, [5, 2000]] = np.inf
            x[3, 1000] = np.nan
            bad += [2, 3]
        d_x, d_y = to_dev(x, torch_dev), torch.empty(M, N, device=torch_dev)
        pkg.check(pkg.lib.cmlb200_gemv(W.q, d_x.data_ptr(), d_y.data_ptr(), M, stream_ptr()), "gemv")
        got = d_y.cpu().numpy()
        with np.errstate(invalid="ignore"):
            want = (x.astype(np.float64)[:, None, :] * Wf.astype(np.float64)[None]).sum(2)
        assert np.array_equal(got[bad], want[bad].astype(np.float32), equal_nan=True)
        rest = [m for m in range(M) if m not in bad]
        assert np.isfinite(got[rest]).all()
        if rest:
            d_c, d_z = to_dev(clean, torch_dev), torch.empty(M, N, device=torch_dev)
            pkg.check(pkg.lib.cmlb200_gemv(W.q, d_c.data_ptr(), d_z.data_ptr(), M, stream_ptr()), "gemv")
            assert np.array_equal(got[rest], d_z.cpu().numpy()[rest])


def test_streams_keep_their_rows_apart(pkg, synth, ob, orc, torch_dev):
    rng = np.random.default_rng(5)
    W, Wf = _weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", 4096, 4096)
    xs = [to_dev(rng.standard_normal((16, 4096)).astype(np.float32), torch_dev) for _ in range(4)]
    alone = []
    for x in xs:
        y = torch.empty(16, 4096, device=torch_dev)
        pkg.check(pkg.lib.cmlb200_gemv(W.q, x.data_ptr(), y.data_ptr(), 16, stream_ptr()), "gemv")
        alone.append(y)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    out = [torch.empty(16, 4096, device=torch_dev) for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, x, y in zip(streams, xs, out):
            pkg.check(pkg.lib.cmlb200_gemv(W.q, x.data_ptr(), y.data_ptr(), 16, s.cuda_stream), "gemv")
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(alone, out))


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("M", [1, 4, 8, 32])
def test_nf4_weights_written_by_the_launch_before(pkg, torch_dev, captured, M):
    """NF4 weights quantized, or given new scales by another product (whose successors begin early), right before the product that reads
    them: the same bits as with a synchronisation between, in order and captured."""
    lib, N, K, block = pkg.lib, 1024, 4096, 64
    g = torch.Generator(torch_dev).manual_seed(M)
    qs, scales = torch.zeros(N * K // 2, dtype=torch.uint8, device=torch_dev), torch.zeros(N * K // block, device=torch_dev)
    W = pkg.QMat(pkg.NF4, N, K, block, qs.data_ptr(), scales.data_ptr(), 0, None)
    maker_qs = torch.randint(0, 256, (4096 * 2048,), dtype=torch.uint8, device=torch_dev, generator=g)
    maker_sc = (torch.rand(4096 * 2048 // 32, device=torch_dev, generator=g) * 0.01).half()
    maker = pkg.QMat(pkg.Q8_0, 4096, 2048, 32, maker_qs.data_ptr(), maker_sc.data_ptr(), 0, None)     # 16 x 4096 results: the scales
    sources = [(torch.randn(N, K, device=torch_dev, generator=g), torch.randn(16, 2048, device=torch_dev, generator=g)) for _ in range(6)]
    x = torch.randn(M, K, device=torch_dev, generator=g)
    w, h, y = torch.empty(N, K, device=torch_dev), torch.empty(16, 2048, device=torch_dev), [torch.empty(M, N, device=torch_dev) for _ in range(2)]

    def run(stream, between):
        pkg.check(lib.cmlb200_quantize_nf4(w.data_ptr(), N * K, block, qs.data_ptr(), scales.data_ptr(), stream), "quantize")
        between()
        pkg.check(lib.cmlb200_gemv(W, x.data_ptr(), y[0].data_ptr(), M, stream), "gemv")
        between()
        pkg.check(lib.cmlb200_gemv(maker, h.data_ptr(), scales.data_ptr(), 16, stream), "scales")
        between()
        pkg.check(lib.cmlb200_gemv(W, x.data_ptr(), y[1].data_ptr(), M, stream), "gemv")

    stream, want = torch.cuda.Stream(), []
    for a, b in sources:
        w.copy_(a)
        h.copy_(b)
        torch.cuda.synchronize()
        run(stream.cuda_stream, torch.cuda.synchronize)
        torch.cuda.synchronize()
        want.append([t.clone() for t in y])
    graph = torch.cuda.CUDAGraph()
    if captured:
        with torch.cuda.graph(graph, stream=stream):
            run(stream.cuda_stream, lambda: None)
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(stream):
        for a, b in sources * 3:
            w.copy_(a)
            h.copy_(b)
            if captured:
                graph.replay()
            else:
                run(stream.cuda_stream, lambda: None)
            got.append([t.clone() for t in y])
    torch.cuda.synchronize()
    for i, pair in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(pair, want[i % len(want)])), i
