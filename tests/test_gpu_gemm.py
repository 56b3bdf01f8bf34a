"""GPU parity of the tcgen05 prefill dequant-GEMM (bf16 activations/outputs, fp32 accumulate
in tensor memory). Tolerance 1e-2 relative to max|y| (bf16 tensor-core prefill), as the path
is specified; the oracle is fed the fp32 values of the bf16-rounded activations."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

from conftest import rel_err_inf
from gpu_util import DevQMat, gemm_status, make_weight, stream_ptr, to_dev

pytestmark = pytest.mark.gpu
TOL = 1e-2


def _gemm(pkg, synth, W, x, N, dev, splits=0):
    M = x.shape[0]
    xb, _ = synth.bf16_round(x)
    d_x = to_dev(xb.reshape(x.shape), dev)
    d_y = torch.zeros((M, N), dtype=torch.uint16, device=dev)
    if splits:
        pkg.check(pkg.lib.cmlb200_gemm_bf16_splitk(W.q, d_x.data_ptr(), d_y.data_ptr(), M, splits, stream_ptr()), "gemm")
    else:
        pkg.check(pkg.lib.cmlb200_gemm_bf16(W.q, d_x.data_ptr(), d_y.data_ptr(), M, stream_ptr()), "gemm")
    assert gemm_status(pkg) == 0, "a bounded wait inside the tensor-core kernel expired"
    return synth.bf16_to_f32(d_y.cpu().numpy())


@pytest.mark.parametrize("kind", ["nf4", "q4_0", "q8_0"])
@pytest.mark.parametrize("M", [1, 16, 64, 100, 256, 300, 513, 1000])
def test_gemm_matches_oracle(pkg, synth, ob, orc, torch_dev, kind, M):
    rng = np.random.default_rng(200 + M)
    N, K = 200, 512                                    # ragged N (tile is 128 rows)
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    got = _gemm(pkg, synth, W, x, N, torch_dev)
    want = ob.linear_nt(orc, xr.reshape(x.shape), Wf)
    assert rel_err_inf(got, want) <= TOL


@pytest.mark.parametrize("splits", [1, 2, 4])
def test_gemm_split_k_agrees(pkg, synth, ob, orc, torch_dev, splits):
    rng = np.random.default_rng(300)
    N, K, M = 256, 2048, 64
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    got = _gemm(pkg, synth, W, x, N, torch_dev, splits=splits)
    assert rel_err_inf(got, ob.linear_nt(orc, xr.reshape(x.shape), Wf)) <= TOL


@pytest.mark.parametrize("M", [64, 512, 2048])
def test_gemm_nf4_config_shape_sampled(pkg, synth, ob, orc, torch_dev, M):
    """NF4 4096 x 4096, block 64 at the benchmark's M values; the oracle checks sampled rows and
    columns (its full triple loop would take minutes)."""
    rng = np.random.default_rng(400 + M)
    N = K = 4096
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, "nf4", N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    got = _gemm(pkg, synth, W, x, N, torch_dev)
    ms = rng.choice(M, 16, replace=False)
    ns = rng.choice(N, 256, replace=False)
    want = ob.linear_nt(orc, xr.reshape(x.shape)[ms], Wf[ns])
    assert np.abs(got[np.ix_(ms, ns)] - want).max() / np.abs(want).max() <= TOL
    # whole-output check against an fp64 matmul of the same dequantised weights
    full = xr.reshape(x.shape).astype(np.float64) @ Wf.T.astype(np.float64)
    assert rel_err_inf(got, full) <= TOL


@pytest.mark.parametrize("kind", ["nf4", "q4_0", "q8_0"])
@pytest.mark.parametrize("K", [64, 320])
@pytest.mark.parametrize("M", [257, 288, 300, 511, 512, 600])
def test_gemm_pairs_of_ctas_at_their_edges(pkg, synth, ob, orc, torch_dev, kind, K, M):
    """More than 256 rows over 74 pairs of 256 weight rows (one round, or two with 600 rows), the last pair ragged: the second MMA's
    smallest and largest number of columns, one slab of K and an odd number of them."""
    rng = np.random.default_rng(K + M)
    N = 18900
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    got = _gemm(pkg, synth, W, x, N, torch_dev)
    want = (to_dev(xr.reshape(x.shape), torch_dev).double() @ to_dev(Wf, torch_dev).double().T).cpu().numpy()
    assert rel_err_inf(got, want) <= TOL


@pytest.mark.parametrize("kind,N,K,M", [("q4_0", 11008, 4096, 512), ("nf4", 4096, 4096, 2000), ("q4_0", 4096, 11008, 2048), ("nf4", 4096, 4096, 4096)])
def test_gemm_large_shapes_repeated(pkg, synth, ob, orc, torch_dev, kind, N, K, M):
    """LLaMA-sized weights with 512 to 4096 activation rows, incl. a ragged last tile; every output
    against an fp64 product, three launches in a row (cold and warm caches: a pipeline race would show
    as whole output columns off by a K slab's worth)."""
    rng = np.random.default_rng(900 + M)
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    full = xr.reshape(x.shape).astype(np.float64) @ Wf.T.astype(np.float64)
    for _ in range(3):
        assert rel_err_inf(_gemm(pkg, synth, W, x, N, torch_dev), full) <= TOL


@pytest.mark.parametrize("kind,K", [("q4_0", 1376), ("q8_0", 96), ("nf4", 1376), ("q4_0", 32)])
@pytest.mark.parametrize("M", [40, 300])
def test_gemm_k_tail_of_half_a_slab(pkg, synth, ob, orc, torch_dev, kind, K, M):
    """cols % 64 == 32 (LLaMA-7B's FFN width split over 8 ranks is 1376): the last 64-wide slab is
    half real, half zero; rows of an odd number of blocks start on odd scale indices."""
    rng = np.random.default_rng(500 + K + M)
    N = 200
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K, block=32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    got = _gemm(pkg, synth, W, x, N, torch_dev)
    assert rel_err_inf(got, ob.linear_nt(orc, xr.reshape(x.shape), Wf)) <= TOL
    if K >= 256:
        got2 = _gemm(pkg, synth, W, x, N, torch_dev, splits=3)
        assert rel_err_inf(got2, ob.linear_nt(orc, xr.reshape(x.shape), Wf)) <= TOL


@pytest.mark.parametrize("kind,N,K,M", [
    ("q4_0", 130, 544, 15), ("q8_0", 127, 1088, 17), ("nf4", 129, 1088, 80), ("q4_0", 1024, 4096, 77),     # clusters, ragged tiles
    ("q4_0", 1030, 1056, 255), ("nf4", 1030, 1088, 257), ("q8_0", 1030, 1056, 272),                        # 256 | 257: one MMA a slab or two
    ("q4_0", 20000, 160, 511), ("q8_0", 20000, 160, 512), ("nf4", 20000, 160, 513), ("q4_0", 20000, 64, 1025)])   # several tiles a CTA
@pytest.mark.parametrize("splits", [0, 2, 8])
def test_gemm_tiles_and_clusters(pkg, synth, ob, orc, torch_dev, kind, N, K, M, splits):
    """The shapes pick_shape and a caller's split come to, at the edges of tiles, slabs and clusters, twice with the same bits. Each
    output is bf16 (2^-9) of a sum over weights that were rounded twice (2^-9 each, as rms over K terms at most that of one):
    3 x 2^-9 of the norm of the outputs."""
    rng = np.random.default_rng(1100 + N + M)
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K, block=32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    _, xr = synth.bf16_round(x)
    want = xr.reshape(x.shape).astype(np.float64) @ Wf.T.astype(np.float64)
    got = _gemm(pkg, synth, W, x, N, torch_dev, splits=splits)
    assert np.linalg.norm(got - want) <= 3 * 2.0 ** -9 * np.linalg.norm(want)
    assert rel_err_inf(got, want) <= TOL
    assert np.array_equal(got, _gemm(pkg, synth, W, x, N, torch_dev, splits=splits))


@pytest.mark.parametrize("M", [48, 300])
def test_gemm_output_modes(pkg, synth, ob, orc, torch_dev, M):
    """The epilogues the LLaMA prefill uses: fp32 output, accumulation onto an fp32 residual, and
    SwiGLU of an earlier gate output (in place), with and without the split-K reduction (M = 48
    takes it on this shape)."""
    rng = np.random.default_rng(700 + M)
    N, K = 384, 1024
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, "q4_0", N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    xb, xr = synth.bf16_round(x)
    want = ob.linear_nt(orc, xr.reshape(x.shape), Wf)
    d_x = to_dev(xb.reshape(x.shape), torch_dev)
    out32 = torch.zeros((M, N), dtype=torch.float32, device=torch_dev)
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 1, out32.data_ptr(), None, stream_ptr()), "out_f32")
    torch.cuda.synchronize()
    assert rel_err_inf(out32.cpu().numpy(), want) <= TOL
    h0 = rng.standard_normal((M, N)).astype(np.float32)
    h = to_dev(h0, torch_dev)
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 2, h.data_ptr(), None, stream_ptr()), "acc_f32")
    torch.cuda.synchronize()
    assert np.abs(h.cpu().numpy() - (h0 + want)).max() <= TOL * np.abs(want).max()
    gate = rng.standard_normal((M, N)).astype(np.float32)
    gb, gr = synth.bf16_round(gate)
    gr = gr.reshape(gate.shape)
    buf = to_dev(gb.reshape(gate.shape), torch_dev)
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 3, buf.data_ptr(), buf.data_ptr(), stream_ptr()), "swiglu")
    torch.cuda.synchronize()
    ref = (gr / (1.0 + np.exp(-gr.astype(np.float64)))) * want
    assert np.abs(synth.bf16_to_f32(buf.cpu().numpy()) - ref).max() <= TOL * np.abs(ref).max()
    assert gemm_status(pkg) == 0
    assert pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 3, buf.data_ptr(), None, stream_ptr()) == -1      # SwiGLU needs the gate
    assert pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 7, buf.data_ptr(), None, stream_ptr()) == -1



@pytest.mark.parametrize("N,K,M,offset", [(384, 128, 33, 0), (384, 1024, 77, 0), (384, 1024, 77, 1), (130, 1024, 45, 0), (1031, 512, 255, 0), (4, 256, 1, 0)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_gemm_cluster_sums_at_their_edges(pkg, synth, ob, orc, torch_dev, mode, N, K, M, offset):
    """What a cluster adds, four weight rows at a time: rows that are no whole fours, outputs off their alignment, every epilogue,
    and nothing written beside them. Twice rounded weights (2^-9 each) and a bf16 output: 3 x 2^-9 of the norm of the outputs."""
    rng = np.random.default_rng(1700 + N + M)
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, "q4_0", N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    xb, xr = synth.bf16_round(x)
    want = xr.reshape(x.shape).astype(np.float64) @ Wf.T.astype(np.float64)
    first = rng.standard_normal((M, N)).astype(np.float32)
    bf16 = mode in (0, 3)
    if mode == 3:
        fb, fr = synth.bf16_round(first)
        g = fr.reshape(first.shape).astype(np.float64)
        want, fill = g / (1.0 + np.exp(-g)) * want, fb.reshape(-1)
    else:
        fill = np.zeros(M * N, np.uint16) if bf16 else first.reshape(-1)
    buf = np.concatenate([fill[:1]] * 8 + [fill] + [fill[:1]] * 8)
    buf = np.roll(buf, offset)
    d = to_dev(buf, torch_dev)
    at = d.data_ptr() + (8 + offset) * buf.itemsize
    d_x = to_dev(xb.reshape(x.shape), torch_dev)
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, mode, at, at if mode == 3 else None, stream_ptr()), "gemm")
    torch.cuda.synchronize()
    assert gemm_status(pkg) == 0
    out = d.cpu().numpy()
    got = out[8 + offset:8 + offset + M * N]
    got = (synth.bf16_to_f32(got) if bf16 else got).reshape(M, N)
    assert np.linalg.norm(got - (first if mode == 2 else 0) - want) <= 3 * 2.0 ** -9 * np.linalg.norm(want)
    assert np.array_equal(out[:8 + offset], buf[:8 + offset]) and np.array_equal(out[8 + offset + M * N:], buf[8 + offset + M * N:])


@pytest.mark.parametrize("N,K,M", [(18900, 320, 300), (18821, 64, 257), (18821, 128, 511), (18900, 64, 600)])
@pytest.mark.parametrize("mode", [1, 2, 3])
def test_gemm_pairs_of_ctas_with_every_epilogue(pkg, synth, ob, orc, torch_dev, mode, N, K, M):
    """fp32 output, a residual, SwiGLU in place, of 74 pairs of CTAs (with 600 rows twice) whose last one ends in its second CTA's first
    rows or in their middle, and nothing written beside them. Bound as with clusters."""
    rng = np.random.default_rng(N + M + mode)
    W, Wf = make_weight(pkg, synth, ob, orc, torch_dev, rng, "q4_0", N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    xb, xr = synth.bf16_round(x)
    d_x = to_dev(xb.reshape(x.shape), torch_dev)
    want = to_dev(xr.reshape(x.shape), torch_dev).double() @ to_dev(Wf, torch_dev).double().T
    first = torch.randn(16 + M * N, device=torch_dev, generator=torch.Generator(torch_dev).manual_seed(M))
    first = first.to(torch.bfloat16) if mode == 3 else first
    before = first[8:-8].double().reshape(M, N)
    if mode == 3:
        want = before * torch.sigmoid(before) * want
    out = first.clone()
    at = out[8:].data_ptr()
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, mode, at, at if mode == 3 else None, stream_ptr()), "gemm")
    torch.cuda.synchronize()
    assert gemm_status(pkg) == 0
    got = out[8:-8].double().reshape(M, N)
    assert ((got - before if mode == 2 else got) - want).norm() <= 3 * 2.0 ** -9 * want.norm()
    assert torch.equal(out[:8], first[:8]) and torch.equal(out[-8:], first[-8:])


@pytest.mark.parametrize("M", [48, 200, 300])
def test_gemm_residual_below_the_normal_range(pkg, synth, ob, orc, torch_dev, M):
    """A residual of subnormal numbers is added to, not flushed: with a cluster's sum, one tile of rows, and two."""
    rng = np.random.default_rng(M)
    N, K = 384, 1024
    W, _ = make_weight(pkg, synth, ob, orc, torch_dev, rng, "q4_0", N, K)
    d_x = torch.zeros(M, K, dtype=torch.bfloat16, device=torch_dev)
    h0 = (rng.standard_normal((M, N)) * 1e-39).astype(np.float32)
    h = to_dev(h0, torch_dev)
    pkg.check(pkg.lib.cmlb200_gemm_bf16_ex(W.q, d_x.data_ptr(), M, 2, h.data_ptr(), None, stream_ptr()), "acc_f32")
    assert np.array_equal(h.cpu().numpy(), h0) and np.count_nonzero(h0) > 0


def test_gemm_q8_0_weights_are_rounded_once(pkg, synth, torch_dev):
    """Unit vectors through a Q8_0 weight with every quant and scales from the smallest to the largest finite half: outputs are the
    products, each rounded to bf16 once. An infinite scale stands for infinite weights."""
    K = N = 256
    scales = np.array([0x0400, 0x0001, 0x3c00, 0x1234, 0x7bff, 0x2e66, 0xbc01, 0x0000], np.uint16)
    blocks = np.zeros((N, K // 32, 34), np.uint8)
    for n in range(N):
        for b in range(K // 32):
            blocks[n, b, :2] = np.frombuffer(scales[(n + b) % 8].tobytes(), np.uint8)
            blocks[n, b, 2:] = (np.arange(32) + 32 * ((n // 8 + b) % 8)).astype(np.uint8)
    W = DevQMat.from_gguf(pkg, torch_dev, pkg.Q8_0, blocks.reshape(-1), N, K)
    s = scales.view(np.float16).astype(np.float32)
    s[1] *= 0.5                                              # C-ML's reading of a subnormal half
    q = blocks[:, :, 2:].view(np.int8).astype(np.float32)
    w = (q * s[(np.arange(N)[:, None] + np.arange(K // 32)[None]) % 8][:, :, None]).reshape(N, K)
    got = _gemm(pkg, synth, W, np.eye(K, dtype=np.float32), N, torch_dev)
    want = synth.bf16_to_f32(synth.bf16_round(np.ascontiguousarray(w.T))[0].reshape(K, N))
    assert np.array_equal(got, want)
    blocks[5, 3, :2] = (0x00, 0x7c)
    blocks[5, 3, 2:] = np.arange(1, 33)
    W = DevQMat.from_gguf(pkg, torch_dev, pkg.Q8_0, blocks.reshape(-1), N, K)
    got = _gemm(pkg, synth, W, np.ones((2, K), np.float32), N, torch_dev)
    assert (got[:, 5] == np.inf).all() and np.isfinite(np.delete(got, 5, 1)).all()


@pytest.fixture(scope="module")
def impatient(tmp_path_factory, pkg):
    """The same source with waits that give up after a single poll."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    root = Path(__file__).resolve().parents[1]
    src, out = root / "c-ml_b200" / "csrc", tmp_path_factory.mktemp("impatient") / "gemm.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-DCML_GEMM_SPIN_LIMIT=1u", "-Xcompiler", "-fPIC", "-shared",
                    "-I", str(root / "include"), "-I", str(src), *(str(src / f) for f in ("gemm_tcgen05.cu", "shim.cu", "call_scratch.cu")),
                    "-Xlinker", "-Bsymbolic", "-o", str(out)], check=True, capture_output=True)
    lib = C.CDLL(str(out))
    for name in ("cmlb200_gemm_bf16", "cmlb200_gemm_status"):
        getattr(lib, name).argtypes = getattr(pkg.lib, name).argtypes
    return lib


@pytest.mark.parametrize("kind,N,K,M", [("q4_0", 4096, 4096, 77), ("nf4", 1024, 2048, 200), ("q8_0", 2048, 4096, 512), ("q4_0", 20000, 1024, 513)])
def test_gemm_waits_that_expire(pkg, synth, ob, orc, torch_dev, impatient, kind, N, K, M):
    """Launches whose waits run out report it and return with nothing of theirs under way: launches in front of and behind them,
    which share their SMs, are right, and so is the next call."""
    rng = np.random.default_rng(1200 + N)
    W, _ = make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K)
    x = to_dev(synth.bf16_round(rng.standard_normal((M, K)).astype(np.float32))[0].reshape(M, K), torch_dev)
    y, want, lost = [torch.zeros((M, N), dtype=torch.uint16, device=torch_dev) for _ in range(3)]
    st = C.c_int(0)
    pkg.check(pkg.lib.cmlb200_gemm_bf16(W.q, x.data_ptr(), want.data_ptr(), M, stream_ptr()), "gemm")
    for _ in range(20):
        y.zero_()
        assert impatient.cmlb200_gemm_bf16(W.q, x.data_ptr(), lost.data_ptr(), M, stream_ptr()) == 0
        pkg.check(pkg.lib.cmlb200_gemm_bf16(W.q, x.data_ptr(), y.data_ptr(), M, stream_ptr()), "gemm")
        torch.cuda.synchronize()
        assert torch.equal(y.view(torch.int16), want.view(torch.int16))
        assert impatient.cmlb200_gemm_status(C.byref(st), 1) == 0 and st.value != 0
    assert gemm_status(pkg) == 0
