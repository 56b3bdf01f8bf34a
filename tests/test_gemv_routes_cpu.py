"""Which kernel a decode product goes to, as the host decides it: without a GPU every route fails at its first CUDA call, and the error
names the source file that made it. The pointers are never dereferenced."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="reads the route from the error of a machine without a GPU")
BASE = 1 << 20


def route(pkg, call):
    rc = call()
    text = pkg.lib.cmlb200_last_error().decode()
    assert rc == -2, (rc, text)
    return text.split("csrc/")[1].split(":")[0]


def pair(pkg, kind, rows, cols, up_qs=0, up_scales=0):
    types = {"q4_0": 2, "q8_0": 7, "nf4": 100}
    block = 64 if kind == "nf4" else 32
    return (pkg.QMat(types[kind], rows, cols, block, BASE, 2 * BASE, 0, None),
            pkg.QMat(types[kind], rows, cols, block, 3 * BASE + up_qs, 4 * BASE + up_scales, 0, None))


FAST = {"gemv_split.cuh", "gemv_split.cu", "call_scratch.cu", "gemv_mma.cu", "gemv_mma8.cu"}      # 16-byte copies of scales


@pytest.mark.parametrize("kind", ["q4_0", "q8_0"])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 32])
def test_both_weights_of_a_pair_have_to_be_aligned(pkg, kind, M):
    """The kernels that copy scales 16 bytes at a time take a gate and an up weight only where both are aligned; a scale plane on a
    4-byte boundary, which every entry point accepts, goes to kernels that read single scales."""
    def swiglu(gate, up):
        return route(pkg, lambda: pkg.lib.cmlb200_gemv_swiglu(gate, up, 5 * BASE, 6 * BASE, M, None))

    def norm(gate, up):
        return route(pkg, lambda: pkg.lib.cmlb200_gemv_rmsnorm(gate, up, 5 * BASE, 7 * BASE, 1e-5, 6 * BASE, M, 2, None))
    for call in [swiglu] + [norm] * (M <= 4):
        if kind != "q8_0" or M > 2:                              # (a Q8_0 pair of one or two rows goes to gemv_dp4a.cu as it is)
            assert call(*pair(pkg, kind, 4096, 1024)) in FAST
        for off in (4, 8):
            assert call(*pair(pkg, kind, 4096, 1024, up_scales=off)) not in FAST


def test_misaligned_quants_of_the_second_weight_are_refused(pkg):
    gate, up = pair(pkg, "q4_0", 4096, 1024, up_qs=8)
    assert pkg.lib.cmlb200_gemv_swiglu(gate, up, 5 * BASE, 6 * BASE, 1, None) == -1
    assert pkg.lib.cmlb200_gemv_rmsnorm(gate, up, 5 * BASE, 7 * BASE, 1e-5, 6 * BASE, 1, 2, None) == -1
    assert b"aligned" in pkg.lib.cmlb200_last_error()


@pytest.mark.parametrize("kind", ["q4_0", "q8_0"])
@pytest.mark.parametrize("rows,cols", [(4096, 1024), (12288, 4096), (4096, 11008), (32000, 4096), (2048, 8192)])
@pytest.mark.parametrize("M", range(1, 9))
def test_normalised_rows_go_where_plain_rows_go(pkg, kind, rows, cols, M):
    """One rule for both entry points (the sources of gemv_dp4a.cu hold the launches of both its kernels and no other)."""
    W = pair(pkg, kind, rows, cols)[0]
    plain = route(pkg, lambda: pkg.lib.cmlb200_gemv(W, 5 * BASE, 6 * BASE, M, None))
    assert route(pkg, lambda: pkg.lib.cmlb200_gemv_rmsnorm(W, None, 5 * BASE, 7 * BASE, 1e-5, 6 * BASE, M, 0, None)) == plain


@pytest.mark.parametrize("kind,M,rows,cols,split", [
    ("q8_0", 2, 6144, 4096, True), ("q8_0", 2, 11008, 4096, False), ("q8_0", 2, 8192, 8192, True), ("q8_0", 2, 3072, 2048, True), ("q8_0", 2, 5632, 2048, False),
    ("q4_0", 3, 6144, 4096, True), ("q4_0", 3, 14336, 4096, False), ("q4_0", 3, 5632, 2048, True), ("q4_0", 3, 4096, 11008, True), ("q8_0", 3, 14336, 4096, True)])
def test_pairs_of_few_rows_of_x(pkg, kind, M, rows, cols, split):
    """Pairs with more row tiles than fit one round of CTAs stay with the digit kernels, with and without the norm."""
    gate, up = pair(pkg, kind, rows, cols)
    taken = [route(pkg, lambda: pkg.lib.cmlb200_gemv_swiglu(gate, up, 5 * BASE, 6 * BASE, M, None)),
             route(pkg, lambda: pkg.lib.cmlb200_gemv_rmsnorm(gate, up, 5 * BASE, 7 * BASE, 1e-5, 6 * BASE, M, 2, None))]
    assert [t == "gemv_split.cuh" for t in taken] == [split, split]
