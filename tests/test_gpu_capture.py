"""Decode products under CUDA graph capture and on many streams: their scratch belongs to the graph that holds the launches, or to the
call in stream order. Outputs are compared bit for bit with the same call outside a capture (the kernels' order of sums is fixed)."""
import ctypes as C

import numpy as np
import pytest
import torch

import __graft_entry__ as entry
from gpu_util import make_block_stream, make_weight, to_dev
from llama_util import TINY, build, device_model

pytestmark = pytest.mark.gpu
STREAM_TYPES = {"q4_1": 3, "q4_k": 12, "q5_k": 13, "q6_k": 14}
KINDS = ["q4_0", "q8_0", "nf4", "q4_1", "q4_k", "q5_k", "q6_k"]


@pytest.fixture(scope="module")
def weights(pkg, synth, ob, orc, torch_dev):
    made = {}

    def get(kind, N=352, K=1024):
        if (kind, N, K) not in made:
            rng = np.random.default_rng(len(kind) + N)
            made[kind, N, K] = (make_block_stream(pkg, synth, ob, orc, torch_dev, rng, STREAM_TYPES[kind], N, K) if kind in STREAM_TYPES
                                else make_weight(pkg, synth, ob, orc, torch_dev, rng, kind, N, K))[0]
        return made[kind, N, K]
    return get


def gemv(pkg, W, x, y, stream):
    pkg.check(pkg.lib.cmlb200_gemv(W.q, x.data_ptr(), y.data_ptr(), x.shape[0], stream), "gemv")


def rows(rng, M, K, dev):
    return to_dev(rng.standard_normal((M, K)).astype(np.float32), dev)


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("kind", KINDS)
def test_every_capture_mode(pkg, weights, torch_dev, kind, mode):
    rng = np.random.default_rng(1)
    W = weights(kind)
    stream = torch.cuda.Stream()
    for M in (1, 5, 9, 32):
        first, second = rows(rng, M, 1024, torch_dev), rows(rng, M, 1024, torch_dev)
        want = [torch.empty(M, 352, device=torch_dev) for _ in range(2)]
        for x, y in zip((first, second), want):
            gemv(pkg, W, x, y, torch.cuda.current_stream().cuda_stream)
        x, y = first.clone(), torch.empty(M, 352, device=torch_dev)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
            gemv(pkg, W, x, y, stream.cuda_stream)
        for i, source in enumerate((first, second, first)):
            x.copy_(source)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, want[i % 2])


@pytest.mark.parametrize("kind,M", [("nf4", 6), ("nf4", 32), ("q8_0", 8), ("q8_0", 20), ("q4_k", 16), ("q4_0", 32)])
def test_two_graphs_of_one_capture_stream_side_by_side(pkg, weights, torch_dev, kind, M):
    rng = np.random.default_rng(2)
    W = weights(kind, 2048, 4096)
    capture, streams = torch.cuda.Stream(), [torch.cuda.Stream(), torch.cuda.Stream()]
    xs = [rows(rng, M, 4096, torch_dev) for _ in streams]
    ys, want, graphs = [torch.empty(M, 2048, device=torch_dev) for _ in xs], [torch.empty(M, 2048, device=torch_dev) for _ in xs], []
    for x, w in zip(xs, want):
        gemv(pkg, W, x, w, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=capture):
            for _ in range(8):
                gemv(pkg, W, x, y, capture.cuda_stream)
        graphs.append(g)
    for _ in range(40):
        for y in ys:
            y.zero_()
        torch.cuda.synchronize()
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want))


def test_branches_of_one_capture(pkg, weights, torch_dev):
    """Two streams of one capture run side by side within its graph."""
    rng = np.random.default_rng(3)
    W = weights("nf4", 2048, 4096)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    xs = [rows(rng, 16, 4096, torch_dev) for _ in range(2)]
    ys, want = [[torch.empty(16, 2048, device=torch_dev) for _ in xs] for _ in range(2)]
    for x, w in zip(xs, want):
        gemv(pkg, W, x, w, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=a):
        b.wait_stream(a)
        for _ in range(6):
            gemv(pkg, W, xs[0], ys[0], a.cuda_stream)
            gemv(pkg, W, xs[1], ys[1], b.cuda_stream)
        a.wait_stream(b)
    for _ in range(20):
        for y in ys:
            y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want))


def test_graph_outlives_its_capture_stream(pkg, weights, torch_dev):
    """The capture stream is destroyed, other streams and captures come and go, and the graph still has its scratch."""
    rng = np.random.default_rng(4)
    lib, W = pkg.lib, weights("q4_k", 2048, 4096)
    x, y, want = rows(rng, 12, 4096, torch_dev), torch.zeros(12, 2048, device=torch_dev), torch.empty(12, 2048, device=torch_dev)
    gemv(pkg, W, x, want, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()

    def captured(x, y):
        s, g = C.c_void_p(), C.c_void_p()
        pkg.check(lib.cmlb200_stream_create(C.byref(s)), "stream")
        pkg.check(lib.cmlb200_graph_begin(s), "begin")
        gemv(pkg, W, x, y, s)
        pkg.check(lib.cmlb200_graph_end(s, C.byref(g)), "end")
        pkg.check(lib.cmlb200_stream_destroy(s), "destroy")
        return g
    kept = captured(x, y)
    run = torch.cuda.Stream()
    other, y2 = rows(rng, 12, 4096, torch_dev), torch.empty(12, 2048, device=torch_dev)
    torch.cuda.synchronize()
    for _ in range(20):
        g = captured(other, y2)
        side = torch.cuda.Stream()
        pkg.check(lib.cmlb200_graph_launch(g, C.c_void_p(side.cuda_stream)), "launch")
        pkg.check(lib.cmlb200_graph_launch(kept, C.c_void_p(run.cuda_stream)), "launch")
        gemv(pkg, W, other, y2, side.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        y.zero_()
        pkg.check(lib.cmlb200_graph_destroy(g), "destroy")
    pkg.check(lib.cmlb200_graph_destroy(kept), "destroy")


def test_graphs_give_their_scratch_back(pkg, weights, torch_dev):
    """200 graphs, of 2 MB of scratch each, one after another: what stays is no more than the pool may keep."""
    rng = np.random.default_rng(5)
    W = weights("nf4", 2048, 4096)
    x, y = rows(rng, 32, 4096, torch_dev), torch.empty(32, 2048, device=torch_dev)
    stream = torch.cuda.Stream()

    def once():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            gemv(pkg, W, x, y, stream.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        g.reset()
    for _ in range(3):
        once()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(200):
        once()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 34 << 20


def test_more_streams_than_a_pool_of_streams(pkg, weights, torch_dev):
    rng = np.random.default_rng(6)
    W = weights("q6_k", 2048, 4096)
    streams = [torch.cuda.Stream() for _ in range(20)]
    xs = [rows(rng, 9, 4096, torch_dev) for _ in streams]
    want, ys = [[torch.zeros(9, 2048, device=torch_dev) for _ in xs] for _ in range(2)]
    for x, w in zip(xs, want):
        gemv(pkg, W, x, w, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for _ in range(5):
        for s, x, y in zip(streams, xs, ys):
            gemv(pkg, W, x, y, s.cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(y, w) for y, w in zip(ys, want))


@pytest.mark.parametrize("gtype", [2, 7, 12])
def test_greedy_loop_of_batches_equals_single_steps(pkg, tmp_path, torch_dev, gtype):
    """The captured loop and uncaptured steps run the same kernels, so their tokens are the same ones."""
    rng = np.random.default_rng(7 + gtype)
    path = tmp_path / "model.gguf"
    build(entry, rng, TINY, path, qtype=gtype, wscale=0.06)
    steps = 6
    for batch in (1, 5, 9, 16):
        prompts = [rng.integers(0, TINY["vocab"], 3 + b % 4).astype(np.int32) for b in range(batch)]
        first = rng.integers(0, TINY["vocab"], batch).astype(np.int32)
        models = [device_model(pkg, TINY, path, max_batch=batch) for _ in range(2)]
        try:
            for m in models:
                for b, p in enumerate(prompts):
                    assert pkg.lib.cml_llama_prefill_sequence(m, b, pkg.np_ptr(p), len(p)) == 0
            want, tokens = [], first
            for _ in range(steps):
                logits = pkg.tensor_to_numpy(pkg.lib.cml_llama_forward_batch(models[0], pkg.np_ptr(tokens), batch))
                tokens = logits.argmax(1).astype(np.int32)
                want.append(tokens)
            out, ms = np.zeros((steps, batch), np.int32), C.c_float(0)
            for half in (0, 1):                                  # the second call replays the graph of the first
                start = first if half == 0 else out[steps // 2 - 1].copy()
                part = np.zeros((steps // 2, batch), np.int32)
                assert pkg.lib.cml_llama_decode_greedy(models[1], pkg.np_ptr(start), batch, steps // 2, pkg.np_ptr(part), C.byref(ms)) == 0
                out[half * (steps // 2):(half + 1) * (steps // 2)] = part
            assert np.array_equal(out, np.array(want))
        finally:
            for m in models:
                pkg.lib.cml_llama_free(m)
