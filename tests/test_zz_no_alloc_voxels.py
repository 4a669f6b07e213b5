"""ppc_bin_agents_noalloc at the sizes where its kernels change path: voxels
with up to 24 agents (their chain), more (a block's sort) and more than 4096
(rank counting), partial tiles, and buffers that are only 4-byte aligned."""
import ctypes as C

import numpy as np
import pytest

from paraphysicell_b200 import build
from paraphysicell_b200.abi import Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("clump,spread,side", [(1, 0, 1), (24, 300, 7), (25, 300, 7), (4096, 1000, 17),
                                               (4097, 77, 16), (60, 131072 - 60, 101)])
def test_crowded_voxels(clump, spread, side, shift):
    import torch

    from paraphysicell_b200 import device

    build.ensure_built()
    L = device.lib()
    L.ppc_bin_agents_noalloc.argtypes = [C.POINTER(Mesh), C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    rng = np.random.default_rng(clump)
    n = clump + spread
    pos = rng.random((n, 3)) * 30 * side
    pos[rng.permutation(n)[:clump]] = 30 * (side // 2) + rng.random((clump, 3)) * 29
    mesh = Mesh.make(3, (0, 0, 0), (30 * side,) * 3)
    key = (pos / 30.0).astype(np.int64)
    key = key[:, 0] + side * (key[:, 1] + side * key[:, 2])
    want_counts = np.bincount(key, minlength=side ** 3)
    want_agents = np.lexsort((-np.arange(n), key))
    dev = torch.from_numpy(pos.ravel()).cuda()
    counts = torch.full((side ** 3 + shift,), -7, dtype=torch.int32, device="cuda")
    agents = torch.full((n + shift,), -7, dtype=torch.int32, device="cuda")
    for _ in range(2):
        rc = L.ppc_bin_agents_noalloc(C.byref(mesh), dev.data_ptr(), n, counts[shift:].data_ptr(),
                                      agents[shift:].data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0, L.ppc_last_error()
        assert np.array_equal(counts.cpu().numpy()[shift:], want_counts)
        assert np.array_equal(agents.cpu().numpy()[shift:], want_agents)
        assert (counts[:shift] == -7).all() and (agents[:shift] == -7).all()


def _case(n, side, seed):
    import torch

    rng = np.random.default_rng(seed)
    pos = rng.random((n, 3)) * 30 * side
    key = (pos / 30.0).astype(np.int64)
    key = key[:, 0] + side * (key[:, 1] + side * key[:, 2])
    return {"mesh": Mesh.make(3, (0, 0, 0), (30 * side,) * 3), "n": n, "pos": torch.from_numpy(pos.ravel()).cuda(),
            "counts": torch.full((side ** 3,), -7, dtype=torch.int32, device="cuda"),
            "agents": torch.full((n,), -7, dtype=torch.int32, device="cuda"),
            "want": (np.bincount(key, minlength=side ** 3), np.lexsort((-np.arange(n), key)))}


def _call(L, c, stream):
    rc = L.ppc_bin_agents_noalloc(C.byref(c["mesh"]), c["pos"].data_ptr(), c["n"], c["counts"].data_ptr(),
                                  c["agents"].data_ptr(), stream.cuda_stream)
    assert rc == 0, L.ppc_last_error()


def _check(c):
    assert np.array_equal(c["counts"].cpu().numpy(), c["want"][0])
    assert np.array_equal(c["agents"].cpu().numpy(), c["want"][1])
    c["counts"].fill_(-7)
    c["agents"].fill_(-7)


def _lib():
    from paraphysicell_b200 import device

    build.ensure_built()
    L = device.lib()
    L.ppc_bin_agents_noalloc.argtypes = [C.POINTER(Mesh), C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


def test_calls_on_two_streams_run_one_after_another():
    """Calls of different grids queued on two streams without a wait between
    them, and calls after them."""
    import torch

    L = _lib()
    cases = [_case(131072, 101, 1), _case(700, 5, 2), _case(20000, 9, 3), _case(1, 3, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for r in range(3):
        for k, c in enumerate(cases):
            _call(L, c, streams[(k + r) % 2])
        torch.cuda.synchronize()
        for c in cases:
            _check(c)
        torch.cuda.synchronize()


def test_captured_call_replays():
    import torch

    L = _lib()
    c, other = _case(30000, 30, 5), _case(4000, 4, 6)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    _call(L, c, stream)
    torch.cuda.synchronize()
    _check(c)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _call(L, c, torch.cuda.current_stream())
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        _check(c)
        _call(L, other, torch.cuda.current_stream())
        torch.cuda.synchronize()
        _check(other)
        torch.cuda.synchronize()


def test_all_agents_in_one_voxel():
    """131,072 agents in the middle one of 27 voxels: compared by the whole
    grid in some 3.4 ms. A walk along the voxel's chain takes 380 ms; the bound
    lies a factor of ten from both."""
    import torch

    L = _lib()
    c = _case(131072, 3, 7)
    c["pos"].copy_(30.0 + c["pos"] / 3.0)
    counts = np.zeros(27, np.int64)
    counts[13] = c["n"]
    c["want"] = (counts, np.arange(c["n"])[::-1])
    stream = torch.cuda.current_stream()
    _call(L, c, stream)
    _check(c)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    _call(L, c, stream)
    b.record()
    torch.cuda.synchronize()
    _check(c)
    assert a.elapsed_time(b) < 35.0


def test_an_error_left_by_another_call_is_not_this_ones():
    """An allocation that failed elsewhere in the program leaves an error
    pending; a call returns its own status and its own bins, and so does the
    next one."""
    import torch

    L = _lib()
    cases = [_case(5000, 9, 8), _case(90000, 60, 9)]
    torch.cuda.synchronize()
    runtime = C.CDLL("libcudart.so.12")
    for _ in range(3):
        for c in cases:
            p = C.c_void_p()
            assert runtime.cudaMalloc(C.byref(p), C.c_size_t(1 << 60)) != 0
            try:
                _call(L, c, torch.cuda.current_stream())
            finally:
                runtime.cudaGetLastError()
            _check(c)
