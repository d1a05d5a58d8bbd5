"""gexs_ctx_upload: bytes arrive unchanged from pageable and pinned sources, at
sizes around a slot (0.5 MiB), the staging threshold (4 MiB) and the ring (8
MiB), with empty and odd pieces; a pageable source may be overwritten as soon
as the call returns; calls from several threads on one context."""
import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

from gexs_b200._capi import GexsUploadPiece as Piece, check, lib

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _upload(ctx, arrays, stream):
    dev = [torch.zeros(max(a.size, 1), dtype=torch.uint8, device="cuda") for a in arrays]
    p = (Piece * len(arrays))()
    for i, (d, a) in enumerate(zip(dev, arrays)):
        p[i] = Piece(d.data_ptr(), a.ctypes.data, a.size, None)
    torch.cuda.synchronize()
    check(lib().gexs_ctx_upload(ctx.h, p, len(arrays), C.c_void_p(stream.cuda_stream)), "upload")
    return dev


@pytest.mark.parametrize("sizes", [
    [0, 1, 7], [4 * MIB - 1], [4 * MIB], [MIB, MIB + 1, 3 * MIB - 1], [16 * MIB + 5, 0, 3],
    [53 * MIB + 11, 1, 17 * MIB]])
def test_bytes_arrive(gpu_ctx, sizes):
    rng = np.random.Generator(np.random.PCG64(len(sizes)))
    want = [rng.integers(0, 256, n, dtype=np.uint8) for n in sizes]
    stream = torch.cuda.Stream()
    src = [w.copy() for w in want]
    dev = _upload(gpu_ctx, src, stream)
    for s in src:
        s[:] = 0                      # pageable: already read
    stream.synchronize()
    pinned = [torch.from_numpy(w).pin_memory() if w.size else torch.empty(0, dtype=torch.uint8)
              for w in want]
    half = [p.numpy() if i % 2 == 0 else w for i, (p, w) in enumerate(zip(pinned, want))]
    dev2 = _upload(gpu_ctx, half, stream)
    stream.synchronize()
    for d, d2, w in zip(dev, dev2, want):
        assert np.array_equal(d.cpu().numpy()[:w.size], w)
        assert np.array_equal(d2.cpu().numpy()[:w.size], w)


def test_threads_share_a_context(gpu_ctx):
    rng = np.random.Generator(np.random.PCG64(9))
    want = [rng.integers(0, 256, 9 * MIB + k, dtype=np.uint8) for k in range(4)]
    got = [None] * 4

    def one(k):
        s = torch.cuda.Stream()
        got[k] = _upload(gpu_ctx, [want[k]], s)[0]
        s.synchronize()

    th = [threading.Thread(target=one, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy()[:w.size], w)


def test_pageable_source_is_refused_under_capture(gpu_ctx):
    """A captured copy would read the staging slot at each replay; later
    uploads are unaffected."""
    rng = np.random.Generator(np.random.PCG64(12))
    want = rng.integers(0, 256, 17 * MIB, dtype=np.uint8)
    dev = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    p = (Piece * 1)(Piece(dev.data_ptr(), want.ctypes.data, want.size, None))
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        status = lib().gexs_ctx_upload(gpu_ctx.h, p, 1, C.c_void_p(stream.cuda_stream))
    assert status != 0
    got = _upload(gpu_ctx, [want], stream)[0]
    stream.synchronize()
    assert np.array_equal(got.cpu().numpy(), want)


def test_waiting_for_the_stream_costs_no_processor_time(gpu_ctx):
    """With other work queued before the copies the threads sleep: the process
    takes far less processor time than one core spinning for that long."""
    stream = torch.cuda.Stream()
    want = np.full(40 * MIB, 7, dtype=np.uint8)
    _upload(gpu_ctx, [want], stream)
    stream.synchronize()
    dev = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    p = (Piece * 1)(Piece(dev.data_ptr(), want.ctypes.data, want.size, None))
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1000000000)                     # about half a second
    wall, cpu = time.perf_counter(), time.process_time()
    check(lib().gexs_ctx_upload(gpu_ctx.h, p, 1, C.c_void_p(stream.cuda_stream)), "upload")
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    stream.synchronize()
    assert wall > 0.2
    assert cpu < 0.5 * wall, (cpu, wall)
    assert np.array_equal(dev.cpu().numpy(), want)
