"""A result compaction does not depend on the calls before it: not on a
captured one that grew the scratch and was never replayed, not on two that
overlapped on different streams."""
import ctypes

import numpy as np
import pytest
import torch

from devmem import cudart

pytestmark = pytest.mark.gpu


class _Call:
    """One compaction with buffers of its own."""

    def __init__(self, gpj, pairs, seed):
        rng = np.random.default_rng(seed)
        self.gpj, self.pairs = gpj, pairs
        self.data = rng.integers(0, 256, 1 << 16, dtype=np.uint8)
        start = rng.integers(0, self.data.size - 40, pairs)
        self.res = np.stack([start, start + rng.integers(0, 24, pairs)], 1).astype(np.int32)
        self.res[rng.random(pairs) < 0.4] = -1
        self.dev = torch.from_numpy(self.res).cuda()
        self.text = torch.from_numpy(self.data).cuda()
        self.matches = torch.zeros(pairs * 5, dtype=torch.int64, device="cuda")
        self.arena = torch.zeros(pairs * 24, dtype=torch.uint8, device="cuda")
        self.counts = torch.zeros(3, dtype=torch.int64, device="cuda")

    def run(self, ctx, stream=0):
        ctx.compact(self.dev.data_ptr(), self.pairs, 1, self.text.data_ptr(), self.data.size, 0,
                    self.matches.data_ptr(), self.pairs, self.arena.data_ptr(),
                    self.arena.numel(), self.counts.data_ptr(), stream)

    def check(self):
        idx = np.flatnonzero(self.res[:, 0] >= 0)
        lengths = (self.res[idx, 1] - self.res[idx, 0]).astype(np.int64)
        assert self.counts.tolist() == [idx.size, int(lengths.sum()), 0]
        got = self.matches.cpu().numpy().view(self.gpj.MATCH_DTYPE)[:idx.size]
        np.testing.assert_array_equal(got["line"], idx)
        np.testing.assert_array_equal(got["start"], self.res[idx, 0])
        np.testing.assert_array_equal(got["text_offset"], np.cumsum(lengths) - lengths)
        text = b"".join(self.data[s:e].tobytes() for s, e in self.res[idx])
        assert self.arena.cpu().numpy()[:len(text)].tobytes() == text


def _dirty_device_memory(size):
    """Leaves ones in the device memory that the next allocation of `size` bytes
    takes; returns blocks that keep it with the process until they are freed."""
    rt, blocks = cudart(), []
    for _ in range(512):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        assert rt.cudaMemset(p, 0xFF, size) == 0
        blocks.append(p)
    torch.cuda.synchronize()
    for p in blocks[1::2]:
        assert rt.cudaFree(p) == 0
    return blocks[::2]


@pytest.mark.parametrize("pairs", [300, 100_000])
def test_a_capture_that_grew_the_scratch_is_never_replayed(gpj, pairs):
    call = _Call(gpj, pairs, 1)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    kept = _dirty_device_memory(256 + (pairs + 511) // 512 * 16)
    with gpj.Context(0) as ctx:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side, capture_error_mode="relaxed"):
            call.run(ctx, side.cuda_stream)
        for _ in range(2):
            call.run(ctx)
            torch.cuda.synchronize()
            call.check()
        call.matches.zero_()
        call.arena.zero_()
        graph.replay()
        torch.cuda.synchronize()
        call.check()
        del graph
    for p in kept:
        assert cudart().cudaFree(p) == 0


def test_calls_after_overlapping_ones(gpj):
    """Overlapping calls share the context's scratch and spoil each other's
    results (all writes stay within the capacities); the ones after them are
    right again."""
    calls = [_Call(gpj, pairs, pairs) for pairs in (400_000, 130_000, 700)]
    streams = [torch.cuda.Stream() for _ in calls]
    with gpj.Context(0) as ctx:
        calls[0].run(ctx)  # the largest: the scratch grows no more
        torch.cuda.synchronize()
        for _ in range(200):
            for call, stream in zip(calls, streams):
                call.run(ctx, stream.cuda_stream)
        torch.cuda.synchronize()
        for call in calls * 2:
            call.run(ctx)
            torch.cuda.synchronize()
            call.check()
