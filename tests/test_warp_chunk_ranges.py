"""The warp-chunk plan of a mesh large enough that the library's builder (am_chunks.hpp) splits
its chunks over host threads: the same plan, chunk by chunk, as each chunk's own, whatever the
number of threads the host offers, and a refusal from whichever range it comes."""
from __future__ import annotations

import os

import numpy as np

from test_warp_chunk_plan import _build_dump, _bytes, _library_plan, chunk_plan

CHUNKS = 5 * 1024 + 7  # ranges of 1024 chunks at least: up to five threads


def test_ranges_give_each_chunk_its_own_plan(tmp_path):
    exe = _build_dump(tmp_path)
    rng = np.random.default_rng(2)
    E = 32 * CHUNKS - 13  # the last chunk is not full
    conn = (np.arange(E)[:, None] + rng.integers(0, 40, size=(E, 4))).astype(np.int32)
    whole = _library_plan(exe, tmp_path, conn)
    ok, ptr, nodes, code, rank = whole
    assert ok and ptr.size == CHUNKS + 1
    cb, rb = _bytes(code).reshape(-1, 128), _bytes(rank).reshape(-1, 128)
    # the chunks beside every boundary of two to five ranges, and a sample of the others
    near = {c for R in range(2, 6) for k in range(R + 1) for c in range(CHUNKS * k // R - 2, CHUNKS * k // R + 2)}
    for c in sorted(c for c in near | set(rng.integers(0, CHUNKS, 200)) if 0 <= c < CHUNKS):
        codes, ranks, order = chunk_plan(conn, c)
        assert list(nodes[ptr[c]:ptr[c + 1]]) == order, c
        assert np.array_equal(cb[c], codes.reshape(-1)) and np.array_equal(rb[c], ranks.reshape(-1)), c
    mine = os.sched_getaffinity(0)
    for n in (1, 2, 3):  # threads follow the cores the process may use
        os.sched_setaffinity(0, set(sorted(mine)[:n]))
        try:
            again = _library_plan(exe, tmp_path, conn)
        finally:
            os.sched_setaffinity(0, mine)
        assert all(np.array_equal(a, b) for a, b in zip(whole, again))


def test_a_refusal_in_any_range(tmp_path):
    exe = _build_dump(tmp_path)
    C = 2 * 1024 + 3
    for bad in (0, 1024, C - 1):
        conn = np.zeros((32 * C, 8), dtype=np.int32)
        conn[32 * bad:32 * bad + 32] = np.arange(256).reshape(32, 8)
        assert not _library_plan(exe, tmp_path, conn)[0]
