"""Host rows through kept pinned buffers: several host threads at once, buffers
released between and during calls, rows longer than a staged piece, results that
come back in pieces."""
import ctypes as C
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from gnomon_b200 import _lib
from gnomon_b200.pipeline import PipelineContext, run
from gnomon_b200.prepare import PreparationResult
from helpers import synth_case
from oracle import oracle

pytestmark = pytest.mark.gpu


def release():
    e = _lib.gnm_error()
    assert _lib.load().gnm_release_cached_memory(0, C.byref(e)) == _lib.GNM_OK, e.message


def test_rows_longer_than_a_piece(cuda):
    """4,500,000 people: 1.1 MB rows and 36 MB of sums."""
    people, variants = 4_500_000, 40
    rng = np.random.default_rng(0)
    rows = rng.integers(0, 256, (variants, people // 4), dtype=np.uint8)
    w = rng.standard_normal(variants).astype(np.float32)
    need = np.arange(0, variants, 3, dtype=np.uint64)
    prep = PreparationResult(w[need.astype(int)], np.zeros(len(need)), np.zeros(len(need)),
                             np.arange(len(need) + 1), ["S"], people, required_bim_indices=need)
    s, c = run(PipelineContext(prep), rows.reshape(-1))
    part = np.r_[0:64, people - 64:people]
    codes = (rows[need.astype(int)][:, part // 4] >> (2 * (part % 4)).astype(np.uint8)) & 3
    want = (w[need.astype(int)][:, None] * np.array([0, 0, 1, 2])[codes]).sum(0)
    np.testing.assert_allclose(s[part], want, rtol=0, atol=1e-5)
    np.testing.assert_array_equal(c[part], (codes == 1).sum(0))


def test_threads_share_the_buffers(cuda):
    cases = [synth_case(p, v, scores=k) for p, v, k in
             [(5_001, 4_003, 1), (20_000, 2_000, 3), (12_345, 3_000, 9), (800, 30_000, 2)]]
    want = [run(PipelineContext(prep), np.ascontiguousarray(rows).reshape(-1))
            for _, prep, rows, _ in cases]
    for (_, prep, rows, _), (s, c) in zip(cases, want):
        es, ec = oracle.score_extended(rows, prep)
        np.testing.assert_array_equal(c, ec)
        assert oracle.rel_err(s, es).max() < 1e-6    # the reference's bar

    def one(i):
        _, prep, rows, _ = cases[i % len(cases)]
        if i % 5 == 0:
            release()
        return i, run(PipelineContext(prep), np.ascontiguousarray(rows).reshape(-1))

    with ThreadPoolExecutor(4) as pool:
        for i, (s, c) in pool.map(one, range(16)):
            np.testing.assert_array_equal(s, want[i % len(cases)][0])
            np.testing.assert_array_equal(c, want[i % len(cases)][1])
    release()
