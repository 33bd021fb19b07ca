"""Host rows of a little over the 1 MB pieces that they are staged in: no pinned buffer is
made for each block."""
import time

import numpy as np
import pytest

from gnomon_b200.pipeline import PipelineContext, run
from gnomon_b200.prepare import PreparationResult

pytestmark = pytest.mark.gpu


def test_rows_just_over_a_piece(cuda):
    """Ten blocks of 16 rows: 4.9 % longer rows take no more than four times as long (31
    times with a buffer per block; host timings vary)."""
    took = []
    for people in (4_100_000, 4_300_000):        # rows of 1,025,000 and 1,075,000 bytes
        rng = np.random.default_rng(people)
        rows = rng.integers(0, 256, 160 * (people // 4), dtype=np.uint8)
        w = rng.standard_normal(160).astype(np.float32)
        prep = PreparationResult(w, np.zeros(160), np.zeros(160), np.arange(161), ["S"], people)
        ctx, ms = PipelineContext(prep), []
        for _ in range(4):
            t0 = time.perf_counter()
            s, c = run(ctx, rows, block_variants=16)
            ms.append(time.perf_counter() - t0)
        took.append(min(ms[1:]))
        codes = (rows.reshape(160, -1)[:, -16:, None] >> np.array([0, 2, 4, 6], np.uint8)) & 3
        codes = codes.reshape(160, 64)
        want = (w[:, None] * np.array([0, 0, 1, 2])[codes]).sum(0)
        # stage tables on a grid of 2^-26 of the largest sum of three terms
        np.testing.assert_allclose(s[-64:], want, rtol=0,
                                   atol=160 / 3 * 2.0 ** -27 * 12 * np.abs(w).max())
        np.testing.assert_array_equal(c[-64:], (codes == 1).sum(0))
    assert took[1] <= 4 * took[0], took
