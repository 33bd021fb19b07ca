"""More score tiles than a grid has rows (65,535): 2,100,000 scores of one cell each."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.device import DevicePlan, row_pitch
from gnomon_b200.prepare import PreparationResult

pytestmark = pytest.mark.gpu


def test_two_million_scores(cuda):
    people, variants, scores = 7, 64, 2_100_000
    rng = np.random.default_rng(1)
    per = np.array([len(range(v, scores, variants)) for v in range(variants)])
    cols = np.concatenate([np.arange(v, scores, variants) for v in range(variants)])
    w = rng.standard_normal(scores).astype(np.float32)        # of cell e, score cols[e]
    flipped = rng.random(scores) < 0.2
    prep = PreparationResult(np.where(flipped, -w, w), np.where(flipped, 2 * w, 0), cols,
                             np.concatenate([[0], np.cumsum(per)]),
                             ["S%d" % k for k in range(scores)], people)
    codes = rng.integers(0, 4, (variants, 8), dtype=np.uint8)
    codes[:, people:] = 0
    q = codes.reshape(variants, 2, 4)
    rows = q[..., 0] | q[..., 1] << 2 | q[..., 2] << 4 | q[..., 3] << 6
    pitch = row_pitch(2)
    d = torch.zeros((variants, pitch), dtype=torch.uint8, device="cuda")
    d[:, :2] = torch.from_numpy(rows).cuda()
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    s, c = plan.score(d, pitch)
    plan.sync()
    plan.close()
    s, c = s.view(people, scores).cpu().numpy(), c.view(people, scores).cpu().numpy()
    mine = codes[np.repeat(np.arange(variants), per), :people].T     # [people][cell]
    x = w.astype(np.float64)
    dosage = np.array([0, 0, 1, 2])[mine]
    want = np.zeros((people, scores))
    want[:, cols] = np.where(mine == 1, 0, np.where(flipped, 2 * x - dosage * x, dosage * x))
    # one cell: its weight to 2^-31.9 and its correction (twice it) likewise
    np.testing.assert_allclose(s, want, rtol=0, atol=4 * 2.0 ** -31.9 * np.abs(x).max())
    missing = np.zeros((people, scores), np.int32)
    missing[:, cols] = mine == 1
    np.testing.assert_array_equal(c, missing)
