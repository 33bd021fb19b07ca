"""Two scores on cohorts so large that one variant split fills the GPU: a plan of few
variants has a single split, and so has any block of at most 30 rows."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("people,variants,blocks", [
    (2_430_001, 30, None),                      # 1,187 tiles of 512 bytes, one stage
    (2_430_001, 650, None),                     # 22 stages in the default shape's one split
    (2_430_001, 3_000, [(0, 1_500), (1_500, 1_470), (2_970, 30)]),   # a short last block
    (2_430_001, 95, [(0, 60), (60, 30), (90, 5)])])
def test_one_split(cuda, people, variants, blocks):
    rng = np.random.default_rng(variants)
    w = rng.standard_normal((variants, 2)).astype(np.float32)
    member = rng.random(w.shape) < np.array([1.0, 0.5])
    flipped = rng.random(w.shape) < 0.2
    w[~member] = 0
    prep = prep_from_dense(w, flipped, member, people)
    pitch = row_pitch(prep.bytes_per_variant)
    gen = torch.Generator(device="cuda").manual_seed(variants)
    d = torch.randint(0, 256, (variants, pitch), dtype=torch.uint8, device="cuda", generator=gen)
    d[:, prep.bytes_per_variant - 1] &= 3       # people % 4 == 1: the rest is padding
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    s, c = plan.outputs()
    plan.reset()
    for v0, n in blocks or [(0, variants)]:
        plan.accumulate(d[v0:], pitch, v0, n)
    plan.finalize(s, c)
    plan.sync()
    plan.close()
    s, c = s.view(people, 2).cpu().numpy(), c.view(people, 2).cpu().numpy()
    part = np.r_[0:300, people // 2:people // 2 + 300, people - 300:people]
    rows = d.cpu().numpy()
    codes = (rows[:, part // 4] >> (2 * (part % 4)).astype(np.uint8)) & 3      # [V][people]
    x = w.astype(np.float64)
    dosage = np.array([0, 0, 1, 2])[codes].T                                   # [people][V]
    called = (codes != 1).T
    want = dosage @ np.where(flipped, -x, x) + called @ np.where(flipped, 2 * x, 0)
    # tables on a grid of 2^-26 of the largest sum of three terms in a 30-row stage:
    # half a step per lookup
    err = variants / 3 * 2.0 ** -27 * 6 * 2 * np.abs(x).max()
    np.testing.assert_allclose(s[part], want, rtol=0, atol=err)
    np.testing.assert_array_equal(c[part], (codes == 1).T.astype(np.int64) @ member)
