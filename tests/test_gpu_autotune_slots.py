"""The autotuner on a plain plan whose partial slots are capped: 1,200 scores x 8,192
people take 118 MB a slot, so 8 GiB hold 72, and every candidate but the shape the
plan has needs at least 74 (148 SMs, half of their CTA slots)."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch

pytestmark = pytest.mark.gpu


def test_every_other_candidate_needs_more_slots_than_allocated(cuda):
    people, variants, scores = 8_192, 2_250, 1_200      # 75 stages
    rng = np.random.default_rng(5)
    w = rng.standard_normal((variants, scores)).astype(np.float32)
    prep = prep_from_dense(w, rng.random(w.shape) < 0.1, np.ones(w.shape, bool), people)
    pitch = row_pitch(prep.bytes_per_variant)
    gen = torch.Generator(device="cuda").manual_seed(1)
    d = torch.randint(0, 256, (variants, pitch), dtype=torch.uint8, device="cuda", generator=gen)
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    try:
        with pytest.raises(_lib.GnomonGpuError):        # 75 slots are not there
            plan.set_shape((513 << 16) | 75)
        default = plan.shape
        s0, c0 = plan.score(d, pitch)
        plan.sync()
        s0, c0 = s0.cpu().numpy(), c0.cpu().numpy()
        assert plan.autotune(d, pitch) == default       # the only shape that fits
        assert default & 0xFFFF <= 72
        s1, c1 = plan.score(d, pitch)
        plan.sync()
        np.testing.assert_array_equal(c1.cpu().numpy(), c0)
        np.testing.assert_array_equal(s1.cpu().numpy(), s0)
    finally:
        plan.close()
