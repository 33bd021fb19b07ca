"""The correction gradient of scores whose dS the 8-bit limbs cannot hold: it is summed
from the dS values of the people missing at each variant, at the edges of that
sum's steps (64 people a lane, 2,048 a warp, 16 scores a tile), with padding
people coded as missing, and in a time near that of finite scores."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch

pytestmark = pytest.mark.gpu


def make(people, variants, scores, missing, seed):
    """(plan, device rows, pitch, codes [variants][people]) with missing padding people."""
    rng = np.random.default_rng(seed)
    padded = (people + 3) // 4 * 4
    codes = rng.choice(np.array([0, 1, 2, 3], np.uint8), (variants, padded),
                       p=[0.6 - missing, missing, 0.3, 0.1])
    codes[:, people:] = 1
    q = codes.reshape(variants, -1, 4)
    rows = q[..., 0] | q[..., 1] << 2 | q[..., 2] << 4 | q[..., 3] << 6
    prep = prep_from_dense(np.ones((variants, scores), np.float32),
                           np.zeros((variants, scores), bool),
                           np.ones((variants, scores), bool), people)
    pitch = row_pitch(prep.bytes_per_variant)
    d = torch.zeros((variants, pitch), dtype=torch.uint8, device="cuda")
    d[:, :rows.shape[1]] = torch.from_numpy(rows).cuda()
    return DevicePlan(prep, engine=_lib.ENGINE_PLAIN), d, pitch, codes[:, :people]


def check_corrections(got, codes, gs):
    """-(sum of dS over the missing), an FP64 sum rounded once to FP32; infinities and
    NaN where a person with one is missing."""
    miss = (codes == 1).astype(np.float64)
    finite = np.where(np.isfinite(gs), gs, 0).astype(np.float64)
    want, size = -(miss @ finite), miss @ np.abs(finite)
    bad = miss @ (~np.isfinite(gs)).astype(np.float64) > 0
    np.testing.assert_array_equal(np.isfinite(got), ~bad)
    assert (np.abs(got - want)[~bad] <= (2.0 ** -24 * np.abs(want) + 1e-12 * size)[~bad]).all()


@pytest.mark.parametrize("missing", [0.02, 0.5])
@pytest.mark.parametrize("people,variants,scores", [
    (1, 1, 1), (63, 19, 2), (64, 20, 15), (65, 21, 16), (515, 257, 17), (2_047, 300, 3),
    (2_048, 256, 33), (2_049, 3_001, 4), (5_003, 700, 16), (40_001, 131, 5)])
def test_scores_that_are_not_finite(cuda, people, variants, scores, missing):
    """Every score, then every second one, holds a NaN or an infinity."""
    plan, d, pitch, codes = make(people, variants, scores, missing, people)
    rng = np.random.default_rng(people + 1)
    for step in (1, 2):
        gs = rng.standard_normal((people, scores)).astype(np.float32)
        for k in range(0, scores, step):
            gs[rng.integers(people), k] = (np.nan, np.inf, -np.inf)[k % 3]
        gw, gc = plan.backward(d, pitch, torch.from_numpy(gs).cuda(), grad_corr=True)
        plan.sync()
        gw, gc = gw.cpu().numpy(), gc.cpu().numpy().astype(np.float64)
        check_corrections(gc[:, ::step], codes, gs[:, ::step])
        if step == 2:                  # their neighbours are finite and on limbs
            assert np.isfinite(gc).sum() >= variants * (scores // 2)
            dosage = np.array([0.0, 0.0, 1.0, 2.0])[codes]
            for got, want in ((gw[:, 1::2], dosage @ gs[:, 1::2].astype(np.float64)),
                              (gc[:, 1::2], -((codes == 1) @ gs[:, 1::2].astype(np.float64)))):
                scale = np.abs(gs[:, 1::2]).sum(axis=0)
                assert (np.abs(got - want) <= 1e-6 * scale).all()
    plan.close()


def test_infinities_keep_their_sign(cuda):
    """One +inf: the correction gradient is -inf exactly where that person is missing."""
    plan, d, pitch, codes = make(3_000, 500, 2, 0.05, 9)
    gs = np.ones((3_000, 2), np.float32)
    gs[1_777, 0], gs[55, 1] = np.inf, -np.inf
    _, gc = plan.backward(d, pitch, torch.from_numpy(gs).cuda(), grad_corr=True)
    plan.sync()
    gc = gc.cpu().numpy()
    np.testing.assert_array_equal(gc[:, 0] == -np.inf, codes[:, 1_777] == 1)
    np.testing.assert_array_equal(gc[:, 1] == np.inf, codes[:, 55] == 1)
    plan.close()


def test_time_with_nan_everywhere(cuda):
    """A loss that turned NaN: no more than eight times a finite step (one thread per
    variant and score over all people took hundreds of times)."""
    plan, d, pitch, _ = make(20_000, 8_192, 16, 0.01, 4)
    took = []
    for gs in (torch.randn(20_000, 16, device="cuda"), torch.full((20_000, 16), torch.nan,
                                                                  device="cuda")):
        ms = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                plan.backward(d, pitch, gs, grad_corr=True)
            b.record()
            plan.sync()
            ms.append(a.elapsed_time(b) / 4)
        took.append(min(ms[1:]))
    plan.close()
    assert took[1] < 8 * took[0], took


@pytest.mark.parametrize("power", [9, 12, 16, 19])
@pytest.mark.parametrize("missing", [0.001, 0.01])
def test_one_dominant_gradient(cuda, power, missing):
    """One person's dS 2^power times the others': where that person is called, the sum
    over the missing is as accurate as its FP32 terms."""
    plan, d, pitch, codes = make(20_000, 400, 4, missing, power)
    gs = np.random.default_rng(power).standard_normal((20_000, 4)).astype(np.float32)
    gs[4_711, 1], gs[4_711, 3] = 2.0 ** power, -2.0 ** power
    gs[5::7, 3] = 0                    # people outside a keep set
    _, gc = plan.backward(d, pitch, torch.from_numpy(gs).cuda(), grad_corr=True)
    plan.sync()
    plan.close()
    gc = gc.cpu().numpy().astype(np.float64)
    check_corrections(gc[:, [1, 3]], codes, gs[:, [1, 3]])


@pytest.mark.parametrize("people,variants,scores", [
    (700, 300, 300), (33, 40, 600), (600_001, 20, 16), (2_100_003, 3, 3)])
def test_scores_of_different_scales(cuda, people, variants, scores):
    """Largest values and spreads are found per score: every third score dominated by
    one person, magnitudes from 2^-60 to 2^60, a score of zeros."""
    plan, d, pitch, codes = make(people, variants, scores, 0.02, scores)
    rng = np.random.default_rng(people)
    gs = rng.standard_normal((people, scores)).astype(np.float32)
    gs *= np.ldexp(np.float32(1), rng.integers(-60, 60, scores)).astype(np.float32)
    gs[rng.integers(people), ::3] *= 2.0 ** 15
    gs[:, 1] = 0
    gw, gc = plan.backward(d, pitch, torch.from_numpy(gs).cuda(), grad_corr=True)
    plan.sync()
    plan.close()
    gw, gc = gw.cpu().numpy().astype(np.float64), gc.cpu().numpy().astype(np.float64)
    check_corrections(gc[:, ::3], codes, gs[:, ::3])
    g = gs.astype(np.float64)
    top = np.abs(g).max(axis=0)
    for got, x in ((gw, np.array([0.0, 0.0, 1.0, 2.0])[codes]), (gc, (codes == 1) * -1.0)):
        want = x @ g
        # limbs leave a value within 2^-31.9 of its score's largest; one rounding to FP32
        err = 2.0 ** -31.9 * (np.abs(x).sum(axis=1)[:, None] * top) + 2.0 ** -24 * np.abs(want)
        assert (np.abs(got - want) <= err).all()
