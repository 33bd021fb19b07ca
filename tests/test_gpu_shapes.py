"""Tensor shape codes with the exact bit (16): they name one kernel at every score count,
where the shape a plan over 64 scores starts with stands for the one that suits it."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.device import DevicePlan, row_pitch
from gnomon_b200.prepare import PreparationResult
from helpers import synth_case
from oracle import oracle

pytestmark = pytest.mark.gpu
EXACT = 16
WIDE, WIDE_SCORES_FIRST, PEOPLE, PAIRS, PAIRS_SCORES_FIRST = 20, 21, 22, 28, 29
TOL = 1e-7     # as the other tests of the 8-bit limbs


def device_rows(rows, bpv):
    pitch = row_pitch(bpv)
    d = torch.zeros((rows.shape[0], pitch), dtype=torch.uint8, device="cuda")
    d[:, :bpv] = torch.from_numpy(np.ascontiguousarray(rows[:, :bpv])).cuda()
    return d, pitch


def run(plan, d, pitch, steps):
    """Blocks (v0, n) and shapes to go on in, reset to finalize."""
    s, c = plan.outputs()
    if isinstance(steps[0], int):
        plan.set_shape(steps[0])
    plan.reset()
    for step in steps:
        if isinstance(step, int):
            plan.set_shape(step)
            assert plan.shape == step
        else:
            plan.accumulate(d[step[0]:], pitch, *step)
    plan.finalize(s, c)
    plan.sync()
    return s.cpu().numpy(), c.cpu().numpy().astype(np.uint32)


def check(prep, rows, got):
    es, ec = oracle.score_extended(rows, prep)
    np.testing.assert_array_equal(got[1], ec)
    assert oracle.rel_err(got[0], es).max() < TOL


@pytest.mark.parametrize("people,variants,scores", [
    (300, 257, 16), (1_000, 640, 64), (257, 129, 65), (700, 900, 128), (129, 65, 129),
    (1_025, 300, 257), (4_099, 700, 520), (600, 500, 700)])
def test_each_code_runs_its_kernel(cuda, people, variants, scores):
    """Up to three pairs of 128-score tiles; the two orders of a wide kernel's tiles
    give the same sums, and SM pairs those of one SM."""
    _, prep, rows, _ = synth_case(people, variants, scores=scores,
                                  config="batched_100k_x_500k_k512")
    d, pitch = device_rows(rows, prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    first = plan.shape
    assert plan.exact_shape == EXACT | 7
    got = {}
    for code in (WIDE, WIDE_SCORES_FIRST, PEOPLE, PAIRS, PAIRS_SCORES_FIRST):
        got[code] = run(plan, d, pitch, [code, (0, variants)])
        assert plan.exact_shape == code
        check(prep, rows, got[code])
    for code in (WIDE_SCORES_FIRST, PAIRS, PAIRS_SCORES_FIRST):
        np.testing.assert_array_equal(got[code][0], got[WIDE][0])
    again = run(plan, d, pitch, [first, (0, variants)])
    np.testing.assert_array_equal(again[0], got[PEOPLE][0])
    assert plan.exact_shape == EXACT | 7
    for code, exact in ((0, 0), (1, 1), (4, WIDE), (12, PAIRS)):
        plan.set_shape(code)
        assert plan.shape == code and plan.exact_shape == exact
    plan.close()


@pytest.mark.parametrize("scores", [100, 150])
def test_shapes_changed_on_the_way(cuda, scores):
    _, prep, rows, _ = synth_case(700, 3_000, scores=scores, config="batched_100k_x_500k_k512")
    d, pitch = device_rows(rows, prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    for steps in ([PEOPLE, (0, 1_024), (1_024, 960), (1_984, 1_016)],      # off a 128-boundary
                  [PAIRS_SCORES_FIRST, (0, 1_024), PEOPLE, (1_024, 1_976)],
                  [PEOPLE, (0, 1_024), PAIRS_SCORES_FIRST, (1_024, 1_024), 0, (2_048, 952)],
                  [WIDE_SCORES_FIRST, (0, 64), (64, 2_936)]):
        check(prep, rows, run(plan, d, pitch, steps))
    plan.close()


def test_plans_that_start_on_sm_pairs(cuda):
    """Over 1 GB of limbs that fill tiles of 256 scores: 512 scores x 240,000 variants,
    one cell per variant.  The default runs SM pairs, score tiles fastest; people
    as M can be pinned."""
    people, variants, scores = 300, 240_000, 512
    rng = np.random.default_rng(2)
    w = rng.standard_normal(variants).astype(np.float32)
    flipped = rng.random(variants) < 0.2
    prep = PreparationResult(np.where(flipped, -w, w), np.where(flipped, 2 * w, 0),
                             rng.integers(0, scores, variants), np.arange(variants + 1),
                             ["S%d" % k for k in range(scores)], people)
    rows = rng.integers(0, 256, (variants, people // 4), dtype=np.uint8)
    d, pitch = device_rows(rows, prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    assert plan.shape == 13 and plan.exact_shape == PAIRS_SCORES_FIRST
    got = {}
    for code in (13, PAIRS_SCORES_FIRST, PAIRS, PEOPLE):
        got[code] = run(plan, d, pitch, [code, (0, variants)])
        check(prep, rows, got[code])
    for code in (PAIRS_SCORES_FIRST, PAIRS):
        np.testing.assert_array_equal(got[code][0], got[13][0])
    plan.close()


@pytest.mark.parametrize("scores", [3, 100])
def test_autotune_keeps_results(cuda, scores):
    _, prep, rows, _ = synth_case(900, 700, scores=scores, config="batched_100k_x_500k_k512")
    d, pitch = device_rows(rows, prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    shape = plan.autotune(d, pitch)
    assert shape == plan.shape
    check(prep, rows, run(plan, d, pitch, [(0, 700)]))
    other = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    other.set_shape(shape)                     # a saved choice
    assert other.exact_shape == plan.exact_shape
    check(prep, rows, run(other, d, pitch, [(0, 700)]))
    plan.close()
    other.close()


@pytest.mark.parametrize("scores", [20, 100])
@pytest.mark.parametrize("bad", [16, 17, 18, 19, 24, 25, 26, 27, 30, 31, 32, 52])
def test_rejected_codes(cuda, bad, scores):
    _, prep, _, _ = synth_case(300, 256, scores=scores, config="batched_100k_x_500k_k512")
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    before = plan.shape
    with pytest.raises(_lib.GnomonGpuError) as ei:
        plan.set_shape(bad)
    assert ei.value.status == _lib.GNM_ERR_INVALID and plan.shape == before
    plan.close()


@pytest.mark.parametrize("scores", [1_000, 1_600, 2_400, 3_000, 4_800])
def test_default_is_not_the_slower_kernel(cuda, scores):
    """Many scores, one cell per variant: the shape a plan starts with takes no more than
    1.15 times the faster of people as M and SM pairs, and all agree."""
    people, variants = 20_000, 20_000
    rng = np.random.default_rng(scores)
    prep = PreparationResult(rng.standard_normal(variants).astype(np.float32), np.zeros(variants),
                             rng.integers(0, scores, variants), np.arange(variants + 1),
                             ["S%d" % k for k in range(scores)], people)
    gen = torch.Generator(device="cuda").manual_seed(scores)
    pitch = row_pitch(prep.bytes_per_variant)
    d = torch.randint(0, 256, (variants, pitch), dtype=torch.uint8, device="cuda", generator=gen)
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    s, c = plan.outputs()
    ms, sums, counts = {}, {}, {}
    for code in (plan.shape, PEOPLE, PAIRS_SCORES_FIRST):
        plan.set_shape(code)
        took = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.score(d, pitch, s, c)
            b.record()
            plan.sync()
            took.append(a.elapsed_time(b))
        ms[code] = min(took[1:])
        sums[code], counts[code] = s.clone(), c.clone()
    plan.close()
    first = next(iter(ms))
    assert ms[first] <= 1.15 * min(ms[PEOPLE], ms[PAIRS_SCORES_FIRST]), ms
    for code in ms:
        assert torch.equal(counts[code], counts[first])
        top = sums[first].abs().max()
        assert (sums[code] - sums[first]).abs().max() <= 1e-7 * top
