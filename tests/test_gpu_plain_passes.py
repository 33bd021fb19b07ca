"""Plain passes of one to three score columns: every kernel shape, scores with
all, some and none of a stage's rows, several calls per run, and the counts'
eight-stage flush.  Sums are compared with the stage tables' own arithmetic,
restated here in numpy: integers on a power-of-two grid per 30-variant stage,
exact but for the FP64 sum across stages."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib, synth
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch
from gnomon_b200.prepare import PreparationResult
from helpers import synth_case
from oracle import oracle

pytestmark = pytest.mark.gpu
KERNELS = [512, 513, 1024, 1025, 2049]
# FP64 sums of at most 1,000 stages in another order: 1,000 x 2^-53 of the sum of
# the stages' magnitudes
TOL = 1e-12


def uneven(prep, K, seed):
    """The same variants with score 0 on all rows, the others on a share of them: runs
    of rows without any (whole stages) and scattered ones."""
    rng = np.random.default_rng(seed)
    V = prep.num_reconciled_variants
    member = rng.random((V, K)) < np.linspace(1.0, 0.3, K)
    member[:, 0] = True
    if K > 1:
        member[30:90, 1:] = False
    rows, cols = np.nonzero(member)
    w = rng.standard_normal(len(rows)).astype(np.float32)
    flip = rng.random(len(rows)) < 0.2
    offs = np.zeros(V + 1, np.uint64)
    np.cumsum(member.sum(axis=1), out=offs[1:])
    return PreparationResult(np.where(flip, -w, w), np.where(flip, 2 * w, 0), cols, offs,
                             [f"S{k}" for k in range(K)], prep.total_people_in_fam)


def run(prep, rows, kernel, splits, blocks=None):
    V, bpv = rows.shape[0], prep.bytes_per_variant
    pitch = row_pitch(bpv)
    d = torch.zeros((V, pitch), dtype=torch.uint8, device="cuda")
    d[:, :bpv] = torch.from_numpy(np.ascontiguousarray(rows[:, :bpv])).cuda()
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    if kernel:
        plan.set_shape((kernel << 16) | splits)
    s, c = plan.outputs()
    plan.reset()
    for v0, n in blocks or [(0, V)]:
        plan.accumulate(d[v0:], pitch, v0, n)
    plan.finalize(s, c)
    plan.sync()
    out = s.cpu().numpy(), c.cpu().numpy().astype(np.uint32)
    plan.close()
    return out


def stage_sums(prep, rows, blocks):
    """(sums [P][K], magnitudes [P][K]) on the stage grids of the given blocks."""
    V, K, P = prep.num_reconciled_variants, prep.num_scores, prep.num_people_to_score
    codes = np.zeros((V + 30, P), np.int64)
    codes[:V] = synth.unpack_codes(rows, P)
    offs = prep.sparse_row_offsets.astype(np.int64)
    at = np.repeat(np.arange(V), np.diff(offs)), prep.sparse_score_columns.astype(np.int64)
    terms = np.zeros((V + 30, K, 4), np.float32)          # by code: 0, missing, het, hom
    terms[at[0], at[1], 1] = -prep.sparse_missing_corrections
    terms[at[0], at[1], 2] = prep.sparse_weights
    terms[at[0], at[1], 3] = np.float32(2) * prep.sparse_weights
    sums, mags = np.zeros((P, K)), np.zeros((P, K))
    for v0, n in blocks:
        for r0 in range(v0, v0 + n, 30):
            rows_in = min(30, v0 + n - r0)
            t = np.zeros((30, K, 4))
            # a block on a 30-row boundary uses the plan's tables, whose last stage
            # goes on past the block
            seen = min(30, V - r0) if v0 % 30 == 0 else rows_in
            t[:seen] = terms[r0:r0 + seen]
            c = np.zeros((30, P), np.int64)
            c[:rows_in] = codes[r0:r0 + rows_in]
            g = t.reshape(10, 3, K, 4)
            table = (g[:, 0, :, :, None, None] + g[:, 1, :, None, :, None]
                     + g[:, 2, :, None, None, :])          # [10][K][4][4][4]
            top = np.abs(table).max(axis=(0, 2, 3, 4))
            up = top.astype(np.float32)
            up = np.where(up.astype(np.float64) < top, np.nextafter(up, np.float32(np.inf)), up)
            q = np.where(up > 0, np.ldexp(1.0, np.frexp(up)[1] - 27), 1.0)
            ints = np.rint(table / q[None, :, None, None, None]).astype(np.int64)
            total = np.zeros((P, K), np.int64)
            for i in range(10):
                total += ints[i][:, c[3 * i], c[3 * i + 1], c[3 * i + 2]].T
            sums += total * q
            mags += np.abs(total * q)
    return sums + prep.baseline, mags + np.abs(prep.baseline)


def check(prep, rows, got, blocks=None):
    s, c = got
    want, mags = stage_sums(prep, rows, blocks or [(0, rows.shape[0])])
    assert (np.abs(s.reshape(want.shape) - want) <= TOL * mags).all()
    np.testing.assert_array_equal(c, oracle.score_extended(rows, prep)[1])


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("kernel", [0] + KERNELS)
def test_passes(cuda, kernel, K):
    """1,003 variants in one split: 34 stages, so the counts flush five times; 2,049
    people: one full and one nearly empty 512-byte tile."""
    _, prep, rows, _ = synth_case(2_049, 1_003, scores=1, config="diff_20k_x_200k_k16")
    prep = uneven(prep, K, 7)
    check(prep, rows, run(prep, rows, kernel, 1))


@pytest.mark.parametrize("people,variants", [(1, 1), (15, 29), (2_048, 31), (8_193, 241),
                                             (40_000, 900)])
@pytest.mark.parametrize("K", [2, 3])
def test_default_shape(cuda, people, variants, K):
    _, prep, rows, _ = synth_case(people, variants, scores=1, config="diff_20k_x_200k_k16")
    prep = uneven(prep, K, people)
    check(prep, rows, run(prep, rows, 0, 0))


def test_two_scores_in_halves(cuda):
    """Two scores and enough splits for two launches of half of them each."""
    _, prep, rows, _ = synth_case(30_000, 24_000, scores=1, config="diff_20k_x_200k_k16")
    prep = uneven(prep, 2, 3)
    got = run(prep, rows, 513, 81)
    one = run(prep, rows, 513, 5)     # one by one: the same integers, other FP64 order
    np.testing.assert_array_equal(got[1], one[1])
    np.testing.assert_allclose(got[0], one[0], rtol=1e-12, atol=1e-12)


def test_calls_off_the_stage_grid(cuda):
    """Blocks off 30-row boundaries build the tables of all scores of a pass into scratch."""
    _, prep, rows, _ = synth_case(3_000, 1_000, scores=1, config="diff_20k_x_200k_k16")
    prep = uneven(prep, 5, 11)
    blocks = [(0, 100), (100, 511), (611, 389)]
    check(prep, rows, run(prep, rows, 512, 7, blocks), blocks)


@pytest.mark.parametrize("people,variants,scores,splits", [
    (183_493, 20_000, 2, 26),    # two launches of 13 splits, two waves each
    (183_493, 9_400, 2, 13),     # too few stages for them: one by one
    (250_001, 6_600, 1, 9)])     # 123 tiles: nine splits fill two waves
def test_default_shape_of_many_tiles(cuda, people, variants, scores, splits):
    """The default shape against other splits of the same rows: stage sums are exact,
    their FP64 sum (<= variants / 30 terms of <= 30 x 2 max|w|) differs in order."""
    rng = np.random.default_rng(people + variants)
    w = rng.standard_normal((variants, scores)).astype(np.float32)
    member = rng.random((variants, scores)) < np.linspace(1.0, 0.2, scores)
    prep = prep_from_dense(np.where(member, w, 0), rng.random(w.shape) < 0.2, member, people)
    bpv = prep.bytes_per_variant
    pitch = row_pitch(bpv)
    gen = torch.Generator(device="cuda").manual_seed(people)
    d = torch.randint(0, 256, (variants, pitch), dtype=torch.uint8, device="cuda", generator=gen)
    if people % 4:                   # padding people are code 00
        d[:, bpv - 1] &= (1 << 2 * (people % 4)) - 1
    out = []
    for pinned in (None, 5):
        plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
        if pinned:
            plan.set_shape((513 << 16) | pinned)
        else:
            assert plan.shape == (513 << 16) | splits
        s, c = plan.score(d, pitch)
        plan.sync()
        out.append((s.cpu().numpy(), c.cpu().numpy()))
        plan.close()
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=0,
                               atol=2 * variants / 30 * 2.0**-53 * variants * 2 * np.abs(w).max())
