"""The narrow 8-bit tensor kernel (people as M, genotypes expanded into tensor
memory) at the sizes where its split can go wrong: edges of the 256- and
512-person tiles, of the 128-variant stages and of the 16-score tiles, one to
many CTAs per tile, several calls per run, and S32 blocks at their limit."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch
from helpers import synth_case
from oracle import oracle

pytestmark = pytest.mark.gpu
NARROW8 = 6
# limbs leave each value within 2^-31.9 of its score's largest one; 1e-7 is the
# 8-bit kernels' tolerance against the extended oracle
TOL = 1e-7


def run(prep, rows, blocks=None):
    V, bpv = rows.shape[0], prep.bytes_per_variant
    pitch = row_pitch(bpv)
    d = torch.zeros((V, pitch), dtype=torch.uint8, device="cuda")
    d[:, :bpv] = torch.from_numpy(np.ascontiguousarray(rows[:, :bpv])).cuda()
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    plan.set_shape(NARROW8)
    out = []
    for _ in range(2):               # a second run writes over the first one's slots
        s, c = plan.outputs()
        plan.reset()
        for v0, n in blocks or [(0, V)]:
            plan.accumulate(d[v0:], pitch, v0, n)
        plan.finalize(s, c)
        plan.sync()
        out.append((s.cpu().numpy(), c.cpu().numpy().astype(np.uint32)))
    plan.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    return out[1]


def check(prep, rows, got):
    s, c = got
    es, ec = oracle.score_extended(rows, prep)
    np.testing.assert_array_equal(c, ec)
    assert oracle.rel_err(s, es).max() < TOL


@pytest.mark.parametrize("people,variants,scores", [
    (1, 1, 1), (3, 127, 2), (64, 128, 16), (255, 129, 15), (256, 257, 17), (257, 1000, 16),
    (511, 640, 33), (512, 385, 64), (513, 900, 8), (769, 131, 48), (1025, 20_000, 9),
    (5_000, 3_001, 16), (40_000, 260, 20)])
def test_tile_edges(cuda, people, variants, scores):
    _, prep, rows, _ = synth_case(people, variants, scores=scores,
                                  config="batched_100k_x_500k_k512")
    check(prep, rows, run(prep, rows))


def test_calls_of_different_lengths(cuda):
    """Later calls meet more, fewer and other slots than the first; one starts
    off a 128-variant boundary and runs on BF16 limbs into the same slots."""
    _, prep, rows, _ = synth_case(700, 9_000, scores=18, config="batched_100k_x_500k_k512")
    for blocks in ([(0, 128), (128, 5_120), (5_248, 256), (5_504, 3_496)],
                   [(0, 4_864), (4_864, 64), (4_928, 4_072)], [(0, 64), (64, 8_936)]):
        check(prep, rows, run(prep, rows, blocks))


@pytest.mark.parametrize("byte,code", [(0xFF, 3), (0x55, 1)], ids=["hom-alt", "missing"])
def test_blocks_at_the_s32_limit(cuda, byte, code):
    """Every weight at the top of the limb range against every person's largest
    dosage (or missing call), more than 2^17 variants per CTA: 127 x 2 x 64 per
    variant, flushed before 2^31.  All sums are equal and known."""
    people, variants, K = 148 * 512 + 1, (1 << 17) + 300, 2
    w = np.full((variants, K), 0.75, np.float32)
    w[:, 1] = -0.75
    flipped = np.zeros((variants, K), bool)
    flipped[:, 1] = code == 1        # missing corrections of 2w on the second score
    prep = prep_from_dense(w, flipped, np.ones((variants, K), bool), people)
    pitch = row_pitch(prep.bytes_per_variant)
    rows = torch.full((variants * pitch,), byte, dtype=torch.uint8, device="cuda")
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    plan.set_shape(NARROW8)
    s, c = plan.score(rows, pitch)
    plan.sync()
    s, c = s.view(people, K).cpu().numpy(), c.view(people, K).cpu().numpy()
    # hom-alt: 2w per variant; missing: baseline 2w per flipped variant, minus 2w
    want = np.array([1.5, -1.5]) * variants if code == 3 else np.zeros(2)
    np.testing.assert_allclose(s, np.broadcast_to(want, s.shape), rtol=0, atol=TOL * variants)
    np.testing.assert_array_equal(c, variants if code == 1 else 0)
    plan.close()


@pytest.mark.parametrize("people,variants,scores,blocks", [
    (38_000, 257, 40, None), (57_000, 140, 64, [(0, 128), (128, 12)]),
    (76_000, 300, 17, [(0, 128), (128, 172)]), (152_000, 130, 3, None)])
def test_whole_tiles_then_shares(cuda, people, variants, scores, blocks):
    """Two and more rounds of people tiles per CTA: whole tiles first, then even
    shares of the rest, with each of the kernel's tile sizes; a second call adds
    to the slots of both."""
    _, prep, rows, _ = synth_case(people, variants, scores=scores,
                                  config="batched_100k_x_500k_k512")
    check(prep, rows, run(prep, rows, blocks))


def default_run(prep, rows, steps):
    """Over 64 scores: a plan in its default shape; a step is a block (v0, n) or a
    shape to continue in.  Two runs, the second over the first one's sums."""
    V, bpv = rows.shape[0], prep.bytes_per_variant
    pitch = row_pitch(bpv)
    d = torch.zeros((V, pitch), dtype=torch.uint8, device="cuda")
    d[:, :bpv] = torch.from_numpy(np.ascontiguousarray(rows[:, :bpv])).cuda()
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    shape = plan.shape
    assert shape == (13 if prep.num_scores > 128 else 5)
    for _ in range(2):
        s, c = plan.outputs()
        plan.set_shape(shape)
        plan.reset()
        for step in steps:
            if isinstance(step, int):
                plan.set_shape(step)
            else:
                plan.accumulate(d[step[0]:], pitch, *step)
        plan.finalize(s, c)
        plan.sync()
    out = s.cpu().numpy(), c.cpu().numpy().astype(np.uint32)
    plan.close()
    return out


@pytest.mark.parametrize("people,variants,scores", [
    (1, 1, 65), (257, 129, 70), (700, 1_000, 97), (513, 385, 128), (5_000, 640, 129),
    (255, 3_001, 200), (1_025, 300, 257), (12_801, 260, 96), (640, 513, 512), (300, 200, 530)])
def test_people_as_m_over_64_scores(cuda, people, variants, scores):
    _, prep, rows, _ = synth_case(people, variants, scores=scores,
                                  config="batched_100k_x_500k_k512")
    check(prep, rows, default_run(prep, rows, [(0, variants)]))


@pytest.mark.parametrize("people,scores", [(700, 100), (700, 150), (9_500, 150)])
def test_wide_blocks_in_the_same_run(cuda, people, scores):
    """Blocks off a 128-variant boundary, and shapes changed on the way, add to the
    wide partials; the finalize sums both."""
    _, prep, rows, _ = synth_case(people, 3_000, scores=scores, config="batched_100k_x_500k_k512")
    pair = 12
    for steps in ([(0, 1_024), (1_024, 960), (1_984, 1_016)], [(0, 64), (64, 2_936)],
                  [(0, 1_024), pair, (1_024, 1_024), 0, (2_048, 952)],
                  [pair, (0, 1_024), 13 if scores > 128 else 5, (1_024, 1_976)], []):
        got = default_run(prep, rows, steps)
        if steps:
            check(prep, rows, got)
        else:                            # nothing accumulated: the baseline alone
            sums = got[0].reshape(people, scores)
            assert not got[1].any() and (sums == sums[0]).all()


def test_captured_wide_blocks_replay_in_any_order(cuda):
    """Over 64 scores: blocks off a 128-variant boundary, each captured by itself,
    replayed in both orders after a reset outside the graphs."""
    _, prep, rows, _ = synth_case(700, 1_000, scores=100, config="batched_100k_x_500k_k512")
    pitch = row_pitch(prep.bytes_per_variant)
    d = torch.zeros((1_000, pitch), dtype=torch.uint8, device="cuda")
    d[:, :prep.bytes_per_variant] = torch.from_numpy(rows[:, :prep.bytes_per_variant]).cuda()
    plan = DevicePlan(prep, engine=_lib.ENGINE_TENSOR)
    s, c = plan.outputs()
    graphs = []
    for v0, n in ((0, 64), (64, 256), (320, 680)):
        plan.reset()
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            plan.accumulate(d[v0:], pitch, v0, n, torch.cuda.current_stream())
    for order in ((0, 1, 2), (2, 1, 0)):
        with torch.cuda.stream(torch.cuda.Stream()):
            stream = torch.cuda.current_stream()
            plan.reset(stream)
            for g in order:
                graphs[g].replay()
            plan.finalize(s, c, stream)
            plan.sync(stream)
        check(prep, rows, (s.cpu().numpy(), c.cpu().numpy().astype(np.uint32)))
    del graphs
    plan.close()
