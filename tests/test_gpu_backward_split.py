"""The 8-bit backward (variants as M, genotypes expanded into tensor memory) where
its split can go wrong: edges of the 256-variant tiles, the 512-person stages
and the 16-score tiles, tiles that span many CTA shares, S32 blocks at their
limit, and scores with infinities."""
import numpy as np
import pytest
import torch

from gnomon_b200 import _lib
from gnomon_b200.autograd import prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch
from helpers import synth_case
from oracle import oracle

pytestmark = pytest.mark.gpu


def device_rows(rows, pitch):
    d = torch.zeros((rows.shape[0], pitch), dtype=torch.uint8, device="cuda")
    d[:, :rows.shape[1]] = torch.from_numpy(np.ascontiguousarray(rows)).cuda()
    return d


@pytest.mark.parametrize("corr", [True, False])
@pytest.mark.parametrize("people,variants,scores", [
    (1, 1, 1), (511, 255, 15), (512, 256, 16), (513, 257, 17), (1025, 129, 33), (700, 3_000, 2),
    (40_000, 300, 16), (3_000, 40_000, 3)])
def test_tile_and_share_edges(cuda, people, variants, scores, corr):
    _, prep, rows, _ = synth_case(people, variants, scores=scores, config="diff_20k_x_200k_k16")
    gs = np.random.default_rng(people).standard_normal((people, scores)).astype(np.float32)
    pitch = row_pitch(prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    d, g = device_rows(rows, pitch), torch.from_numpy(gs).cuda()
    for _ in range(2):
        gw, gc = plan.backward(d, pitch, g, grad_corr=corr)
    plan.sync()
    plan.close()
    ew, ec = oracle.backward_extended(rows, prep, gs)
    # limbs to 2^-31.9 of the score's largest |dS|, one rounding to FP32: 1e-6 of the
    # largest possible sum, as the other backward tests
    scale = np.abs(gs).sum(axis=0).max()
    assert np.abs(gw.cpu().numpy() - ew).max() / scale < 1e-6
    if corr:
        assert np.abs(gc.cpu().numpy() - ec).max() / scale < 1e-6


@pytest.mark.parametrize("byte", [0xFF, 0x55], ids=["hom-alt", "missing"])
def test_blocks_at_the_s32_limit(cuda, byte):
    """More than 2^17 people per share, every dS at the top of the limb range:
    127 x 2 x 64 per person, flushed before 2^31."""
    people, variants = (1 << 17) + 700, 148 * 256
    prep = prep_from_dense(np.zeros((variants, 1), np.float32), np.zeros((variants, 1), bool),
                           np.ones((variants, 1), bool), people)
    pitch = row_pitch(prep.bytes_per_variant)
    rows = torch.full((variants * pitch,), byte, dtype=torch.uint8, device="cuda")
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    gw, gc = plan.backward(rows, pitch, torch.ones(people, 1, device="cuda"), grad_corr=True)
    plan.sync()
    plan.close()
    want = (2.0 * people, 0.0) if byte == 0xFF else (0.0, -float(people))
    # four limbs of 1.0: residual below 2^-31.9 per person, then FP32
    np.testing.assert_allclose(gw.cpu().numpy(), want[0], rtol=1e-6, atol=1e-3)
    np.testing.assert_allclose(gc.cpu().numpy(), want[1], rtol=1e-6, atol=1e-3)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_score_that_is_not_finite(cuda, bad):
    """Only variants at which the person with the bad dS is missing get a bad
    correction gradient; the other score is untouched."""
    people, variants = 1_300, 700
    _, prep, rows, _ = synth_case(people, variants, scores=2, config="diff_20k_x_200k_k16")
    gs = np.random.default_rng(3).standard_normal((people, 2)).astype(np.float32)
    gs[1_234, 1] = bad
    pitch = row_pitch(prep.bytes_per_variant)
    plan = DevicePlan(prep, engine=_lib.ENGINE_PLAIN)
    gw, gc = plan.backward(device_rows(rows, pitch), pitch, torch.from_numpy(gs).cuda(),
                           grad_corr=True)
    plan.sync()
    plan.close()
    gw, gc = gw.cpu().numpy(), gc.cpu().numpy()
    missing = ((rows[:, 1_234 // 4] >> (2 * (1_234 % 4))) & 3) == 1
    np.testing.assert_array_equal(np.isfinite(gc[:, 1]), ~missing)
    clean = np.where(np.isfinite(gs), gs, 0).astype(np.float32)
    ew, ec = oracle.backward_extended(rows, prep, clean)
    scale = np.abs(clean).sum(axis=0).max()
    assert np.abs(gc[~missing] - ec[~missing]).max() / scale < 1e-6
    assert np.abs(gw[:, 0] - ew[:, 0]).max() / scale < 1e-6
