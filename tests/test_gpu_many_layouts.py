"""ksvd_denoise_many where images of different patch sizes, hence different
shared-memory layouts, sweep one after the other on the same CTAs, some CTAs
having no entries in the first: every image within 0.02 dB of the one-image
path, and the same bits from run to run."""

import numpy as np
import pytest

SPEC = [(22, 200), (22, 200), (22, 200), (22, 90), (12, 110)]  # patch side, image side


def _params(ksvd, patch):
    return ksvd.make_params(patch_width_dim=patch, patch_height_dim=patch, sliding_width=2, sliding_height=2, atoms=24,
                            omp_iter=3, ksvd_iter=3, compat=1, precision=ksvd.PREC_FP16_RESCORE)


def test_plan_shares_ctas(ksvd, built_lib):
    """The last image follows one of larger patches on its CTAs, with more of them at work."""
    begin, ctas, order, _ = ksvd.many_plan([(_params(ksvd, p), s, s) for p, s in SPEC])
    assert (begin[3], ctas[3]) == (begin[4], ctas[4]) and order.index(3) < order.index(4)
    entries = [((s - p) // 2 + 1) ** 2 * 3 / 24 for p, s in SPEC]  # per atom, on average
    assert entries[4] > 1.5 * entries[3] and ctas[4] > entries[4] / 64 > entries[3] / 64


@pytest.mark.gpu
def test_layouts_in_turn(torch_cuda, ksvd, synth):
    jobs, clean = [], []
    for i, (p, s) in enumerate(SPEC):
        clean.append(synth.clean_image(s, 80 + i))
        jobs.append((_params(ksvd, p), synth.add_gaussian(clean[-1], 20.0, 80 + i), 400.0))
    outs, _ = ksvd.denoise_many(jobs, tune=False)
    again, _ = ksvd.denoise_many(jobs, tune=False)
    for (params, noisy, s2), c, a, b in zip(jobs, clean, outs, again):
        np.testing.assert_array_equal(a, b)
        with ksvd.Context(params) as ctx:
            single, _ = ctx.denoise(noisy, s2)
        assert abs(synth.psnr(c, single) - synth.psnr(c, a)) <= 0.02


# patch side, image side: 49 to 484 values, not all a multiple of four
SMALL = [[(22, 64), (8, 40), (12, 48), (7, 39)], [(22, 64), (8, 44), (12, 50)]]


@pytest.mark.parametrize("spec", SMALL)
def test_small_plan_leaves_slices(ksvd, built_lib, spec):
    """Every image of these batches has a CTA for each 64 of its patches, so its atoms are
    cut into the same slices as on the whole GPU."""
    _, ctas, _, _ = ksvd.many_plan([(_params(ksvd, p), s, s) for p, s in spec])
    assert all(64 * c >= ((s - p) // 2 + 1) ** 2 for c, (p, s) in zip(ctas, spec))


@pytest.mark.gpu
@pytest.mark.parametrize("spec", SMALL)
def test_mixed_batch_same_bits(torch_cuda, ksvd, synth, spec):
    """The same slices, hence the same sums in the same order, whatever the widest
    patch of the launch: the images of the batch equal the one-image path's."""
    jobs = [(_params(ksvd, p), synth.add_gaussian(synth.clean_image(s, 90 + i), 20.0, 90 + i), 400.0)
            for i, (p, s) in enumerate(spec)]
    outs, _ = ksvd.denoise_many(jobs, tune=False)
    for (params, noisy, s2), a in zip(jobs, outs):
        with ksvd.Context(params) as ctx:
            single, _ = ctx.denoise(noisy, s2)
        np.testing.assert_array_equal(a, single)
