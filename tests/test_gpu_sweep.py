"""The update sweep in each way it shares an atom among CTAs (one CTA alone,
partials as tagged words, partials behind a counter), with columns in shared
memory and beyond it, against the FP64 oracle.  Tolerances are those of the
update elsewhere: atoms within 1e-4, coefficients within 1e-4 of the largest."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,side,step,K,L", [
    (2, 2, 40, 1, 4, 2),      # one float4 per row
    (8, 8, 96, 1, 40, 4),     # rows of 16-byte pieces
    (7, 5, 90, 1, 130, 3),    # 35 values: no bulk copies; more atoms than one table of slices
    (12, 12, 90, 1, 32, 3),   # 14 column groups, 48 words
    (16, 16, 80, 1, 24, 3),   # 8 column groups: features split over warps
    (22, 21, 80, 1, 16, 3),   # 462 values, 4 column groups
])
@pytest.mark.parametrize("entries_per_cta", [4096, 64, 8])
def test_update_any_split(torch_cuda, ksvd, oracle, synth, pw, ph, side, step, K, L, entries_per_cta):
    torch = torch_cuda
    img = synth.add_gaussian(synth.clean_image(side, 8), 20.0, 8)
    Y = oracle.extract_patches(img, pw, ph, step, step)
    D = oracle.init_dictionary(Y, K, int_norm=True, dtype=np.float32)
    idx, coef = oracle.omp(Y, D, L, dtype=np.float32)
    c = ksvd.Context(ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=step, sliding_height=step,
                                      atoms=K, omp_iter=L, compat=1))
    c.set_update_slice(entries_per_cta)
    Yd, Dd, id_, cd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (Y, D, idx, coef))
    c.update_dictionary(Yd, Dd, id_, cd)
    torch.cuda.synchronize()
    Dr, cr = oracle.update_dictionary(Y.astype(np.float64), D.astype(np.float64), idx, coef.astype(np.float64),
                                      q1_cap=False)
    assert np.abs(Dd.cpu().numpy() - Dr).max() < 1e-4
    assert np.abs(cd.cpu().numpy() - cr).max() < 1e-4 * np.abs(cr).max()
    c.close()
