"""The rebuild over its pixel tiles (rectangular, from 64 pixels a side down
to the gather without tiles) against the oracle, within 1e-5 relative."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,sw,sh,w,h", [
    (3, 3, 3, 3, 70, 131),    # 64 x 64 tiles, the last ones partial
    (8, 8, 2, 2, 65, 64),
    (8, 8, 2, 2, 128, 128),
    (8, 8, 2, 2, 200, 200),   # tiles of exactly 48 KB among the candidates
    (12, 12, 3, 3, 100, 90),  # 32 x 16 tiles, uncovered border
    (6, 14, 4, 2, 90, 70),
    (16, 16, 2, 2, 60, 50),   # no tile fits
])
def test_build_image_tiles(torch_cuda, ksvd, oracle, synth, pw, ph, sw, sh, w, h):
    torch = torch_cuda
    img = np.ascontiguousarray(synth.add_gaussian(synth.clean_image(max(w, h), 62)[:h, :w], 20.0, 62))
    Y = oracle.extract_patches(img, pw, ph, sw, sh)
    D = oracle.init_dictionary(Y, 24, dtype=np.float32)
    idx, coef = oracle.omp(Y, D, 3, dtype=np.float32)
    with ksvd.Context(ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=sw, sliding_height=sh,
                                       atoms=24, omp_iter=3)) as c:
        out = torch.empty(img.shape, dtype=torch.float32, device="cuda")
        lam = c.build_image(*(torch.from_numpy(img).cuda(), 400.0),
                            *(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (D, idx, coef)), out)
    ref, rlam = oracle.build_image(img, pw, ph, sw, sh, D, idx, coef, 400.0, dtype=np.float32)
    assert lam == pytest.approx(rlam, rel=1e-5)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-5, atol=1e-3)
