"""The rebuild's two ways over the geometries where its model changes between
them, against the oracle, within 1e-5 relative."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,sw,sh,w,h,K,L", [
    (8, 8, 8, 8, 128, 96, 24, 3),     # every pixel covered once: no tiles
    (6, 6, 4, 4, 300, 200, 24, 5),    # at most four times: no tiles
    (3, 3, 5, 4, 90, 70, 24, 2),      # pixels between the patches
    (12, 12, 3, 3, 500, 400, 24, 3),  # tiles beyond 110 KB
    (20, 20, 4, 4, 150, 140, 24, 3),  # large patches in tiles
    (4, 4, 1, 1, 130, 120, 24, 3),
    (22, 22, 5, 5, 120, 100, 24, 5),
    (16, 16, 2, 2, 90, 80, 24, 8),    # one tile of few pixels fits
])
def test_build_image_paths(torch_cuda, ksvd, oracle, synth, pw, ph, sw, sh, w, h, K, L):
    torch = torch_cuda
    img = np.ascontiguousarray(synth.add_gaussian(synth.clean_image(max(w, h), 62)[:h, :w], 20.0, 62))
    Y = oracle.extract_patches(img, pw, ph, sw, sh)
    D = oracle.init_dictionary(Y, K, dtype=np.float32)
    idx, coef = oracle.omp(Y, D, L, dtype=np.float32)
    with ksvd.Context(ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=sw, sliding_height=sh,
                                       atoms=K, omp_iter=L)) as c:
        out = torch.empty(img.shape, dtype=torch.float32, device="cuda")
        lam = c.build_image(*(torch.from_numpy(img).cuda(), 400.0),
                            *(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (D, idx, coef)), out)
    ref, rlam = oracle.build_image(img, pw, ph, sw, sh, D, idx, coef, 400.0, dtype=np.float32)
    assert lam == pytest.approx(rlam, rel=1e-5)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-5, atol=1e-3)
