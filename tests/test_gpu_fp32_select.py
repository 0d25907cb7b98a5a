"""The FP32 OMP on the tensor cores (its FP16 correlation only narrows the
atoms down) against the FP32 SIMT kernels, which ksvd_omp_noalloc runs: the
same argmax over the same sums, so the same codes, bit for bit, for any scale
and offset of the data."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(oracle, synth, pw, ph, K, kind):
    # more than two waves of the SIMT kernel's tiles of 32 patches on 148 SMs, a
    # ragged number: what the tensor cores take
    img = synth.add_gaussian(synth.clean_image(80, 11), 20.0, 11)
    Y = oracle.extract_patches(img, pw, ph, 2, 2)
    Y = np.concatenate([Y * np.float32(1.0 + 0.01 * i) for i in range(9500 // Y.shape[0] + 1)])[:9501]
    D = oracle.init_dictionary(Y, K, int_norm=True, dtype=np.float32)
    if kind == "small atoms":
        D *= np.float32(1e-3)
    elif kind == "large atoms":
        D *= np.float32(300.0)
    elif kind == "tiny atoms":  # outside the range of the 16-bit dictionary's scale
        D *= np.float32(1e-20)
    elif kind == "offset":
        Y += np.float32(1e6)
    elif kind == "ties":
        Y[:] = 128.0
        D[:] = D[0]
    elif kind == "mixed":
        D[3] = 0.0
        D[5] = D[4]
        D[7] *= np.float32(1e4)
        Y[:40] = 0.0
        Y[40:80] *= np.float32(1e-6)
        Y[100, 3] = np.nan
    return Y, D


@pytest.mark.parametrize("pw,ph,K,L", [
    (12, 12, 256, 5),   # resident 16-bit dictionary, the largest
    (8, 8, 200, 16),    # the most atoms per patch
    (5, 5, 16, 3),      # 25 values: no 16-byte rows
    (8, 8, 257, 5),     # streamed dictionary, one atom beyond the resident one
    (16, 16, 512, 8),   # streamed, the most atoms
    (22, 21, 64, 5),    # 462 values
])
@pytest.mark.parametrize("kind", ["plain", "small atoms", "large atoms", "tiny atoms", "offset", "ties", "mixed"])
def test_fp32_codes_equal_simt(torch_cuda, ksvd, oracle, synth, pw, ph, K, L, kind):
    torch = torch_cuda
    Y, D = _inputs(oracle, synth, pw, ph, K, kind)
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2, atoms=K,
                              omp_iter=L, precision=ksvd.PREC_FP32)
    Yd, Dd = torch.from_numpy(Y).cuda(), torch.from_numpy(D).cuda()
    N = Y.shape[0]
    codes = []
    with ksvd.Context(params) as ctx:
        for run in (ctx.omp, lambda *a: ksvd.omp_noalloc(params, *a)):
            idx = torch.empty((N, L), dtype=torch.int32, device="cuda")
            coef = torch.empty((N, L), device="cuda")
            run(Yd, Dd, idx, coef)
            torch.cuda.synchronize()
            codes.append((idx.cpu().numpy(), coef.cpu().numpy()))
    np.testing.assert_array_equal(codes[0][0], codes[1][0])
    np.testing.assert_array_equal(codes[0][1], codes[1][1])
