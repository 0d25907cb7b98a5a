"""The residual rows that the FP32 form's tensor-core OMP writes for the update
sweep inside K-SVD iterations, against the separate residual pass: the same
dictionary and codes, bit for bit.  (Fewer patches take the SIMT kernel, whose
rows test_gpu_parity.py compares.)"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,K,L", [
    (12, 12, 128, 5),  # resident 16-bit dictionary, 16-byte rows
    (7, 7, 100, 4),    # 49 values: rows of single floats
    (5, 6, 33, 3),     # 30 values, a ragged tile of atoms
    (8, 8, 256, 5),    # the most atoms of the resident dictionary
    (9, 9, 300, 4),    # streamed dictionary, 81 values
])
def test_fused_rows_equal_separate_pass(torch_cuda, ksvd, synth, pw, ph, K, L):
    torch = torch_cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    side = 2 * int(np.ceil(np.sqrt(64 * sms))) + max(pw, ph) + 3
    noisy = synth.add_gaussian(synth.clean_image(side, 31), 20.0, 31).astype(np.float32)
    noisy[:36, :36] = 0.0  # patches that stop after one atom
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2, atoms=K,
                              omp_iter=L, precision=ksvd.PREC_FP32, compat=ksvd.COMPAT_INT_NORM)
    N = ksvd.num_patches(params, side, side)
    assert N > 64 * sms  # more than two waves of the SIMT kernel's tiles of 32 patches
    out = []
    with ksvd.Context(params) as c:
        Y = torch.empty((N, pw * ph), device="cuda")
        c.extract_patches(torch.from_numpy(np.ascontiguousarray(noisy)).cuda(), Y)
        D0 = torch.empty((K, pw * ph), device="cuda")
        c.init_dictionary(Y, D0)
        for fused in (True, False):
            D = D0.clone()
            idx = torch.empty((N, L), dtype=torch.int32, device="cuda")
            coef = torch.empty((N, L), device="cuda")
            for _ in range(2):
                if fused:
                    c.iterate(Y, D, idx, coef, 1)
                else:
                    c.omp(Y, D, idx, coef)
                    c.update_dictionary(Y, D, idx, coef)
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in (D, idx, coef)])
    stopped = np.count_nonzero(out[0][1][:, 1] < 0)
    assert 0 < stopped < N // 2  # rows of both kinds
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
