"""Which kernels take the FP32 form's few patches: the SIMT ones where they are
the faster, else the tensor cores (whose exact scores the profile counts); the
codes are the same either way."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,K,L,waves,simt", [
    (8, 8, 512, 5, 1, True),      # beyond 256 atoms, dictionary resident in the SIMT kernel: one wave
    (8, 8, 512, 5, 2, False),
    (8, 8, 384, 3, 2, True),      # and two of few steps
    (7, 7, 300, 5, 2, True),
    (9, 9, 512, 8, 1, True),
    (13, 13, 300, 3, 1, True),    # streamed, rows of single floats
    (13, 13, 300, 3, 2, False),
    (10, 10, 384, 3, 1, True),    # streamed, short rows
    (16, 16, 512, 5, 1, False),   # streamed, long rows
    (8, 8, 256, 5, 2, True),      # up to 256 atoms
    (8, 8, 256, 5, 3, False),
    (13, 13, 200, 3, 2, True),
    (16, 16, 256, 5, 1, True),
    (16, 16, 256, 5, 2, False),
])
def test_route_of_few_patches(torch_cuda, ksvd, synth, oracle, pw, ph, K, L, waves, simt):
    torch = torch_cuda
    N = 32 * waves * torch.cuda.get_device_properties(0).multi_processor_count - 5
    img = synth.add_gaussian(synth.clean_image(80, 13), 20.0, 13)
    Y = oracle.extract_patches(img, pw, ph, 2, 2)
    Y = np.concatenate([Y * np.float32(1.0 + 0.01 * i) for i in range(N // Y.shape[0] + 1)])[:N]
    D = oracle.init_dictionary(Y, K, int_norm=True, dtype=np.float32)
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2, atoms=K,
                              omp_iter=L, precision=ksvd.PREC_FP32)
    Yd, Dd = (torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda() for a in (Y, D))
    codes = []
    with ksvd.Context(params) as ctx:
        ctx.profile_reset()
        ctx.profile(2)
        for run in (ctx.omp, lambda *a: ksvd.omp_noalloc(params, *a)):
            idx = torch.empty((N, L), dtype=torch.int32, device="cuda")
            coef = torch.empty((N, L), device="cuda")
            run(Yd, Dd, idx, coef)
            torch.cuda.synchronize()
            codes.append((idx.cpu().numpy(), coef.cpu().numpy()))
        assert (ctx.profile_counters()["omp_exact_rescores"] == 0) == simt
    np.testing.assert_array_equal(codes[0][0], codes[1][0])
    np.testing.assert_array_equal(codes[0][1], codes[1][1])
