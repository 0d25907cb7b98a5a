"""The FP32 OMP on the tensor cores with patches or dictionaries that do not
start on a 16-byte boundary (rows of a multiple of 16 bytes): the codes of the
aligned buffers, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph,K,L", [(12, 12, 128, 5), (16, 16, 320, 4), (22, 22, 64, 3)])
@pytest.mark.parametrize("off_y,off_d", [(1, 0), (0, 1), (2, 3)])
def test_fp32_codes_unaligned(torch_cuda, ksvd, synth, oracle, pw, ph, K, L, off_y, off_d):
    torch = torch_cuda
    img = synth.add_gaussian(synth.clean_image(80, 12), 20.0, 12)
    Y = oracle.extract_patches(img, pw, ph, 2, 2)
    # more than two waves of the SIMT kernel's tiles of 32 patches on 148 SMs
    Y = np.concatenate([Y * np.float32(1.0 + 0.01 * i) for i in range(9500 // Y.shape[0] + 1)])[:9501]
    D = oracle.init_dictionary(Y, K, int_norm=True, dtype=np.float32)
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2, atoms=K,
                              omp_iter=L, precision=ksvd.PREC_FP32)
    codes = []
    with ksvd.Context(params) as ctx:
        for oy, od in ((0, 0), (off_y, off_d)):
            dev = []
            for a, o in ((Y, oy), (D, od)):
                buf = torch.empty(a.size + o, device="cuda")
                v = buf[o:].view(a.shape)
                v.copy_(torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)))
                assert v.data_ptr() % 16 == 4 * o
                dev.append(v)
            idx = torch.empty((Y.shape[0], L), dtype=torch.int32, device="cuda")
            coef = torch.empty((Y.shape[0], L), device="cuda")
            ctx.omp(*dev, idx, coef)
            torch.cuda.synchronize()
            codes.append((idx.cpu().numpy(), coef.cpu().numpy()))
    np.testing.assert_array_equal(codes[0][0], codes[1][0])
    np.testing.assert_array_equal(codes[0][1].view(np.uint32), codes[1][1].view(np.uint32))
