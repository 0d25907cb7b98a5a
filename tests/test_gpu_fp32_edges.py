"""The FP32 OMP on the tensor cores against the FP32 SIMT kernels (which
ksvd_omp_noalloc runs) where the window of atoms or the stop test is at its
limits: the same codes, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (8, 8, 200, 16),    # resident 16-bit dictionary
    (5, 5, 16, 3),      # 25 values: no 16-byte rows
    (8, 8, 257, 5),     # streamed 16-bit dictionary
    (12, 12, 512, 5),   # the SIMT kernel streams too
    (22, 21, 64, 5),    # 462 values
]


def _data(oracle, synth, pw, ph, K):
    # more than two waves of the SIMT kernel's tiles of 32 patches on 148 SMs:
    # what the tensor cores take
    img = synth.add_gaussian(synth.clean_image(80, 11), 20.0, 11)
    Y = oracle.extract_patches(img, pw, ph, 2, 2)
    Y = np.concatenate([Y * np.float32(1.0 + 0.01 * i) for i in range(9500 // Y.shape[0] + 1)])[:9501]
    return Y, oracle.init_dictionary(Y, K, int_norm=True, dtype=np.float32)


def _both(torch, ksvd, pw, ph, L, Y, D):
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2,
                              atoms=D.shape[0], omp_iter=L, precision=ksvd.PREC_FP32)
    Yd, Dd = (torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda() for a in (Y, D))
    codes = []
    with ksvd.Context(params) as ctx:
        for run in (ctx.omp, lambda *a: ksvd.omp_noalloc(params, *a)):
            idx = torch.empty((Y.shape[0], L), dtype=torch.int32, device="cuda")
            coef = torch.empty((Y.shape[0], L), device="cuda")
            run(Yd, Dd, idx, coef)
            torch.cuda.synchronize()
            codes.append((idx.cpu().numpy(), coef.cpu().numpy()))
    return codes


def _assert_same(codes):
    np.testing.assert_array_equal(codes[0][0], codes[1][0])
    np.testing.assert_array_equal(codes[0][1], codes[1][1])


@pytest.mark.parametrize("pw,ph,K,L", SHAPES)
@pytest.mark.parametrize("scale", [1e-18, 1e-22, 1e-25, 1e-26, 1e-30, 1e-36])
@pytest.mark.parametrize("centred", [False, True])
def test_tiny_patches(torch_cuda, ksvd, oracle, synth, pw, ph, K, L, scale, centred):
    """Patches whose squares leave the FP32 range."""
    Y, D = _data(oracle, synth, pw, ph, K)
    if centred:
        Y = Y - Y.mean(1, keepdims=True)
    _assert_same(_both(torch_cuda, ksvd, pw, ph, L, Y * np.float32(scale), D))


@pytest.mark.parametrize("pw,ph,K,L", SHAPES)
def test_infinite_values(torch_cuda, ksvd, oracle, synth, pw, ph, K, L):
    """Infinite values: an atom whose correlation is infinite is the largest, one
    whose correlation is NaN is never chosen before a number (checked for the
    first atom of a pursuit against the same sums in numpy)."""
    Y, D = _data(oracle, synth, pw, ph, K)
    D = D - D.mean(1, keepdims=True)
    D /= np.linalg.norm(D, axis=1, keepdims=True)
    D[7] = np.abs(D[7])  # one atom of one sign
    D[0, 5] = 0.0        # infinity times zero
    Y[:40] = np.inf
    Y[40:80] = -np.inf
    Y[80:120, 5] = np.inf
    Y[120:160, 0] = np.inf
    Y[120:160, 1] = -np.inf
    Y[160:200, pw * ph - 1] = -np.inf
    Y[200] = np.nan
    codes = _both(torch_cuda, ksvd, pw, ph, L, Y, D)
    _assert_same(codes)
    with np.errstate(invalid="ignore"):
        c = np.abs(np.add.reduce(D[None].astype(np.float64) * Y[:201, None].astype(np.float64), axis=2))
    want = np.argmax(np.where(np.isnan(c), -1.0, c), axis=1)
    np.testing.assert_array_equal(codes[0][0][:200, 0], want[:200])


def _near_stop(rng, D, N):
    """Patches of one atom and a rest of norm 1e-3 but for rounding, orthogonal to it."""
    a = rng.integers(0, D.shape[0], N)
    d = D[a].astype(np.float64)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e = rng.standard_normal(d.shape)
    e -= (e * d).sum(1, keepdims=True) * d
    e *= 1e-3 * (1 + 1e-6 * rng.uniform(-1, 1, (N, 1))) / np.linalg.norm(e, axis=1, keepdims=True)
    return (0.05 * d + e).astype(np.float32)


@pytest.mark.parametrize("pw,ph,K,L", SHAPES + [(16, 16, 512, 8)])
def test_stop_threshold(torch_cuda, ksvd, oracle, synth, pw, ph, K, L):
    """Residual norms that the order of their sum decides."""
    _, D = _data(oracle, synth, pw, ph, K)
    Y = _near_stop(np.random.default_rng(3), D, 9501)
    codes = _both(torch_cuda, ksvd, pw, ph, L, Y, D)
    stopped = np.count_nonzero(codes[1][0][:, 1] < 0)
    assert 500 < stopped < 9000  # both sides of the threshold
    _assert_same(codes)


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("pw,ph,K,L", [(8, 8, 200, 4), (5, 5, 16, 3), (8, 8, 300, 5), (16, 16, 512, 8)])
@pytest.mark.parametrize("precision", [1, 2])
def test_stop_threshold_16bit(torch_cuda, ksvd, oracle, synth, pw, ph, K, L, precision):
    """The 16-bit forms' stop test after the first atom, whose norm is summed over
    the 8-feature chunks of a padded row in four parts (in numpy; a product and
    sum rounded twice instead of once may move one patch in 2000)."""
    _, D = _data(oracle, synth, pw, ph, K)
    n = pw * ph
    Y = _near_stop(np.random.default_rng(4), D, 4000)
    params = ksvd.make_params(patch_width_dim=pw, patch_height_dim=ph, sliding_width=2, sliding_height=2, atoms=K,
                              omp_iter=L, precision=precision)
    with ksvd.Context(params) as ctx:
        idx = torch_cuda.empty((Y.shape[0], L), dtype=torch_cuda.int32, device="cuda")
        coef = torch_cuda.empty((Y.shape[0], L), device="cuda")
        ctx.omp(torch_cuda.from_numpy(Y).cuda(), torch_cuda.from_numpy(D).cuda(), idx, coef)
        torch_cuda.cuda.synchronize()
        idx = idx.cpu().numpy()
    d = D[idx[:, 0]]
    g = ((d.astype(np.float64) * Y).sum(1) / (d.astype(np.float64) ** 2).sum(1)).astype(np.float32)
    r = _fma(-g[:, None], d, Y)
    nkc = 2 * ((n + 15) // 16)
    total = np.zeros(Y.shape[0], np.float32)
    for q in range(4):
        t = np.zeros_like(total)
        for k in range(8 * (nkc * q // 4), min(n, 8 * (nkc * (q + 1) // 4))):
            t = _fma(r[:, k], r[:, k], t)
        total += t
    stops = np.sqrt(total) < np.float32(1e-3)
    assert 200 < np.count_nonzero(stops) < 3800  # both sides of the threshold
    assert np.count_nonzero(stops != (idx[:, 1] < 0)) <= 2
