"""The learned proposal's gradients with the batch split over the SMs, from one
split to the most and with parts of unequal length, against the float64
oracle with the same BF16 rounding points (each block within 2e-2 relative, the
bound of the unsplit gradients)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n_side,K", [(16, 12, 256), (80, 8, 100), (1040, 12, 256), (2064, 9, 33)])
def test_grad_splits(torch_cuda, ksvd, synth, oracle, batch, n_side, K):
    from ksvd_loader import load_oracle
    load_oracle()
    import mlp_oracle as mlp
    torch = torch_cuda
    n = n_side * n_side
    img = synth.add_gaussian(synth.clean_image(110, 41), 20.0, 41)
    Yall = oracle.extract_patches(img, n_side, n_side, 2, 2)
    D = oracle.init_dictionary(Yall, K, int_norm=True, dtype=np.float32)
    Y = np.ascontiguousarray(Yall[:batch])
    assert Y.shape[0] == batch
    sup, _ = oracle.omp(Y, D, 5, dtype=np.float32)
    with ksvd.Context(ksvd.make_params(patch_width_dim=n_side, patch_height_dim=n_side, sliding_width=2,
                                       sliding_height=2, atoms=K, omp_iter=5, precision=3)) as c:
        c.proposal_init(7)
        params = c.proposal_get_params()
        grad = torch.zeros(params.size, dtype=torch.float32, device="cuda")
        loss = c.proposal_loss_grad(torch.from_numpy(Y).cuda(), torch.from_numpy(sup).cuda(), grad)
    rl, rg = mlp.loss_grad(params.astype(np.float64), Y, sup, K, emulate=True)
    assert abs(loss - rl) <= 1e-4 * abs(rl)
    g = grad.cpu().numpy().astype(np.float64)
    o = np.cumsum([0, 512 * n, 512, 512 * 512, 512, K * 512, K])
    for name, a, b in zip(("W1", "b1", "W2", "b2", "W3", "b3"), o[:-1], o[1:]):
        err = np.linalg.norm(g[a:b] - rg[a:b]) / (np.linalg.norm(rg[a:b]) + 1e-30)
        assert err <= 2e-2, (name, err)
