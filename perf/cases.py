"""Timed cases of the library: what programs call, over the sizes they call it with.

The sizes come from the workloads of synth.py and bench.py (512^2 and 2048^2 images with 12 x 12 patches at stride 3
and 256 atoms; 16 x 16 patches at stride 2 and 512 atoms; uneven batches of 8, 12 and 22-pixel patches), from the
library's default parameters (8 x 8 patches at stride 2, 256 atoms, 5 OMP atoms, 10 iterations) and from the ragged
geometries of the tests.  Images are the gratings and rectangles of synth.py under Gaussian or speckle noise, drawn on
the GPU.

A case is a dict: `kind` (below), the image `w` x `h`, the patch `pw` x `ph` and its steps `sw`, `sh`, `atoms`, `omp`
(atoms per patch), `prec` (the arithmetic form), `cap` (the reference's cap of 1024 patches per atom in the update; the
library's default) and, for whole calls, `iters` and `speckle`.

  denoise   ksvd_denoise on host buffers
  many      ksvd_denoise_many on host buffers, `count` images of uneven size and patch shape
  iterate   one K-SVD iteration (OMP + dictionary update) on resident patches
  omp       sparse coding of resident patches with a given dictionary (`prec` 3: the learned proposal's)
  rebuild   the denoised image from the codes
  learn     loss and weight gradients of the learned proposal on one training batch (`batch` patches)
"""

import math

import numpy as np
import torch

from ksvd_loader import load

KS = load().ksvd
FP32, BF16, FP16, LEARNED = KS.PREC_FP32, KS.PREC_BF16_RESCORE, KS.PREC_FP16_RESCORE, KS.PREC_BF16_LEARNED


def _case(kind, w, h, pw, ph, sw, sh, atoms, omp, prec, cap=True, **more):
    return dict(kind=kind, w=w, h=h, pw=pw, ph=ph, sw=sw, sh=sh, atoms=atoms, omp=omp, prec=prec, cap=cap, **more)


def listed():
    return [
        # a thumbnail or a tile with every parameter at its default: the smallest call, bound by launches and latency
        dict(_case("denoise", 128, 128, 8, 8, 2, 2, 256, 5, FP32, iters=10, speckle=False), name="denoise_128_p8_fp32"),
        # an ordinary photograph through the fast form: the 512^2 workload
        dict(_case("denoise", 512, 512, 12, 12, 3, 3, 256, 5, FP16, iters=10, speckle=False),
             name="denoise_512_p12_fp16"),
        # a folder of uneven images, some of them speckled, in one call
        dict(kind="many", count=8, side=512, atoms=256, omp=5, prec=FP16, cap=True, iters=5, name="many_8_uneven"),
        # the headline: one iteration of the 2048^2 workload, whole update
        dict(_case("iterate", 2048, 2048, 12, 12, 3, 3, 256, 5, FP16, cap=False), name="iterate_2048_p12_fp16"),
        # one iteration with the default parameters on an ordinary image
        dict(_case("iterate", 512, 512, 8, 8, 2, 2, 256, 5, FP32), name="iterate_512_p8_fp32"),
        # a ragged geometry: rectangular image, patches and steps, atoms no multiple of a tile, patch values no
        # multiple of four
        dict(_case("iterate", 1000, 777, 10, 11, 3, 2, 200, 4, BF16, cap=False), name="iterate_1000x777_p10x11_bf16"),
        # sparse coding of a large image with the plain form
        dict(_case("omp", 2048, 2048, 12, 12, 3, 3, 256, 5, FP32), name="omp_2048_p12_fp32"),
        # sparse coding with a large dictionary (beyond shared memory): the largest case, and the plain form of it
        dict(_case("omp", 2048, 2048, 16, 16, 2, 2, 512, 8, FP16), name="omp_2048_p16_k512_fp16"),
        dict(_case("omp", 1024, 1024, 16, 16, 2, 2, 512, 8, FP32), name="omp_1024_p16_k512_fp32"),
        # sparse coding through the learned proposal (network, restricted pursuit, fallback)
        dict(_case("omp", 1024, 1024, 12, 12, 3, 3, 256, 5, LEARNED), name="omp_1024_p12_learned"),
        # the last stage of a call on a large image
        dict(_case("rebuild", 2048, 2048, 12, 12, 3, 3, 256, 5, FP32), name="rebuild_2048_p12"),
        # one training step's forward and backward pass at the library's own batch size
        dict(_case("learn", 512, 512, 12, 12, 3, 3, 256, 5, LEARNED, batch=4096), name="learn_4096_p12"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: image sides, patch shapes, steps, dictionary sizes and forms of the listed ranges."""
    kind = rng.choice(["denoise", "many", "iterate", "iterate", "iterate", "omp", "omp", "omp", "rebuild", "learn"])
    if kind == "many":
        return dict(kind="many", count=rng.randint(2, 8), side=_log_int(rng, 128, 512), atoms=rng.choice([64, 128, 200, 256]),
                    omp=rng.randint(3, 6), prec=rng.choice([FP32, BF16, FP16]), cap=rng.random() < 0.5,
                    iters=rng.randint(1, 5))
    while True:
        atoms = rng.choice([64, 100, 128, 200, 256, 256, 256, 384, 512])
        omp = rng.randint(3, 8)
        prec = rng.choice([FP32, FP32, BF16, FP16, FP16])
        pw = rng.choice([6, 8, 8, 9, 10, 12, 12, 16, 22])
        ph = pw if rng.random() < 0.7 else max(5, pw + rng.choice([-2, -1, 1]))
        if rng.random() < 0.5:
            sw = sh = 3 if pw >= 12 else 2
        else:
            sw, sh = rng.randint(2, 4), rng.randint(2, 4)
        w = _log_int(rng, 128, 512 if kind == "denoise" else 2048)
        h = w if rng.random() < 0.5 else max(128, min(2048, int(w * rng.uniform(0.6, 1.6))))
        more = {}
        if kind == "denoise":
            more = dict(iters=rng.randint(1, 10), speckle=rng.random() < 0.3)
        if kind == "omp" and rng.random() < 0.2:
            prec = LEARNED
        if kind == "learn":
            prec, w, h = LEARNED, 512, 512
            more = dict(batch=16 * rng.randint(32, 512))
        if prec == LEARNED and (atoms > 256 or pw * ph > 144):  # what the proposal and its fallback take
            continue
        case = _case(kind, w, h, pw, ph, sw, sh, atoms, omp, prec, cap=rng.random() < 0.5, **more)
        N = _patches(case)
        # no more work than the listed cases of the kind and form
        most = {"denoise": 5e10 / more.get("iters", 1), "iterate": 2.5e11}.get(kind, 1e12)
        if prec != FP16:
            most = min(most, 1.7e11)
        if N >= 4 * atoms and N * pw * ph * atoms * omp <= most and N >= more.get("batch", 0):
            return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _params(c, **kw):
    compat = KS.COMPAT_INT_NORM | (KS.COMPAT_Q1_CAP if c["cap"] else 0)
    kw.setdefault("ksvd_iter", c.get("iters", 10))
    return KS.make_params(patch_width_dim=c["pw"], patch_height_dim=c["ph"], sliding_width=c["sw"],
                          sliding_height=c["sh"], atoms=c["atoms"], omp_iter=c["omp"], precision=c["prec"],
                          speckle=int(c.get("speckle", False)), compat=compat, **kw)


def _grid(c):
    return (c["w"] - c["ph"]) // c["sh"] + 1, (c["h"] - c["pw"]) // c["sw"] + 1


def _patches(c):
    nx, ny = _grid(c)
    return nx * ny


def _image(w, h, seed, sigma, speckle=False):
    """Gratings and flat rectangles in [0, 255] with Gaussian noise, or speckle of 4 looks (strictly positive)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = np.random.default_rng(seed)
    yy = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    img = torch.zeros((h, w), device="cuda")
    for _ in range(12):
        th, per, ph, amp = r.uniform(0, np.pi), r.uniform(4, 64), r.uniform(0, 2 * np.pi), r.uniform(0.5, 1)
        img += amp * torch.sin((xx * np.cos(th) + yy * np.sin(th)) * (2 * np.pi / per) + ph)
    img = (img - img.min()) / (img.max() - img.min()) * 255
    side = min(w, h)
    for _ in range(40):
        rw, rh = (int(r.integers(max(1, side // 32), max(2, side // 6) + 1)) for _ in range(2))
        x0, y0 = int(r.integers(0, w - rw + 1)), int(r.integers(0, h - rh + 1))
        img[y0:y0 + rh, x0:x0 + rw] = r.uniform(0, 255)
    if speckle:
        looks = -torch.log(torch.rand((4, h, w), generator=g, device="cuda").clamp_min(1e-7)).mean(0)
        return (img + 1) * looks
    return img + sigma * torch.randn((h, w), generator=g, device="cuda")


SIGMA = 25.0
SPECKLE_VAR = (math.pi ** 2 / 6 - (1 + 1 / 4 + 1 / 9)) / math.log(2) ** 2  # of log2 of Gamma(4, 1/4) noise


def _sigma2(c):
    return SPECKLE_VAR if c.get("speckle") else SIGMA * SIGMA


def _many_shapes(c):
    """The uneven batch: sides down to half of `side`, patches of 8, 12 and 22 at stride 3, every fourth speckled."""
    shapes = []
    for i in range(c["count"]):
        r = np.random.default_rng(7919 * c["count"] + c["side"] + i)
        patch = int(r.choice([8, 12, 22]))
        w, h = (int(r.uniform(0.5, 1) * c["side"]) + 66 for _ in range(2))
        j = dict(c, kind="denoise", w=w, h=h, pw=patch, ph=patch, sw=3, sh=3, speckle=i % 4 == 3)
        while _patches(j) < 4 * j["atoms"]:
            j["w"] += 32
            j["h"] += 32
        shapes.append(j)
    return shapes


def _many_jobs(c, seed):
    r = np.random.default_rng(seed)
    return [(j, _image(j["w"], j["h"], int(r.integers(1 << 30)), SIGMA, j["speckle"]).cpu().numpy())
            for j in _many_shapes(c)]


def prepare(case, seed):
    c = case
    if c["kind"] == "many":
        jobs = [(_params(j), img, _sigma2(j)) for j, img in _many_jobs(c, seed)]
        outs = [np.empty_like(img) for _, img, _ in jobs]
        return dict(case=c, jobs=jobs, outs=outs)
    ctx = KS.Context(_params(c))
    img = _image(c["w"], c["h"], seed, SIGMA, c.get("speckle", False))
    if c["kind"] == "denoise":
        img = img.cpu().numpy()
        return dict(case=c, ctx=ctx, img=img, out=np.empty_like(img))
    N, n, K, L = _patches(c), c["pw"] * c["ph"], c["atoms"], c["omp"]
    Y = torch.empty((N, n), device="cuda")
    D = torch.empty((K, n), device="cuda")
    idx = torch.empty((N, L), dtype=torch.int32, device="cuda")
    coef = torch.empty((N, L), device="cuda")
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    ctx.extract_patches(img, Y)
    ctx.init_dictionary(Y, D)
    s = dict(case=c, ctx=ctx, img=img, Y=Y, D0=D, D=D.clone(), idx=idx, coef=coef)
    if c["prec"] == LEARNED:
        ctx.set_noise_variance(_sigma2(c))
        ctx.proposal_init(seed)
    if c["kind"] == "rebuild":
        ctx.omp(Y, D, idx, coef)
        s["out"] = torch.empty_like(img)
    if c["kind"] == "learn":
        plain = KS.Context(_params(dict(c, prec=FP32)))
        plain.omp(Y, D, idx, coef)
        plain.close()
        rows = torch.randperm(N, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")[:c["batch"]]
        s["batch"], s["supports"] = Y[rows].contiguous(), idx[rows].contiguous()
        s["grad"] = torch.empty(ctx.proposal_num_params(), device="cuda")
    torch.cuda.synchronize()
    return s


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "many":
        KS.denoise_many(s["jobs"], tune=False, outs=s["outs"])
        return s["outs"]
    if kind == "denoise":
        out, stats = s["ctx"].denoise(s["img"], _sigma2(s["case"]), s["out"])
        return out, stats["lambda_"]
    if kind == "iterate":
        s["D"].copy_(s["D0"])  # an iteration works on its dictionary in place
        s["ctx"].iterate(s["Y"], s["D"], s["idx"], s["coef"], 1)
        return s["D"], s["idx"], s["coef"]
    if kind == "omp":
        s["ctx"].omp(s["Y"], s["D0"], s["idx"], s["coef"])
        return s["idx"], s["coef"]
    if kind == "rebuild":
        lam = s["ctx"].build_image(s["img"], _sigma2(s["case"]), s["D0"], s["idx"], s["coef"], s["out"])
        return s["out"], lam
    loss = s["ctx"].proposal_loss_grad(s["batch"], s["supports"], s["grad"])
    return s["grad"], loss


# ---------------------------------------------------------------------------
# the work no implementation can do without
# ---------------------------------------------------------------------------
def _omp_flops(c, N, n):
    if c["prec"] != LEARNED:
        return 2.0 * n * c["atoms"] * c["omp"] * N
    return 2.0 * N * (512 * (n + 512 + c["atoms"]) + 16 * n)


def work(case):
    c = case
    if c["kind"] == "many":
        parts = [work(j) for j in _many_shapes(c)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    N, n, K, L, P = _patches(c), c["pw"] * c["ph"], c["atoms"], c["omp"], c["w"] * c["h"]
    omp, sweep = _omp_flops(c, N, n), 6.0 * n * L * N
    if c["kind"] == "denoise":
        return dict(bytes=8.0 * P, flops=c["iters"] * (omp + sweep) + omp + 2.0 * N * n * L)
    if c["kind"] == "iterate":
        return dict(bytes=4.0 * N * n + 8.0 * N * L + 8.0 * K * n, flops=omp + sweep)
    if c["kind"] == "omp":
        return dict(bytes=4.0 * N * n + 8.0 * N * L + 4.0 * K * n, flops=omp)
    if c["kind"] == "rebuild":
        return dict(bytes=8.0 * P + 8.0 * N * L + 4.0 * K * n, flops=2.0 * N * n * L)
    params = 512.0 * (n + 512 + K)
    return dict(bytes=4.0 * c["batch"] * (n + L) + 8.0 * params, flops=6.0 * c["batch"] * params)


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _x_gather(c, img):
    nx, ny = _grid(c)
    p = img.unfold(1, c["ph"], c["sh"]).unfold(0, c["pw"], c["sw"])  # (ny, nx, ph, pw)
    return p.permute(1, 0, 2, 3).reshape(nx * ny, c["ph"] * c["pw"])


def _x_init(c, Y):
    """The initial atoms: middle patches over their norm, whose sum of squares the reference truncates term by term."""
    A = Y[Y.shape[0] // 2:Y.shape[0] // 2 + c["atoms"]]
    a = A.float().cpu().numpy()
    acc = np.zeros(a.shape[0], np.int64)
    for i in range(a.shape[1]):
        acc = (acc.astype(np.float32) + a[:, i] * a[:, i]).astype(np.int64)
    return A / torch.from_numpy(acc.astype(np.float64)).to(A.device).sqrt()[:, None]


def _x_omp(c, Y, D):
    N, K, L = Y.shape[0], c["atoms"], c["omp"]
    G = D @ D.T
    idx = torch.full((N, L), -1, dtype=torch.int64, device=Y.device)
    coef = torch.zeros((N, L), dtype=torch.float64, device=Y.device)
    lowest = torch.arange(K, device=Y.device)
    step = max(1, (1 << 26) // K)
    for p0 in range(0, N, step):
        y = Y[p0:p0 + step]
        B = y.shape[0]
        S = torch.zeros((B, L), dtype=torch.int64, device=Y.device)
        g = torch.zeros((B, L), dtype=torch.float64, device=Y.device)
        C = torch.zeros((B, L, L), dtype=torch.float64, device=Y.device)  # Cholesky factor of the support's Gram
        z = torch.zeros((B, L), dtype=torch.float64, device=Y.device)
        cnt = torch.zeros(B, dtype=torch.int64, device=Y.device)
        live = torch.ones(B, dtype=torch.bool, device=Y.device)
        r = y.clone()
        for k in range(L):
            a = r @ D.T
            a.abs_()
            a = torch.where(a == a.max(1, keepdim=True).values, lowest, K).min(1).values.clamp_max(K - 1)
            live = live & ~(S[:, :k] == a[:, None]).any(1)
            row = torch.zeros((B, L), dtype=torch.float64, device=Y.device)
            for i in range(k):
                row[:, i] = (G[S[:, i], a] - (C[:, i, :i] * row[:, :i]).sum(1)) / C[:, i, i]
            piv = G[a, a] - (row * row).sum(1)
            live = live & (piv > 0)
            row[:, k] = piv.clamp_min(1e-300).sqrt()
            C[:, k] = torch.where(live[:, None], row, C[:, k])
            C[:, k, k] = torch.where(live, C[:, k, k], torch.ones_like(piv))
            S[:, k] = torch.where(live, a, S[:, k])
            z[:, k] = torch.where(live, ((D[a] * y).sum(1) - (row[:, :k] * z[:, :k]).sum(1)) / row[:, k], z[:, k])
            new = torch.zeros_like(g)
            for i in range(k, -1, -1):
                new[:, i] = (z[:, i] - (C[:, i + 1:k + 1, i] * new[:, i + 1:k + 1]).sum(1)) / C[:, i, i]
            g = torch.where(live[:, None], new, g)
            cnt = cnt + live
            if k + 1 < L:
                r = y.clone()
                for i in range(k + 1):
                    r -= g[:, i, None] * D[S[:, i]]
                live = live & (r.norm(dim=1) >= 1e-3)
        used = torch.arange(L, device=Y.device)[None] < cnt[:, None]
        idx[p0:p0 + step] = torch.where(used, S, -1)
        coef[p0:p0 + step] = torch.where(used, g, 0.0)
    return idx, coef


def _x_update(c, Y, D, idx, coef):
    D, coef, L = D.clone(), coef.clone(), c["omp"]
    R = Y.clone()
    for s in range(L):
        R -= coef[:, s, None] * D[idx[:, s].clamp_min(0)]
    flat, x = idx.reshape(-1), coef.reshape(-1)
    flat = torch.where(x != 0, flat, -1)
    order = torch.sort(flat, stable=True).indices
    ends = torch.searchsorted(flat[order].contiguous(), torch.arange(-1, c["atoms"], device=Y.device), right=True).tolist()
    for j in range(c["atoms"]):
        e = order[ends[j]:ends[j + 1]]
        if not e.numel():
            continue
        p = e // L
        E = R[p] + x[e, None] * D[j]
        T = E[:1024] if c["cap"] else E
        M = T.T @ T
        for _ in range(12):  # the top eigenvector by squaring
            M = M @ M
            M = M / M.diagonal().sum().clamp_min(1e-300)
        u = M @ D[j]
        u = u / u.norm().clamp_min(1e-300)
        u = torch.where((u @ D[j]) < 0, -u, u)
        v = E @ u
        if c["cap"]:
            v[1024:] = 0
        D[j] = u
        x[e] = v
        R[p] = E - v[:, None] * u
    return D, x.reshape(coef.shape)


def _x_rebuild(c, img, sigma2, D, idx, coef):
    nx, ny = _grid(c)
    acc, w = torch.zeros_like(img), torch.zeros_like(img)
    X = torch.zeros((idx.shape[0], D.shape[1]), dtype=D.dtype, device=D.device)
    for s in range(idx.shape[1]):
        X += torch.where(idx[:, s, None] >= 0, coef[:, s, None] * D[idx[:, s].clamp_min(0)], 0.0)
    X = X.reshape(nx, ny, c["ph"], c["pw"])
    for r in range(c["ph"]):
        for q in range(c["pw"]):
            at = (slice(q, q + (ny - 1) * c["sw"] + 1, c["sw"]), slice(r, r + (nx - 1) * c["sh"] + 1, c["sh"]))
            acc[at] += X[:, :, r, q].T
            w[at] += 1
    d = torch.where(w > 0, acc / w.clamp_min(1) - img, 0.0)
    lam = abs(math.sqrt(float((d * d).sum()) / (sigma2 * img.numel())) - 1)
    out = torch.where(w > 0, (lam * img + acc) / (lam + w), img)
    return (torch.exp2(out) if c.get("speckle") else out), lam


def _x_denoise(c, img):
    y = torch.from_numpy(img).cuda().double()
    if c["speckle"]:
        y = torch.where(y == 0, 0.0, torch.log2(y))
    Y = _x_gather(c, y)
    D = _x_init(c, Y)
    for _ in range(c["iters"]):
        idx, coef = _x_omp(c, Y, D)
        D, _ = _x_update(c, Y, D, idx, coef)
    idx, coef = _x_omp(c, Y, D)
    return _x_rebuild(c, y, _sigma2(c), D, idx, coef)


def _x_learn(c, w, Y, sup):
    """Binary cross-entropy of the network n -> 512 -> 512 -> atoms and its gradient, parameters as the library's."""
    n, K, H = Y.shape[1], c["atoms"], 512
    sizes = [(H, n), (H,), (H, H), (H,), (K, H), (K,)]
    parts, at = [], 0
    for sz in sizes:
        parts.append(w[at:at + math.prod(sz)].reshape(sz).clone().requires_grad_())
        at += math.prod(sz)
    d = Y - Y.mean(1, keepdim=True)
    norm = d.norm(dim=1, keepdim=True)
    x = torch.where(norm > 0, d * math.sqrt(n) / norm.clamp_min(1e-300), 0.0)
    f = torch.nn.functional
    hid = f.gelu(f.linear(f.gelu(f.linear(x, parts[0], parts[1])), parts[2], parts[3]))
    t = torch.zeros((Y.shape[0], K + 1), dtype=torch.float64, device=Y.device)
    t.scatter_(1, torch.where(sup >= 0, sup, K).long(), 1.0)
    loss = f.binary_cross_entropy_with_logits(f.linear(hid, parts[4], parts[5]), t[:, :K])
    loss.backward()
    return torch.cat([p.grad.reshape(-1) for p in parts]), float(loss.detach())


def exact(case, seed):
    """What run() returns, in 64 bits.  The learned OMP has no such value: which atoms it picks among depends on its
    16-bit network."""
    c = case
    if c["prec"] == LEARNED and c["kind"] == "omp":
        return None
    if c["kind"] == "many":
        return [_x_denoise(j, img)[0].cpu().numpy() for j, img in _many_jobs(c, seed)]
    s = prepare(case, seed)
    if c["kind"] == "denoise":
        return _x_denoise(c, s["img"])
    if c["kind"] == "learn":
        w = torch.from_numpy(s["ctx"].proposal_get_params()).cuda().double()
        return _x_learn(c, w, s["batch"].double(), s["supports"])
    Y, D = s["Y"].double(), s["D0"].double()
    if c["kind"] == "rebuild":
        return _x_rebuild(c, s["img"].double(), _sigma2(c), D, s["idx"].long(), s["coef"].double())
    idx, coef = _x_omp(c, Y, D)
    if c["kind"] == "omp":
        return idx.int(), coef
    D, coef = _x_update(c, Y, D, idx, coef)
    return D, idx.int(), coef
