"""Performance cases of the signature-kernel engine: calls of `sigpde_b200.torch` as programs make them.

A case names the call ("kind"), the path counts, lengths, dimension, dyadic order, static kernel,
input type and cell precision.  Paths are Brownian (increments N(0, 1/(L-1))), the engine's benchmark
inputs; robust calls scale each path by a factor log-uniform in [0.5, 4].

Kinds
  pairwise  SigPDE.pairwise(x, y): k(x_b, y_b) of a batch
  gram      SigPDE.gram(x, y), or the symmetric Gram where "sym" is true
  robust    RobustSigPDE.gram(x): the root-find for every path's scale, then the symmetric Gram
  scales    RobustSigPDE.normalization(x): the scales alone
  uneven    sig.ragged.RaggedPairwise: a batch of pairs with their own lengths and orders, new values
            loaded into a kept plan each pass
  train     forward and backward of sum(w * gram(x, y)): the values and both gradients
  step      forward and backward of sum(w * pairwise(x, y))
"""
import math

import torch

import sigpde_b200.torch as sig

DTYPES = {"float32": torch.float32, "float64": torch.float64}
SIGMA = 1.0  # RBF bandwidth


def listed():
    return [
        # the smallest call: a batch of short paths, where launches and host latency are the cost
        dict(name="pairwise8", kind="pairwise", nx=8, lx=20, ly=20, d=5, order=1, kernel="linear", dtype="float32",
             precision="fp64"),
        # a serving-sized small symmetric Gram (a few paths of odd length)
        dict(name="gram_sym24", kind="gram", nx=24, ny=24, sym=True, lx=65, ly=65, d=3, order=1, kernel="linear",
             dtype="float32", precision="fp64"),
        # an ordinary two-sample batch in float64, uneven lengths, no refinement
        dict(name="pairwise1000", kind="pairwise", nx=1000, lx=101, ly=77, d=4, order=0, kernel="linear",
             dtype="float64", precision="fp64"),
        # the headline Gram, float64 cells (the default) and tensor-core increments
        dict(name="gram256", kind="gram", nx=256, ny=256, sym=False, lx=128, ly=128, d=8, order=2, kernel="linear",
             dtype="float32", precision="fp64"),
        dict(name="gram256_tc64", kind="gram", nx=256, ny=256, sym=False, lx=128, ly=128, d=8, order=2,
             kernel="linear", dtype="float32", precision="tc64"),
        # a wide-path symmetric Gram of serving size, odd counts and lengths
        dict(name="gram_wide195", kind="gram", nx=195, ny=195, sym=True, lx=196, ly=196, d=32, order=1,
             kernel="linear", dtype="float32", precision="tc32"),
        # a static kernel evaluated on the device
        dict(name="rbf_gram200", kind="gram", nx=200, ny=170, sym=False, lx=128, ly=111, d=8, order=1, kernel="rbf",
             dtype="float32", precision="fp64"),
        # the robust benchmark, and a robust request of few long wide paths (latency of the root-find)
        dict(name="robust512", kind="robust", nx=512, lx=64, d=16, order=1, kernel="linear", dtype="float32",
             precision="fp64"),
        dict(name="scales24_long", kind="scales", nx=24, lx=220, d=8, order=1, kernel="linear", dtype="float32",
             precision="fp64"),
        # uneven pairs in one launch
        dict(name="uneven4096", kind="uneven", nx=4096, lmin=16, lmax=512, d=32, orders=3, dtype="float32",
             precision="tc64"),
        # training steps: the Gram loss of the gradient benchmark, and a small batch with an RBF kernel
        dict(name="train128", kind="train", nx=128, ny=128, lx=128, ly=128, d=8, order=2, kernel="linear",
             dtype="float64", precision="fp64"),
        dict(name="step64_rbf", kind="step", nx=64, lx=50, ly=50, d=4, order=1, kernel="rbf", dtype="float32",
             precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# refined cells of the largest listed case of each kind
_MOST_CELLS = {"pairwise": 4.0e9, "gram": 1.6e10, "robust": 2.0e9, "scales": 1.6e8, "uneven": 4.0e9, "train": 4.0e9,
               "step": 4.0e8}


def draw(rng):
    kind = rng.choice(["pairwise", "gram", "gram", "gram", "robust", "scales", "uneven", "train", "train", "step"])
    c = dict(kind=kind, d=_log_int(rng, 2, 32), dtype=rng.choice(["float32", "float32", "float64"]))
    if kind == "uneven":
        c.update(nx=_log_int(rng, 64, 4096), lmin=rng.randint(8, 32), lmax=_log_int(rng, 64, 512),
                 orders=rng.randint(0, 3), precision=rng.choice(["fp64", "tc64"]))
        return c
    c["order"] = rng.choice([0, 1, 1, 2, 2, 3]) if kind in ("pairwise", "gram") else rng.choice([0, 1, 2])
    c["lx"] = _log_int(rng, 16, 128) if kind in ("train", "step") else _log_int(rng, 20, 256)
    c["nx"] = {"pairwise": lambda: _log_int(rng, 8, 1024), "gram": lambda: _log_int(rng, 8, 256),
               "robust": lambda: _log_int(rng, 8, 512), "scales": lambda: _log_int(rng, 8, 512),
               "train": lambda: _log_int(rng, 8, 128), "step": lambda: _log_int(rng, 8, 512)}[kind]()
    c["kernel"] = "linear" if kind in ("robust", "scales") else rng.choice(["linear", "linear", "linear", "rbf"])
    c["precision"] = "fp64" if kind in ("scales", "train", "step") else rng.choice(
        ["fp64", "fp64", "fp64", "tc64", "tc64", "fp32", "tc32"])
    if kind in ("pairwise", "step"):
        c["ly"] = max(16, int(c["lx"] * rng.uniform(0.5, 1.5)))
    elif kind in ("gram", "train"):
        c["sym"] = kind == "gram" and rng.random() < 0.4
        c["ly"] = c["lx"] if c["sym"] else max(16, int(c["lx"] * rng.uniform(0.6, 1.4)))
        c["ny"] = c["nx"] if c["sym"] else max(4, int(c["nx"] * rng.uniform(0.5, 1.5)))
        if kind == "train" and c["kernel"] == "rbf":  # torch builds these increments: batches of moderate size
            c["nx"], c["ny"] = min(c["nx"], 48), min(c["ny"], 48)
    while _cells(c) > _MOST_CELLS[kind]:
        c["nx"] = max(4, int(c["nx"] * 0.8))
        if "ny" in c:
            c["ny"] = c["nx"] if c.get("sym") else max(4, int(c["ny"] * 0.8))
    return c


# ------------------------------------------------------------------ inputs
def _brownian(g, n, length, d, dtype, scale=None):
    inc = torch.randn(n, length - 1, d, generator=g, device="cuda", dtype=torch.float64) / math.sqrt(length - 1)
    x = torch.zeros(n, length, d, device="cuda", dtype=torch.float64)
    torch.cumsum(inc, 1, out=x[:, 1:])
    if scale is not None:
        x = x * scale[:, None, None]
    return x.to(DTYPES[dtype])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uneven_lengths(c, seed):
    g = torch.Generator().manual_seed(int(seed))
    def lens():
        return torch.randint(c["lmin"], c["lmax"] + 1, (c["nx"],), generator=g)
    return lens(), lens(), torch.randint(0, c["orders"] + 1, (c["nx"],), generator=g)


def _uneven_pack(g, lens, d, dtype):
    """Brownian paths of the given lengths, packed back to back."""
    lens = lens.to("cuda")
    top = int(lens.max())
    inc = torch.randn(len(lens), top, d, generator=g, device="cuda", dtype=torch.float32)
    inc /= (lens - 1).to(torch.float32).sqrt()[:, None, None]
    inc[:, 0] = 0
    x = torch.cumsum(inc, 1, dtype=torch.float64)
    keep = torch.arange(top, device="cuda")[None, :] < lens[:, None]
    return x[keep].to(DTYPES[dtype])


def _inputs(c, seed):
    """The case's tensors, from the seed alone."""
    g = _gen(seed)
    if c["kind"] == "uneven":
        lx, ly, orders = _uneven_lengths(c, seed)
        return dict(lx=lx, ly=ly, orders=orders, x=_uneven_pack(g, lx, c["d"], c["dtype"]),
                    y=_uneven_pack(g, ly, c["d"], c["dtype"]))
    if c["kind"] in ("robust", "scales"):
        f = torch.exp(torch.rand(c["nx"], generator=g, device="cuda", dtype=torch.float64) * math.log(8.0)) * 0.5
        return dict(x=_brownian(g, c["nx"], c["lx"], c["d"], c["dtype"], f))
    s = dict(x=_brownian(g, c["nx"], c["lx"], c["d"], c["dtype"]))
    if not c.get("sym"):
        s["y"] = _brownian(g, c.get("ny", c["nx"]), c["ly"], c["d"], c["dtype"])
    if c["kind"] in ("train", "step"):
        shape = (c["nx"], c["ny"]) if c["kind"] == "train" else (c["nx"],)
        s["w"] = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64).to(DTYPES[c["dtype"]])
    return s


def _static_kernel(c):
    return sig.kernels.LinearKernel() if c["kernel"] == "linear" else sig.kernels.RBFKernel(SIGMA)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "uneven":
        s["solver"] = sig.ragged.RaggedPairwise(s["lx"].tolist(), s["ly"].tolist(), s["orders"].tolist(), case["d"],
                                                DTYPES[case["dtype"]], "cuda", case["precision"])
    elif case["kind"] in ("robust", "scales"):
        s["solver"] = sig.RobustSigPDE(_static_kernel(case), case["order"], precision=case["precision"])
    else:
        s["solver"] = sig.SigPDE(_static_kernel(case), case["order"], precision=case["precision"])
    if case["kind"] in ("train", "step"):
        s["x"].requires_grad_()
        s["y"].requires_grad_()
    return s


def run(state):
    kind, k = state["case"]["kind"], state["solver"]
    if kind == "uneven":
        k.load_packed(state["x"], state["y"])
        return k.solve()
    if kind == "robust":
        return k.gram(state["x"])
    if kind == "scales":
        return k.normalization(state["x"])
    x, y = state["x"], state.get("y")
    if kind == "pairwise":
        return k.pairwise(x, y)
    if kind == "gram":
        return k.gram(x, y)
    values = k.gram(x, y) if kind == "train" else k.pairwise(x, y)
    gx, gy = torch.autograd.grad((state["w"] * values).sum(), (x, y))
    return {"values": values.detach(), "grad_x": gx, "grad_y": gy}


# ------------------------------------------------------------------ work
def _pairs(c):
    if c["kind"] in ("pairwise", "step", "uneven", "scales"):
        return c["nx"]
    if c["kind"] == "robust" or c.get("sym"):
        return c["nx"] * (c["nx"] + 1) // 2
    return c["nx"] * c["ny"]


def _cells(c):
    """Refined cells of all pairs (uneven batches: their mean)."""
    if c["kind"] == "uneven":
        mean = ((c["lmin"] + c["lmax"]) / 2 - 1) ** 2
        return c["nx"] * mean * sum(4 ** o for o in range(c["orders"] + 1)) / (c["orders"] + 1)
    ly = c.get("ly", c["lx"])
    return _pairs(c) * (c["lx"] - 1) * (ly - 1) * 4.0 ** c["order"]


def work(case):
    c = case
    el = 8 if c["dtype"] == "float64" else 4
    cells, pairs, d = _cells(c), _pairs(c), c["d"]
    if c["kind"] == "uneven":
        coarse = c["nx"] * ((c["lmin"] + c["lmax"]) / 2 - 1) ** 2
        points = c["nx"] * (c["lmin"] + c["lmax"])
        return {"bytes": el * (points * d + c["nx"]), "flops": 4 * cells + 2 * d * coarse}
    coarse = cells / 4.0 ** c["order"]
    path_values = c["nx"] * c["lx"] * d
    if c["kind"] not in ("robust", "scales") and not c.get("sym"):
        path_values += c.get("ny", c["nx"]) * c["ly"] * d
    outs = {"scales": c["nx"], "robust": c["nx"] ** 2, "pairwise": c["nx"], "step": c["nx"]}.get(
        c["kind"], c["nx"] * c.get("ny", c["nx"]))
    # a cell: add, multiply, fused multiply-add (4 operations); a coarse cell: its d-term increment
    flops = 4 * cells + (2 * d + 8) * coarse
    if c["kind"] in ("robust", "scales"):  # the root-find: one solve for k(x, x) and about eight of the bracket's
        self_cells = c["nx"] * (c["lx"] - 1) ** 2 * 4.0 ** c["order"]
        flops = (flops if c["kind"] == "robust" else 0) + 9 * 4 * self_cells
    moved = el * (path_values + outs)
    if c["kind"] in ("train", "step"):  # the adjoint's cell and the derivative's two sums; the contractions
        flops += 8 * cells + (4 * d + 8) * coarse
        moved = el * (2 * path_values + 2 * outs)
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------ values in 64 bits
def _increments(c, x, y, pairwise):
    """Coarse increments / 4^order of pairs, cells first: (ncx, ncy, pairs...)."""
    if c["kernel"] == "linear":
        dx, dy = x[:, 1:] - x[:, :-1], y[:, 1:] - y[:, :-1]
        inc = torch.einsum("aik,ajk->ija" if pairwise else "aik,bjk->ijab", dx, dy)
    else:
        ip = torch.einsum("aik,ajk->ija" if pairwise else "aik,bjk->ijab", x, y)
        xx, yy = (x * x).sum(-1).t(), (y * y).sum(-1).t()  # (points, paths)
        sq = xx[:, None] + yy[None] if pairwise else xx[:, None, :, None] + yy[None, :, None, :]
        G = torch.exp(-(sq - 2 * ip) / SIGMA)
        inc = G[1:, 1:] + G[:-1, :-1] - G[1:, :-1] - G[:-1, 1:]
    return inc / 4.0 ** c["order"]


def _diagonals(ncx, ncy, order):
    """For every anti-diagonal: its rows [p0, p1) and the coarse cell of each (1-based fine rows p, columns k - p)."""
    n, m = ncx << order, ncy << order
    for k in range(2, n + m + 1):
        p0, p1 = max(1, k - m), min(n, k - 1) + 1
        p = torch.arange(p0, p1, device="cuda")
        yield k, p0, p1, ((p - 1) >> order) * ncy + ((k - p - 1) >> order)


def _solve(inc, order, keep=None):
    """K[n][m] of every pair from increments (ncx, ncy, P), anti-diagonal by anti-diagonal; `keep` takes them all."""
    ncx, ncy, P = inc.shape
    n = ncx << order
    flat = inc.reshape(ncx * ncy, P)
    A, B = 1 + flat / 2 + flat * flat / 12, 1 - flat * flat / 12
    # row p of a diagonal holds K(p, k - p); rows outside it hold the boundary value 1
    older, old = (torch.ones(n + 2, P, dtype=torch.float64, device="cuda") for _ in range(2))
    for k, p0, p1, at in _diagonals(ncx, ncy, order):
        new = torch.ones_like(old)
        new[p0:p1] = (old[p0:p1] + old[p0 - 1:p1 - 1]) * A[at] - older[p0 - 1:p1 - 1] * B[at]
        if keep is not None:
            keep.append(new)
        older, old = old, new
    return old[n].clone()


def _solve_backward(inc, order, w):
    """K[n][m], and d(sum w K)/d inc."""
    ncx, ncy, P = inc.shape
    n = ncx << order
    one = torch.ones(n + 2, P, dtype=torch.float64, device="cuda")
    keep = [one, one]
    value = _solve(inc, order, keep)
    flat = inc.reshape(ncx * ncy, P)
    grad = torch.zeros_like(flat)
    Pr, Qr, Qrr = (torch.zeros(n + 2, P, dtype=torch.float64, device="cuda") for _ in range(3))
    diags = list(_diagonals(ncx, ncy, order))
    for i, (k, p0, p1, at) in reversed(list(enumerate(diags))):
        lam = Pr[p0:p1] + Pr[p0 + 1:p1 + 1] - Qrr[p0 + 1:p1 + 1]
        if i == len(diags) - 1:
            lam = lam + w
        c = flat[at]
        old, older = keep[i + 1], keep[i]
        dk = (old[p0:p1] + old[p0 - 1:p1 - 1]) * (0.5 + c / 6) + older[p0 - 1:p1 - 1] * (c / 6)
        grad.index_add_(0, at, lam * dk)
        Pn, Qn = torch.zeros_like(Pr), torch.zeros_like(Pr)
        Pn[p0:p1], Qn[p0:p1] = lam * (1 + c / 2 + c * c / 12), lam * (1 - c * c / 12)
        Pr, Qr, Qrr = Pn, Qn, Qr
    return value, grad.reshape(inc.shape)


def _exact_scales(c, x):
    """lambda with k(lambda x, lambda x) = f(k(x, x)), f(s) = 2 - 1 / (1 + log s), by Ridders' method."""
    inc = _increments(c, x, x, True)
    k = _solve(inc, c["order"])
    f = 2 - 1 / (1 + torch.log(k))
    lo, hi = torch.zeros_like(k), torch.ones_like(k)
    flo, fhi = 1 - f, k - f
    best = hi.clone()
    for _ in range(24):
        mid = (lo + hi) / 2
        fm = _solve(inc * mid * mid, c["order"]) - f
        s = torch.sqrt((fm * fm - flo * fhi).clamp_min(1e-300))
        new = (mid + (mid - lo) * torch.sign(flo - fhi) * fm / s).clamp(lo, hi)
        fn = _solve(inc * new * new, c["order"]) - f
        done = (new - best).abs().max() < 1e-15
        best = new
        for a, fa in ((mid, fm), (new, fn)):  # keep the sign change inside [lo, hi]
            inside = (a > lo) & (a < hi)
            low = inside & (fa < 0)
            high = inside & (fa >= 0)
            lo, flo = torch.where(low, a, lo), torch.where(low, fa, flo)
            hi, fhi = torch.where(high, a, hi), torch.where(high, fa, fhi)
        if done:
            break
    return torch.where(k < 1, torch.zeros_like(k), best)


def _parts(n, per, most=2.0e8):
    step = max(1, int(most / per))
    return [(i, min(n, i + step)) for i in range(0, n, step)]


def _exact_gram(c, x, y):
    n, m = (x.shape[1] - 1) << c["order"], (x.shape[1] - 1) * (y.shape[1] - 1)
    return torch.cat([_solve(_increments(c, x[i:j], y, False).flatten(2), c["order"]).reshape(j - i, -1)
                      for i, j in _parts(x.shape[0], y.shape[0] * max(n, m))])


def _exact_uneven(c, s):
    d = c["d"]
    out = torch.empty(c["nx"], dtype=torch.float64, device="cuda")
    def padded(pack, lens):  # rows beyond a path's end repeat its last point: increments 0 leave K unchanged
        lens = lens.to("cuda")
        start = torch.cumsum(lens, 0) - lens
        at = start[:, None] + torch.minimum(torch.arange(int(lens.max()), device="cuda")[None], lens[:, None] - 1)
        return pack.double()[at.reshape(-1)].reshape(len(lens), -1, d)
    x, y = padded(s["x"], s["lx"]), padded(s["y"], s["ly"])
    for o in range(c["orders"] + 1):
        idx = (s["orders"] == o).nonzero().reshape(-1)
        if not len(idx):
            continue
        idx = idx[torch.argsort((torch.maximum(s["lx"], s["ly"]))[idx])]
        for part in idx.split(max(1, -(-len(idx) // 4))):
            a, b = int(s["lx"][part].max()), int(s["ly"][part].max())
            at = part.to("cuda")
            inc = _increments(dict(kernel="linear", order=o), x[at, :a], y[at, :b], True)
            out[at] = _solve(inc, o)
    return out


def exact(case, seed):
    c, s = case, _inputs(case, seed)
    if c["kind"] == "uneven":
        return _exact_uneven(c, s)
    x = s["x"].double()
    if c["kind"] == "scales":
        return _exact_scales(c, x)
    if c["kind"] == "robust":
        x = x * _exact_scales(c, x)[:, None, None]
        return _exact_gram(c, x, x)
    y = s["y"].double() if "y" in s else x
    if c["kind"] == "gram":
        return _exact_gram(c, x, y)
    if c["kind"] == "pairwise":
        return _solve(_increments(c, x, y, True), c["order"])
    x.requires_grad_()
    y.requires_grad_()
    pairwise, w = c["kind"] == "step", s["w"].double()
    n, m = (c["lx"] - 1) << c["order"], (c["ly"] - 1) << c["order"]
    values = []
    for i, j in _parts(c["nx"], (1 if pairwise else c["ny"]) * n * (n + m), 8.0e8):
        inc = _increments(c, x[i:j], y[i:j] if pairwise else y, pairwise)
        v, g = _solve_backward(inc.detach().flatten(2), c["order"], w[i:j].reshape(-1))
        inc.backward(g.reshape(inc.shape))
        values.append(v.reshape(w[i:j].shape))
    return {"values": torch.cat(values), "grad_x": x.grad, "grad_y": y.grad}
