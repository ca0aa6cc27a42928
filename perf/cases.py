"""The library's working set: the calls a user of the GP framework makes, over the sizes they are made at.

Every case is one call through a public entry point (``gprat_b200.capi``, ``gprat_b200.autograd``,
``gprat_b200.serving``) on a model that already holds its training data.  Series and targets follow the
benchmark's generator: x ~ N(0, 1), y_i = sum_j sin(x_{i+j}) / 8 + N(0, 0.01^2), test series ~ N(0, 1).
"""
import math

import numpy as np
import torch

from gprat_b200 import autograd, capi, serving

PRECISION = {"fp64": capi.PREC_FP64, "int8": capi.PREC_FP64_INT8, "tf32": capi.PREC_MIXED_TF32,
             "bf16": capi.PREC_MIXED_BF16}
ADAM = (0.1, 0.9, 0.999, 1e-8)  # learning rate, beta1, beta2, epsilon: the reference's defaults
GIB = 1 << 30


def _case(kind, precision, n_tiles, tile, d, m=0, name=None):
    c = {"kind": kind, "precision": precision, "n_tiles": n_tiles, "tile": tile, "d": d, "m": m}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest regression in use (16 tiles of 64 points): launches and the serial chain count
        _case("predict", "fp64", 16, 64, 8, 512, "predict fp64 n=1024"),
        # a data set whose size nobody rounded: 13 tiles of 250 points, an odd number of regressors and test points
        _case("predict", "fp64", 13, 250, 21, 777, "predict fp64 n=3250"),
        # the larger single-call regression of the benchmark (32 tiles of 512), host buffers in and out
        _case("predict", "fp64", 32, 512, 8, 4096, "predict fp64 n=16384"),
        # the benchmark's largest workload in the default precision, inputs and outputs resident on the GPU
        _case("device", "fp64", 32, 1024, 64, 8192, "device fp64 n=32768"),
        # the same workload in the benchmark's headline precision
        _case("device", "int8", 32, 1024, 64, 8192, "device int8 n=32768"),
        # the single-call regression in the headline precision, host buffers
        _case("predict", "int8", 32, 512, 8, 4096, "predict int8 n=16384"),
        # the low-precision factor with refined weights, at both ends of where it is used
        _case("predict", "tf32", 32, 512, 8, 4096, "predict tf32 n=16384"),
        _case("predict", "bf16", 16, 256, 16, 1024, "predict bf16 n=4096"),
        # hyper-parameter training: one Adam step of the optimisation benchmark (loss, gradient, update)
        _case("optimize", "fp64", 16, 512, 8, 0, "optimize_step n=8192"),
        # the loss as a torch function, forward and backward, at the size of a quick experiment
        _case("autograd", "fp64", 8, 256, 8, 0, "nlml forward+backward n=2048"),
        # serving: a fitted model answers a burst of requests of uneven sizes
        _case("serve", "int8", 16, 512, 8, 1500, "serve int8 n=8192"),
        # the factor itself, as the reference returns it: tiles in host memory
        _case("cholesky", "fp64", 8, 256, 8, 0, "cholesky n=2048"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["predict", "predict", "predict", "device", "device", "optimize", "autograd", "serve",
                       "cholesky"])
    precision = rng.choice(["fp64", "fp64", "int8", "tf32", "bf16"]) if kind in ("predict", "device") else "fp64"
    if kind == "serve":
        precision = rng.choice(["fp64", "int8"])
    top = {"predict": 16384, "device": 24576, "optimize": 10240, "autograd": 6144, "serve": 10240,
           "cholesky": 3072}[kind]
    n = _log_int(rng, 700, top)
    # the tensor-core modes are for problems whose posterior variance is not tiny next to the prior: 8 regressors up
    d = rng.choice([8, 11, 16, 21, 32, 64] if precision != "fp64" else [1, 4, 7, 8, 16, 21, 32, 64])
    m = 0 if kind in ("optimize", "autograd", "cholesky") else _log_int(rng, 60, 6000)
    n_tiles = rng.randint(3, 10) if kind == "cholesky" else rng.randint(4, 32)
    tile = max(1, n // n_tiles)
    if precision != "fp64":  # the tensor-core modes take training sets of a multiple of 128 points
        n_tiles, tile = max(6, n // 128), 128
    return _case(kind, precision, n_tiles, tile, d, m)


# lengthscale, vertical lengthscale, noise variance: the benchmark's for many and for few regressors
def _hyper(case):
    return (4.0, 1.0, 0.01) if case["d"] >= 32 else (1.0, 1.0, 0.1)


def _size(case):
    return case["n_tiles"] * case["tile"]


def _burst(case):
    """Request sizes of a serving burst: half of the points in one request, the rest halved again and again."""
    sizes, left = [], case["m"]
    while left > 0 and len(sizes) < 7:
        take = max(1, left // 2)
        sizes.append(take)
        left -= take
    return sizes


def _data(case, seed):
    rng = np.random.default_rng(seed)
    n, d, m = _size(case), case["d"], case["m"]
    x = rng.standard_normal(n + d - 1)
    windows = np.lib.stride_tricks.sliding_window_view(np.sin(x), d)[:n]
    y = windows.sum(axis=1) / 8.0 + 0.01 * rng.standard_normal(n)
    xt = rng.standard_normal(max(m, 1) + d - 1)
    theta0 = np.array([0.5, 2.0, 0.5]) * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, 3))
    return x, y, xt, theta0


def prepare(case, seed):
    x, y, xt, theta0 = _data(case, seed)
    s = {"case": case, "hyper": np.array(_hyper(case)), "xt": xt}
    if case["kind"] == "serve":
        s["server"] = serving.Server(0, 8 * GIB, PRECISION[case["precision"]])
        s["model"] = s["server"].add_model(x, y, case["n_tiles"], case["tile"], case["d"], s["hyper"])
        at, parts = 0, []
        for size in _burst(case):
            parts.append((np.ascontiguousarray(xt[at:at + size + case["d"] - 1]), size))
            at += size
        s["requests"] = parts
        return s
    gp = capi.CudaGP(x, y, case["n_tiles"], case["tile"], case["d"])
    gp.set_precision(PRECISION[case["precision"]])
    s["gp"] = gp
    if case["kind"] == "device":
        s["d_xt"] = torch.from_numpy(xt).cuda()
        s["mean"] = torch.empty(case["m"], dtype=torch.float64, device="cuda")
        s["var"] = torch.empty(case["m"], dtype=torch.float64, device="cuda")
    elif case["kind"] == "optimize":
        s["params"] = np.concatenate([theta0, np.zeros(6)])
    elif case["kind"] == "autograd":
        s["theta"] = torch.tensor(theta0, dtype=torch.float64, requires_grad=True)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "predict":
        return s["gp"].predict_with_uncertainty(s["hyper"], s["xt"], 1, case["m"])
    if kind == "device":
        s["gp"].fit_predict_device(s["hyper"], s["d_xt"].data_ptr(), s["d_xt"].numel(), case["m"],
                                   s["mean"].data_ptr(), s["var"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        return s["mean"], s["var"]
    if kind == "optimize":
        return s["gp"].optimize_step(s["params"], ADAM, (1, 1, 1), 0)
    if kind == "autograd":
        theta = s["theta"]
        theta.grad = None
        loss = autograd.nlml(s["gp"], theta)
        loss.backward()
        return loss.detach(), theta.grad
    if kind == "serve":
        ids = [s["server"].submit_predict(s["model"], xt, size) for xt, size in s["requests"]]
        return [s["server"].wait(i)[:2] for i in ids]
    return s["gp"].cholesky(s["hyper"])


def work(case):
    n, d, m = float(_size(case)), case["d"], float(case["m"])
    factor, series = n ** 3 / 3, 8 * (2 * n + d)
    kind = case["kind"]
    if kind in ("predict", "device"):
        return {"bytes": series + 8 * (3 * m + d), "flops": factor + 2 * n * n + n * n * m + 2 * n * m}
    if kind == "optimize":
        return {"bytes": series + 8 * 19, "flops": 3 * factor + 2 * n * n}
    if kind == "autograd":
        return {"bytes": series + 8 * 7, "flops": 3 * factor + 2 * n * n}
    if kind == "serve":  # the resident factor and weights are read, nothing is factored
        return {"bytes": 4 * n * n + series + 8 * 3 * m, "flops": n * n * m + 2 * n * m}
    return {"bytes": series + 4 * n * (n + 1), "flops": factor}


# --- the same quantities from torch in 64 bits ------------------------------------------------------------


def _squared_distances(xa, xb, d):
    out = torch.empty((xa.numel() - d + 1, xb.numel() - d + 1), dtype=torch.float64, device=xa.device)
    cols = out.shape[1]
    for r0 in range(0, out.shape[0], 2048):
        rows = min(2048, out.shape[0] - r0)
        part = out[r0:r0 + rows]
        part.zero_()
        for k in range(d):
            z = xa[r0 + k:r0 + k + rows, None] - xb[None, k:k + cols]
            part.addcmul_(z, z)
    return out


def _covariance(xa, xb, d, theta):
    r2 = _squared_distances(xa, xb, d)
    return r2.mul_(-0.5 / (theta[0] * theta[0])).exp_().mul_(theta[1])


def _softplus_inverse(t):
    return math.log(math.expm1(t))


def _loss_and_gradient(x, y, d, theta):
    """NLML per point and its gradient in the constrained parameters."""
    n = y.numel()
    r2 = _squared_distances(x, x, d)
    e = torch.exp(r2 * (-0.5 / theta[0] ** 2))
    K = theta[1] * e
    K.diagonal().add_(theta[2])
    L = torch.linalg.cholesky(K)
    del K
    alpha = torch.cholesky_solve(y[:, None], L)[:, 0]
    loss = 0.5 * (torch.dot(y, alpha) + 2 * torch.log(L.diagonal()).sum() + n * math.log(2 * math.pi)) / n
    Q = torch.cholesky_inverse(L)
    del L
    Q -= torch.outer(alpha, alpha)
    e.mul_(Q)
    scale = 0.5 / n
    g_v = scale * e.sum()
    g_l = scale * theta[1] / theta[0] ** 3 * e.mul_(r2).sum()
    g_s = scale * Q.diagonal().sum()
    return float(loss), [float(g_l), float(g_v), float(g_s)]


def exact(case, seed):
    x, y, xt, theta0 = _data(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    xs, ys, ts = (torch.from_numpy(v).to(dev) for v in (x, y, xt))
    n, d, kind, theta = _size(case), case["d"], case["kind"], _hyper(case)
    if kind in ("optimize", "autograd"):
        loss, grad = _loss_and_gradient(xs, ys, d, theta0)
        if kind == "autograd":
            return torch.tensor(loss, dtype=torch.float64), torch.tensor(grad, dtype=torch.float64)
        lr, b1, b2, eps = ADAM
        out = np.zeros(9)
        for q in range(3):  # one Adam step from zero moments on the softplus-unconstrained parameters
            shift = 1e-6 if q == 2 else 0.0
            u = _softplus_inverse(theta0[q] - shift)
            g = grad[q] / (1.0 + math.exp(-u))
            out[3 + q], out[6 + q] = (1 - b1) * g, (1 - b2) * g * g
            u -= lr * math.sqrt(1 - b2) / (1 - b1) * out[3 + q] / (math.sqrt(out[6 + q]) + eps)
            out[q] = math.log1p(math.exp(u)) + shift
        return loss, out
    K = _covariance(xs, xs, d, theta)
    K.diagonal().add_(theta[2])
    L = torch.linalg.cholesky(K)
    if kind == "cholesky":
        nt, t = case["n_tiles"], case["tile"]
        full = (torch.tril(L) + torch.triu(K, 1)).cpu().numpy()
        return [full[i * t:(i + 1) * t, j * t:(j + 1) * t].reshape(-1) if j <= i else None
                for i in range(nt) for j in range(nt)]
    del K
    alpha = torch.cholesky_solve(ys[:, None], L)[:, 0]

    def predict(series):
        Ks = _covariance(series, xs, d, theta)
        mean = Ks @ alpha
        V = torch.linalg.solve_triangular(L, Ks.T, upper=False)
        return mean.cpu(), (theta[1] - V.square_().sum(dim=0)).cpu()

    if kind != "serve":
        return predict(ts)
    out, at = [], 0
    for size in _burst(case):
        out.append(predict(ts[at:at + size + d - 1]))
        at += size
    return out
