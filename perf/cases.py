"""The framework's work as a user's program has it done, as cases that can be timed.

Each case is a dict of plain values.  ``prepare`` makes what the program holds before the
call (lattice, plan, strikes, workspace, weights, tables), ``run`` is one pass through the
public entry points, ``work`` states what a pass cannot do without, ``exact`` restates the
result in 64 bits with torch alone.  Kinds:

  solve      European quotes of one local-vol or stochastic-vol lattice (Lattice.solve)
  bermudan   Bermudan / down-and-out contracts by induction (Lattice.bermudan)
  batch      many uneven lattices in one plan (Batch.execute)
  calibrate  one pricing call of a calibration: parameters in, prices out, host to host
  mc         step kernel, cumulative rows, guide table and the Monte Carlo over them
  paths      Monte Carlo over rows that are already there, every state kept
  infer      surrogate quotes of a whole book (Surrogate.predict)
  train      one step of surrogate training: gradient and Adam
  grouped    the drop-in grouped FP32 products through a task table (opcuda_sgemm4)
"""
import math

import numpy as np
import torch

from oplib_b200 import _lib
from oplib_b200.calibrate import BOX_HI, LVBatchPricer
from oplib_b200.model import Batch, Lattice, bind_stream, cumulative_rows, guide_table, mc_run
from oplib_b200.surrogate import Surrogate

DEV = "cuda"
F64 = torch.float64
X_LO, X_HI = 0.05, 5.0
MLP_SIZES = [(8, 256), (256, 256), (256, 256), (256, 256), (256, 1)]


# ------------------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest solve: a coarse lattice priced while somebody waits (smoke-test size)
        dict(name="solve_lv256", kind="solve", model="lv", n=256, nk=64, nmat=4, period=0.25, dt0_log2=14,
             mode="bf16x3", all_states=False),
        # the plain local-vol configuration: 512 nodes, 64 strikes, 8 quarterly maturities
        dict(name="solve_lv512", kind="solve", model="lv", n=512, nk=64, nmat=8, period=0.25, dt0_log2=14,
             mode="bf16x3", all_states=False),
        # a size off the tile grid with an odd strike count and the values of every state
        dict(name="solve_lv1000_states", kind="solve", model="lv", n=1000, nk=37, nmat=5, period=0.25, dt0_log2=14,
             mode="fp16x3", all_states=True),
        # the stochastic-vol configuration: 48 x 128 states, 128 strikes, 16 maturities
        dict(name="solve_sv6144", kind="solve", model="sv", n=128, nv=48, nk=128, nmat=16, period=0.25, dt0_log2=16,
             mode="bf16x3", all_states=False),
        # Bermudan puts on a middle-sized stochastic-vol lattice
        dict(name="bermudan_sv3072", kind="bermudan", model="sv", n=128, nv=24, nk=128, nmat=16, period=0.25,
             dt0_log2=16, mode="fp16x3", put=True, barrier=0.0),
        # half of the calibration sweep: sizes 256..2048 in steps of 128, 32 strikes x 8 maturities
        dict(name="sweep_256_lattices", kind="batch", nlat=256, n_lo=256, n_hi=2048, n_step=128, nk=32, nmat=8,
             period=0.25, mode="bf16x3"),
        # one pricing call of a small calibration: 8 problems, trial point and six bumps each
        dict(name="calibrate_8", kind="calibrate", problems=8, n_lo=256, n_hi=640, nk=16, nmat=4, period=0.25,
             mode="fp16x3"),
        # the Monte Carlo configuration from the generator on: 2^20 paths x 504 daily steps
        dict(name="mc_2p20_504", kind="mc", n=512, npaths=1 << 20, nsteps=504, mode="fp32"),
        # a ragged number of long paths with every state written out
        dict(name="paths_700", kind="paths", n=512, npaths=100_003, nsteps=700),
        # the surrogate over 2^20 quotes, four members
        dict(name="surrogate_2p20", kind="infer", rows=1 << 20, members=4),
        # one training step at the training batch size
        dict(name="train_step_4096", kind="train", rows=4096),
        # the reference's grouped-product benchmark shape: 40 products of 576^3
        dict(name="grouped_40x576", kind="grouped", count=40, m=576, n=576, k=576),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "bermudan", "batch", "calibrate", "mc", "paths", "infer", "train",
                       "grouped"])
    mode = rng.choice(["bf16x3", "bf16x3", "fp16x3"])
    if kind in ("solve", "bermudan"):
        c = dict(kind=kind, nk=_log_int(rng, 4, 128), nmat=rng.randint(1, 16), period=rng.choice([0.125, 0.25, 0.5]))
        if rng.random() < 0.6:
            n = _log_int(rng, 200, 2048)
            if rng.random() < 0.5:
                n = max(256, n // 128 * 128)
            if kind == "solve" and rng.random() < 0.15:
                mode, n = "fp32", min(n, 1024)
            c.update(model="lv", n=n, dt0_log2=14)
        else:
            c.update(model="sv", n=rng.choice([48, 64, 96, 128]), nv=rng.randint(8, 48), dt0_log2=16)
        c["mode"] = mode
        if kind == "solve":
            c["all_states"] = rng.random() < 0.25
        else:
            c.update(put=rng.random() < 0.6, barrier=rng.choice([0.0, 0.0, 0.7]))
        return c
    if kind == "batch":
        n_hi = _log_int(rng, 384, 2048)
        return dict(kind=kind, nlat=_log_int(rng, 4, 128), n_lo=256, n_hi=n_hi, n_step=rng.choice([128, 128, 100]),
                    nk=_log_int(rng, 8, 64), nmat=rng.randint(2, 8), period=0.25, mode=mode)
    if kind == "calibrate":
        return dict(kind=kind, problems=rng.randint(2, 16), n_lo=256, n_hi=_log_int(rng, 300, 1024),
                    nk=rng.randint(5, 32), nmat=rng.randint(1, 8), period=0.25, mode=mode)
    if kind == "mc":
        return dict(kind=kind, n=_log_int(rng, 128, 1024), npaths=_log_int(rng, 1000, 1 << 20),
                    nsteps=rng.randint(20, 623), mode=rng.choice(["fp32", "fp16x3"]))
    if kind == "paths":
        return dict(kind=kind, n=_log_int(rng, 128, 1024), npaths=_log_int(rng, 1000, 1 << 18),
                    nsteps=_log_int(rng, 20, 1008))
    if kind == "infer":
        return dict(kind=kind, rows=_log_int(rng, 1000, 1 << 20), members=rng.choice([2, 4]))
    if kind == "train":
        return dict(kind=kind, rows=rng.choice([512, 1000, 1024, 2048, 4096, 8192]))
    return dict(kind=kind, count=_log_int(rng, 1, 40), m=_log_int(rng, 32, 640), n=_log_int(rng, 16, 640),
                k=_log_int(rng, 32, 640))


# ------------------------------------------------------------------- inputs from the seed

def _lv_params(r):
    return dict(level=float(r.uniform(0.1, 0.4)), skew=float(r.uniform(-0.3, 0.3)), width=float(r.uniform(0.2, 1.0)),
                rate=float(r.uniform(0.0, 0.05)), floor=0.01)


def _sv_params(r):
    return dict(rate=float(r.uniform(0.0, 0.05)), kappa=float(r.uniform(1.5, 2.5)), theta=float(r.uniform(0.03, 0.06)),
                xi=float(r.uniform(0.4, 0.7)), rho=float(r.uniform(-0.8, -0.3)))


def _model(case, seed):
    r = np.random.default_rng(seed)
    p = _lv_params(r) if case["model"] == "lv" else _sv_params(r)
    lo, hi = r.uniform(0.45, 0.6), r.uniform(1.4, 1.6)
    return p, np.linspace(lo, hi, case["nk"])


def _lattice(case, p):
    if case["model"] == "lv":
        return Lattice.local_vol(n=case["n"], device=DEV, **p)
    return Lattice.stoch_vol(nx=case["n"], nv=case["nv"], device=DEV, **p)


def _sweep(case, seed):
    r = np.random.default_rng(seed)
    sizes = np.arange(case["n_lo"], case["n_hi"] + 1, case["n_step"])
    # the sizes are those of the case and not of the seed, so that every seed is the same work
    n = np.random.default_rng(1).choice(sizes, size=case["nlat"])
    n[0] = sizes[-1]
    return [dict(n=int(v), **_lv_params(r)) for v in n], np.linspace(r.uniform(0.45, 0.6), r.uniform(1.4, 1.6), case["nk"])


def _calibration(case, seed):
    r = np.random.default_rng(seed)
    n = np.random.default_rng(1).integers(case["n_lo"], case["n_hi"] + 1, size=case["problems"])
    rate = r.uniform(0.0, 0.05, case["problems"])
    at = np.stack([r.uniform(0.1, 0.4, case["problems"]), r.uniform(-0.3, 0.3, case["problems"]),
                   r.uniform(0.2, 1.0, case["problems"])], axis=1)
    pts = np.repeat(at[:, None, :], 7, axis=1)
    for j, h in enumerate((1e-3, 1e-3, 2e-3)):
        pts[:, 1 + 2 * j, j] += h
        pts[:, 2 + 2 * j, j] -= h
    return [int(v) for v in n], [float(v) for v in rate], np.linspace(0.6, 1.4, case["nk"]), pts


def _network(gen, scale=0.8):
    """Weights as a few epochs leave them: He-uniform, somewhat shrunk, with biases."""
    out = []
    for i, o in MLP_SIZES:
        a = scale * math.sqrt(6.0 / i) if o > 1 else 0.1
        out.append(((torch.rand(o * i, generator=gen, device=DEV) * 2 - 1) * a))
        out.append((torch.rand(o, generator=gen, device=DEV) * 2 - 1) * 0.1)
    return torch.cat(out)


def _features(gen, rows):
    lo = torch.tensor([0.1, -0.3, 0.2, 0.0, 0.0, 0.0, -0.7, 0.05], dtype=F64, device=DEV)
    hi = torch.tensor([0.4, 0.3, 1.0, 0.0, 0.0, 0.05, 0.4, 2.0], dtype=F64, device=DEV)
    return lo + (hi - lo) * torch.rand(rows, 8, generator=gen, device=DEV, dtype=F64)


def _scaled(feat):
    lo = torch.tensor([0.1, -0.3, 0.2, 0.0, -1.0, 0.0, -0.7, 0.05], dtype=F64, device=DEV)
    hi = torch.tensor([0.4, 0.3, 1.0, 4.0, 1.0, 0.05, 0.4, 2.0], dtype=F64, device=DEV)
    return 2.0 * (feat - lo) / (hi - lo) - 1.0


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _infer_inputs(case, seed):
    g = _gen(seed)
    theta = torch.stack([_network(g) for _ in range(case["members"])])
    return theta, _features(g, case["rows"]), 0.05 + 0.4 * torch.rand(case["rows"], generator=g, device=DEV, dtype=F64)


def _train_inputs(case, seed):
    g = _gen(seed)
    theta = _network(g)
    X = _scaled(_features(g, case["rows"])).float().contiguous()
    t = 0.5 * torch.randn(case["rows"], generator=g, device=DEV)
    mom = 1e-3 * torch.randn(theta.numel(), generator=g, device=DEV)
    var = 1e-6 + 1e-5 * torch.rand(theta.numel(), generator=g, device=DEV)
    return theta, X, t, mom, var


def _grouped_inputs(case, seed):
    """Rows that sum to 1, as kernels to be chained have; column-major as the entry takes them."""
    g = _gen(seed)
    A = torch.rand(case["count"], case["m"], case["k"], generator=g, device=DEV)
    A /= A.sum(-1, keepdim=True)
    B = torch.rand(case["count"], case["k"], case["n"], generator=g, device=DEV)
    B /= B.sum(-1, keepdim=True)
    return A, B


# ------------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k in ("solve", "bermudan"):
        p, strikes = _model(case, seed)
        lat = _lattice(case, p)
        dt0 = 2.0 ** -case["dt0_log2"]
        mode = {"fp32": 1, "bf16x3": 2, "fp16x3": 3}[case["mode"]]
        s.update(lat=lat, dt0=dt0, strikes=torch.as_tensor(strikes, dtype=F64, device=DEV),
                 plan=lat.plan(case["period"], dt0), ws=lat.workspace(case["nk"], mode))
    elif k == "batch":
        params, strikes = _sweep(case, seed)
        lats = [Lattice.local_vol(device=DEV, **p) for p in params]
        s["batch"] = Batch(lats, strikes, case["nmat"], case["period"], 2.0 ** -14, mode=case["mode"])
    elif k == "calibrate":
        n, rate, strikes, pts = _calibration(case, seed)
        s["pricer"] = LVBatchPricer(n, rate, strikes, case["nmat"], case["period"], mode=case["mode"], device=DEV)
        s["pts"] = pts
    elif k in ("mc", "paths"):
        p = _lv_params(np.random.default_rng(seed))
        lat = Lattice.local_vol(n=case["n"], device=DEV, **p)
        s.update(lat=lat, plan=lat.plan(1 / 252, 2.0 ** -14), seed=int(seed) & 0x7fffffff,
                 disc=math.exp(-p["rate"] * case["nsteps"] / 252))
        if k == "paths":
            s["rows"] = cumulative_rows(lat.kernel(1 / 252, 2.0 ** -14, plan=s["plan"]))
            s["guide"] = guide_table(s["rows"])
    elif k == "infer":
        theta, feat, base = _infer_inputs(case, seed)
        net = Surrogate(members=case["members"], device=DEV)
        net.theta.copy_(theta)
        bind_stream(net.device)
        for m in range(case["members"]):
            _lib.call("opb_mlp_pack", net.theta[m].data_ptr(), net.packed[m * net.stride:].data_ptr())
        n = int(net.lib.opb_mlp_infer_workspace_bytes(case["rows"], case["members"]))
        s.update(net=net, feat=feat, base=base, ws=torch.empty(n, dtype=torch.uint8, device=DEV))
    elif k == "train":
        theta, X, t, mom, var = _train_inputs(case, seed)
        lib = _lib.load()
        s.update(theta=theta, thb=torch.empty_like(theta), X=X, t=t, mom=mom, var=var, grad=torch.empty_like(theta),
                 loss=torch.zeros(1, dtype=F64, device=DEV), step=torch.full((1,), 500, dtype=torch.int32, device=DEV),
                 lr=torch.full((1 << 20,), 3e-4, device=DEV),
                 ws=torch.empty(int(lib.opb_mlp_workspace_floats(case["rows"])), device=DEV))
        bind_stream(theta.device)
        _lib.call("opb_mlp_round", theta.data_ptr(), s["thb"].data_ptr(), None)
    else:
        A, B = _grouped_inputs(case, seed)
        Ac, Bc = A.transpose(1, 2).contiguous(), B.transpose(1, 2).contiguous()
        C = torch.empty(case["count"], case["n"], case["m"], device=DEV)
        m, n, kk = case["m"], case["n"], case["k"]
        bx, by = -(-m // 64), -(-n // 16)
        words = _lib.load().opb_sgemm4_task_size() // 8
        rec = np.zeros((case["count"], bx, by, words), dtype=np.int64)
        ints = rec.view(np.int32).reshape(case["count"], bx, by, 2 * words)
        ints[..., 0] = np.arange(case["count"])[:, None, None]
        ints[..., 1] = np.arange(bx)[None, :, None]
        ints[..., 2] = np.arange(by)[None, None, :]
        ints[..., 3], ints[..., 4], ints[..., 5] = m, n, kk
        for i in range(case["count"]):
            rec[i, ..., 3:6] = (Ac[i].data_ptr(), Bc[i].data_ptr(), C[i].data_ptr())
        nb = case["count"] * bx * by
        drec = torch.from_numpy(rec.reshape(-1)).to(DEV)
        s.update(A=Ac, B=Bc, C=C, rec=drec, nb=nb, ptrs=torch.arange(nb, dtype=torch.int64, device=DEV) * (8 * words)
                 + drec.data_ptr())
    return s


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "solve":
        quotes, V = s["lat"].solve(s["strikes"], c["nmat"], c["period"], s["dt0"], mode=c["mode"], plan=s["plan"],
                                   all_states=c["all_states"], workspace=s["ws"])
        return {"quotes": quotes, "states": V} if c["all_states"] else {"quotes": quotes}
    if k == "bermudan":
        return s["lat"].bermudan(s["strikes"], c["nmat"], c["period"], s["dt0"], mode=c["mode"], put=c["put"],
                                 barrier=c["barrier"], plan=s["plan"], workspace=s["ws"])
    if k == "batch":
        return s["batch"].execute()
    if k == "calibrate":
        return s["pricer"](s["pts"])
    if k == "mc":
        rows = cumulative_rows(s["lat"].kernel(1 / 252, 2.0 ** -14, mode=c["mode"], plan=s["plan"]))
        sums, _ = mc_run(rows, s["lat"].y0, c["nsteps"], s["seed"], c["npaths"], guide=guide_table(rows),
                         x=s["lat"].x, disc=s["disc"])
        return {"rows": rows, "sums": sums}
    if k == "paths":
        sums, states = mc_run(s["rows"], s["lat"].y0, c["nsteps"], s["seed"], c["npaths"], guide=s["guide"],
                              x=s["lat"].x, disc=s["disc"], want_paths=True)
        return {"sums": sums, "states": states}
    if k == "infer":
        iv, spread = s["net"].predict(s["feat"], s["base"], ws=s["ws"])
        return {"iv": iv, "spread": spread}
    if k == "train":
        bind_stream(s["theta"].device)
        _lib.call("opb_mlp_loss_grad", s["thb"].data_ptr(), s["X"].data_ptr(), s["t"].data_ptr(), c["rows"],
                  s["ws"].data_ptr(), s["grad"].data_ptr(), s["loss"].data_ptr())
        _lib.call("opb_mlp_adam_sched", s["theta"].data_ptr(), s["mom"].data_ptr(), s["var"].data_ptr(),
                  s["grad"].data_ptr(), s["step"].data_ptr(), s["lr"].data_ptr(), 0.9, 0.999, 1e-8,
                  s["thb"].data_ptr())
        return {"grad": s["grad"], "loss": s["loss"], "theta": s["theta"], "mom": s["mom"], "var": s["var"]}
    bind_stream(s["C"].device)
    _lib.call("opcuda_sgemm4", s["nb"], s["ptrs"].data_ptr())
    return s["C"]


# ----------------------------------------------------------------------------------- work

def _squarings_flops(n, half, niter):
    """Useful flops of niter squarings of an n x n matrix of half-bandwidth ``half``, the band
    doubling each time: outputs within the doubled band, each a sum over the overlap."""
    total = 0.0
    for _ in range(niter):
        total += 2.0 * n * min(n, 4 * half + 1) * min(n, 2 * half + 1) / (1.0 if 2 * half >= n else 2.0)
        half = min(2 * half, n)
    return total


def work(case):
    k = case["kind"]
    if k in ("solve", "bermudan"):
        d = case["n"] * case.get("nv", 1)
        w, half, niter = (3, 1, 13) if case["model"] == "lv" else (7, case["n"] + 1, 14)
        out = 8.0 * case["nk"] * (case["nmat"] if k == "solve" else 1)
        if case.get("all_states"):
            out += 8.0 * case["nk"] * case["nmat"] * d
        return dict(bytes=12.0 * w * d + 8.0 * d + 8.0 * case["nk"] + out,
                    flops=_squarings_flops(d, half, niter) + 2.0 * d * d * case["nk"] * case["nmat"])
    if k in ("batch", "calibrate"):
        if k == "batch":
            n = [p["n"] for p in _sweep(case, 0)[0]]
        else:
            n = [v for v in _calibration(case, 0)[0] for _ in range(7)]
        return dict(bytes=44.0 * sum(n) + 8.0 * len(n) * case["nk"] * case["nmat"],
                    flops=sum(_squarings_flops(v, 1, 14) + 2.0 * v * v * case["nk"] * case["nmat"] for v in n))
    if k in ("mc", "paths"):
        # a path-step: the generator's output, the uniform and its search, the payoff's running values
        steps = float(case["npaths"]) * case["nsteps"]
        n = case["n"]
        if k == "mc":
            return dict(bytes=44.0 * n + 4.0 * n * n + 16, flops=40.0 * steps + 2.0 * n ** 3)
        return dict(bytes=8.0 * n * n + 2.0 * steps + 16, flops=40.0 * steps)
    macs = sum(i * o for i, o in MLP_SIZES)
    params = sum(i * o + o for i, o in MLP_SIZES)
    if k == "infer":
        return dict(bytes=88.0 * case["rows"] + 2.0 * params * case["members"],
                    flops=2.0 * macs * case["rows"] * case["members"])
    if k == "train":
        return dict(bytes=36.0 * case["rows"] + 36.0 * params, flops=6.0 * macs * case["rows"])
    m, n, kk = case["m"], case["n"], case["k"]
    return dict(bytes=4.0 * case["count"] * (m * kk + kk * n + m * n), flops=2.0 * case["count"] * m * n * kk)


# ---------------------------------------------------------------- the results in 64 bits

def _lv_dense(n, level, skew, width, rate, floor):
    """The birth-death generator that matches drift r x and variance (sigma x)^2 on log-spaced
    nodes, the end nodes absorbing."""
    i = torch.arange(n, dtype=F64, device=DEV)
    x = X_LO * (X_HI / X_LO) ** (i / (n - 1))
    sig = torch.clamp(level + skew * torch.exp(-((x - 1.0) / width) ** 2), min=floor)
    mu, var = rate * x[1:-1], (sig[1:-1] * x[1:-1]) ** 2
    dn, up = x[1:-1] - x[:-2], x[2:] - x[1:-1]
    down, rise = (var - up * mu) / (dn * (dn + up)), (var + dn * mu) / (up * (dn + up))
    L = torch.zeros(n, n, dtype=F64, device=DEV)
    j = torch.arange(1, n - 1, device=DEV)
    L[j, j - 1], L[j, j + 1], L[j, j] = down, rise, -(down + rise)
    return L, x


def _sv_dense(nx, nv, rate, kappa, theta, xi, rho):
    """The (spot, variance) generator: the covariance on two diagonal moves at a capped common
    rate, the remaining moments on the axes, negative rates cut off and the spot's drift
    mended; absorbing at the spot's ends, drift alone at the variance's."""
    ix, iv = np.arange(nx), np.arange(nv)
    xs = X_LO * (X_HI / X_LO) ** (ix / (nx - 1))
    V = (0.05 * (1.0 / 0.05) ** (iv / (nv - 1))) ** 2
    x, v = xs[None, 1:-1], V[:, None]
    dm, dp = xs[None, :-2] - x, xs[None, 2:] - x
    vm = np.concatenate([[0.0], V[:-1] - V[1:]])[:, None]   # step down in variance
    vp = np.concatenate([V[1:] - V[:-1], [0.0]])[:, None]
    inner = ((iv > 0) & (iv < nv - 1))[:, None]
    var_x, var_v, mu_x, mu_v = v * x * x, xi * xi * v, rate * x + 0 * v, kappa * (theta - v) + 0 * x
    a, b = (vm, vp) if rho < 0 else (vp, vm)                # the variance move that goes with spot up, down
    with np.errstate(all="ignore"):
        q = np.minimum(rho * xi * v * x / (dp * a + dm * b), var_x / (dp ** 2 + dm ** 2))
        q = np.minimum(q, var_v / (a ** 2 + b ** 2))
        q = np.where(inner & (rho != 0.0), np.maximum(q, 0.0), 0.0)
    ax, bx = mu_x - q * (dp + dm), var_x - q * (dp ** 2 + dm ** 2)
    av, bv = mu_v - q * (a + b), var_v - q * (a ** 2 + b ** 2)

    def axial(m1, m2, lo, hi):
        return (hi * m1 - m2) / (lo * (hi - lo)), (m2 - lo * m1) / (hi * (hi - lo))

    xm, xp = axial(ax, bx, dm, dp)
    with np.errstate(all="ignore"):
        um, up = axial(av, bv, vm, vp)
        up = np.where(inner, up, np.where(iv[:, None] == 0, np.maximum(mu_v, 0.0) / vp, 0.0))
        um = np.where(inner, um, np.where(iv[:, None] == nv - 1, np.minimum(mu_v, 0.0) / vm, 0.0))
    xm, xp, um, up = (np.maximum(r, 0.0) for r in (xm, xp, um, up))
    drift = q * (dp + dm) + xm * dm + xp * dp
    xm = xm + np.where(drift > mu_x, (drift - mu_x) / -dm, 0.0)
    xp = xp + np.where(drift > mu_x, 0.0, (mu_x - drift) / dp)
    d = nx * nv
    L = torch.zeros(d, d, dtype=F64, device=DEV)
    y = (ix[None, 1:-1] + nx * iv[:, None])
    s = -1 if rho < 0 else 1
    for rate_, to in ((xm, -1), (xp, 1), (um, -nx), (up, nx), (q, 1 + s * nx), (q, -1 - s * nx)):
        on = rate_ != 0
        src = torch.from_numpy(y[on]).to(DEV)
        val = torch.from_numpy(rate_[on]).to(DEV)
        L.index_put_((src, src + to), val, accumulate=True)
        L.index_put_((src, src), -val, accumulate=True)
    return L, torch.from_numpy(np.tile(xs, nv)).to(DEV)


def _spot_state(case):
    """The quoted state: the spot node nearest 1, at the volatility nearest sqrt(theta)."""
    xs = X_LO * (X_HI / X_LO) ** (np.arange(case["n"]) / (case["n"] - 1))
    return int(np.argmin(np.abs(xs - 1.0)))


def _period_kernel(L, period, dt0, dt_max=None):
    dt = 0.5 / (float(L.diagonal().abs().max()) if dt_max is None else dt_max)
    niter = math.ceil(math.log(period / min(dt, dt0)) / math.log(2.0))
    P = torch.eye(L.shape[0], dtype=F64, device=DEV) + period * 2.0 ** -niter * L
    for _ in range(niter):
        P = P @ P
        P /= P.sum(1, keepdim=True)
    return P


def _european(P, x, strikes, rate, period, nmat):
    """Discounted call values [nmat, states, strikes]."""
    V = torch.clamp(x[:, None] - torch.as_tensor(strikes, dtype=F64, device=DEV)[None, :], min=0.0)
    out = []
    for m in range(1, nmat + 1):
        V = P @ V
        out.append(V * math.exp(-rate * m * period))
    return torch.stack(out)


def _forward(theta, X):
    off, h = 0, X
    for i, o in MLP_SIZES:
        W, b = theta[off:off + i * o].view(o, i), theta[off + i * o:off + i * o + o]
        off += i * o + o
        h = h @ W.T + b
        if o > 1:
            h = 0.5 * h * (1.0 + torch.erf(h / math.sqrt(2.0)))
    return h[:, 0]


def exact(case, seed):
    k = case["kind"]
    if k in ("solve", "bermudan"):
        p, strikes = _model(case, seed)
        if case["model"] == "lv":
            L, x = _lv_dense(case["n"], **p)
            y0 = _spot_state(case)
        else:
            L, x = _sv_dense(case["n"], case["nv"], **p)
            vols = 0.05 * 20.0 ** (np.arange(case["nv"]) / (case["nv"] - 1))
            y0 = _spot_state(case) + case["n"] * int(np.argmin(np.abs(vols - math.sqrt(p["theta"]))))
        P = _period_kernel(L, case["period"], 2.0 ** -case["dt0_log2"])
        if k == "solve":
            V = _european(P, x, strikes, p["rate"], case["period"], case["nmat"])
            return {"quotes": V[:, y0], "states": V} if case["all_states"] else {"quotes": V[:, y0]}
        K = torch.as_tensor(strikes, dtype=F64, device=DEV)[None, :]
        ex = torch.clamp(K - x[:, None] if case["put"] else x[:, None] - K, min=0.0)
        out = (x <= case["barrier"])[:, None] if case["barrier"] > 0 else torch.zeros_like(x, dtype=torch.bool)[:, None]
        V = torch.where(out, 0.0, ex)
        for m in range(case["nmat"] - 1, -1, -1):
            V = math.exp(-p["rate"] * case["period"]) * (P @ V)
            if m >= 1:
                V = torch.where(out, 0.0, torch.maximum(V, ex))
        return V[y0]
    if k == "batch":
        params, strikes = _sweep(case, seed)
        got = []
        for p in params:
            L, x = _lv_dense(**p)
            V = _european(_period_kernel(L, case["period"], 2.0 ** -14), x, strikes, p["rate"], case["period"],
                          case["nmat"])
            got.append(V[:, _spot_state(p)])
        return torch.stack(got)
    if k == "calibrate":
        n, rate, strikes, pts = _calibration(case, seed)
        vmax = float(BOX_HI[0] + BOX_HI[1])
        got = []
        for i, v in enumerate(n):
            top, _ = _lv_dense(v, vmax, 0.0, 1.0, rate[i], 0.01)
            dmax = float(top.diagonal().abs().max())
            for q in pts[i]:
                L, x = _lv_dense(v, float(q[0]), float(q[1]), float(q[2]), rate[i], 0.01)
                V = _european(_period_kernel(L, case["period"], 2.0 ** -14, dmax), x, strikes, rate[i],
                              case["period"], case["nmat"])
                got.append(V[:, _spot_state(dict(n=v))].reshape(-1))
        return torch.stack(got).view(len(n), 7, -1)
    if k == "mc":
        p = _lv_params(np.random.default_rng(seed))
        L, _ = _lv_dense(case["n"], **p)
        P = _period_kernel(L, 1 / 252, 2.0 ** -14)
        return {"rows": torch.cumsum(P, 1), "sums": None}
    if k == "paths":
        return None
    if k == "infer":
        theta, feat, base = _infer_inputs(case, seed)
        X = _scaled(feat)
        ys = torch.stack([torch.cat([_forward(th.double(), x) for x in X.split(1 << 17)]) for th in theta])
        return {"iv": base + 0.05 * ys.mean(0), "spread": 0.05 * (ys.max(0).values - ys.min(0).values)}
    if k == "train":
        theta, X, t, mom, var = (v.double() for v in _train_inputs(case, seed))
        th = theta.float().bfloat16().double().requires_grad_()
        loss = ((_forward(th, X) - t) ** 2).sum()
        g, = torch.autograd.grad(loss / case["rows"], th)
        mom, var = 0.9 * mom + 0.1 * g, 0.999 * var + 0.001 * g * g
        step = 501
        theta = theta - 3e-4 * (mom / (1 - 0.9 ** step)) / (torch.sqrt(var / (1 - 0.999 ** step)) + 1e-8)
        return {"grad": g, "loss": loss.detach().view(1), "theta": theta, "mom": mom, "var": var}
    A, B = _grouped_inputs(case, seed)
    return (A.double() @ B.double()).transpose(1, 2).contiguous()
