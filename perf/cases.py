"""What a user of cppe_gb300 has it do, as timed cases.

The inputs are the package's seeded water boxes (density 1.0 g/cm^3, the benchmark's multipoles,
polarizabilities and exclusions) and right-hand sides made of the field of 12 point charges plus a static
field of each site's own, drawn with the standard deviation that the boxes' static multipole fields have
(0.015 a.u.).  Every case goes through the package's public entry points: cppe_gb300.capi's System, Batch, Mlp
and multipole_fields (the C ABI).  `kind` says which:

  solve    induced dipoles of one system: the first-call solve of an SCF, to ||F - B mu||_2 < 1e-8
  apply    the operator B on one vector (BMatrix::apply, what a caller's own iteration uses)
  fields   the static multipole fields (charges, dipoles and quadrupoles) at all sites
  batch    snapshots x right-hand sides solved together
  train    loss and gradients of the learned guess' network on one batch of rows

Sizes follow the benchmark's configurations (999 sites direct; 30,000 sites at order 5; 300,000 and 1,000,002
sites at order 6; snapshots of 500 to 20,000 sites with 8 right-hand sides, direct below 4,000) and the test
systems (18 and 8,805 sites).
"""
import math
import os

import numpy as np
import torch

from cppe_gb300 import capi, learned, synthetic

DAMPING = 2.1304
STATIC_FIELD = 0.015
MODEL = os.path.join(os.path.dirname(os.path.abspath(synthetic.__file__)), "data", "learned_water.npz")


def listed():
    return [
        # the smallest system of the tests (six waters), undamped, with the default options: launches and latency
        dict(name="solve_18", kind="solve", waters=6, summation="direct", precision="fp64", damp=False, order=5,
             learned=False, host=True),
        # the CPU-runnable configuration: 333 waters by direct summation in the default precision
        dict(name="solve_999", kind="solve", waters=333, summation="direct", precision="fp64", damp=True, order=5,
             learned=False, host=True),
        # static fields of the 8,805-site protein-sized test system, direct summation, undamped (the defaults)
        dict(name="fields_8805", kind="fields", waters=2935, summation="direct", damp=False, order=5),
        # static fields by FMM at the middle size
        dict(name="fields_fmm_30k", kind="fields", waters=9999, summation="fmm", damp=False, order=5),
        # one application of the operator in the default precision, ragged size, order 6, host vectors
        dict(name="apply_100k", kind="apply", waters=33334, summation="fmm", arith="fp64", damp=True, order=6),
        # the default-precision solver at the middle size
        dict(name="solve_30k", kind="solve", waters=10000, summation="fmm", precision="fp64", damp=True, order=5,
             learned=False, host=False),
        # the same with mixed precision and the shipped model
        dict(name="solve_mixed_30k", kind="solve", waters=10000, summation="fmm", precision="mixed", damp=True,
             order=5, learned=True, host=False),
        # the precision configuration: 300,000 sites, no model
        dict(name="solve_mixed_300k", kind="solve", waters=100000, summation="fmm", precision="mixed", damp=True,
             order=6, learned=False, host=False),
        # the headline: 1,000,002 sites with the shipped model
        dict(name="solve_mixed_1m", kind="solve", waters=333334, summation="fmm", precision="mixed", damp=True,
             order=6, learned=True, host=False),
        # snapshots of a trajectory with 8 right-hand sides each
        dict(name="batch_mixed_32x8", kind="batch", snapshots=32, lo=500, hi=20000, nrhs=8, precision="mixed",
             damp=True, order=5, host=False),
        # the three unit-field solves of an electric-field response (induced_moments_eef): one system, 3 fields
        dict(name="batch_eef_2997", kind="batch", snapshots=1, lo=2997, hi=2997, nrhs=3, precision="fp64",
             damp=True, order=5, host=True),
        # a training step's forward and backward pass
        dict(name="train_16k", kind="train", rows=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "fmm64", "mixed", "mixed", "apply", "fields", "fields_fmm", "batch", "train"])
    if kind == "direct":
        return dict(kind="solve", waters=_log(rng, 6, 1300), summation="direct", precision="fp64",
                    damp=rng.random() < 0.7, order=5, learned=False, host=True)
    if kind == "fmm64":
        return dict(kind="solve", waters=_log(rng, 1334, 15000), summation="fmm", precision="fp64", damp=True,
                    order=rng.choice([5, 6]), learned=False, host=False)
    if kind == "mixed":
        return dict(kind="solve", waters=_log(rng, 1334, 150000), summation="fmm", precision="mixed", damp=True,
                    order=rng.choice([5, 6]), learned=rng.random() < 0.5, host=False)
    if kind == "apply":
        return dict(kind="apply", waters=_log(rng, 400, 50000), summation="fmm",
                    arith=rng.choice(["fp64", "fp64", "fp32", "dd"]), damp=rng.random() < 0.7,
                    order=rng.choice([5, 6]))
    if kind == "fields":
        return dict(kind="fields", waters=_log(rng, 6, 3500), summation="direct", damp=rng.random() < 0.3, order=5)
    if kind == "fields_fmm":
        return dict(kind="fields", waters=_log(rng, 1334, 20000), summation="fmm", damp=rng.random() < 0.3,
                    order=rng.choice([5, 6]))
    if kind == "batch":
        return dict(kind="batch", snapshots=_log(rng, 1, 24), lo=500, hi=_log(rng, 2000, 20000),
                    nrhs=rng.randint(1, 9), precision=rng.choice(["mixed", "mixed", "fp64"]), damp=True, order=5,
                    host=rng.random() < 0.3)
    return dict(kind="train", rows=_log(rng, 700, 30000))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _rhs(box, seed, count=1):
    """`count` right-hand sides: point-charge fields plus a static field."""
    rng = np.random.default_rng([seed, 17])
    fields = learned.generator_rhs(box, count, seed)
    static = STATIC_FIELD * rng.standard_normal(3 * box.n)
    return [f + static for f in fields]


def _snapshots(case, seed):
    # the sizes belong to the case, the boxes to the seed
    sizes = [int(n) // 3 for n in synthetic.snapshot_sizes(case["snapshots"], seed=1000, lo=case["lo"], hi=case["hi"])]
    boxes = [synthetic.water_box(w, seed=1000 * (seed % 10 ** 6) + k) for k, w in enumerate(sizes)]
    return boxes, [_rhs(b, seed + k, case["nrhs"]) for k, b in enumerate(boxes)]


def _train_inputs(case, seed):
    """Descriptor rows with the shipped model's means and spreads, and target rows of their usual sizes."""
    d = np.load(MODEL)
    rng = np.random.default_rng([seed, 29])
    n = case["rows"]
    std = np.where(d["inv_std"] > 0, 1.0 / np.maximum(d["inv_std"], 1e-12), 0.0)
    feats = (d["mean"] + std * rng.standard_normal((n, capi.N_IN))).astype(np.float32)
    rows = np.zeros((n, capi.TROW), np.float32)
    rows[:, 0:3] = 0.1 * rng.standard_normal((n, 3))
    rows[:, 3:6] = 0.4 * rows[:, 0:3] + 0.02 * rng.standard_normal((n, 3))
    rows[:, 6:9] = 0.4 * rows[:, 3:6] + 0.01 * rng.standard_normal((n, 3))
    rows[:, 9:12] = rows[:, 0:3] + rows[:, 3:6] + 0.6 * rows[:, 6:9] + 0.005 * rng.standard_normal((n, 3))
    rows[:, 12:15] = 0.02 * rng.standard_normal((n, 3))
    rows[:, 15:18] = 0.3 * rows[:, 12:15] + 0.005 * rng.standard_normal((n, 3))
    rows[:, 18:21] = rows[:, 12:15] + 0.7 * rows[:, 15:18] + 0.003 * rng.standard_normal((n, 3))
    for col, v in ((21, rows[:, 0:3]), (22, rows[:, 12:15])):
        s = (v * v).sum(axis=1)
        rows[:, col] = s + 0.01 * s.mean()
    return feats, rows


def _options(case):
    return dict(damp=case["damp"], damping=DAMPING, order=case["order"], ncrit=64, theta=0.5, thresh=1e-8,
                precision=capi.MIXED if case.get("precision") == "mixed" else capi.FP64)


def _device(vectors):
    d = torch.from_numpy(np.ascontiguousarray(np.concatenate(vectors))).cuda()
    return d, torch.empty_like(d)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        feats, rows = _train_inputs(case, seed)
        return dict(case=case, model=learned.load(MODEL), feats=feats, rows=rows)
    if kind == "batch":
        boxes, rhs = _snapshots(case, seed)
        flat = [f for fs in rhs for f in fs]
        s = dict(case=case, batch=capi.Batch(boxes, case["nrhs"], direct_below=4000, **_options(case)))
        if case["host"]:
            s["rhs"] = np.concatenate(flat)
        else:
            s["rhs"], s["mu"] = _device(flat)
        return s
    box = synthetic.water_box(case["waters"], seed=seed)
    if kind == "fields":
        return dict(case=case, box=box, polarizable=np.ones(box.n, np.int32))
    system = capi.System(box.xyz, box.alpha6, box.excl_ptr, box.excl_idx,
                         summation=capi.FMM if case["summation"] == "fmm" else capi.DIRECT, **_options(case))
    s = dict(case=case, system=system)
    if kind == "apply":
        s["v"] = 0.1 * np.random.default_rng([seed, 5]).standard_normal(3 * box.n)
        return s
    if case["learned"]:
        s["model"] = learned.load(MODEL)
        system.set_model(s["model"])
    rhs = _rhs(box, seed)
    if case["host"]:
        s["rhs"] = rhs[0]
    else:
        s["rhs"], s["mu"] = _device(rhs)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        loss, grads = state["model"].loss_grad(state["feats"], state["rows"])
        return [loss, grads]
    if kind == "batch":
        b = state["batch"]
        if case["host"]:
            return [b.solve(state["rhs"])[0]]
        b.solve_device(state["rhs"].data_ptr(), state["mu"].data_ptr())
        return [state["mu"]]
    if kind == "fields":
        b = state["box"]
        return [capi.multipole_fields(b.xyz, b.q, b.mu, b.quad, 2, state["polarizable"], b.alpha_iso, b.excl_ptr,
                                      b.excl_idx, fmm=case["summation"] == "fmm", ncrit=64, order=case["order"],
                                      theta=0.5, damp=case["damp"], damping=DAMPING)]
    s = state["system"]
    if kind == "apply":
        return [s.apply(state["v"], fp32=case["arith"] == "fp32", dd=case["arith"] == "dd")]
    if case["host"]:
        return [s.solve(state["rhs"])[0]]
    s.solve_device(state["rhs"].data_ptr(), state["mu"].data_ptr())
    return [state["mu"]]


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _operator(n, fmm, order):
    """Floating-point operations of one application: a damped dipole pair takes 45, an order-p translation
    2 * ((p + 1)(p + 2)(p + 3) / 6)^2 / 5 or so; at theta 0.5 and ncrit 64 a site has some 3,000 near sites and
    its leaf's share of about 10 translations."""
    if not fmm:
        return 45.0 * n * n
    terms = (order + 1) * (order + 2) * (order + 3) / 6
    return n * (45.0 * min(n, 3000) + 10 * 0.4 * terms * terms)


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["rows"]
        mac = n * (64 * 128 + 128 * 128 + 128 * 4)
        return dict(bytes=4.0 * n * (64 + 24) + 2 * 4.0 * 25220, flops=2.0 * mac * 3)
    if kind == "batch":
        sizes = synthetic.snapshot_sizes(case["snapshots"], seed=1000, lo=case["lo"], hi=case["hi"])
        flops = sum(14 * case["nrhs"] * _operator(int(n), n >= 4000, case["order"]) for n in sizes)
        return dict(bytes=float(sum(int(n) for n in sizes)) * (80 + 48 * case["nrhs"]), flops=float(flops))
    n = 3 * case["waters"]
    fmm = case["summation"] == "fmm"
    per_site = 24 + 48 + 12 + 24 + 24  # position, polarizability, exclusions, vector in, vector out
    if kind == "fields":
        # charges, dipoles and quadrupoles: 14, 45 and 70 operations a pair
        return dict(bytes=n * (per_site + 80.0), flops=_operator(n, fmm, case["order"]) * 129 / 45)
    applies = 1 if kind == "apply" else 14
    return dict(bytes=float(n * per_site), flops=float(applies * _operator(n, fmm, case["order"])))


# ---------------------------------------------------------------------------
# The values in 64 bits, by direct summation in torch
# ---------------------------------------------------------------------------
def _cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), device="cuda" if torch.cuda.is_available() else "cpu").to(dtype)


def _pairs(box, i0, i1, damp, excl):
    """Separations (target - source) of the targets i0..i1 to all sites, 1/R (0 where a pair is left out) and
    the Thole factors of the field and its gradients."""
    xyz = box["xyz"]
    d = xyz[i0:i1, None, :] - xyz[None, :, :]
    r2 = (d * d).sum(-1)
    rows = torch.arange(i0, i1, device=xyz.device)
    r2[rows - i0, rows] = math.inf
    e0, e1 = int(box["ptr"][i0]), int(box["ptr"][i1])
    if excl and e1 > e0:
        t = torch.repeat_interleave(rows, (box["ptr"][i0 + 1:i1 + 1] - box["ptr"][i0:i1]).to(rows.device))
        r2[t - i0, box["idx"][e0:e1].to(rows.device)] = math.inf
    ir = r2.rsqrt()
    fE = fT = fD = None
    if damp:
        v = DAMPING * box["s"][i0:i1, None] * box["s"][None, :] * torch.where(ir > 0, r2 * ir, torch.full_like(ir, 100.0))
        v = torch.nan_to_num(v, nan=100.0, posinf=100.0)
        e = torch.exp(-v)
        fE = 1 - (1 + v + 0.5 * v * v) * e
        fT = fE - v ** 3 / 6 * e
        fD = fT - v ** 4 / 30 * e
    return d, ir, fE, fT, fD


def _box64(box):
    ptr = torch.as_tensor(np.asarray(box.excl_ptr, np.int64))
    return dict(xyz=_cuda(box.xyz), s=_cuda(box.alpha_iso ** (-1.0 / 6.0)), ptr=ptr,
                idx=torch.as_tensor(np.asarray(box.excl_idx, np.int64)))


def _apply64(box, damp, v):
    """(alpha^-1 - T) v."""
    b, n = _box64(box), box.n
    v = _cuda(v).reshape(n, 3)
    out = torch.empty_like(v)
    step = max(1, 40_000_000 // n)
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        d, ir, fE, fT, _ = _pairs(b, i0, i1, damp, True)
        A, B = ir ** 3, 3 * ir ** 5
        if damp:
            A, B = A * fE, B * fT
        dot = (d * v[None]).sum(-1) * B
        out[i0:i1] = A @ v - (dot[:, :, None] * d).sum(1)
    a = _cuda(box.alpha6)[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    return out + torch.linalg.solve(a, v[:, :, None])[:, :, 0]


def _dense64(box, damp):
    b, n = _box64(box), box.n
    B = torch.zeros(n, 3, n, 3, dtype=torch.float64, device=b["xyz"].device)
    eye = torch.eye(3, dtype=torch.float64, device=B.device)
    for i0 in range(0, n, 500):
        i1 = min(n, i0 + 500)
        d, ir, fE, fT, _ = _pairs(b, i0, i1, damp, True)
        A, C = ir ** 3, 3 * ir ** 5
        if damp:
            A, C = A * fE, C * fT
        t = A[:, :, None, None] * eye - C[:, :, None, None] * d[..., :, None] * d[..., None, :]
        B[i0:i1] = t.permute(0, 2, 1, 3)
    a = _cuda(box.alpha6)[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    at = torch.arange(n, device=B.device)
    B[at, :, at, :] = torch.linalg.inv(a)
    return B.reshape(3 * n, 3 * n)


def _fields64(box, damp):
    """-grad of q/R + mu.r/R^3 + 1/2 Theta:(3 r r/R^5 - 1/R^3), summed over the sources."""
    b, n = _box64(box), box.n
    q, mu = _cuda(box.q), _cuda(box.mu)
    th = _cuda(box.quad)[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    tr = th.diagonal(dim1=1, dim2=2).sum(-1)
    out = torch.empty(n, 3, dtype=torch.float64, device=b["xyz"].device)
    step = max(1, 30_000_000 // n)
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        d, ir, fE, fT, fD = _pairs(b, i0, i1, damp, True)
        g3, g5, g7 = ir ** 3, 3 * ir ** 5, 15 * ir ** 7
        if damp:
            g3, g5, g7 = g3 * fE, g5 * fT, g7 * fD
        td = torch.einsum("jab,ijb->ija", th, d)
        dtd = (d * td).sum(-1)
        along = q[None] * g3 + (d * mu[None]).sum(-1) * g5 + 0.5 * dtd * g7 - 0.5 * tr[None] * g5
        out[i0:i1] = (along[:, :, None] * d).sum(1) - g3 @ mu - (g5[:, :, None] * td).sum(1)
    return out


def _train64(case, seed):
    feats, rows = (_cuda(x) for x in _train_inputs(case, seed))
    m = np.load(MODEL)
    sizes = [(128, 64), (128,), (128, 128), (128,), (4, 128), (4,)]
    at, W = 0, []
    for shape in sizes:
        k = int(np.prod(shape))
        W.append(_cuda(m["params"][at:at + k]).reshape(shape).requires_grad_(True))
        at += k
    x = (feats - _cuda(m["mean"])) * _cuda(m["inv_std"])
    h = torch.nn.functional.gelu(x @ W[0].T + W[1])
    h = torch.nn.functional.gelu(h @ W[2].T + W[3])
    y = h @ W[4].T + W[5]
    v1, v2, v3, mu, a, w, e = (rows[:, 3 * k:3 * k + 3] for k in range(7))
    dg = y[:, 0:1] * v1 + y[:, 1:2] * v2 + y[:, 2:3] * v3 - mu
    dp = a + y[:, 3:4] * w - e
    loss = ((dg * dg).sum(1) / rows[:, 21] + (dp * dp).sum(1) / rows[:, 22]).mean()
    loss.backward()
    return [float(loss.detach()), torch.cat([p.grad.reshape(-1) for p in W])]


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, seed)
    if kind == "batch":
        sizes = synthetic.snapshot_sizes(case["snapshots"], seed=1000, lo=case["lo"], hi=case["hi"])
        if sizes.max() >= 4000 or sum(int(n) ** 3 for n in sizes) > 3e10:
            return None
        boxes, rhs = _snapshots(case, seed)
        return [torch.cat([torch.linalg.solve(_dense64(b, case["damp"]), _cuda(np.stack(fs, axis=1))).T.reshape(-1)
                           for b, fs in zip(boxes, rhs)])]
    box = synthetic.water_box(case["waters"], seed=seed)
    if kind == "fields":
        return [_fields64(box, case["damp"]).reshape(-1)]
    if kind == "apply":
        v = 0.1 * np.random.default_rng([seed, 5]).standard_normal(3 * box.n)
        return [_apply64(box, case["damp"], v).reshape(-1)]
    if case["summation"] == "direct":
        return [torch.linalg.solve(_dense64(box, case["damp"]), _cuda(_rhs(box, seed)[0])[:, None])[:, 0]]
    return None
