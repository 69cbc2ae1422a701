"""Workloads the library's speed is measured on.

Three groups, all through the calls of `openmxp_b200`:

* `solve`: what a program does with one system -- generate it, factor it and
  refine the solution -- from an order where launches and latency count
  (n = 1024) to one that fills the GPU (n = 61440), in the three precision
  forms and with both refinement methods;
* `batch`: many systems of uneven orders generated and solved in one call,
  a large batch and one of a few small systems;
* the single steps a program (a grid driver, another refinement loop) calls by
  themselves, at ragged sizes: the diagonal block with its inverses, the FP32
  panel solves, the casts with the trailing update, the triangular solves of a
  factor the library did not make, and the regenerating matrix product.

`listed()` is the fixed list, `draw()` gives more cases of the same ranges.
"""
from __future__ import annotations

import math

import torch

import openmxp_b200 as mxp

_DEV = "cuda"
_MASK = (1 << 64) - 1
_LCG_A, _LCG_C = 6364136223846793005, 1
_LCG_SCALE = float.fromhex("0x1.fffffffffffffp-65")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest solve the tests and the smoke check run: launches and latency
        {"name": "solve_1024_fp16", "kind": "solve", "n": 1024, "b": 128, "form": "fp16", "ir": "classic", "rule": 0},
        # a small system of the CPU baseline's size, refined by GMRES
        {"name": "solve_8192_fp16_gmres", "kind": "solve", "n": 8192, "b": 256, "form": "fp16", "ir": "gmres", "rule": 0},
        # the stress matrix (weak diagonal) in the most accurate form
        {"name": "solve_32768_bf16x2", "kind": "solve", "n": 32768, "b": 1024, "form": "bf16x2", "ir": "classic", "rule": 1},
        # the largest orders: the plain form with GMRES, and the FP8 form of the headline run
        {"name": "solve_61440_fp16_gmres", "kind": "solve", "n": 61440, "b": 2560, "form": "fp16", "ir": "gmres", "rule": 0},
        {"name": "solve_61440_fp8", "kind": "solve", "n": 61440, "b": 2560, "form": "fp8", "ir": "classic", "rule": 0},
        # systems of orders 256..4096, several per SM, in the configuration the autotuner picks
        {"name": "batch_512", "kind": "batch", "count": 512, "max_order": 4096, "b": 256},
        # fewer small systems than SMs: one system's chain decides
        {"name": "batch_96_small", "kind": "batch", "count": 96, "max_order": 1024, "b": 256},
        # one diagonal block and its two triangular inverses, ragged order and pitch
        {"name": "diag_inv_1000", "kind": "diag", "n": 1000, "pad": 24},
        # the plain FP32 panel solves, left and right, ragged
        {"name": "panel_solves_5003", "kind": "panel", "m": 5003, "b": 500},
        # casts and trailing update of one step in FP8, ragged
        {"name": "update_fp8_5003", "kind": "update", "form": "fp8", "m": 5003, "n": 4001, "k": 640},
        # triangular solves with a factor made elsewhere
        {"name": "factor_solve_9999", "kind": "trsv", "n": 9999},
        # residual of the FP64 system, regenerated
        {"name": "residual_30011", "kind": "gemv", "n": 30011},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "batch", "diag", "panel", "update", "trsv", "gemv"])
    if kind == "solve":
        form = rng.choice(["fp16", "bf16x2", "fp8"])
        top = 32768 if form == "bf16x2" else 49152
        b = 64 * max(1, _log_int(rng, 64, 2560) // 64)
        nb = rng.randint(4, max(5, min(48, top // b)))
        return {"kind": kind, "n": b * nb, "b": b, "form": form, "ir": rng.choice(["classic", "gmres"]),
                "rule": rng.randint(0, 1)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 1, 512), "max_order": 128 * rng.randint(2, 32),
                "b": rng.choice([64, 128, 256, 256])}
    if kind == "diag":
        return {"kind": kind, "n": _log_int(rng, 50, 2560), "pad": rng.randint(0, 40)}
    if kind == "panel":
        return {"kind": kind, "m": _log_int(rng, 200, 20000), "b": _log_int(rng, 40, 1024)}
    if kind == "update":
        return {"kind": kind, "form": rng.choice(["fp16", "bf16x2", "fp8"]), "m": _log_int(rng, 100, 12000),
                "n": _log_int(rng, 100, 12000), "k": 64 * max(1, _log_int(rng, 64, 2560) // 64)}
    if kind == "trsv":
        return {"kind": kind, "n": _log_int(rng, 100, 20000)}
    return {"kind": kind, "n": _log_int(rng, 100, 40000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(seed)
    return g


def _randn(g, n, scale=1.0):
    return torch.randn(n, generator=g, device=_DEV, dtype=torch.float32) * scale


def _batch_orders(case):
    """Orders 128 * u, u uniform from the smallest to the largest of the case (the batch's own draw
    for the full range, 256 .. 4096); the matrices' seeds differ from pass to pass, not the orders."""
    top = case["max_order"] // 128
    if top == 32:
        return mxp.batch_sizes(case["count"], 3)
    g = torch.Generator()
    g.manual_seed(top)
    return [128 * int(u) for u in torch.randint(1, top + 1, (case["count"],), generator=g)]


def _block(g, n, ld, factored=False):
    """A diagonal block as the LU meets it (off-diagonals in [-1/2, 1/2], a dominant diagonal) or,
    factored, leaves it (the entries of L are smaller by the pivot).  Column-major with leading
    dimension ld, as a (n, ld) tensor of columns."""
    a = torch.rand(n, ld, generator=g, device=_DEV, dtype=torch.float32) - 0.5
    i = torch.arange(n, device=_DEV)
    a[i, i] = 0.25 * n + 2.0 + torch.rand(n, generator=g, device=_DEV)
    if factored:
        for c in range(0, n, 2048):
            part = a[c:c + 2048]
            cols = torch.arange(c, c + len(part), device=_DEV)
            part[torch.arange(ld, device=_DEV)[None, :] > cols[:, None]] *= 4.0 / n
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        form = case["form"]
        ws = mxp.Workspace(case["n"], case["b"], form, trsm_single=form == "fp8")
        n, dev = case["n"], _DEV
        p = mxp.Problem(n, seed, case["rule"], torch.empty(n * n, dtype=torch.float32, device=dev), n,
                        *(torch.empty(n, dtype=torch.float64, device=dev) for _ in range(3)))
        return {"case": case, "ws": ws, "p": p, "x": torch.empty(n, dtype=torch.float64, device=dev)}
    if kind == "batch":
        sizes = _batch_orders(case)
        bt = mxp.Batch(sizes, [1000 + 4096 * seed + i for i in range(len(sizes))])
        bt.set_config(case["b"], 128, 3)
        return {"case": case, "bt": bt}
    g = _rng(seed)
    if kind == "diag":
        n, ld = case["n"], case["n"] + case["pad"]
        a0 = _block(g, n, ld)
        return {"case": case, "a0": a0, "a": torch.empty_like(a0), "xu": torch.zeros(n, n, device=_DEV),
                "xl": torch.zeros(n, n, device=_DEV), "ws": mxp.Workspace(max(n, 128), n)}
    if kind == "panel":
        m, b = case["m"], case["b"]
        return {"case": case, "t": _block(g, b, b, factored=True), "r0": _randn(g, m * b), "l0": _randn(g, m * b),
                "r": torch.empty(m * b, device=_DEV), "l": torch.empty(m * b, device=_DEV)}
    if kind == "update":
        m, n, k, form = case["m"], case["n"], case["k"], mxp.FORMS[case["form"]]
        ldk = 3 * k if form == mxp.FORM_BF16X2 else k
        dt = torch.uint8 if form == mxp.FORM_FP8 else torch.int16
        tiles = lambda rows: torch.zeros(-(-rows // 128) * -(-k // 128), dtype=torch.uint8, device=_DEV)  # noqa: E731
        return {"case": case, "L": _randn(g, m * k, 1e-2), "U": _randn(g, k * n, 0.5), "C": _randn(g, (m + 3) * n),
                "lp": torch.zeros(m * ldk, dtype=dt, device=_DEV), "rp": torch.zeros(n * ldk, dtype=dt, device=_DEV),
                "ls": tiles(m), "rs": tiles(n), "ldk": ldk, "ws": mxp.Workspace(max(m, n) + k, k, form)}
    if kind == "trsv":
        n = case["n"]
        lu = _block(g, n, n, factored=True)
        b = torch.randn(n, generator=g, device=_DEV, dtype=torch.float64)
        return {"case": case, "lu": lu, "b": b, "x": torch.empty_like(b), "ws": mxp.Workspace(n, min(n, 256))}
    n = case["n"]
    return {"case": case, "seed": seed, "d": 0.25 * n + torch.rand(n, generator=g, device=_DEV, dtype=torch.float64),
            "x": torch.randn(n, generator=g, device=_DEV, dtype=torch.float64) / n,
            "b": torch.randn(n, generator=g, device=_DEV, dtype=torch.float64),
            "y": torch.empty(n, dtype=torch.float64, device=_DEV), "ws": mxp.Workspace(n, min(n, 256))}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        p = s["p"]
        mxp.regenerate(p)
        mxp.solve(p, case["b"], s["ws"], x=s["x"], method=mxp.IR_GMRES if case["ir"] == "gmres" else mxp.IR_CLASSIC)
        return {"x": s["x"], "lu": p.A}
    if kind == "batch":
        bt = s["bt"]
        bt.matgen()
        bt.solve()
        return {"x": bt.x, "lu": bt.A}
    if kind == "diag":
        n, ld = case["n"], case["n"] + case["pad"]
        s["a"].copy_(s["a0"])
        mxp.getrf_nopiv_inv(s["a"], n, ld, s["xu"], s["xl"], n, s["ws"])
        return {"lu": s["a"], "inv_u": s["xu"], "inv_l": s["xl"]}
    if kind == "panel":
        m, b = case["m"], case["b"]
        s["r"].copy_(s["r0"])
        s["l"].copy_(s["l0"])
        mxp.trsm_right_upper(m, b, s["t"], b, s["r"], m)
        mxp.trsm_left_lower_unit(b, m, s["t"], b, s["l"], b)
        return {"right": s["r"], "left": s["l"]}
    if kind == "update":
        m, n, k, form, ldk = case["m"], case["n"], case["k"], mxp.FORMS[case["form"]], s["ldk"]
        ls, rs = (s["ls"], s["rs"]) if form == mxp.FORM_FP8 else (None, None)
        mxp.panel_cast_left(form, m, k, s["L"], m, s["lp"], ldk, ls)
        mxp.panel_cast_right(form, n, k, s["U"], k, s["rp"], ldk, rs)
        mxp.schur_update(form, m, n, k, s["lp"], ldk, s["rp"], ldk, s["C"], m + 3, s["ws"], ls, rs)
        return {"c": s["C"], "l": s["lp"], "r": s["rp"], "ls": s["ls"], "rs": s["rs"]}
    if kind == "trsv":
        s["x"].copy_(s["b"])
        mxp.lu_solve(s["lu"], case["n"], case["n"], s["x"], s["ws"])
        return s["x"]
    s["y"].copy_(s["b"])
    mxp.otf_gemv(case["n"], s["seed"], s["d"], -1.0, s["x"], 1.0, s["y"], s["ws"])
    return s["y"]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far a correct result may be off
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        ns = [case["n"]] if kind == "solve" else _batch_orders(case)
        # the factors are written once; the matrix itself is generated, not read
        return {"bytes": float(sum(4 * n * n + 24 * n for n in ns)), "flops": float(sum(mxp.hpl_flops(n) for n in ns))}
    if kind == "diag":
        n = case["n"]
        return {"bytes": 16.0 * n * n, "flops": 4.0 / 3.0 * n ** 3}
    if kind == "panel":
        m, b = case["m"], case["b"]
        return {"bytes": 16.0 * m * b + 4.0 * b * b, "flops": 2.0 * m * b * b}
    if kind == "update":
        m, n, k = case["m"], case["n"], case["k"]
        es = {"fp16": 2, "bf16x2": 6, "fp8": 1}[case["form"]]
        return {"bytes": float((4 + es) * (m + n) * k + 8 * m * n), "flops": 2.0 * m * n * k}
    if kind == "trsv":
        n = case["n"]
        return {"bytes": 4.0 * n * n + 16.0 * n, "flops": 2.0 * n * n}
    n = case["n"]
    return {"bytes": 32.0 * n, "flops": 2.0 * n * n}


def tolerance(case):
    kind = case["kind"]
    # about four times what the results are off the 64-bit ones by: FP8 factors 1.9e-5 (rounding of the
    # panels, relative to the dominant diagonal), FP16 and split BF16 ones 2e-7, FP32 steps 1e-7, FP64
    # ones 3e-15 (a sum of n terms in another order)
    if kind == "solve" and case["form"] == "fp8":
        return {"rel": 1e-4, "max": 1e-2}
    if kind in ("solve", "batch"):
        return {"rel": 1e-6, "max": 1e-3}
    if kind in ("diag", "panel", "update"):
        return {"rel": 5e-7, "max": 1e-4}
    return {"rel": 1e-13, "max": 1e-11}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _signed(v):
    v &= _MASK
    return v - (1 << 64) if v >> 63 else v


def _lcg_pow(a, c, k):
    """The affine map x -> a x + c applied k times, mod 2^64."""
    ra, rc = 1, 0
    while k:
        if k & 1:
            ra, rc = ra * a & _MASK, (ra * c + rc) & _MASK
        a, c = a * a & _MASK, (a * c + c) & _MASK
        k >>= 1
    return ra, rc


def _states(start, a, c, count):
    out = []
    for _ in range(count):
        out.append(start)
        start = (a * start + c) & _MASK
    return out


def _columns(n, seed, c0, c1):
    """Columns c0 .. c1 of the generated FP64 matrix, as a (c1 - c0, n) tensor (the diagonal holds
    generator values), and column n (the right-hand side) when c0 == c1 == n."""
    s00 = (_LCG_A * seed + _LCG_C) & _MASK
    ia, ic = [], []
    a, c = 1, 0
    for _ in range(n):
        ia.append(_signed(a))
        ic.append(_signed(c))
        a, c = _LCG_A * a & _MASK, (_LCG_A * c + _LCG_C) & _MASK
    ia, ic = torch.tensor(ia, device=_DEV), torch.tensor(ic, device=_DEV)
    ja, jc = _lcg_pow(_LCG_A, _LCG_C, n)
    sa, sc = _lcg_pow(_LCG_A, _LCG_C, n * c0)
    base = torch.tensor([_signed(v) for v in _states((sa * s00 + sc) & _MASK, ja, jc, max(1, c1 - c0))], device=_DEV)
    out = torch.empty(len(base), n, dtype=torch.float64, device=_DEV)
    for q in range(0, len(base), 1024):
        out[q:q + 1024] = (base[q:q + 1024, None] * ia[None, :] + ic[None, :]).double() * _LCG_SCALE
    return out


def _system(n, seed, rule):
    """(A, A as the LU meets it, rhs) in FP64; matrices as tensors of columns."""
    a = _columns(n, seed, 0, n)
    i = torch.arange(n, device=_DEV)
    a[i, i] = 0.0
    d = torch.zeros(n, dtype=torch.float64, device=_DEV)
    for q in range(0, n, 2048):
        d += a[q:q + 2048].abs().sum(0)
    if rule == 1:
        d = 0.55 * d + 1.0
    a[i, i] = d
    return a, a.float().double(), _columns(n, seed, n, n)[0]


def _factor(a):
    """No-pivot LU (compact) of the matrix whose columns are the rows of a; returned the same way."""
    lu, _ = torch.linalg.lu_factor(a.t(), pivot=False)
    return lu


def _solve64(lu, b):
    y = torch.linalg.solve_triangular(lu, b[:, None], upper=False, unitriangular=True)
    return torch.linalg.solve_triangular(lu, y, upper=True)[:, 0]


def _exact_system(n, seed, rule):
    a, a32, rhs = _system(n, seed, rule)
    lu = _factor(a32)
    del a32
    x = _solve64(lu, rhs)
    for _ in range(3):
        x = x + _solve64(lu, rhs - a.t() @ x)
    return x, lu.t().contiguous().reshape(-1)


def _quantised(x, form, left):
    """The values the low-precision panels stand for, FP64; x: rows x K.  BF16X2: (hi, lo)."""
    if form == "fp16":
        return x.half().double()
    if form == "bf16x2":
        hi = x.bfloat16()
        return hi.double(), (x - hi.float()).bfloat16().double()
    rows, k = x.shape
    p = torch.zeros(-(-rows // 128) * 128, -(-k // 128) * 128, device=x.device)
    p[:rows, :k] = x
    t = p.view(p.shape[0] // 128, 128, p.shape[1] // 128, 128)
    amax = t.abs().amax(dim=(1, 3), keepdim=True).double()
    e = 8 - torch.floor(torch.log2(amax))
    e = torch.where(amax * torch.exp2(e) > 448.0, e - 1, e)
    q = (t * torch.exp2(e).float()).to(torch.float8_e4m3fn).double() * torch.exp2(-e)
    return q.view(p.shape)[:rows, :k]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        if case["n"] > 20000:
            return None
        x, lu = _exact_system(case["n"], seed, case["rule"])
        return {"x": x, "lu": lu}
    if kind == "batch":
        sizes = _batch_orders(case)
        if sum(n * n * (n + 4096) for n in sizes) > 4e11:
            return None
        got = [_exact_system(n, 1000 + 4096 * seed + i, 0) for i, n in enumerate(sizes)]
        return {"x": torch.cat([g[0] for g in got]), "lu": torch.cat([g[1] for g in got])}
    s = prepare(case, seed)
    if kind == "diag":
        n = case["n"]
        full = s["a0"].double()
        lu = _factor(full[:, :n])
        eye = torch.eye(n, dtype=torch.float64, device=_DEV)
        out = full.clone()
        out[:, :n] = lu.t()
        return {"lu": out, "inv_u": torch.linalg.solve_triangular(lu, eye, upper=True).t().contiguous(),
                "inv_l": torch.linalg.solve_triangular(lu, eye, upper=False, unitriangular=True).t().contiguous()}
    if kind == "panel":
        m, b = case["m"], case["b"]
        t = s["t"].double().t()
        right = torch.linalg.solve_triangular(t, s["r0"].double().view(b, m).t(), upper=True, left=False)
        left = torch.linalg.solve_triangular(t, s["l0"].double().view(m, b).t(), upper=False, unitriangular=True)
        return {"right": right.t().contiguous().view(-1), "left": left.t().contiguous().view(-1)}
    if kind == "update":
        m, n, k = case["m"], case["n"], case["k"]
        left = _quantised(s["L"].view(k, m).t().contiguous(), case["form"], True)
        right = _quantised(s["U"].view(n, k), case["form"], False)
        if case["form"] == "bf16x2":
            upd = right[0] @ left[0].t() + right[1] @ left[0].t() + right[0] @ left[1].t()
        else:
            upd = right @ left.t()
        c = s["C"].double().view(n, m + 3)
        c[:, :m] -= upd
        return {"c": c.reshape(-1), "l": None, "r": None, "ls": None, "rs": None}
    if kind == "trsv":
        return _solve64(s["lu"].double().t(), s["b"])
    n = case["n"]
    y = s["b"] - s["d"] * s["x"]
    for c in range(0, n, 4096):
        cols = _columns(n, seed, c, min(c + 4096, n))
        i = torch.arange(len(cols), device=_DEV)
        cols[i, c + i] = 0.0
        y -= s["x"][c:c + len(cols)] @ cols
    return y
