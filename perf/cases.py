"""The calls whose speed on a GPU matters to a user of this library, as data.

Each case is one call (or the few calls a program makes together) through the
public entry points: the rounding of a sum of trains, of one train and of a
batch of uneven ones, the reaction-Burgers step in its plain and its learned
form, the formal arithmetic, the inner product, and the reference-signature
API on host cores.  Sizes follow the benchmark's configurations (d = 20..40,
n = 64..256, ranks to 96) and the small and odd sizes of the tests.

A rounded train's cores are only defined up to an orthogonal matrix per bond,
so the rounding cases return what a program reads from the train: its values.
A tensor of at most FULL_MAX entries is returned whole; a larger one by its
values on the cross fibers of NPTS left and NPTS right multi-indices of every
mode (X[p_1..p_{k-1}, j, q_{k+1}..q_d] for all p, j, q), and its ranks.

Layout: core k of a train is a tensor of shape (r_{k+1}, n_k, r_k), row-major,
which is the library's column-major r_k x n_k x r_{k+1}.
"""
import math
import random

import numpy as np
import torch

import paratt_b200 as P
from paratt_b200 import capi as H
from paratt_b200.learned import LearnedStepper

FULL_MAX = 1 << 21
NPTS = 8
BOX, NU, DT = 10.0, 0.05, 1e-3
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # smallest: a rounding of a four-mode train with odd sizes, as in the tests: launches and latency only
        {"name": "round_sum_small", "op": "round_sum", "d": 4, "n": 17, "r": 5, "cap": 10, "ragged": True, "rtol": 1e-10},
        # an ordinary rounding after an addition, at the sizes of configuration 0 (ranks to 32)
        {"name": "round_sum_c0", "op": "round_sum", "d": 20, "n": 64, "r": 10, "cap": 20, "ragged": False, "rtol": 1e-8},
        # the rounding of configuration 1: ranks 32 + 32 back to 32
        {"name": "round_sum_c1", "op": "round_sum", "d": 40, "n": 256, "r": 32, "cap": 32, "ragged": False, "rtol": 1e-10},
        # a train with a decaying spectrum and odd ranks between 65 and 96, as the batch workload has them
        {"name": "round_one_r96", "op": "round_one", "d": 12, "n": 101, "r": 95, "cap": 47, "ragged": True, "rtol": 1e-8},
        # many independent uneven trains at once
        {"name": "round_batch_12", "op": "round_batch", "count": 12, "shapes": 4, "nmax": 512, "rmax": 96, "rtol": 1e-8},
        # time steps: configuration 0, and the benchmark's configuration 4 by the plain and the learned method
        {"name": "step_c0", "op": "step", "d": 20, "n": 64, "maxrank": 20, "ngauss": 1},
        {"name": "step_c4", "op": "step", "d": 40, "n": 256, "maxrank": 64, "ngauss": 3},
        {"name": "learned_step_c4", "op": "learned_step", "d": 40, "n": 256, "maxrank": 64, "ngauss": 3},
        # formal arithmetic at full rank: the all-modes difference operator, and the product of two trains
        {"name": "op_sum_r64", "op": "op_sum", "d": 40, "n": 256, "r": 64},
        {"name": "hadamard_r8", "op": "hadamard", "d": 40, "n": 256, "r": 8, "r2": 8},
        # the inner product of two trains (norms and error estimates)
        {"name": "dot_r64", "op": "dot", "d": 40, "n": 256, "r": 64, "r2": 64},
        # a driver written against the reference: add and truncate trains whose cores are in host memory
        {"name": "host_add_truncate", "op": "host", "d": 20, "n": 128, "r": 16, "cap": 16, "rtol": 1e-8},
    ]


def _log_int(rng, a, b):
    return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))


def draw(rng):
    op = rng.choice(["round_sum"] * 3 + ["round_one"] * 3 + ["round_batch", "step", "step", "learned_step", "op_sum",
                                                            "hadamard", "dot", "host"])
    d = rng.randint(3, 40)
    if op == "round_sum":
        n, r = _log_int(rng, 8, 300), _log_int(rng, 2, 32)
        return {"op": op, "d": d, "n": n, "r": r, "cap": rng.randint(r, 2 * r), "ragged": rng.random() < 0.5,
                "rtol": rng.choice([1e-6, 1e-8, 1e-10])}
    if op == "round_one":
        n, r = _log_int(rng, 16, 256), rng.randint(6, 96)
        return {"op": op, "d": min(d, 20), "n": n, "r": r, "cap": max(2, r // 2), "ragged": rng.random() < 0.7,
                "rtol": rng.choice([1e-6, 1e-8])}
    if op == "round_batch":
        return {"op": op, "count": rng.randint(3, 12), "shapes": rng.randint(5, 10 ** 6), "nmax": rng.choice([64, 128, 256]),
                "rmax": rng.randint(24, 96), "rtol": 1e-8}
    if op == "step":
        return {"op": op, "d": rng.randint(4, 32), "n": _log_int(rng, 24, 256), "maxrank": rng.randint(20, 48),
                "ngauss": rng.randint(1, 4)}
    if op == "learned_step":
        return {"op": op, "d": rng.randint(20, 40), "n": _log_int(rng, 64, 256), "maxrank": rng.randint(32, 48),
                "ngauss": rng.randint(2, 4)}
    if op == "op_sum":
        return {"op": op, "d": d, "n": _log_int(rng, 16, 256), "r": _log_int(rng, 3, 64)}
    if op == "hadamard":
        return {"op": op, "d": d, "n": _log_int(rng, 16, 256), "r": rng.randint(2, 9), "r2": rng.randint(2, 9)}
    if op == "dot":
        return {"op": op, "d": d, "n": _log_int(rng, 16, 256), "r": _log_int(rng, 3, 64), "r2": _log_int(rng, 3, 64)}
    return {"op": op, "d": min(d, 20), "n": _log_int(rng, 16, 128), "r": _log_int(rng, 3, 16),
            "cap": rng.randint(16, 32), "rtol": 1e-8}


# ---------------------------------------------------------------------------
# sizes and inputs
# ---------------------------------------------------------------------------
def _dims(c):
    return [max(4, c["n"] + ((7 * k) % 5 - 2 if c.get("ragged") else 0)) for k in range(c["d"])]


def _clamp(r, n):
    """Ranks of a valid train: r_k <= r_{k-1} n_{k-1} and r_k <= n_k r_{k+1}."""
    r, d = list(r), len(n)
    for k in range(1, d):
        r[k] = min(r[k], r[k - 1] * n[k - 1])
    for k in range(d - 1, 0, -1):
        r[k] = min(r[k], r[k + 1] * n[k])
    return r


def _ranks(c, key="r"):
    n = _dims(c)
    return _clamp([1] + [max(1, c[key] - ((5 * k) % 4 if c.get("ragged") else 0)) for k in range(1, c["d"])] + [1], n)


def _shapes(c):
    """(dims, ranks, caps) of the trains of a batch: d 10..40, one mode size, ranks 8..rmax per bond, caps half of them."""
    rng, out = random.Random(c["shapes"]), []
    for _ in range(c["count"]):
        d = rng.randint(10, 40)
        n = [rng.choice([v for v in (32, 64, 128, 256, 512) if v <= c["nmax"]])] * d
        r = _clamp([1] + [rng.randint(8, c["rmax"]) for _ in range(d - 1)] + [1], n)
        out.append((n, r, [1] + [max(1, v // 2) for v in r[1:-1]] + [1]))
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _gauss_train(n, r, g):
    """N(0, 1 / r) cores: those of configuration 1 scaled to entries of order one."""
    return [torch.randn(r[k + 1], n[k], r[k], dtype=F64, device="cuda", generator=g) / math.sqrt(r[k])
            for k in range(len(n))]


def _decay_train(n, r, g):
    """Left-orthonormal cores, bond column j scaled by 2^-j, as in the batch workload."""
    out = []
    for k in range(len(n)):
        q = torch.linalg.qr(torch.randn(r[k] * n[k], r[k + 1], dtype=F64, device="cuda", generator=g))[0]
        if k < len(n) - 1:
            q = q * torch.pow(2.0, -torch.arange(r[k + 1], dtype=F64, device="cuda"))
        out.append(q.t().reshape(r[k + 1], n[k], r[k]).contiguous())
    return out


def _bumps(c, seed):
    """Sum of Gaussians on the periodic box: centres U[-2, 2]^d, widths U[0.3, 0.8]; its train and the centres' grid points."""
    rng, d, n, G = np.random.default_rng(seed), c["d"], c["n"], c["ngauss"]
    ctr, wid = rng.uniform(-2.0, 2.0, (G, d)), rng.uniform(0.3, 0.8, G)
    x = -BOX / 2 + np.arange(n) * (BOX / n)
    cores = []
    for k in range(d):
        v = np.exp(-(x[None, :] - ctr[:, k, None]) ** 2 / (2 * wid[:, None] ** 2))
        if G == 1:
            m = v.reshape(1, n, 1)
        elif k == 0:
            m = v.reshape(G, n, 1)
        elif k == d - 1:
            m = v.T.reshape(1, n, G)
        else:
            m = np.zeros((G, n, G))
            for j in range(G):
                m[j, :, j] = v[j]
        cores.append(torch.from_numpy(np.ascontiguousarray(m)).cuda())
    at = np.clip(np.rint((ctr + BOX / 2) / (BOX / n)).astype(int), 0, n - 1)
    return cores, at


def _points(c, n, seed):
    """NPTS left and NPTS right multi-indices (d x NPTS each): around the Gaussians' centres, or anywhere."""
    rng = np.random.default_rng([int(seed), 7])
    if "ngauss" in c:
        at = _bumps(c, seed)[1]
        pl, pr = [np.stack([at[m % len(at)] for m in range(NPTS)], 1) + rng.integers(-1, 2, (len(n), NPTS)) for _ in "lr"]
        return pl % np.array(n)[:, None], pr % np.array(n)[:, None]
    return [np.stack([rng.integers(0, v, NPTS) for v in n]) for _ in "lr"]


def _rank_of(cores):
    return [1] + [int(c.shape[0]) for c in cores]


def _rms(cores):
    a = torch.ones(1, 1, dtype=F64, device=cores[0].device)
    for c in cores:
        t = torch.matmul(c, a)
        a = torch.matmul(t.reshape(t.shape[0], -1), c.reshape(c.shape[0], -1).t()) / c.shape[1]
    return math.sqrt(max(float(a[0, 0]), 0.0))


# ---------------------------------------------------------------------------
# reading a train: its values
# ---------------------------------------------------------------------------
def _full(cores):
    t = cores[0].reshape(cores[0].shape[0], -1)
    for c in cores[1:]:
        t = (c.reshape(-1, c.shape[2]) @ t).reshape(c.shape[0], -1)
    return t.reshape(-1)


def _is_small(n):
    return math.prod(n) <= FULL_MAX


def _crosses(cores, pl, pr, cols):
    d, M = len(cores), cols.numel()
    R = [None] * (d + 1)
    R[d] = torch.ones(1, M, dtype=F64, device=cores[0].device)
    for k in range(d - 1, 0, -1):
        R[k] = torch.bmm(cores[k].index_select(1, pr[k]).permute(1, 2, 0), R[k + 1].t().unsqueeze(2)).squeeze(2).t()
    L = torch.ones(1, M, dtype=F64, device=cores[0].device)
    out = []
    for k, c in enumerate(cores):
        p = torch.mm(c.reshape(-1, c.shape[2]), L).reshape(c.shape[0], c.shape[1], M)
        out.append(torch.mm(R[k + 1].t(), p.reshape(c.shape[0], -1)).reshape(-1))
        L = p[:, pl[k], cols]
    return torch.cat(out)


def _points_on(c, n, seed, device="cuda"):
    pl, pr = _points(c, n, seed)
    return [list(torch.from_numpy(np.ascontiguousarray(p)).to(device)) for p in (pl, pr)] + [torch.arange(NPTS, device=device)]


def _values(cores, pts):
    return _full(cores) if pts is None else _crosses(cores, *pts)


# ---------------------------------------------------------------------------
# the library's side
# ---------------------------------------------------------------------------
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = P.Context(0)
    return _ctx


class _Closed:
    """Closes what it holds when the last reference goes."""

    def __init__(self, close, *things):
        self.close, self.things = close, things

    def __del__(self):
        self.close(*self.things)


class _Memory:
    """One of a train's buffers, for torch; keeps the train."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 3}


class _Train:
    """A train on the device and torch views of its cores (one view per buffer the library hands out)."""

    def __init__(self, n, cap, cores=None):
        self.tt = P.TT(_context(), n, cap)
        self.owner = _Closed(lambda t: t.close(), self.tt)
        self.n, self.count, self.view = n, [cap[k] * n[k] * cap[k + 1] for k in range(len(n))], {}
        if cores is not None:
            cores = [c.contiguous() for c in cores]
            torch.cuda.synchronize()
            self.tt.set_device(_rank_of(cores), [c.data_ptr() for c in cores])

    def cores(self):
        """Views of the current cores, 1-D over each core's actual elements."""
        ptrs = (P._dp * len(self.n))()
        P._check(P.lib().ptt_tt_device_cores(self.tt.h, ptrs, None))
        r, out = self.tt.ranks(), []
        addr = np.ctypeslib.as_array(P.C.cast(ptrs, P.C.POINTER(P.C.c_size_t)), (len(self.n),)).tolist()
        for k, a in enumerate(addr):
            v = self.view.get((k, a))
            if v is None:
                v = self.view[(k, a)] = torch.as_tensor(_Memory(self.owner, a, self.count[k]), device="cuda")
            out.append(v.as_strided((r[k + 1], self.n[k], r[k]), (self.n[k] * r[k], r[k], 1)))
        return r, out


def prepare(case, seed):
    op, ctx = case["op"], _context()
    if op in ("round_sum", "round_one"):
        n, r = _dims(case), _ranks(case)
        a, b, tol = _round_input(case, seed)
        s = {"cap": case["cap"], "tol": tol, "pts": None if _is_small(n) else _points_on(case, n, seed), "x": _Train(n, r, a)}
        if op == "round_sum":
            s["y"] = _Train(n, r, b)
        s["z"] = _Train(n, [1] + [2 * v for v in r[1:-1]] + [1] if op == "round_sum" else r)
    elif op == "round_batch":
        s = {"x": [], "z": [], "cap": [], "tol": [], "pts": []}
        for i, (n, r, cap) in enumerate(_shapes(case)):
            a, tol = _batch_input(case, seed, i)
            s["x"].append(_Train(n, r, a))
            s["z"].append(_Train(n, r))
            s["cap"].append(cap)
            s["tol"].append(tol)
            s["pts"].append(_points_on({}, n, seed + i))
    elif op in ("step", "learned_step"):
        d, n, m = case["d"], [case["n"]] * case["d"], case["maxrank"]
        u0 = _bumps(case, seed)[0]
        tol = 1e-8 * _rms(u0)
        cap = [1] + [2 * m] * (d - 1) + [1]
        s = {"u0": _Train(n, cap, u0), "u": _Train(n, cap), "pts": None if _is_small(n) else _points_on(case, n, seed)}
        if op == "step":
            s["sim"] = P.RxnBurgers(ctx, d, case["n"], maxrank=m, dt=DT, tol=tol, nu=NU, L=BOX, seed=7)
            s["end"] = _Closed(lambda t: t.close(), s["sim"])
        else:  # the method's first step is a plain one, which records the spectra the proposal reads
            s["ls"] = LearnedStepper(ctx, d, case["n"], m, DT, tol, seed=3)
            s["ls"].step(s["u0"].tt)
            s["spec"] = [(g.copy(), dl, list(rk)) for g, dl, rk in s["ls"].spec]
            s["end"] = _Closed(lambda t: t.close(), s["ls"])
    elif op == "op_sum":
        n, r = _dims(case), _ranks(case)
        s = {"x": _Train(n, r, _gauss_train(n, r, _gen(seed))), "z": _Train(n, [1] + [2 * v for v in r[1:-1]] + [1])}
    elif op in ("hadamard", "dot"):
        n, r, r2 = _dims(case), _ranks(case), _ranks(case, "r2")
        a, b = _pair_input(case, seed)
        s = {"x": _Train(n, r, a), "y": _Train(n, r2, b)}
        if op == "hadamard":
            s["z"] = _Train(n, [p * q for p, q in zip(r, r2)])
    else:  # host
        n, r = _dims(case), _ranks(case)
        a, b, tol = _round_input(case, seed)
        host = [[np.asfortranarray(c.cpu().numpy().transpose(2, 1, 0)) for c in t] for t in (a, b)]
        s = {"x": H.HostTT(host[0]), "y": H.HostTT(host[1]), "tol": tol, "cap": H._iarr([case["cap"]] * (case["d"] + 1)),
             "z": H.HostTT(dims=n, ranks=[1] * (case["d"] + 1), capacity=[1] + [2 * v for v in r[1:-1]] + [1]),
             "pts": None if _is_small(n) else _points_on(case, n, seed, "cpu")}
        s["end"] = _Closed(lambda *t: [v.free() for v in t], s["x"], s["y"], s["z"])
    s["op"] = op
    return s


def _read(train, pts):
    r, cores = train.cores()
    with torch.cuda.stream(torch.cuda.ExternalStream(_context().stream)):
        return np.array(r), _values(cores, pts)


def _stencil(case_n):
    h = BOX / case_n
    return [NU / h ** 2, -2.0 * NU / h ** 2, NU / h ** 2]


def run(s):
    op = s["op"]
    if op == "round_sum":
        P.axpby(1.0, s["x"].tt, 1.0, s["y"].tt, s["z"].tt)
        s["z"].tt.round(s["tol"], s["cap"])
        return _read(s["z"], s["pts"])
    if op == "round_one":
        s["z"].tt.copy_from(s["x"].tt)
        s["z"].tt.round(s["tol"], s["cap"])
        return _read(s["z"], s["pts"])
    if op == "round_batch":
        for x, z in zip(s["x"], s["z"]):
            z.tt.copy_from(x.tt)
        P.round_batch([z.tt for z in s["z"]], s["tol"], s["cap"])
        return [_read(z, p) for z, p in zip(s["z"], s["pts"])]
    if op == "step":
        s["u"].tt.copy_from(s["u0"].tt)
        s["sim"].step(s["u"].tt)
        return _read(s["u"], s["pts"])
    if op == "learned_step":
        s["u"].tt.copy_from(s["u0"].tt)
        s["ls"].seed_from(s["spec"])
        s["ls"].step(s["u"].tt)
        return _read(s["u"], s["pts"])
    if op == "op_sum":
        P.op_sum(s["x"].tt, _stencil(s["x"].n[0]), 1.0, s["z"].tt)
        return s["z"].cores()[1]
    if op == "hadamard":
        P.hadamard(s["x"].tt, s["y"].tt, s["z"].tt)
        return s["z"].cores()[1]
    if op == "dot":
        return np.array([s["x"].tt.dot(s["y"].tt), s["x"].tt.dot(s["x"].tt)])
    L = H.capi()
    L.attac_tt_axpby(1.0, s["x"].p.contents.x, 1.0, s["y"].p.contents.x, s["z"].p.contents.x)
    L.paratt_truncate(s["z"].p, s["tol"], s["cap"])
    cores = [torch.from_numpy(c.transpose(2, 1, 0)) for c in s["z"].cores()]
    return np.array(s["z"].ranks()), _values(cores, s["pts"])


# ---------------------------------------------------------------------------
# inputs shared by prepare() and exact()
# ---------------------------------------------------------------------------
def _round_input(case, seed):
    n, r, g = _dims(case), _ranks(case), _gen(seed)
    if case["op"] == "round_one":
        a = _decay_train(n, r, g)
        return a, None, case["rtol"] * _rms(a)
    a, b = _gauss_train(n, r, g), _gauss_train(n, r, g)
    return a, b, case["rtol"] * _rms(_add(a, b))


def _batch_input(case, seed, i):
    n, r, _ = _shapes(case)[i]
    a = _decay_train(n, r, _gen(1000 * seed + i))
    return a, case["rtol"] * _rms(a)


def _pair_input(case, seed):
    n, g = _dims(case), _gen(seed)
    a = _gauss_train(n, _ranks(case), g)
    b = _gauss_train(n, _ranks(case, "r2"), g)
    for k in range(len(b)):  # a product of related trains: its value is not one of cancellation
        m, w = (min(p, q) for p, q in zip(b[k].shape[::2], a[k].shape[::2]))
        b[k][:m, :, :w] += a[k][:m, :, :w]
    return a, b


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _add(a, b):
    d, out = len(a), []
    for k, (x, y) in enumerate(zip(a, b)):
        if k == 0:
            out.append(torch.cat([x, y], 0))
        elif k == d - 1:
            out.append(torch.cat([x, y], 2))
        else:
            z = torch.zeros(x.shape[0] + y.shape[0], x.shape[1], x.shape[2] + y.shape[2], dtype=F64, device=x.device)
            z[:x.shape[0], :, :x.shape[2]] = x
            z[x.shape[0]:, :, x.shape[2]:] = y
            out.append(z)
    return out


def _apply_all(u, sten, shift):
    """sum_i S_i u + shift u as the train [[u_k, S u_k], [0, u_k]] (first core: block row 0, last: block column 1)."""
    d, out = len(u), []
    for k, c in enumerate(u):
        s = sum(sten[t] * torch.roll(c, 1 - t, 1) for t in range(3))
        if k == 0:
            out.append(torch.cat([c, s + shift * c], 0))
        elif k == d - 1:
            out.append(torch.cat([s, c], 2))
        else:
            z = torch.zeros(2 * c.shape[0], c.shape[1], 2 * c.shape[2], dtype=F64, device=c.device)
            z[:c.shape[0], :, :c.shape[2]] = c
            z[c.shape[0]:, :, :c.shape[2]] = s
            z[c.shape[0]:, :, c.shape[2]:] = c
            out.append(z)
    return out


def _times(a, b):
    """Formal product: row index i_y + r_y i_x, column index j_y + r_y' j_x."""
    return [torch.einsum("lji,mjk->lmjik", x, y).reshape(x.shape[0] * y.shape[0], x.shape[1], x.shape[2] * y.shape[2])
            for x, y in zip(a, b)]


def _rounded(u, tol, cap):
    u, d = list(u), len(u)
    cap = cap if hasattr(cap, "__len__") else [cap] * (d + 1)
    for k in range(d - 1):
        q, r = torch.linalg.qr(u[k].reshape(u[k].shape[0], -1).t())
        u[k] = q.t().reshape(q.shape[1], u[k].shape[1], u[k].shape[2])
        u[k + 1] = torch.matmul(u[k + 1], r.t())
    delta = tol / math.sqrt(d - 1.0) * math.exp(0.5 * sum(math.log(c.shape[1]) for c in u))
    for k in range(d - 1, 0, -1):
        c = u[k]
        q, r = torch.linalg.qr(c.reshape(-1, c.shape[2]))
        w, sv, v = np.linalg.svd(r.cpu().numpy().T, full_matrices=False)
        keep = int(np.sum(sv >= math.sqrt(len(sv)) * 2.0 ** -53 * sv[0]))
        tail = 0.0
        rank = keep
        for j in range(keep - 1, -1, -1):
            tail += float(sv[j]) ** 2
            if math.sqrt(tail) >= delta:
                break
            rank = j
        rank = max(1, min(rank, cap[k]))
        u[k] = (q @ torch.from_numpy(v[:rank].T.copy()).to(q)).reshape(c.shape[0], c.shape[1], rank)
        us = torch.from_numpy((w[:, :rank] * sv[:rank]).T.copy()).to(q)
        u[k - 1] = (us @ u[k - 1].reshape(u[k - 1].shape[0], -1)).reshape(rank, u[k - 1].shape[1], u[k - 1].shape[2])
    return u


def _step(u, case, tol):
    d, m, h = case["d"], case["maxrank"], BOX / case["n"]
    d1 = [1.0 / (4.0 * d * h), 0.0, -1.0 / (4.0 * d * h)]

    def scaled(a, v):
        return [a * v[0]] + v[1:]

    def field(v):
        w = _rounded(_times(v, v), tol, m)
        a = _rounded(_apply_all(v, _stencil(case["n"]), 1.0), tol, m)
        b = _rounded(_apply_all(w, d1, -1.0), tol, m)
        return _rounded(_add(a, b), tol, m)

    us = _rounded(_add(u, scaled(0.5 * DT, field(u))), tol, m)
    return _rounded(_add(u, scaled(DT, field(us))), tol, m)


def _dot(a, b):
    t = torch.ones(1, 1, dtype=F64, device=a[0].device)  # t[y index, x index]
    for x, y in zip(a, b):
        v = torch.matmul(x, t.t())  # (x', n, y)
        t = torch.matmul(y.reshape(y.shape[0], -1), v.reshape(v.shape[0], -1).t()) / x.shape[1]
    return float(t[0, 0])


def exact(case, seed):
    op, n = case["op"], _dims(case) if "d" in case else None
    if op in ("round_sum", "round_one", "host"):
        a, b, tol = _round_input(case, seed)
        z = _rounded(a if b is None else _add(a, b), tol, case["cap"])
        return None, _values(z, None if _is_small(n) else _points_on(case, n, seed))
    if op == "round_batch":
        out = []
        for i, (n, r, cap) in enumerate(_shapes(case)):
            a, tol = _batch_input(case, seed, i)
            out.append((None, _values(_rounded(a, tol, cap), _points_on({}, n, seed + i))))
        return out
    if op in ("step", "learned_step"):
        u = _bumps(case, seed)[0]
        tol = 1e-8 * _rms(u)
        for _ in range(1 if op == "step" else 2):
            u = _step(u, case, tol)
        return None, _values(u, None if _is_small(n) else _points_on(case, n, seed))
    if op == "op_sum":
        return _apply_all(_gauss_train(n, _ranks(case), _gen(seed)), _stencil(case["n"]), 1.0)
    a, b = _pair_input(case, seed)
    if op == "hadamard":
        return _times(a, b)
    return np.array([_dot(a, b), _dot(a, a)])


# ---------------------------------------------------------------------------
# what a call cannot do without
# ---------------------------------------------------------------------------
def _size(n, r):
    return 8.0 * sum(r[k] * n[k] * r[k + 1] for k in range(len(n)))


def _round_flops(n, r, kept):
    """QR with Q of every left unfolding and R into the next core, then LQ with Q, U S and V over the kept ranks."""
    f, d = 0.0, len(n)
    for k in range(d - 1):
        f += 4.0 * r[k] * n[k] * r[k + 1] ** 2 + 2.0 * r[k + 1] ** 2 * n[k + 1] * r[k + 2]
    for k in range(1, d):
        m = n[k] * kept[k + 1]
        f += 2.0 * m * r[k] ** 2 + 12.0 * r[k] ** 3 + 4.0 * m * r[k] * kept[k] + 2.0 * r[k - 1] * n[k - 1] * r[k] * kept[k]
    return f


def _kept(r, cap, rtol):
    return [1] + [min(v, c, 2 - int(math.log2(rtol))) for v, c in zip(r[1:-1], cap[1:-1])] + [1]


def work(case):
    op = case["op"]
    if op == "round_batch":
        b = f = 0.0
        for n, r, cap in _shapes(case):
            k = _kept(r, cap, case["rtol"])
            b, f = b + _size(n, r) + _size(n, k), f + _round_flops(n, r, k)
        return {"bytes": b, "flops": f}
    n, d = _dims(case), case["d"]
    if op in ("step", "learned_step"):  # ranks of a state of G Gaussians: about 2 G + 1; field ones twice that
        m = case["maxrank"]
        r, f = min(m, 2 * case["ngauss"] + 1), 0.0
        for rin, rout in 2 * [(r * (r + 1) // 2, r), (2 * r, 2 * r), (2 * r, 2 * r), (4 * r, 2 * r), (3 * r, r)]:
            full = [1] + [min(v, 128) for v in [rin] * (d - 1)] + [1]
            f += _round_flops(n, full, [1] + [min(rout, m)] * (d - 1) + [1])
        u = [1] + [r] * (d - 1) + [1]
        return {"bytes": 2 * _size(n, u), "flops": f}
    r = _ranks(case)
    if op == "op_sum":
        z = [1] + [2 * v for v in r[1:-1]] + [1]
        return {"bytes": _size(n, r) + _size(n, z), "flops": 5.0 * _size(n, r) / 8}
    if op in ("hadamard", "dot"):
        r2 = _ranks(case, "r2")
        if op == "hadamard":
            z = [p * q for p, q in zip(r, r2)]
            return {"bytes": _size(n, r) + _size(n, r2) + _size(n, z), "flops": _size(n, z) / 8}
        f = 0.0
        for x, y in ((r, r2), (r, r)):
            f += sum(2.0 * n[k] * x[k] * y[k + 1] * (y[k] + x[k + 1]) for k in range(d))
        return {"bytes": _size(n, r) + _size(n, r2), "flops": f}
    pair = op in ("round_sum", "host")
    z = [1] + [2 * v for v in r[1:-1]] + [1] if pair else r
    k = [1] + [min(v, case["cap"]) for v in z[1:-1]] + [1] if pair else _kept(z, [case["cap"]] * (d + 1), case["rtol"])
    return {"bytes": (2 if pair else 1) * _size(n, r) + _size(n, k), "flops": _round_flops(n, z, k)}
