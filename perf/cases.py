"""Timing cases: what a program built on this library has it do.

A quantum Monte Carlo program solves its orbitals' grid data into a
coefficient table once (``solve``), then evaluates all orbitals at electron
positions, over and over: one position a call through the CPU-shaped entry
(``point``), batches of positions in flat device buffers (``flat``), batches
through the pointer-array GPU entries (``ptrs``), and the determinant step
that consumes the orbitals: the ratio of a proposed move (``ratio``) and the
rank-1 update of the inverse after an accepted one (``update``).

``op`` names the path; the other keys are its sizes, types and options.
Grids are given by their points per axis; the box is the unit cube.
"""
import ctypes as C
import math

import numpy as np
import torch

from einspline_gb300 import _lib as L
from einspline_gb300 import api

DEV = "cuda"
BC = {"periodic": api.PERIODIC, "antiperiodic": api.ANTIPERIODIC, "natural": api.NATURAL, "flat": api.FLAT}
STORE = {"native": api.STORE_NATIVE, "f16": api.STORE_F16, "bf16": api.STORE_BF16, "i16": api.STORE_I16}
ELEM = {"native": {"s": 4, "c": 4, "d": 8, "z": 8}, "f16": 2, "bf16": 2, "i16": 2}


def listed():
    return [
        # one electron moved at a time by a program written for the CPU
        # library: one position a call, results in host arrays; the 32^3 x
        # 128 table of the parity configuration
        dict(name="point_s_32x128", op="point", kind="s", store="native", gx=32, gy=32, gz=32, bc="periodic", n=128,
             form="vgh"),
        # one small walker's positions, the smallest request that the
        # serving configuration sees is 32 points
        dict(name="walker_f16_64x1024", op="flat", kind="s", store="f16", gx=64, gy=64, gz=64, bc="periodic",
             n=1024, npts=48, form="vgh", sort=False),
        # the headline step: 64 walkers of 32..512 positions, F16 table
        dict(name="step_f16_64x1024", op="flat", kind="s", store="f16", gx=64, gy=64, gz=64, bc="periodic", n=1024,
             npts=17509, form="vgh", sort=False),
        # the same orbitals as an FP32 table through the pointer-array GPU
        # entry that programs written for the reference's GPU path call
        dict(name="ptrs_s_vgh_64x1024", op="ptrs", kind="s", store="native", gx=64, gy=64, gz=64, bc="periodic",
             n=1024, npts=16384, form="vgh"),
        # double precision batches (48^3 x 512)
        dict(name="ptrs_d_vgh_48x512", op="ptrs", kind="d", store="native", gx=48, gy=48, gz=48, bc="periodic",
             n=512, npts=8192, form="vgh"),
        # complex orbitals (twisted boundary conditions), visited in cell order
        dict(name="sorted_c_64x256", op="flat", kind="c", store="native", gx=64, gy=64, gz=64, bc="periodic", n=256,
             npts=32768, form="vgh", sort=True),
        # value, gradient and laplacian rows as QMC drivers take them, on an
        # odd, non-periodic grid with an odd number of orbitals
        dict(name="ptrs_s_vgl_ragged", op="ptrs", kind="s", store="native", gx=45, gy=37, gz=51, bc="natural",
             n=203, npts=3001, form="vgl"),
        # values alone (pseudopotential quadrature: many points, no
        # derivatives) from a 16-bit fixed-point table
        dict(name="value_i16_56x777", op="flat", kind="s", store="i16", gx=56, gy=60, gz=52, bc="antiperiodic",
             n=777, npts=24000, form="value", sort=False),
        # the largest batch: a population of walkers in one launch, visited in
        # cell order
        dict(name="large_f16_96x1024", op="flat", kind="s", store="f16", gx=96, gy=96, gz=96, bc="periodic", n=1024,
             npts=160000, form="vgh", sort=True),
        # the ratio of a proposed move for a population, with gradient,
        # laplacian and the new rows, in the reference's inverse layout
        dict(name="ratio_f16_64x1024", op="ratio", kind="s", store="f16", gx=64, gy=64, gz=64, bc="periodic", n=1024,
             walkers=2048, trans=0),
        # the accepted walkers' inverse updates
        dict(name="update_512x768", op="update", n=768, walkers=512, trans=0),
        # reading a wave function: grid data in, coefficient table out
        dict(name="solve_s_64x512", op="solve", kind="s", store="native", gx=64, gy=64, gz=64, bc="periodic", n=512),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["point", "flat", "flat", "flat", "ptrs", "ptrs", "ptrs", "ratio", "update", "solve"])
    if op == "update":
        n = _logint(rng, 16, 1024)
        return dict(op=op, n=n, walkers=_logint(rng, 1, max(2, min(2048, int(3e8 // (n * n))))),
                    trans=rng.randrange(2))
    grid = [_logint(rng, 8, 80) for _ in range(3)]
    case = dict(op=op, gx=grid[0], gy=grid[1], gz=grid[2],
                bc=rng.choice(["periodic", "periodic", "periodic", "antiperiodic", "natural", "flat"]))
    if op == "ratio":
        case.update(kind="s", store=rng.choice(["native", "f16", "bf16"]), n=_logint(rng, 16, 1024),
                    walkers=_logint(rng, 1, 4096), trans=rng.randrange(2))
        return case
    kind = rng.choice("sssccdz")
    store = rng.choice(["native", "native", "f16", "bf16", "i16"]) if kind in "sc" and op in ("flat", "point") else "native"
    cells = math.prod(g + 3 for g in grid)
    ncomp = 2 if kind in "cz" else 1
    nmax = max(4, min(1024, int(6e8 // (cells * ncomp))))
    case.update(kind=kind, store=store, n=_logint(rng, 4, nmax))
    if op == "solve":
        return case
    if op == "point":
        case.update(form=rng.choice(["value", "vgh"]))
        return case
    # evaluations bounded by the largest listed case's; FP64 arithmetic by less
    evals = 2e7 if kind in "dz" else 1e8
    case.update(npts=_logint(rng, 1, max(2, min(150000, int(evals // (case["n"] * ncomp))))))
    if op == "flat":
        case.update(form=rng.choice(["vgh", "vgh", "value"]), sort=rng.random() < 0.4)
    else:
        case.update(form=rng.choice(["vgh", "vgl", "value"]))
    return case


# ------------------------------------------------------------------ inputs
def _gen(seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + what) & 0x7FFFFFFF)
    return g


def _grid_data(case, seed):
    """[n, gx, gy, gz(, 2)]: uniform in [-1, 1]; orbitals of a determinant
    around 1, so that ratios of small moves stay near 1 as in a real run."""
    dt = torch.float32 if case["kind"] in "sc" else torch.float64
    shape = (case["n"], case["gx"], case["gy"], case["gz"]) + ((2,) if case["kind"] in "cz" else ())
    d = torch.rand(shape, dtype=dt, device=DEV, generator=_gen(seed, 1)).mul_(2).sub_(1)
    return d.mul_(0.5).add_(1.0) if case["op"] == "ratio" else d


def _points(case, seed, count, dt):
    # strictly inside the box: the upper edge belongs to no cell
    return torch.rand((count, 3), dtype=dt, device=DEV, generator=_gen(seed, 2)).mul_(0.999)


def _spline(case, data):
    grids = [(0.0, 1.0, case[a]) for a in ("gx", "gy", "gz")]
    bcs = [(BC[case["bc"]],) * 2] * 3
    s = api.MultiUBspline3D(case["kind"], grids, bcs, case["n"], storage=STORE[case["store"]])
    if data is not None:
        s.set_device(0, data)
        s.flush()
        torch.cuda.synchronize()
    return s


class _DeviceArray:
    """A spline's device table as torch sees it; keeps the spline alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 3}


def _ptr_array(t, rows):
    step = t.numel() // rows * t.element_size()
    return torch.arange(rows, dtype=torch.int64, device=DEV) * step + t.data_ptr()


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _lattice(seed, dt):
    # a slightly skewed cell's transform to Cartesian derivatives
    g = torch.eye(3, dtype=dt, device=DEV) + 0.1 * (torch.rand((3, 3), dtype=dt, device=DEV, generator=_gen(seed, 5)) - 0.5)
    return g.contiguous()


def _update_inputs(case, seed):
    n, W, ld = case["n"], case["walkers"], case["n"]
    rng = np.random.default_rng(seed)
    base = min(2, W)
    A, B = [], []
    for _ in range(base):
        a = np.eye(n) + 0.3 * rng.standard_normal((n, n)) / math.sqrt(n)
        A.append(a)
        B.append(np.linalg.inv(a))
    A = torch.from_numpy(np.stack(A)).to(DEV)
    B = torch.from_numpy(np.stack(B)).to(DEV)
    g = _gen(seed, 3)
    # walker w: a base matrix with its rows scaled, and the scaled inverse
    s = 0.5 + 1.5 * torch.rand((W, n), dtype=torch.float64, device=DEV, generator=g)
    which = torch.arange(W, device=DEV) % base
    Aw = torch.empty((W, n, ld), dtype=torch.float32, device=DEV)
    Bw = torch.empty((W, n, ld), dtype=torch.float32, device=DEV)
    for w0 in range(0, W, 64):
        sl = slice(w0, w0 + 64)
        Aw[sl] = (s[sl, :, None] * A[which[sl]]).float()
        inv = B[which[sl]] / s[sl, None, :]
        Bw[sl] = (inv.transpose(1, 2) if case["trans"] else inv).float()
    k = n // 3
    rows = Aw[:, k, :] + (0.2 / math.sqrt(n)) * torch.randn((W, n), device=DEV, generator=g) * s[:, k, None].float()
    return Aw, Bw, rows.contiguous(), k


def prepare(case, seed):
    op = case["op"]
    st = {"case": case}
    if op == "update":
        A, B, rows, k = _update_inputs(case, seed)
        st.update(det=api.Determinants(A, B, case["n"], case["trans"]), rows=rows, k=k,
                  accepted=torch.arange(case["walkers"], device=DEV))
        return st
    data = _grid_data(case, seed)
    if op == "solve":
        st.update(data=data, spline=_spline(case, None))
        ti = st["spline"].info()
        f64 = ti.elem_bytes == 8
        st["table"] = torch.as_tensor(_DeviceArray(st["spline"], ti.coefs, (ti.nx, ti.ny, ti.nz, ti.ncol_pad),
                                                   "<f8" if f64 else "<f4"))
        assert st["table"].data_ptr() == ti.coefs  # a view: the program reads the table in place
        return st
    sp = _spline(case, data)
    del data
    st["spline"] = sp
    kind, n = case["kind"], case["n"]
    ncomp = 2 if kind in "cz" else 1
    dt = torch.float32 if kind in "sc" else torch.float64
    if op == "point":
        ndt = np.float32 if kind in "sc" else np.float64
        st["xyz"] = np.random.default_rng(seed).random(3) * 0.999
        st["out"] = tuple(np.zeros(n * ncomp * m, ndt) for m in ((1, 3, 9) if case["form"] == "vgh" else (1,)))
        return st
    if op == "flat":
        st["pos"] = _points(case, seed, case["npts"], torch.float64)
        vgh = case["form"] == "vgh"
        shp = sp.out_shapes(case["npts"], 0)
        st["out"] = tuple(torch.empty(x, dtype=dt, device=DEV) if i == 0 or vgh else None for i, x in enumerate(shp))
        return st
    if op == "ptrs":
        P = case["npts"]
        st["handle"] = sp.to_cuda()
        st["spline"] = None  # the device handle has its own table
        sp.destroy()
        st["pos"] = _points(case, seed, P, dt)
        per = {"vgh": (1, 3, 6), "vgl": (1, 4), "value": (1,)}[case["form"]]
        st["out"] = tuple(torch.empty((P, m * n * ncomp), dtype=dt, device=DEV) for m in per)
        st["ptrs"] = tuple(_ptr_array(o, P) for o in st["out"])
        st["linv"] = _lattice(seed, dt)
        return st
    # ratio
    W = case["walkers"]
    g = _gen(seed, 3)
    # as much memory as W inverses of the leading dimension take; the ratio
    # reads one column (or row) of each
    inv = torch.empty((W, n, n), dtype=torch.float32, device=DEV)
    for w0 in range(0, W, 256):
        inv[w0:w0 + 256].normal_(0.0, 0.5 / n, generator=g).add_(1.0 / n)
    st["det"] = api.Determinants(inv, inv, n, case["trans"])
    st["rows"] = torch.empty((W, n), dtype=torch.float32, device=DEV)
    st["pos"] = _points(case, seed, W, torch.float32)
    st["k"] = n // 3
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "flat":
        return st["spline"].eval(st["pos"], vgh=case["form"] == "vgh", sort=case["sort"], out=st["out"])
    if op == "point":
        x, y, z = (float(v) for v in st["xyz"])
        bufs = [o.ctypes.data for o in st["out"]]
        suffix = "_vgh" if case["form"] == "vgh" else ""
        getattr(L.load(), "eval_multi_UBspline_3d_%s%s" % (case["kind"], suffix))(st["spline"].ptr, x, y, z, *bufs)
        L.check()
        return st["out"]
    if op == "ptrs":
        P, h = case["npts"], st["handle"]
        suffix = {"vgh": "_vgh", "vgl": "_vgl", "value": ""}[case["form"]]
        f = getattr(L.load(), "eval_multi_multi_UBspline_3d_%s%s_cuda" % (case["kind"], suffix))
        ptrs = [_ptr(p) for p in st["ptrs"]]
        if case["form"] == "vgl":
            f(h.ptr, _ptr(st["pos"]), _ptr(st["linv"]), *ptrs, P, case["n"])
        else:
            f(h.ptr, _ptr(st["pos"]), *ptrs, P)
        L.check()
        return st["out"]
    if op == "ratio":
        r, gr, lap = st["det"].ratio(st["spline"], st["pos"], st["k"], grad_lapl=True, rows=st["rows"])
        return r, gr, lap, st["rows"]
    if op == "update":
        st["det"].update(st["k"], st["accepted"], st["rows"])
        return st["det"].A, st["det"].ainv
    st["spline"].set_device(0, st["data"])
    st["spline"].flush()
    return st["table"]


def work(case):
    op, n = case["op"], case["n"]
    if op == "update":
        W = case["walkers"]
        # the inverse read and written, the row of A read and written, the new row read
        return {"bytes": W * 4.0 * (2 * n * n + 3 * n), "flops": 4.0 * W * n * n}
    ncomp = 2 if case["kind"] in "cz" else 1
    es = ELEM[case["store"]]
    es = es[case["kind"]] if isinstance(es, dict) else es
    acc = 4 if case["kind"] in "sc" else 8
    cyc = case["bc"] in ("periodic", "antiperiodic")
    cells = math.prod(case[a] + (3 if cyc else 2) for a in ("gx", "gy", "gz"))
    pts = math.prod(case[a] for a in ("gx", "gy", "gz"))
    cols = n * ncomp
    if op == "solve":
        # two multiply-adds a coefficient and axis (forward, back)
        return {"bytes": float(cols) * (pts * acc + cells * es), "flops": 12.0 * cols * cells}
    P = case["walkers"] if op == "ratio" else 1 if op == "point" else case["npts"]
    rows = min(64 * P, cells)
    if op == "ratio":
        return {"bytes": cols * (rows * es + P * 4.0 * 2) + P * (12 + 20.0), "flops": 2.0 * P * cols * (64 + 48 + 20 + 5)}
    outs = {"value": 1, "vgl": 5, "vgh": 13 if op == "point" else 10}[case["form"]]
    fma = 84 if case["form"] == "value" else 328
    return {"bytes": float(cols) * (rows * es + P * outs * acc) + 24.0 * P, "flops": 2.0 * fma * P * cols}


# ------------------------------------------------------- 64-bit evaluation
def _axis_matrix(M, bc):
    """Coefficients from data along one axis, [coefficients, M]."""
    d = float(M if bc in ("periodic", "antiperiodic") else M - 1)  # 1 / spacing
    if bc in ("periodic", "antiperiodic"):
        s = 1.0 if bc == "periodic" else -1.0
        A = np.zeros((M, M))
        # data i = (c_i + 4 c_{i+1} + c_{i+2}) / 6; unknowns u_i = c_{i+1}
        for i in range(M):
            A[i, i] += 4.0 / 6.0
            A[i, (i - 1) % M] += (1.0 if i > 0 else s) / 6.0
            A[i, (i + 1) % M] += (1.0 if i < M - 1 else s) / 6.0
        U = np.linalg.inv(A)
        return np.concatenate([s * U[M - 1:], U, s * U[:2]], axis=0)
    A = np.zeros((M + 2, M + 2))
    for i in range(M):
        A[i + 1, i:i + 3] = np.array([1.0, 4.0, 1.0]) / 6.0
    edge = np.array([-0.5, 0.0, 0.5]) * d if bc == "flat" else np.array([1.0, -2.0, 1.0]) * d * d
    A[0, :3] = edge
    A[M + 1, M - 1:] = edge
    return np.linalg.inv(A)[:, 1:M + 1]


def _exact_coefs(case, data):
    """FP64 coefficients [Nx, Ny, Nz, columns] of data [columns', gx, gy, gz(, 2)]."""
    d = data.double()
    if d.dim() == 5:
        d = d.permute(0, 4, 1, 2, 3).reshape(-1, *d.shape[1:4])
    for axis, a in enumerate(("gx", "gy", "gz")):
        m = torch.from_numpy(_axis_matrix(case[a], case["bc"])).to(DEV)
        d = torch.movedim(torch.matmul(torch.movedim(d, axis + 1, -1), m.T), -1, axis + 1)
    return torch.movedim(d, 0, -1).contiguous()


def _basis(t):
    v = torch.stack([(1 - t) ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6,
                     t ** 3 / 6], -1)
    g = torch.stack([-(1 - t) ** 2 / 2, (3 * t ** 2 - 4 * t) / 2, (-3 * t ** 2 + 2 * t + 1) / 2, t ** 2 / 2], -1)
    h = torch.stack([1 - t, 3 * t - 2, 1 - 3 * t, t], -1)
    return v, g, h


def _exact_eval(case, data, pos, nout):
    """FP64 value, gradient and Hessian of every column: [P, columns, nout] in
    the order v, x, y, z, xx, xy, xz, yy, yz, zz."""
    cyc = case["bc"] in ("periodic", "antiperiodic")
    P = pos.shape[0]
    B, idx = [], []
    for axis, a in enumerate(("gx", "gy", "gz")):
        d = float(case[a] if cyc else case[a] - 1)
        u = pos[:, axis].double() * d
        i = u.floor().clamp(0, case[a] - 1 if cyc else case[a] - 2)
        v, g, h = _basis(u - i)
        B.append((v, g * d, h * d * d))
        idx.append(i.long())
    order = ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2))
    cols = case["n"] * (2 if case["kind"] in "cz" else 1)
    out = torch.empty((P, cols, nout), dtype=torch.float64, device=DEV)
    off = torch.arange(4, device=DEV)
    ncomp = 2 if case["kind"] in "cz" else 1
    for s0 in range(0, case["n"], 32):
        c = _exact_coefs(case, data[s0:s0 + 32])
        ny, nz = c.shape[1], c.shape[2]
        flat = c.reshape(-1, c.shape[3])
        for p0 in range(0, P, 16384):
            sl = slice(p0, min(P, p0 + 16384))
            r = (((idx[0][sl, None] + off)[:, :, None, None] * ny + (idx[1][sl, None] + off)[:, None, :, None]) * nz
                 + (idx[2][sl, None] + off)[:, None, None, :]).reshape(-1, 64)
            w = torch.stack([(B[0][q[0]][sl][:, :, None, None] * B[1][q[1]][sl][:, None, :, None]
                              * B[2][q[2]][sl][:, None, None, :]).reshape(-1, 64) for q in order[:nout]], -1)
            out[sl, s0 * ncomp:s0 * ncomp + flat.shape[1]] = torch.matmul(flat[r].transpose(1, 2), w)
    return out


def exact(case, seed):
    op, n = case["op"], case["n"]
    if op == "update":
        A, B, rows, k = _update_inputs(case, seed)
        A2, B2 = A.double(), B.double()
        if case["trans"]:
            B2 = B2.transpose(1, 2)
        x = torch.matmul((rows.double() - A2[:, k, :])[:, None, :], B2)          # [W, 1, n]
        colk = B2[:, :, k:k + 1].clone()
        B2 = B2 - colk * (x / (1.0 + x[:, :, k:k + 1]))
        A2[:, k, :] = rows.double()
        return A2, B2.transpose(1, 2).contiguous() if case["trans"] else B2
    data = _grid_data(case, seed)
    if op == "solve":
        c = torch.cat([_exact_coefs(case, data[s0:s0 + 64]) for s0 in range(0, n, 64)], -1)
        per_row = 128 // (4 if case["kind"] in "sc" else 8)  # rows are padded to 128 bytes with zeros
        pad = -c.shape[-1] % per_row
        return torch.nn.functional.pad(c, (0, pad))
    kind = case["kind"]
    ncomp = 2 if kind in "cz" else 1
    if op == "ratio":
        W, k = case["walkers"], n // 3
        g = _gen(seed, 3)
        col = torch.empty((W, n), dtype=torch.float64, device=DEV)
        for w0 in range(0, W, 256):
            inv = torch.empty((min(256, W - w0), n, n), dtype=torch.float32, device=DEV)
            inv.normal_(0.0, 0.5 / n, generator=g).add_(1.0 / n)
            col[w0:w0 + 256] = (inv[:, k, :] if case["trans"] else inv[:, :, k]).double()
        e = _exact_eval(case, data, _points(case, seed, W, torch.float32), 10)
        s = (e * col[:, :, None]).sum(1)
        return (s[:, 0], s[:, 1:4] / s[:, :1], (s[:, 4] + s[:, 7] + s[:, 9]) / s[:, 0], e[:, :, 0].contiguous())
    if op == "point":
        xyz = np.random.default_rng(seed).random(3) * 0.999
        vgh = case["form"] == "vgh"
        e = _exact_eval(case, data, torch.from_numpy(xyz[None]).to(DEV), 10 if vgh else 1)[0]
        if not vgh:
            return (e[:, 0].cpu().numpy(),)
        # CPU layout: the components of a complex entry side by side
        e = e.reshape(n, ncomp, 10)
        full = e[:, :, [4, 5, 6, 5, 7, 8, 6, 8, 9]]
        return tuple(x.transpose(1, 2).reshape(-1).contiguous().cpu().numpy() for x in (e[:, :, :1], e[:, :, 1:4], full))
    dt = torch.float64 if op == "flat" or kind in "dz" else torch.float32
    P = case["npts"]
    e = _exact_eval(case, data, _points(case, seed, P, dt), 1 if case["form"] == "value" else 10)
    val = e[:, :, 0].contiguous()
    if op == "flat":
        ext = (2,) if ncomp == 2 else ()
        val = val.reshape((P, n) + ext)
        if case["form"] == "value":
            return val, None, None
        return val, e[:, :, 1:4].reshape((P, n) + ext + (3,)), e[:, :, 4:].reshape((P, n) + ext + (6,))
    if case["form"] == "value":
        return (val,)
    if case["form"] == "vgh":
        return val, e[:, :, 1:4].reshape(P, -1), e[:, :, 4:].reshape(P, -1)
    G = _lattice(seed, torch.float32 if kind in "sc" else torch.float64).double()
    grad = torch.einsum("rc,pnc->prn", G, e[:, :, 1:4])
    GG = G.T @ G
    H = e[:, :, 4:][:, :, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(P, -1, 3, 3)
    lap = torch.einsum("ab,pnab->pn", GG, H)
    return val, torch.cat([grad, lap[:, None, :]], 1).reshape(P, -1)
