"""Performance cases of the matrix powers kernel: what a program that uses
the library has it do, through the Python mirror of the C API.

A pass is one exec call on a plan the program keeps, with a new x in level 0
of its basis buffer (or, for the solver, one whole solve).  The plans keep
the matrix on the GPU, as a program that calls them many times does.

The matrices are built here in numpy, so that `exact` needs nothing of the
library: 5/7-point Laplacians, 7/9-point variable-coefficient diffusion
(log-normal edge coefficients, symmetric, weakly diagonally dominant) and
random banded operators, the kinds of the repository's benchmark.
"""
import numpy as np
import torch

import mpk_gb300 as M
from mpk_gb300 import shifts as S

_ARITH = {"fma": M.ARITH_FMA, "separate": M.ARITH_SEPARATE, "df64": M.ARITH_DF64}
_VALUE = {"f32": M.VALUE_F32, "bf16": M.VALUE_BF16}
_BATCH = {"default": M.BATCH_DEFAULT, "staged": M.BATCH_STAGED, "staged2": M.BATCH_STAGED2,
          "staged4": M.BATCH_STAGED4}
_stream = None


def stream():
    """The program's own stream: every device exec call goes to it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


# ---------------------------------------------------------------- cases
def listed():
    return [
        # The smallest ordinary call: the reference's 1/deg operator on a
        # 100 x 100 mesh, 4 powers, which launches and waits dominate.
        dict(name="deg_mesh_100", kind="wave", op="deg", arith="fma", nx=100, ny=100, nz=1, k=4),
        # The repository's headline workload: 128^3, 8 powers, bit-exact FP64.
        dict(name="deg_cube_128", kind="wave", op="deg", arith="fma", nx=128, ny=128, nz=128, k=8),
        # A valued operator of odd sizes: 9-point diffusion in FP64.
        dict(name="val_diff9_1023x769", kind="wave", op="diff", arith="fma", nx=1023, ny=769, nz=1, k=5),
        # Double-float rows, the fast form that is not bit-exact, odd 3-D box.
        dict(name="df64_box_101x97x89", kind="wave", op="deg", arith="df64", nx=101, ny=97, nz=89, k=8),
        # The chain of separate SpMVs (verify_val's gold), the x86 rounding.
        dict(name="spmv_diff7_97x96x95", kind="spmv", op="diff", arith="separate", nx=97, ny=96, nz=95, k=6),
        # Mixed precision on a 3-D operator whose values stay in L2.
        dict(name="mixed_f32_box_120x110x100", kind="mixed", op="diff", value="f32", nx=120, ny=110, nz=100, k=8),
        # ... and in BF16 on a ragged 2-D mesh with few powers.
        dict(name="mixed_bf16_701x699", kind="mixed", op="diff", value="bf16", nx=701, ny=699, nz=1, k=4),
        # Temporal blocking on PA1 tiles, for 2-D operators of many values.
        dict(name="tiles_f32_1400x1300", kind="tiles", op="diff", value="f32", nx=1400, ny=1300, nz=1, k=8),
        # Many matrices x 16 right-hand sides (stencils and random banded), in
        # the configuration the autotuner finds for them, fixed, as a program
        # that makes a plan per set of matrices has it.
        dict(name="batch_48x16", kind="batch", mode="staged4", count=48, nmin=1000, nmax=30000, nrhs=16, k=6),
        # The same at its smallest: a handful of little matrices, 4 sides,
        # the untimed default configuration.
        dict(name="batch_6x4", kind="batch", mode="default", count=6, nmin=300, nmax=3000, nrhs=4, k=4),
        # A whole solve from host arrays: s-step CG on 3-D diffusion, to the
        # accuracy that the FP64 Gram and residual are there for.
        dict(name="sstep_64", kind="sstep", op="diff", nx=64, ny=64, nz=64, s=8),
        # The host call: x and every power in the program's own numpy array.
        dict(name="host_deg_cube_64", kind="host", op="deg", arith="fma", nx=64, ny=64, nz=64, k=8),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _dims(rng, nlo, nhi, three):
    """A box of about n cells, n log-uniform, sides within 20 % of each other."""
    n = _log(rng, nlo, nhi)
    if three:
        s = n ** (1 / 3)
        nx, ny = (max(4, round(s * rng.uniform(0.9, 1.1))) for _ in range(2))
        return nx, ny, max(4, round(n / (nx * ny)))
    nx = max(4, round(n ** 0.5 * rng.uniform(0.85, 1.15)))
    return nx, max(4, round(n / nx)), 1


def draw(rng):
    kind = rng.choice(["wave", "wave", "wave", "spmv", "mixed", "mixed", "tiles", "batch", "batch", "sstep", "host"])
    if kind == "batch":
        nmax = round(_log(rng, 2000, 30000))
        return dict(kind=kind, mode=rng.choice(list(_BATCH)), count=rng.randint(4, 48), nmin=rng.randint(300, 1000),
                    nmax=nmax,
                    nrhs=rng.choice([4, 8, 16, 32]) if nmax < 12000 else rng.choice([4, 8, 16]), k=rng.randint(2, 6))
    three = rng.random() < 0.5
    k = rng.randint(2, 8)
    if kind == "sstep":
        nx, ny, nz = _dims(rng, 30000, 260000, three)
        return dict(kind=kind, op="diff", nx=nx, ny=ny, nz=nz, s=rng.choice([6, 8]))
    if kind == "tiles":
        nx, ny, nz = _dims(rng, 300000, 1.8e6, False)
        return dict(kind=kind, op="diff", value=rng.choice(["f32", "bf16"]), nx=nx, ny=ny, nz=nz, k=rng.randint(4, 8))
    if kind == "mixed":
        nx, ny, nz = _dims(rng, 10000, 1.3e6, three)
        return dict(kind=kind, op="diff", value=rng.choice(["f32", "bf16"]), nx=nx, ny=ny, nz=nz, k=k)
    if kind == "host":
        nx, ny, nz = _dims(rng, 10000, 260000, three)
        return dict(kind=kind, op="deg", arith=rng.choice(["fma", "separate"]), nx=nx, ny=ny, nz=nz, k=k)
    op = rng.choice(["deg", "diff"])
    nx, ny, nz = _dims(rng, 10000, 1.5e6 if op == "deg" else 900000, three)
    arith = rng.choice(["fma", "fma", "separate", "df64"]) if kind == "wave" else rng.choice(["fma", "separate"])
    return dict(kind=kind, op=op, arith=arith, nx=nx, ny=ny, nz=nz, k=k)


# ---------------------------------------------------------------- matrices
def _mesh(nx, ny, nz, nine, val=None):
    """CSR of a (2d+1)-point (nine: 9-point, 2-D) mesh operator, ascending
    columns.  val(offset, mask) gives the values of one diagonal."""
    n = nx * ny * nz
    i = np.arange(n, dtype=np.int32)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    if nine:
        d = [(dx, dy, 0) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    elif nz == 1:
        d = [(0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0)]
    else:
        d = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    ok = np.empty((n, len(d)), dtype=bool)
    col = np.empty((n, len(d)), dtype=np.int32)
    for t, (dx, dy, dz) in enumerate(d):
        m = np.ones(n, dtype=bool)
        if dx:
            m &= (x + dx >= 0) & (x + dx < nx)
        if dy:
            m &= (y + dy >= 0) & (y + dy < ny)
        if dz:
            m &= (z + dz >= 0) & (z + dz < nz)
        ok[:, t] = m
        col[:, t] = i + (dx + nx * (dy + ny * dz))
    ptr = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(ok.sum(axis=1), out=ptr[1:])
    if val is None:
        return ptr, col[ok], None
    # symmetric edge coefficients: one log-normal number per edge, stored
    # at the edge's lower cell; diagonal = sum of the row's edges * 1.01
    v = np.zeros((n, len(d)))
    mid = len(d) // 2
    for t in range(mid + 1, len(d)):
        dx, dy, dz = d[t]
        o = dx + nx * (dy + ny * dz)
        c = -val.lognormal(0.0, 1.0, n)
        m = ok[:, t]
        v[m, t] = c[m]
        back = np.flatnonzero(m) + o
        v[back, len(d) - 1 - t] = c[m]
    v[:, mid] = -1.01 * v.sum(axis=1)
    return ptr, col[ok], v[ok]


def _matrix(case, seed):
    if case["op"] == "deg":
        return _mesh(case["nx"], case["ny"], case["nz"], False)
    return _mesh(case["nx"], case["ny"], case["nz"], case["nz"] == 1, np.random.default_rng(seed))


def _banded(n, rng):
    """Random banded rows: about 5 to 30 entries within 64 of the diagonal."""
    p = rng.uniform(5.0, 30.0, (n, 1)).astype(np.float32) / 129
    ok = rng.random((n, 129), dtype=np.float32) < p
    off = np.arange(-64, 65, dtype=np.int32)
    i = np.arange(n, dtype=np.int32)[:, None]
    col = i + off
    ok &= (col >= 0) & (col < n)
    ok[:, 64] = True
    ptr = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(ok.sum(axis=1), out=ptr[1:])
    val = rng.normal(size=int(ptr[-1])) * 0.2
    val[np.flatnonzero((col == i)[ok])] = 1.0
    return ptr, col[ok], val


def _batch(case, seed):
    """The sizes and kinds are the case's, the values the seed's."""
    shape = np.random.default_rng(case["count"] * 1000003 + case["nmax"])
    rng = np.random.default_rng(seed)
    mats = []
    for m in range(case["count"]):
        n = int(np.exp(shape.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        three = shape.random() < 0.25
        if m % 2:
            mats.append(_banded(n, rng))
            continue
        s = max(2, round(n ** (1 / 3 if three else 1 / 2)))
        ptr, col, val = _mesh(s, s, max(2, n // (s * s)) if three else 1, not three, rng)
        mats.append((ptr, col, val * 0.1))
    return mats


def _batch_rows(case):
    shape = np.random.default_rng(case["count"] * 1000003 + case["nmax"])
    rows, nnz = 0, 0.0
    for m in range(case["count"]):
        n = int(np.exp(shape.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        three = shape.random() < 0.25
        if m % 2:
            rows, nnz = rows + n, nnz + 18.4 * n
            continue
        s = max(2, round(n ** (1 / 3 if three else 1 / 2)))
        z = max(2, n // (s * s)) if three else 1
        rows += s * s * z
        nnz += (7 * s * s * z - 4 * s * z - 2 * s * s) if three else (3 * s - 2) ** 2
    return rows, nnz


def _nnz(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if nz == 1 and case["op"] == "diff":
        return (3 * nx - 2) * (3 * ny - 2)
    return n + 2 * (3 * n - ny * nz - nx * nz - nx * ny) if nz > 1 else n + 2 * (2 * n - nx - ny)


def _x(case, seed, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, dtype=dtype, device="cuda", generator=g) * 2 - 1


def _host_x(seed, n):
    return np.random.default_rng(seed + 1).uniform(-1.0, 1.0, n)


# ---------------------------------------------------------------- a pass
def prepare(case, seed):
    kind, k = case["kind"], case.get("k")
    if kind == "batch":
        mats = _batch(case, seed)
        plan = M.Plan.batch([M.Csr(*m) for m in mats], case["nrhs"], k, tune=_BATCH[case["mode"]])
        vb = torch.zeros((k + 1, plan.n, case["nrhs"]), dtype=torch.float32, device="cuda")
        vb[0] = _x(case, seed, vb[0].numel(), torch.float32).view(plan.n, case["nrhs"])
        torch.cuda.synchronize()
        return dict(kind=kind, plan=plan, vv=vb)
    ptr, col, val = _matrix(case, seed)
    a = M.Csr(ptr, col, val)
    if kind == "sstep":
        b = _host_x(seed, a.n)
        return dict(kind=kind, a=a, b=b, s=case["s"], shifts=S.from_lanczos(a, case["s"]))
    if kind in ("mixed", "tiles"):
        if kind == "mixed":
            plan = M.Plan.mixed(a, k, _VALUE[case["value"]])
        else:
            nx, ny = case["nx"], case["ny"]
            i = np.arange(a.n, dtype=np.int32)
            npart = -(-a.n // 1024)
            part = M.partition_rcb(np.stack([i % nx, i // nx], axis=1), npart)
            plan = M.Plan.mixed_tiles(a, part, npart, k, _VALUE[case["value"]])
        vv = torch.zeros((k + 1, a.n), dtype=torch.float32, device="cuda")
    else:
        make = M.Plan.spmv if kind == "spmv" else M.Plan.wave
        plan = make(a, k, arith=_ARITH[case["arith"]])
        if kind == "host":
            vv = np.zeros((k + 1) * a.n)
            vv[:a.n] = _host_x(seed, a.n)
            return dict(kind=kind, plan=plan, vv=vv)
        vv = torch.zeros((k + 1, a.n), dtype=torch.float64, device="cuda")
    vv[0] = _x(case, seed, a.n, vv.dtype)
    torch.cuda.synchronize()
    return dict(kind=kind, plan=plan, vv=vv)


def run(state):
    kind = state["kind"]
    if kind == "sstep":
        x, _ = M.sstep_cg(state["a"], state["b"], state["s"], shifts=state["shifts"], tol=1e-11)
        return x
    plan, vv = state["plan"], state["vv"]
    if kind == "host":
        return plan.exec_host(vv)[plan.n:]
    if kind == "batch":
        plan.exec_batch_device(vv.data_ptr(), stream())
    elif kind in ("mixed", "tiles"):
        plan.exec_mixed_device(vv.data_ptr(), stream())
    else:
        plan.exec_device(vv.data_ptr(), stream())
    return vv[1:]


def work(case):
    """The matrix once, x once, every power once.  The solver: its matrix,
    b and x once over the host link, and the solve's vectors and matrix
    read once per iteration (78 outer iterations of s steps)."""
    kind, k = case["kind"], case.get("k", 0)
    if kind == "batch":
        rows, nnz = _batch_rows(case)
        return dict(bytes=8 * nnz + 4 * rows + 4 * rows * case["nrhs"] * (k + 1), flops=2 * nnz * case["nrhs"] * k)
    n, nnz = case["nx"] * case["ny"] * case["nz"], _nnz(case)
    if kind == "sstep":
        s = case["s"]
        m = 2 * s + 1
        per = 8 * nnz + 4 * n * m + 8 * n * 6 + 12 * nnz
        return dict(bytes=78 * per, flops=78 * (2 * nnz * (2 * s - 1) + 2 * n * m * (m + 1) / 2 + 4 * n * m + 2 * nnz))
    entry = 4 if case["op"] == "deg" else 4 + (8 if "arith" in case else 4 if case["value"] == "f32" else 2)
    vec = 8 if "arith" in case else 4
    return dict(bytes=entry * nnz + 4 * (n + 1) + vec * n * (k + 1), flops=2 * nnz * k)


# ---------------------------------------------------------------- 64 bits
def _sparse(ptr, col, val):
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (ptr, col, val)]
    n = len(ptr) - 1
    return torch.sparse_csr_tensor(t[0].long(), t[1].long(), t[2], size=(n, n))


def exact(case, seed):
    kind, k = case["kind"], case.get("k")
    if kind == "batch":
        mats = _batch(case, seed)
        N = sum(len(m[0]) - 1 for m in mats)
        X = _x(case, seed, N * case["nrhs"], torch.float32).view(N, case["nrhs"]).double()
        out = torch.empty((k,) + X.shape, dtype=torch.float64, device="cuda")
        r = 0
        for ptr, col, val in mats:
            A = _sparse(ptr, col, val.astype(np.float32).astype(np.float64))
            v = X[r:r + len(ptr) - 1]
            for l in range(k):
                v = A @ v
                out[l, r:r + len(ptr) - 1] = v
            r += len(ptr) - 1
        return out
    ptr, col, val = _matrix(case, seed)
    n = len(ptr) - 1
    if val is None:
        val = np.repeat(1.0 / np.diff(ptr), np.diff(ptr))
    A = _sparse(ptr, col, val)
    if kind == "sstep":
        b = torch.from_numpy(_host_x(seed, n)).cuda()
        x, r = torch.zeros_like(b), b.clone()
        p, rr, bb = r.clone(), b @ b, float(b @ b)
        for it in range(4000):  # textbook CG to the end of 64 bits
            q = A @ p
            a = rr / (p @ q)
            x += a * p
            r -= a * q
            new = r @ r
            p = r + (new / rr) * p
            rr = new
            if it % 50 == 0 and float(rr) < 1e-28 * bb:
                break
        return x.cpu().numpy()
    if kind in ("mixed", "tiles"):
        e = int(np.ceil(np.log2(np.add.reduceat(np.abs(val), ptr[:-1]).max())))
        v, scale = _x(case, seed, n, torch.float32).double(), 2.0 ** -e
    elif kind == "host":
        v, scale = torch.from_numpy(_host_x(seed, n)).cuda(), 1.0
    else:
        v, scale = _x(case, seed, n, torch.float64), 1.0
    out = torch.empty((k, n), dtype=torch.float64, device="cuda")
    for l in range(k):
        v = (A @ v) * scale
        out[l] = v
    return out.view(-1).cpu().numpy() if kind == "host" else out
