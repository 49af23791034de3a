"""The work this framework is used for, as a list of timed cases.

A reconstruction with it is: rows of the system matrix from the scanner's
geometry (`Context.build`), its transpose, and MLEM over the rows or through
the transpose, in FP32, with the matrix in FP16, or for a batch of frames; or
the whole of it in one call from host buffers (`reco_host`).  Programs that
keep the reference's own loop call the candidate search and the two SpMV
directions instead.  Every one of these has its listed cases, over the three
scanner grids of the configuration (40^3, 70^3 and 100^3 voxels).

The builds get the geometry itself.  The passes over a matrix get rows of the
same shape made here (tubes of voxels around the lines of consecutive
channels of a few views), so that their results can be computed in 64 bits
without the framework.
"""
import ctypes
import math

import numpy as np
import torch

import raptr_b200 as R

DEV = "cuda"
GRIDS = {40: R.SMALL, 70: R.FULL, 100: R.FINE}
NAT = 13 ** 4  # channels of one view (two heads of 13 x 13 crystals)


# ---- cases -------------------------------------------------------------------


def listed():
    return [
        # rows of a handful of measured channels on the small scanner: the
        # latency of a build, as a program that refreshes a few rows sees it
        dict(name="build_few_rows_40", kind="build", grid=40, rows=500, nrays=100),
        # the build that dominates a reconstruction: rows from all views of
        # the full scanner, 1000 rays each
        dict(name="build_70", kind="build", grid=70, rows=60000, nrays=1000),
        # the fine grid, an odd number of rows and rays
        dict(name="build_100", kind="build", grid=100, rows=12345, nrays=999),
        # the reference's getWorkqueue: a chunk of the candidates of a channel list
        dict(name="candidates_70", kind="candidates", grid=70, rows=3001),
        # CSR -> CSC in back-projection order before gather MLEM: 7 views
        dict(name="transpose_70", kind="transpose", grid=70, rows=7 * NAT),
        # one forward projection of one view of the small scanner, a matrix
        # that stays in L2: launch latency and the row loop
        dict(name="forward_40", kind="spmv", grid=40, rows=NAT, op=R.OP_N),
        # the back projection of the reference's loop (transposed SpMV over
        # the rows, no transpose kept), an odd number of rows
        dict(name="back_70", kind="spmv", grid=70, rows=100001, op=R.OP_T),
        # the small workload's MLEM as the reference runs it, over the rows
        dict(name="mlem_rows_40", kind="mlem", form="rows", grid=40, rows=5 * NAT, iters=20),
        # MLEM through the transpose, FP32: the resident iterations of a
        # reconstruction on the full grid
        dict(name="mlem_70", kind="mlem", form="gather", grid=70, rows=7 * NAT, iters=8),
        # the same with the matrix in FP16
        dict(name="mlem_half_70", kind="mlem", form="half", grid=70, rows=7 * NAT, iters=8),
        # 64 frames that share the FP16 matrix, as a dynamic series or the
        # serving loop's full batches
        dict(name="mlem_batch64_70", kind="mlem", form="batch", grid=70, rows=2 * NAT, iters=2, frames=64),
        # the whole small reconstruction in one call from host buffers
        dict(name="reco_host_40", kind="reco", grid=40, nrays=100, iters=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges, sizes spread over their logarithm."""
    kind = rng.choice(["build", "build", "build", "candidates", "transpose", "spmv", "spmv", "mlem", "mlem", "mlem",
                       "mlem", "reco"])
    grid = rng.choice([40, 70, 100])
    if kind == "build":
        nrays = _log(rng, 64, 1000)
        most = min(60000, int(60e6 * 70 / (nrays * grid)))
        if grid == 100:
            most = min(most, 30000)
        return dict(kind=kind, grid=grid, rows=_log(rng, 300, most), nrays=nrays)
    if kind == "candidates":
        return dict(kind=kind, grid=grid, rows=_log(rng, 100, {40: 3001, 70: 3001, 100: 1000}[grid]))
    most = {40: 5 * NAT, 70: 7 * NAT, 100: 2 * NAT}[grid]
    if kind == "transpose":
        return dict(kind=kind, grid=grid, rows=_log(rng, 2000, most))
    if kind == "spmv":
        return dict(kind=kind, grid=grid, rows=_log(rng, 500, most), op=rng.choice([R.OP_N, R.OP_T]))
    if kind == "mlem":
        form = rng.choice(["rows", "gather", "half", "batch"])
        rows, iters = _log(rng, 1000, most), rng.randint(1, 8)
        if form == "batch":
            frames = 4 * rng.randint(1, 16)
            rows = min(rows, 2 * NAT if grid == 70 else (NAT // 2 if grid == 100 else 3 * NAT))
            return dict(kind=kind, form=form, grid=grid, rows=rows, iters=rng.randint(1, 2), frames=frames)
        return dict(kind=kind, form=form, grid=grid, rows=rows, iters=iters)
    return dict(kind="reco", grid=40, nrays=rng.randint(40, 100), iters=rng.randint(2, 20))


# ---- inputs ------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _measured(g, rows, seed):
    """A sorted list of distinct channels spread over all views."""
    rng = np.random.Generator(np.random.PCG64(seed))
    step = g.n_channels / rows
    ids = np.floor((np.arange(rows) + rng.random(rows)) * step).astype(np.int64)
    return torch.from_numpy(np.minimum(ids, g.n_channels - 1).astype(np.int32)).to(DEV)


def _activity(g):
    """Background 0.1 with a warm and a hot sphere."""
    n, p = g.grid_n[0], g.grid_d[0]
    a = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 - n / 2) * p
    X, Y, Z = torch.meshgrid(a, a, a, indexing="ij")
    x = torch.full((n, n, n), 0.1, device=DEV, dtype=torch.float64)
    x[X * X + Y * Y + Z * Z < 0.015 ** 2] = 1.0
    x[(X - 0.02) ** 2 + Y * Y + Z * Z < 0.008 ** 2] = 4.0
    return x.reshape(-1).float()


class Rows:
    """A system matrix that the program holds itself (CSR, and CSC in the
    back-projection order when asked for), with a measurement of it."""

    row_order = row_rank = col_ptr = row_idx = tval = hval = rscale = htval = pscale = None
    has_transpose = False

    def __init__(self, case, seed):
        g = GRIDS[case["grid"]]
        n, pitch, rows = g.grid_n[0], g.grid_d[0], case["rows"]
        gen = _gen(seed)
        act = _activity(g)
        views = min(-(-rows // NAT), g.na)
        chans, cols, vals, lens, lams = [], [], [], [], []
        for v in range(views):
            k = min(NAT, rows - v * NAT)
            cnl = int(v * g.na / views) * NAT + torch.arange(k, device=DEV)
            for lo in range(0, k, 14281):
                self._view(g, n, pitch, cnl[lo:lo + 14281], act, gen, cols, vals, lens, lams)
            chans.append(cnl)
        self.m, self.n = rows, n ** 3
        self.col, self.val = torch.cat(cols), torch.cat(vals)
        self.nnz = self.col.numel()
        self.row_ptr = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
        self.row_ptr[1:] = torch.cumsum(torch.cat(lens), 0)
        lam = torch.cat(lams)
        frames = case.get("frames", 1)
        # about 20 counts per channel, frame by frame a little different
        rate = (lam * (20.0 / lam.mean()))[:, None] * torch.linspace(0.7, 1.3, frames, device=DEV)
        self.y = torch.poisson(rate, generator=gen).contiguous()
        self._order(g, torch.cat(chans))

    @staticmethod
    def _view(g, n, pitch, cnl, act, gen, cols, vals, lens, lams):
        """Tubes of voxels around the channels' centre lines."""
        t = cnl % NAT
        i0z, i0y, i1z, i1y = t // 2197, t // 169 % 13, t // 13 % 13, t % 13
        a = math.radians(int(cnl[0]) // NAT * g.da)
        s, c = math.sin(a), math.cos(a)

        def centre(x, iz, iy):
            z = (iz - 6.0) * g.segz
            return torch.stack([c * x + s * z, (iy - 6.0) * g.segy, -s * x + c * z], 1)

        p, q = centre(g.pos0x, i0z, i0y), centre(g.pos1x, i1z, i1y)
        A = 0 if abs(c) >= abs(s) else 2
        axes = (1, 2) if A == 0 else (0, 1)
        slab = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 - n / 2) * pitch
        tt = (slab[None] - p[:, A:A + 1]) / (q - p)[:, A:A + 1]
        h = 0.0032 / pitch
        W = int(math.ceil(2 * h)) + 1
        cell, wgt = [], []
        for d in axes:
            f = ((p[:, d:d + 1] + tt * (q - p)[:, d:d + 1]) / pitch + n / 2).float()
            i = torch.floor(f - h + 0.5).int()[:, :, None] + torch.arange(W, device=DEV, dtype=torch.int32)
            w = 1 - (i + 0.5 - f[:, :, None]).abs() / h
            cell.append(i)
            wgt.append(torch.where((i >= 0) & (i < n), w, torch.zeros_like(w)).clamp_(min=0))
        iu, iv = cell[0][:, :, :, None], cell[1][:, :, None, :]
        ia = torch.arange(n, device=DEV, dtype=torch.int32)[None, :, None, None]
        col = (ia * n + iu) * n + iv if A == 0 else (iu * n + iv) * n + ia
        w = wgt[0][:, :, :, None] * wgt[1][:, :, None, :]
        w, col = w.reshape(len(cnl), -1), col.reshape(len(cnl), -1)
        keep = w > 1e-3
        w = w * (torch.rand(w.shape, device=DEV, generator=gen) * 0.8 + 0.6) * pitch
        lams.append((torch.where(keep, w, torch.zeros_like(w)) * act[torch.where(keep, col, 0)]).sum(1))
        lens.append(keep.sum(1))
        cc, ww = col[keep], w[keep]
        if A != 0:
            key = torch.repeat_interleave(torch.arange(len(cnl), device=DEV), lens[-1]) * n ** 3 + cc
            key, o = torch.sort(key)
            cc, ww = (key % n ** 3).int(), ww[o]
        cols.append(cc.int())
        vals.append(ww)

    def _order(self, g, cnl):
        """Back-projection order: view, then midpoint, then slope."""
        t = cnl % NAT
        z0, y0, z1, y1 = t // 2197, t // 169 % 13, t // 13 % 13, t % 13
        key = ((cnl // NAT * 32 + z0 + z1) * 32 + y0 + y1) * 1024 + (z0 - z1 + 13) * 32 + y0 - y1 + 13
        self.order = torch.argsort(key).int()
        self.rank = torch.empty_like(self.order)
        self.rank[self.order.long()] = torch.arange(self.m, device=DEV, dtype=torch.int32)

    def rows(self):
        return torch.repeat_interleave(torch.arange(self.m, device=DEV, dtype=torch.int32),
                                       self.row_ptr[1:] - self.row_ptr[:-1])

    def transpose(self):
        """CSC with row positions ascending in every column."""
        key = self.col.long() * 2 ** 23 + self.rank[self.rows().long()]
        key, self.perm = torch.sort(key)
        self.col_ptr = torch.searchsorted(key, torch.arange(self.n + 1, device=DEV) * 2 ** 23)
        self.row_idx = (key % 2 ** 23).int()
        self.tval = self.val[self.perm]
        self.row_order, self.row_rank, self.has_transpose = self.order, self.rank, True
        return self

    def half(self):
        """Values as rscale_i * h_ij, h in binary16."""
        row = self.rows().long()
        top = torch.zeros(self.m, device=DEV).scatter_reduce_(0, row, self.val, "amax")
        self.rscale = torch.where(top > 0, top * 2.0 ** -15, torch.ones_like(top))
        self.hval = (self.val / self.rscale[row]).half()
        self.htval = self.hval[self.perm]
        self.pscale = self.rscale[self.order.long()]
        return self

    def sensitivity(self):
        """Column sums normalised to sum 1 (summed as whole numbers, so that
        every preparation gets the same bits)."""
        s = torch.zeros(self.n, dtype=torch.int64, device=DEV)
        s.index_add_(0, self.col, (self.val.double() * 2.0 ** 44).long())
        return (s.double() / s.sum().double()).float()


def _matrix(case, seed):
    A = Rows(case, seed)
    if case.get("form") in ("gather", "half", "batch"):
        A.transpose()
    if case.get("form") in ("half", "batch"):
        A.half()
    return A


def prepare(case, seed):
    kind, g = case["kind"], GRIDS[case["grid"]]
    if kind == "reco":
        A = Rows(dict(case, rows=g.n_channels), seed)
        return dict(case=case, geom=g, seed=seed, y=A.y[:, 0].cpu().numpy())
    if kind in ("build", "candidates"):
        st = dict(case=case, ctx=R.Context(g), cnl=_measured(g, case["rows"], seed), seed=seed)
        if kind == "build":
            # the program's own matrix arrays, with room for the longest rows
            room = _room(case)
            st.update(rp=torch.zeros(case["rows"] + 1, dtype=torch.int64, device=DEV),
                      col=torch.zeros(room, dtype=torch.int32, device=DEV), val=torch.zeros(room, device=DEV))
        return st
    A = _matrix(case, seed)
    st = dict(case=case, A=A)
    if kind == "spmv":
        st["x"] = _activity(g) if case["op"] == R.OP_N else A.y[:, 0].contiguous()
    if kind == "mlem":
        frames = case.get("frames")
        st.update(ctx=R.Context(g), s=A.sensitivity(),
                  x0=torch.full((A.n, frames) if frames else (A.n,), 1.0 / A.n, device=DEV))
        st["y"] = A.y if frames else A.y[:, 0].contiguous()
    return st


# ---- one pass ----------------------------------------------------------------


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "build":
        status, _ = st["ctx"].build_into(st["cnl"], case["nrays"], st["seed"], st["rp"], st["col"], st["val"])
        if status != R.RAPTR_OK:
            raise RuntimeError("the matrix arrays are too small")
        return st["rp"], st["col"], st["val"]
    if kind == "candidates":
        # a chunk of the queue, as much as the program's arrays take
        most = int(0.75 * case["rows"] * _candidates(case["grid"]) / 1.2)
        cnl, vxl, _ = st["ctx"].workqueue(st["cnl"], max_out=most)
        return cnl, vxl
    if kind == "reco":
        return R.reco_host(st["geom"], st["y"], case["nrays"], st["seed"], case["iters"])[0]
    A = st["A"]
    if kind == "transpose":
        return R.csr_transpose_ordered(A.m, A.n, A.row_ptr, A.col, A.val, A.order)
    if kind == "spmv":
        return R.spmv(case["op"], A.m, A.n, A.row_ptr, A.col, A.val, st["x"])
    x = st["x0"].clone()
    form, ctx = case["form"], st["ctx"]
    if form == "half":
        ctx.mlem_half(A, st["y"], st["s"], x, case["iters"])
    elif form == "batch":
        ctx.mlem_batch(A, st["y"], st["s"], x, case["iters"])
    else:
        ctx.mlem(A, st["y"], st["s"], x, case["iters"])
    return x


# ---- what a pass cannot do without -------------------------------------------


def _per_row(grid):
    """Entries of a matrix row, on average (measured: 40^3 at 100 rays, 70^3
    and 100^3 at 1000 rays)."""
    return {40: 320, 70: 725, 100: 1535}[grid]


def _room(case):
    """Entries that the matrix arrays of a build have room for."""
    return int(1.6 * case["rows"] * _per_row(case["grid"]))


def _candidates(grid):
    """Voxels of a channel's enclosing cylinder: radius half the voxel's and
    the crystal's diagonals, up to 1.2 grid edges long."""
    p = GRIDS[grid].grid_d[0]
    r = 0.5 * (math.sqrt(3) * p + math.sqrt(0.020 ** 2 + 2 * 0.004 ** 2))
    return math.pi * r * r * 1.2 * grid * p / p ** 3


def work(case):
    kind, grid = case["kind"], case["grid"]
    N = grid ** 3
    if kind == "candidates":
        c = 0.75 * case["rows"] * _candidates(grid) / 1.2
        return dict(bytes=8 * c + 4 * case["rows"], flops=20 * c)
    if kind in ("build", "reco"):
        rows = case["rows"] if kind == "build" else GRIDS[grid].n_channels
        nnz = rows * _per_row(grid)
        # a crossing: the next plane's parameter, the length, its sum
        w = dict(bytes=8.0 * nnz + 12 * rows, flops=12.0 * rows * case["nrays"] * 1.35 * grid)
        if kind == "reco":
            w = dict(bytes=w["bytes"] + 16.0 * nnz * case["iters"], flops=w["flops"] + 4.0 * nnz * case["iters"])
        return w
    rows = case["rows"]
    nnz = rows * _per_row(grid)
    if kind == "transpose":
        return dict(bytes=16.0 * nnz + 8 * (rows + N) + 4 * rows, flops=0)
    if kind == "spmv":
        return dict(bytes=8.0 * nnz + 12 * rows + 4 * N, flops=2.0 * nnz)
    K, form = case.get("frames", 1), case["form"]
    per = {"rows": 8, "gather": 16, "half": 12, "batch": 12}[form]
    return dict(bytes=case["iters"] * (float(per) * nnz + 8 * rows * (K + 1) + 12 * N * K),
                flops=case["iters"] * 4.0 * nnz * K)


# ---- the same in 64 bits -----------------------------------------------------


def _csr64(ptr, idx, val, n):
    return torch.sparse_csr_tensor(ptr, idx.long(), val, size=(ptr.numel() - 1, n))


def exact(case, seed):
    kind = case["kind"]
    if kind == "build":
        planes = 3 * (case["grid"] + 1)
        if case["rows"] * case["nrays"] * planes > 4e9:
            return None  # minutes
        g = GRIDS[case["grid"]]
        val = _build64(g, _measured(g, case["rows"], seed), case["nrays"], seed)
        return None, None, torch.nn.functional.pad(val, (0, _room(case) - val.numel()))
    if kind in ("candidates", "reco"):
        return None  # whole numbers; a build of all channels
    A = _matrix(case, seed)
    if kind == "transpose":
        A.transpose()
        return None, None, A.tval.double()
    if kind == "spmv":
        if case["op"] == R.OP_N:
            x = _activity(GRIDS[case["grid"]])
            return (_csr64(A.row_ptr, A.col, A.val.double(), A.n) @ x.double()[:, None])[:, 0]
        out = torch.zeros(A.n, dtype=torch.float64, device=DEV)
        return out.index_add_(0, A.col, A.val.double() * A.y[:, 0].double()[A.rows().long()])
    val = A.val.double()
    if case["form"] in ("half", "batch"):
        val = A.hval.double() * A.rscale.double()[A.rows().long()]
    if not A.has_transpose:
        A.transpose()
    F = _csr64(A.row_ptr, A.col, val, A.n)
    B = _csr64(A.col_ptr, A.order[A.row_idx.long()], val[A.perm], A.m)
    y, s = A.y.double(), A.sensitivity().double()[:, None]
    x = torch.full((A.n, y.shape[1]), 1.0 / A.n, device=DEV).double()
    for _ in range(case["iters"]):
        e = torch.where(y == 0, torch.zeros_like(y), y / (F @ x))
        x = x * (B @ e) / (s + (s == 0))
        x = x / x.sum(0)
    return x if case.get("frames") else x[:, 0]


def _f32(v):
    return torch.tensor(v, dtype=torch.float32, device=DEV)


def _trafo(g, posx, iz, iy, ny, nz, s, c, u):
    """Points of a crystal in scanner coordinates, in float32 as the matrix is
    defined (each operation rounded); u: (channels, rays, 3) in [0, 1]."""
    p1 = (iy - _f32(0.5) * (ny - 1)) * _f32(g.segy)
    p2 = (iz - _f32(0.5) * (nz - 1)) * _f32(g.segz)
    hx = _f32(posx) - _f32(0.5) * _f32(g.segx)
    hz = p2 - _f32(0.5) * _f32(g.segz)
    sx, sy, sz = _f32(g.segx), _f32(g.segy), _f32(g.segz)
    col = [t[:, None] if t.dim() else t for t in (c * sx, s * sz, c * hx + s * hz, p1 - _f32(0.5) * sy, -s * sx, c * sz,
                                                  -s * hx + c * hz)]
    x = col[0] * u[..., 0] + col[1] * u[..., 2] + col[2]
    y = sy * u[..., 1] + col[3]
    z = col[4] * u[..., 0] + col[5] * u[..., 2] + col[6]
    return torch.stack([x, y, z], -1)


def _philox(key0, key1, ctr, half):
    """Philox4x32-10 with key (key0, key1) and counter (ctr, half, 0, 0)."""
    m = 0xFFFFFFFF
    c = [ctr.expand(key1.shape[0], -1), torch.full_like(ctr, half).expand(key1.shape[0], -1)]
    c += [torch.zeros_like(c[0]), torch.zeros_like(c[0])]
    k0, k1 = key0, key1[:, None]
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return [((v >> 8) + 1).float() * 2.0 ** -24 for v in c]


def _norm(v):
    return torch.sqrt(v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1] + v[..., 2] * v[..., 2])


def _build64(g, cnl, nrays, seed):
    """Mean path length of the channels' rays per voxel, in 64 bits: which
    voxels a row holds follows from the plane parameters in float32 (that is
    how the matrix is defined), the lengths are those of the same rays."""
    lib = ctypes.CDLL("libm.so.6")
    for f in (lib.sinf, lib.cosf):
        f.restype, f.argtypes = ctypes.c_float, [ctypes.c_float]
    n, N = g.grid_n[0], g.n_voxels
    args = [np.float32(np.float32(np.float32(math.pi) * np.float32(a)) * np.float32(g.da)) / np.float32(180)
            for a in range(g.na)]
    sins, coss = _f32([lib.sinf(float(a)) for a in args]), _f32([lib.cosf(float(a)) for a in args])
    ray = torch.arange(nrays, device=DEV)[None]
    plane = [_f32(g.grid_o[d]) + torch.arange(n + 1, device=DEV).float() * _f32(g.grid_d[d]) for d in range(3)]
    centre = [_f32(g.grid_o[d]) + (torch.arange(n, device=DEV).float() + 0.5) * _f32(g.grid_d[d]) for d in range(3)]
    radius = 0.5 * (_norm(_f32(g.grid_d)) + _norm(_f32([g.segx, g.segy, g.segz])))
    out = []
    per = max(1, min(int(2e8 / N), int(2.5e7 / (nrays * 3 * (n + 1)))))
    for lo in range(0, cnl.numel(), per):
        ch = cnl[lo:lo + per].long()
        t = ch % NAT
        iz0, iy0, iz1, iy1 = ((t // k % 13).float() for k in (2197, 169, 13, 1))
        s, c = sins[ch // NAT], coss[ch // NAT]
        u, w = _philox(seed & 0xFFFFFFFF, ch, ray, 0), _philox(seed & 0xFFFFFFFF, ch, ray, 1)
        r0 = _trafo(g, g.pos0x, iz0, iy0, 13, 13, s, c, torch.stack(u[:3], -1))
        r1 = _trafo(g, g.pos1x, iz1, iy1, 13, 13, s, c, torch.stack([u[3], w[0], w[1]], -1))
        d = r1 - r0
        a = torch.stack([(plane[k] - r0[..., k:k + 1]) / d[..., k:k + 1] for k in range(3)], -2)
        amin = torch.minimum(a[..., 0], a[..., n]).amax(-1)[..., None]
        amax = torch.maximum(a[..., 0], a[..., n]).amin(-1)[..., None]
        a, o = torch.sort(a.flatten(-2), dim=-1, stable=True)
        ok = (a[..., :-1] >= amin) & (a[..., 1:] <= amax) & (a[..., :-1] < a[..., 1:])
        axis = o // (n + 1)
        vox = torch.zeros_like(o[..., :-1])
        for k in range(3):
            cnt = torch.cumsum((axis == k).int(), -1)[..., :-1]
            vox = vox * n + torch.where(d[..., k:k + 1] > 0, cnt - 1, n - cnt)
        a64 = torch.stack([(plane[k].double() - r0[..., k:k + 1].double()) /
                           (r1[..., k:k + 1].double() - r0[..., k:k + 1].double()) for k in range(3)], -2)
        a64 = torch.gather(a64.flatten(-2), -1, o)
        length = (a64[..., 1:] - a64[..., :-1]) * _norm(r1.double() - r0.double())[..., None]
        at = (vox + torch.arange(len(ch), device=DEV)[:, None, None] * N)[ok]
        acc = torch.zeros(len(ch) * N, dtype=torch.float64, device=DEV).index_add_(0, at, length[ok])
        hit = torch.zeros(len(ch) * N, dtype=torch.bool, device=DEV)
        hit[at] = True
        at = torch.nonzero(hit)[:, 0]
        row, v = at // N, at % N
        mid = _f32([[0.5, 0.5, 0.5]])[None].expand(len(ch), 1, 3)
        c0 = _trafo(g, g.pos0x, iz0, iy0, 13, 13, s, c, mid)[:, 0]
        ab = _trafo(g, g.pos1x, iz1, iy1, 13, 13, s, c, mid)[:, 0] - c0
        ap = torch.stack([centre[0][v // (n * n)], centre[1][v // n % n], centre[2][v % n]], -1) - c0[row]
        b = ab[row]
        cr = torch.stack([b[:, 1] * ap[:, 2] - b[:, 2] * ap[:, 1], b[:, 2] * ap[:, 0] - b[:, 0] * ap[:, 2],
                          b[:, 0] * ap[:, 1] - b[:, 1] * ap[:, 0]], -1)
        out.append(acc[at[_norm(cr) / _norm(ab)[row] < radius]] / nrays)
    return torch.cat(out)
