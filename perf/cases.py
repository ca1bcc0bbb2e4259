"""Performance cases: passes over the suite's loop kernels through the C ABI.

Every case is one rep of a group of kernels as a user's program runs it: the
arrays and the workspaces are on the device before the call, run() makes the
calls on the current stream.  Sizes follow the suite's defaults (about 10^6
elements), the graph batch of small kernels and the large sets of bench.py;
values are uniform in [0.5, 1.5) unless a kernel needs others.
"""
import ctypes
import math

import torch

import rajaperf_gb300 as rp

F64, I64 = torch.float64, torch.int64
DEV = "cuda"


def listed():
    return [
        # the smallest calls: sixteen 1-D kernels of a few thousand elements
        # replayed as one CUDA graph (the suite's launch-bound small sizes)
        {"name": "loops_small_graph", "family": "loops", "n": 4099, "graph": True},
        # the same kernels called one by one at the suite's default size
        {"name": "loops_default", "family": "loops", "n": 1000003, "graph": False},
        # a rep of the Stream group on arrays far larger than L2
        {"name": "stream_large", "family": "stream", "n": (1 << 27) + 7},
        # the suite's SCAN (FP64 prefix sum), large
        {"name": "scan_f64_large", "family": "scan", "n": (1 << 26) + 1001, "dtype": "f64"},
        # integer scan, index list, histogram and per-bin sums with the
        # suite's ten bins
        {"name": "index_bins", "family": "index", "n": (1 << 24) + 4093, "bins": 10},
        # a hydro step on a 2-D mesh: HYDRO_2D, DEL_DOT_VEC_2D, PRESSURE, ENERGY
        {"name": "mesh_2d", "family": "mesh2d", "kn": 1999, "jn": 2003},
        # a 3-D mesh at the suite's default 100^3: halo exchange of three
        # variables with 26 neighbours, then zone volumes
        {"name": "mesh_3d", "family": "mesh3d", "dim": 100, "width": 1, "vars": 3},
        # time-stepped stencils: the suite's default size, ...
        {"name": "jacobi_2d", "family": "jacobi", "n": 1002, "steps": 40},
        # ... bench.py's 256^3 grid, ...
        {"name": "heat_3d", "family": "heat", "n": 258, "steps": 20},
        # ... and a ragged 2-D grid
        {"name": "fdtd_2d", "family": "fdtd", "nx": 2003, "ny": 1501, "steps": 40},
        # split-precision GEMM on tensor cores, the suite's nk = 1.2 ni
        {"name": "gemm_split", "family": "gemm_split", "m": 3500, "n": 3500, "k": 4200},
        # native FP64 3MM at the suite's default size
        {"name": "mm3_f64", "family": "mm3", "ni": 1000, "nj": 1100, "nk": 1010, "nl": 1200,
         "nm": 1000},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["loops", "stream", "scan", "index", "mesh2d", "mesh3d", "jacobi",
                         "heat", "fdtd", "gemm_split", "mm3"])
    if family == "loops":
        return {"family": family, "n": size(4097, 1 << 22), "graph": rng.random() < 0.5}
    if family == "stream":
        return {"family": family, "n": size(1 << 20, 1 << 27)}
    if family == "scan":
        return {"family": family, "n": size(1 << 14, 1 << 26),
                "dtype": rng.choice(["f64", "f64", "i64"])}
    if family == "index":
        return {"family": family, "n": size(1 << 14, 1 << 24), "bins": size(4, 20000)}
    if family == "mesh2d":
        return {"family": family, "kn": size(60, 2000), "jn": size(60, 2000)}
    if family == "mesh3d":
        return {"family": family, "dim": size(16, 200), "width": rng.choice([1, 1, 2]),
                "vars": rng.choice([1, 3, 3, 5])}
    if family == "jacobi":
        return {"family": family, "n": size(66, 4000), "steps": rng.choice([10, 20, 40])}
    if family == "heat":
        return {"family": family, "n": size(18, 258), "steps": rng.choice([10, 20])}
    if family == "fdtd":
        return {"family": family, "nx": size(64, 3000), "ny": size(64, 3000),
                "steps": rng.choice([10, 20, 40])}
    if family == "gemm_split":
        return {"family": family, "m": size(250, 4000), "n": size(250, 4000),
                "k": size(250, 4800)}
    return {"family": family, "ni": size(100, 1100), "nj": size(100, 1100),
            "nk": size(100, 1100), "nl": size(100, 1100), "nm": size(100, 1100)}


class Family:
    """The state of a case.  A subclass makes its inputs (from the seed alone)
    in inputs(), its outputs and workspaces in buffers(), calls the library in
    call() and names what a pass returns in outputs(); exact_values() gives
    the same from the inputs in plain torch."""

    def __init__(self, case, seed):
        self.case = case
        self.gen = torch.Generator(device=DEV).manual_seed(seed)
        self.inputs()

    def uniform(self, *shape, lo=0.5, hi=1.5):
        t = torch.rand(*shape, dtype=F64, device=DEV, generator=self.gen)
        return t if (lo, hi) == (0.0, 1.0) else t.mul_(hi - lo).add_(lo)

    def integers(self, lo, hi, n, dtype=I64):
        return torch.randint(lo, hi, (n,), dtype=dtype, device=DEV, generator=self.gen)

    def ready(self):
        self.lib = rp.b200()
        self.buffers()
        self.result = self.outputs()
        return self

    def workspace(self, nbytes):
        ws = torch.zeros(max(int(nbytes), 256), dtype=torch.uint8, device=DEV)
        return ws, ws.numel()

    def run(self):
        self.call(torch.cuda.current_stream().cuda_stream)
        return self.result


def zeros(*shape, dtype=F64):
    return torch.zeros(*shape, dtype=dtype, device=DEV)


def ptrs(*tensors):
    return [t.data_ptr() for t in tensors]


def ok(*status):
    for s in status:
        rp.check(s)


# STREAM's alpha: sqrt(2) - 1 keeps a[] constant over any number of reps.
ALPHA = math.sqrt(2.0) - 1.0


class Stream(Family):
    """COPY, MUL, ADD, TRIAD, DOT on three shared arrays, as STREAM does."""

    def inputs(self):
        self.n = self.case["n"]
        self.a = self.uniform(self.n)

    def buffers(self):
        self.b, self.c, self.dot = zeros(self.n), zeros(self.n), zeros(1)
        self.ws, self.wb = self.workspace(self.lib.b200_reduce_workspace_bytes(self.n, None))

    def call(self, s):
        L, n = self.lib, self.n
        a, b, c, dot, ws = ptrs(self.a, self.b, self.c, self.dot, self.ws)
        ok(L.b200_stream_copy(a, c, n, None, s), L.b200_stream_mul(b, c, ALPHA, n, None, s),
           L.b200_stream_add(a, b, c, n, None, s),
           L.b200_stream_triad(a, b, c, ALPHA, n, None, s),
           L.b200_stream_dot(a, b, n, 0.0, dot, ws, self.wb, None, s))

    def outputs(self):
        return {"a": self.a, "b": self.b, "c": self.c, "dot": self.dot}

    def exact_values(self):
        b = ALPHA * self.a
        c = self.a + b
        a = b + ALPHA * c
        return {"a": a, "b": b, "c": c, "dot": (a * b).sum().reshape(1)}

    @staticmethod
    def work(c):
        return {"bytes": 8 * 12 * c["n"], "flops": 6 * c["n"]}


class Loops(Family):
    """The 1-D kernels of the Stream, Basic, LCALS and Algorithm groups."""

    def inputs(self):
        self.n = n = self.case["n"]
        self.stream = Stream(self.case, int(self.gen.initial_seed()))
        self.x, self.y, self.z, self.u = (self.uniform(n + 12) for _ in range(4))
        self.acc, self.px = self.uniform(n), self.uniform(13 * n)
        self.dx, self.cx = self.uniform(14 * n), self.uniform(14 * n)
        self.xmin = self.uniform(n)
        self.xmin[n // 3] = -0.5

    def buffers(self):
        n = self.n
        self.stream.ready()
        self.init3 = [zeros(n) for _ in range(3)]
        self.mas = [zeros(n) for _ in range(3)]
        self.h1, self.eos, self.diff, self.py, self.pw = (zeros(n) for _ in range(5))
        self.loc, self.sum = zeros(1, dtype=I64), zeros(1)
        self.ws, self.wb = self.workspace(self.lib.b200_reduce_workspace_bytes(n, None))
        self.graph = None
        if self.case["graph"]:
            self.graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(self.graph):
                self.kernels(torch.cuda.current_stream().cuda_stream)

    def kernels(self, s):
        L, n, wb = self.lib, self.n, self.wb
        x, y, z, u, acc, px, ws = ptrs(self.x, self.y, self.z, self.u, self.acc, self.px,
                                       self.ws)
        dx, cx, xmin, loc, tot = ptrs(self.dx, self.cx, self.xmin, self.loc, self.sum)
        h1, eos, diff, py, pw = ptrs(self.h1, self.eos, self.diff, self.py, self.pw)
        self.stream.call(s)
        ok(L.b200_basic_daxpy(acc, x, 0.5, n, None, s),
           L.b200_basic_init3(*ptrs(*self.init3), x, y, n, None, s),
           L.b200_basic_muladdsub(*ptrs(*self.mas), x, y, n, None, s),
           L.b200_lcals_hydro_1d(h1, y, z, 0.0979, 0.1958, 0.0979, n, None, s),
           L.b200_lcals_eos(eos, y, z, u, 0.0979, 0.1958, 0.0979, n, None, s),
           L.b200_lcals_first_diff(diff, y, n, None, s),
           L.b200_lcals_int_predict(px, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6, 0.7, 0.8, n, None, s),
           L.b200_lcals_first_min(xmin, n, 0.5, 0, loc, None, ws, wb, None, s),
           L.b200_lcals_diff_predict(dx, cx, n, None, s),
           L.b200_lcals_planckian(x, py, u, y, pw, n, None, s),
           L.b200_algorithm_reduce_sum(x, n, 0.0, tot, ws, wb, None, s))

    def call(self, s):
        if self.graph is None:
            self.kernels(s)
        else:
            self.graph.replay()

    def outputs(self):
        return {"stream": self.stream.outputs(), "daxpy": self.acc, "init3": self.init3,
                "muladdsub": self.mas, "hydro_1d": self.h1, "eos": self.eos,
                "first_diff": self.diff, "int_predict": self.px, "first_min": self.loc,
                "diff_predict": self.dx, "planckian": [self.py, self.pw], "sum": self.sum}

    def exact_values(self):
        n = self.n
        x, y, z, u = self.x, self.y, self.z, self.u
        q, r, t = 0.0979, 0.1958, 0.0979
        in1, in2 = x[:n], y[:n]
        us = [u[k:k + n] for k in range(7)]
        eos = us[0] + r * (z[:n] + r * y[:n]) + t * (
            us[3] + r * (us[2] + r * us[1]) + t * (us[6] + q * (us[5] + q * us[4])))
        px = self.px.clone().view(13, n)
        dm = {22: 0.1, 23: 0.2, 24: 0.3, 25: 0.4, 26: 0.5, 27: 0.6, 28: 0.7}
        px[0] = (sum(dm[16 + k] * px[k] for k in range(12, 5, -1)) +
                 0.8 * (px[4] + px[5]) + px[2])
        dp, d = self.dx.clone().view(14, n), self.cx.view(14, n)[4]
        for k in range(4, 13):
            new, d = d, d - dp[k]
            dp[k] = new
        dp[13] = d
        py = u[:n] / y[:n]
        return {"stream": self.stream.exact_values(), "daxpy": self.acc + 0.5 * x[:n],
                "init3": [-in1 - in2] * 3, "muladdsub": [in1 * in2, in1 + in2, in1 - in2],
                "hydro_1d": q + y[:n] * (r * z[10:10 + n] + t * z[11:11 + n]), "eos": eos,
                "first_diff": y[1:n + 1] - y[:n], "int_predict": px.reshape(-1),
                "first_min": None, "diff_predict": dp.reshape(-1),
                "planckian": [py, x[:n] / (torch.exp(py) - 1.0)],
                "sum": x[:n].sum().reshape(1)}

    @staticmethod
    def work(c):
        # arrays read and written per element: 12 Stream, 3 DAXPY, 5 INIT3, 5
        # MULADDSUB, 3 HYDRO_1D, 4 EOS, 2 FIRST_DIFF, 11 INT_PREDICT, 1
        # FIRST_MIN, 20 DIFF_PREDICT, 5 PLANCKIAN, 1 REDUCE_SUM
        return {"bytes": 8 * 72 * c["n"], "flops": 70 * c["n"]}


class Scan(Family):
    """Exclusive prefix sum; FP64 over [0, 1) as the suite's, or int64."""

    def inputs(self):
        self.n, self.f64 = self.case["n"], self.case["dtype"] == "f64"
        self.x = (self.uniform(self.n, lo=0.0, hi=1.0) if self.f64
                  else self.integers(0, 100, self.n))

    def buffers(self):
        self.y = zeros(self.n, dtype=self.x.dtype)
        self.ws, self.wb = self.workspace(self.lib.b200_scan_workspace_bytes(self.n))
        self.fn = (self.lib.b200_algorithm_scan if self.f64
                   else self.lib.b200_algorithm_scan_i64)

    def call(self, s):
        x, y, ws = ptrs(self.x, self.y, self.ws)
        ok(self.fn(x, y, self.n, 0, ws, self.wb, None, s))

    def outputs(self):
        return {"y": self.y}

    def exact_values(self):
        if not self.f64:
            return {"y": None}
        # whole numbers of 2^-26 and of 2^-53 are summed apart, both exactly
        hi = (self.x * 2.0 ** 26).floor()
        lo = ((self.x * 2.0 ** 26 - hi) * 2.0 ** 27).to(I64)
        hi = hi.to(I64)
        hi = hi.cumsum(0) - hi
        lo = lo.cumsum(0) - lo
        return {"y": hi.to(F64) * 2.0 ** -26 + lo.to(F64) * 2.0 ** -53}

    @staticmethod
    def work(c):
        return {"bytes": 16 * c["n"], "flops": c["n"]}


class Index(Family):
    """SCAN over integers, INDEXLIST, HISTOGRAM, MULTI_REDUCE."""

    def inputs(self):
        self.n, self.nb = self.case["n"], self.case["bins"]
        self.count = self.integers(0, 100, self.n)
        self.sign = self.uniform(self.n, lo=-0.5, hi=0.5)
        self.bin = self.integers(0, self.nb, self.n)
        self.data = self.uniform(self.n)

    def buffers(self):
        n, nb, L = self.n, self.nb, self.lib
        self.offsets = zeros(n, dtype=I64)
        self.list, self.len = zeros(n, dtype=torch.int32), zeros(1, dtype=I64)
        self.counts0, self.counts = zeros(nb, dtype=I64), zeros(nb, dtype=I64)
        self.sums0, self.sums = zeros(nb), zeros(nb)
        self.ws = [self.workspace(b) for b in (L.b200_scan_workspace_bytes(n),
                                               L.b200_indexlist_workspace_bytes(n),
                                               L.b200_multi_reduce_workspace_bytes(n, nb))]

    def call(self, s):
        L, n, nb = self.lib, self.n, self.nb
        (w0, b0), (w1, b1), (w2, b2) = [(w.data_ptr(), b) for w, b in self.ws]
        count, offsets, sign, lst, length = ptrs(self.count, self.offsets, self.sign,
                                                 self.list, self.len)
        bins, c0, c1, data, s0, s1 = ptrs(self.bin, self.counts0, self.counts, self.data,
                                          self.sums0, self.sums)
        ok(L.b200_algorithm_scan_i64(count, offsets, n, 0, w0, b0, None, s),
           L.b200_basic_indexlist(sign, lst, n, length, w1, b1, None, s),
           L.b200_algorithm_histogram(bins, n, nb, c0, c1, None, s),
           L.b200_basic_multi_reduce(bins, data, n, nb, s0, s1, w2, b2, None, s))

    def outputs(self):
        return {"offsets": self.offsets, "list": self.list, "len": self.len,
                "counts": self.counts, "sums": self.sums}

    def exact_values(self):
        return {"offsets": None, "list": None, "len": None, "counts": None,
                "sums": zeros(self.nb).index_add_(0, self.bin, self.data)}

    @staticmethod
    def work(c):
        # scan 16, index list 8 + 4 for the half selected, histogram 8, sums 16
        return {"bytes": 50 * c["n"] + 32 * c["bins"], "flops": 2 * c["n"]}


class Mesh2D(Family):
    """HYDRO_2D on a kn x jn grid, DEL_DOT_VEC_2D on a jittered mesh of about
    as many zones, PRESSURE and ENERGY on the zones."""

    def inputs(self):
        self.kn, self.jn = kn, jn = self.case["kn"], self.case["jn"]
        self.n = n = kn * jn
        # za zb zm zp zq zr zu zv zz zrout zzout
        self.hydro = [self.uniform(n) for _ in range(11)]
        # nodes of a jn-1 x kn-1 zone mesh with the suite's ghost layers
        self.jp, rows = jn + 3, kn + 3
        nodes = self.jp * rows
        ii = torch.arange(self.jp, device=DEV, dtype=F64).repeat(rows)
        jj = torch.arange(rows, device=DEV, dtype=F64).repeat_interleave(self.jp)
        self.x = 0.2 * (ii + self.uniform(nodes, lo=-0.1, hi=0.1))
        self.y = 0.1 * (jj + self.uniform(nodes, lo=-0.1, hi=0.1))
        zi = torch.arange(2, jn + 1, device=DEV, dtype=I64)
        zj = torch.arange(2, kn + 1, device=DEV, dtype=I64)
        self.zones = (zj[:, None] * self.jp + zi[None, :]).reshape(-1).contiguous()
        self.xd, self.yd = self.uniform(nodes), self.uniform(nodes)
        self.en = [self.uniform(n) for _ in range(13)]

    def buffers(self):
        self.div = zeros(self.x.numel())
        self.bvc, self.p_new, self.e_new, self.q_new = (zeros(self.n) for _ in range(4))

    def call(self, s):
        L, n = self.lib, self.n
        eo, dv, pn, po, qo, wk, ch, ph, bv, pb, ql, qq, vn = ptrs(*self.en)
        bvc, p_new, e_new, q_new = ptrs(self.bvc, self.p_new, self.e_new, self.q_new)
        ok(L.b200_lcals_hydro_2d(*ptrs(*self.hydro), 0.0041, 0.0037, self.kn, self.jn, None, s),
           L.b200_apps_del_dot_vec_2d(*ptrs(self.x, self.y, self.xd, self.yd, self.div,
                                            self.zones), self.zones.numel(), self.jp, 1e-20,
                                      0.5, None, s),
           L.b200_apps_pressure(ch, bvc, p_new, eo, vn, 0.5, 1e-7, 0.0, 1.2, n, None, s),
           L.b200_apps_energy(e_new, eo, dv, pn, po, q_new, qo, wk, ch, ph, bv, pb, ql, qq, vn,
                              1.1, 1e-7, 0.0, 1e-7, n, None, s))

    def outputs(self):
        za, zb, _, _, _, _, zu, zv, _, zrout, zzout = self.hydro
        return {"hydro": [za, zb, zu, zv, zrout, zzout], "div": self.div,
                "pressure": [self.bvc, self.p_new], "energy": [self.e_new, self.q_new]}

    def exact_values(self):
        za, zb, zm, zp, zq, zr, zu, zv, zz, zrout, zzout = [
            t.clone().view(self.kn, self.jn) for t in self.hydro]

        def at(t, k=0, j=0):  # the interior, shifted by k rows and j columns
            return t[1 + k:self.kn - 1 + k, 1 + j:self.jn - 1 + j]

        pq = zp + zq
        za_in = ((at(pq, 1, -1) - at(zp, 0, -1) - at(zq, 0, -1)) * (at(zr) + at(zr, 0, -1)) /
                 (at(zm, 0, -1) + at(zm, 1, -1)))
        zb_in = ((at(pq, 0, -1) - at(zp) - at(zq)) * (at(zr) + at(zr, -1)) /
                 (at(zm) + at(zm, 0, -1)))
        at(za).copy_(za_in)
        at(zb).copy_(zb_in)
        for v, f, out, base in ((zu, zz, zrout, zr), (zv, zr, zzout, zz)):
            new = at(v) + 0.0041 * (at(za) * (at(f) - at(f, 0, 1)) -
                                    at(za, 0, -1) * (at(f) - at(f, 0, -1)) -
                                    at(zb) * (at(f) - at(f, -1)) +
                                    at(zb, 1) * (at(f) - at(f, 1)))
            at(v).copy_(new)
            at(out).copy_(at(base) + 0.0037 * new)

        def corners(t):
            z = self.zones
            return t[z + 1], t[z + 1 + self.jp], t[z + self.jp], t[z]

        def halves(t):
            t1, t2, t3, t4 = corners(t)
            return 0.5 * (t1 + t2 - t3 - t4), 0.5 * (t2 + t3 - t4 - t1), t1 + t2 + t3 + t4

        (xi, xj, _), (yi, yj, ysum) = halves(self.x), halves(self.y)
        (fxi, fxj, _), (fyi, fyj, fysum) = halves(self.xd), halves(self.yd)
        rarea = 1.0 / (xi * yj - xj * yi + 1e-20)
        div = zeros(self.x.numel())
        div[self.zones] = (rarea * (fxi * yj - fxj * yi) + rarea * (fyj * xi - fyi * xj) +
                           fysum / ysum)

        eo, dv, pn, po, qo, wk, ch, ph, bv, pb, ql, qq, vn = self.en
        bvc = 0.5 * (ch + 1.0)
        p = bvc * eo
        p = torch.where((p.abs() < 1e-7) | (vn >= 1.2), torch.zeros_like(p), p).clamp(min=0.0)

        def cut(e):
            return torch.where(e.abs() < 1e-7, torch.zeros_like(e), e).clamp(min=0.0)

        # delvc is positive: the artificial viscosities q are zero
        e = eo - 0.5 * dv * (po + qo) + 0.5 * wk
        e = cut(e + 0.5 * dv * (3.0 * (po + qo) - 4.0 * ph) + 0.5 * wk)
        e = cut(e - (7.0 * (po + qo) - 8.0 * ph + pn) * dv / 6.0)
        return {"hydro": [t.reshape(-1) for t in (za, zb, zu, zv, zrout, zzout)], "div": div,
                "pressure": [bvc, p], "energy": [e, torch.zeros_like(e)]}

    @staticmethod
    def work(c):
        # doubles per point: HYDRO_2D 9 read, 6 written; DEL_DOT_VEC_2D 5 and
        # 1; PRESSURE 3 and 2; ENERGY (positive delvc) 7 and 2
        n = c["kn"] * c["jn"]
        return {"bytes": 8 * 35 * n, "flops": (44 + 54 + 3 + 25) * n}


class Seg(ctypes.Structure):
    """b200_halo_seg of include/b200.h."""
    _fields_ = [("var", ctypes.c_void_p), ("list", ctypes.c_void_p),
                ("buffer", ctypes.c_void_p), ("len", ctypes.c_int64)]


class Mesh3D(Family):
    """HALO_PACKING of `vars` variables on a dim^3 grid with 26 neighbours, and
    VOL3D on a jittered mesh of dim^3 nodes."""

    def inputs(self):
        dim, w, nv = self.case["dim"], self.case["width"], self.case["vars"]
        full = dim + 2 * w
        self.vars = [self.uniform(full ** 3) for _ in range(nv)]
        cells = torch.arange(full ** 3, dtype=torch.int32, device=DEV).view(full, full, full)
        send = {-1: slice(w, 2 * w), 0: slice(w, w + dim), 1: slice(dim, dim + w)}
        recv = {-1: slice(0, w), 0: slice(w, w + dim), 1: slice(w + dim, full)}
        offsets = [(k, j, i) for k in (-1, 0, 1) for j in (-1, 0, 1) for i in (-1, 0, 1)
                   if (k, j, i) != (0, 0, 0)]
        self.pack = [cells[tuple(send[d] for d in o)].reshape(-1).clone() for o in offsets]
        self.unpack = [cells[tuple(recv[d] for d in o)].reshape(-1).clone() for o in offsets]
        self.received = self.uniform(nv * sum(t.numel() for t in self.unpack))
        self.jp = jp = dim + 4  # nodes per row with the suite's ghost layers
        line = torch.arange(jp, device=DEV, dtype=F64)
        self.x, self.y, self.z = (
            (h * line.view(shape)).expand(jp, jp, jp).reshape(-1) +
            h * self.uniform(jp ** 3, lo=-0.1, hi=0.1)
            for h, shape in ((0.3, (1, 1, jp)), (0.2, (1, jp, 1)), (0.1, (jp, 1, 1))))
        corner = 1 + jp + jp * jp
        self.first, self.last = corner, (dim + 2) * corner  # zones, ghost zones among them

    def segments(self, lists, buffer):
        segs, at = [], 0
        for lst in lists:
            for var in self.vars:
                segs.append(Seg(var.data_ptr(), lst.data_ptr(), buffer.data_ptr() + 8 * at,
                                lst.numel()))
                at += lst.numel()
        return (Seg * len(segs))(*segs)

    def buffers(self):
        self.sent = zeros(self.received.numel())
        self.vol = zeros(self.jp ** 3)
        self.ps = self.segments(self.pack, self.sent)
        self.us = self.segments(self.unpack, self.received)

    def call(self, s):
        L = self.lib
        ok(L.b200_comm_halo_packing(ctypes.addressof(self.ps), len(self.ps),
                                    ctypes.addressof(self.us), len(self.us), None, s),
           L.b200_apps_vol3d(*ptrs(self.x, self.y, self.z, self.vol), 0.083333333333333333,
                             self.jp, self.jp ** 2, self.first, self.last + 1, None, s))

    def outputs(self):
        return {"vars": self.vars, "sent": self.sent, "vol": self.vol}

    def exact_values(self):
        new, sent, at = [v.clone() for v in self.vars], [], 0
        for lst in self.pack:
            sent += [v[lst.long()] for v in self.vars]
        for lst in self.unpack:
            for v in new:
                v[lst.long()] = self.received[at:at + lst.numel()]
                at += lst.numel()
        i = torch.arange(self.first, self.last + 1, device=DEV)
        off = [0, 1, self.jp, 1 + self.jp]
        off += [o + self.jp ** 2 for o in off]
        P = [torch.stack([t[i + o] for t in (self.x, self.y, self.z)]) for o in off]

        def triple(a, b, c):
            return (a * torch.linalg.cross(b, c, dim=0)).sum(0)

        v71, v72, v74 = P[7] - P[1], P[7] - P[2], P[7] - P[4]
        v30, v50, v60 = P[3] - P[0], P[5] - P[0], P[6] - P[0]
        vol = zeros(self.jp ** 3)
        # the suite's third block repeats the second block's cross product
        vol[i] = 0.083333333333333333 * (
            triple(v71 + v60, v72, v30) + triple(v72 + v50, v74, v60) +
            triple(v74 + v30, v74, v60) + triple(v74 + v30, v71, v50))
        return {"vars": new, "sent": torch.cat(sent), "vol": vol}

    @staticmethod
    def work(c):
        d, w = c["dim"], c["width"]
        halo = (d + 2 * w) ** 3 - d ** 3
        # each halo cell is sent and received: an index, a value read and written
        return {"bytes": 2 * (4 + 16 * c["vars"]) * halo + 32 * d ** 3,
                "flops": 72 * d ** 3}


class Jacobi(Family):
    def inputs(self):
        n = self.case["n"]
        self.a, self.b = self.uniform(n, n), self.uniform(n, n)

    def buffers(self):
        pass

    def call(self, s):
        ok(self.lib.b200_polybench_jacobi_2d(*ptrs(self.a, self.b), self.case["n"],
                                             self.case["steps"], None, s))

    def outputs(self):
        return {"A": self.a, "B": self.b}

    def exact_values(self):
        a, b = self.a.clone(), self.b.clone()
        for _ in range(self.case["steps"]):
            for s, d in ((a, b), (b, a)):
                d[1:-1, 1:-1] = 0.2 * (s[1:-1, 1:-1] + s[1:-1, :-2] + s[1:-1, 2:] +
                                       s[2:, 1:-1] + s[:-2, 1:-1])
        return {"A": a, "B": b}

    @staticmethod
    def work(c):
        # each array read and written once: the steps need not go to memory
        return {"bytes": 8 * 4 * c["n"] ** 2, "flops": 10 * c["steps"] * (c["n"] - 2) ** 2}


class Heat(Family):
    def inputs(self):
        n = self.case["n"]
        self.a, self.b = self.uniform(n, n, n), self.uniform(n, n, n)

    def buffers(self):
        pass

    def call(self, s):
        ok(self.lib.b200_polybench_heat_3d(*ptrs(self.a, self.b), self.case["n"],
                                           self.case["steps"], None, s))

    def outputs(self):
        return {"A": self.a, "B": self.b}

    def exact_values(self):
        a, b = self.a.clone(), self.b.clone()
        mid, up, dn = slice(1, -1), slice(2, None), slice(None, -2)
        axes = [((up, mid, mid), (dn, mid, mid)), ((mid, up, mid), (mid, dn, mid)),
                ((mid, mid, up), (mid, mid, dn))]
        for _ in range(self.case["steps"]):
            for s, d in ((a, b), (b, a)):
                c = s[mid, mid, mid]
                ti, tj, tk = (0.125 * (s[hi] - 2.0 * c + s[lo]) for hi, lo in axes)
                d[mid, mid, mid] = ti + tj + tk + c
        return {"A": a, "B": b}

    @staticmethod
    def work(c):
        return {"bytes": 8 * 4 * c["n"] ** 3, "flops": 30 * c["steps"] * (c["n"] - 2) ** 3}


class Fdtd(Family):
    def inputs(self):
        nx, ny = self.case["nx"], self.case["ny"]
        self.ex, self.ey, self.hz = (self.uniform(nx, ny) for _ in range(3))
        self.fict = self.uniform(self.case["steps"])

    def buffers(self):
        self.ws, self.wb = self.workspace(
            self.lib.b200_fdtd_2d_workspace_bytes(self.case["nx"], self.case["ny"]))

    def call(self, s):
        c = self.case
        ex, ey, hz, fict, ws = ptrs(self.ex, self.ey, self.hz, self.fict, self.ws)
        ok(self.lib.b200_polybench_fdtd_2d_ws(ex, ey, hz, fict, c["nx"], c["ny"], c["steps"],
                                              ws, self.wb, None, s))

    def outputs(self):
        return {"ex": self.ex, "ey": self.ey, "hz": self.hz}

    def exact_values(self):
        ex, ey, hz = self.ex.clone(), self.ey.clone(), self.hz.clone()
        for t in range(self.case["steps"]):
            ey[0] = self.fict[t]
            ey[1:] -= 0.5 * (hz[1:] - hz[:-1])
            ex[:, 1:] -= 0.5 * (hz[:, 1:] - hz[:, :-1])
            hz[:-1, :-1] -= 0.7 * (ex[:-1, 1:] - ex[:-1, :-1] + ey[1:, :-1] - ey[:-1, :-1])
        return {"ex": ex, "ey": ey, "hz": hz}

    @staticmethod
    def work(c):
        n = c["nx"] * c["ny"]
        return {"bytes": 8 * 6 * n, "flops": 11 * c["steps"] * n}


class GemmSplit(Family):
    """C = 1.5 A B + 1.2 C in split precision, entries in [-1, 1)."""

    def inputs(self):
        m, n, k = self.case["m"], self.case["n"], self.case["k"]
        self.a, self.b = self.uniform(m, k, lo=-1.0, hi=1.0), self.uniform(k, n, lo=-1.0, hi=1.0)
        self.c = self.uniform(m, n, lo=-1.0, hi=1.0)

    def buffers(self):
        self.size = self.case["m"], self.case["n"], self.case["k"]
        self.ws, self.wb = self.workspace(
            self.lib.b200_gemm_split_workspace_bytes(*self.size, None))

    def call(self, s):
        a, b, c, ws = ptrs(self.a, self.b, self.c, self.ws)
        ok(self.lib.b200_gemm_split(a, b, c, *self.size, 1.5, 1.2, ws, self.wb, None, s))

    def outputs(self):
        return {"C": self.c}

    def exact_values(self):
        return {"C": 1.5 * (self.a @ self.b) + 1.2 * self.c}

    @staticmethod
    def work(c):
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 8 * (m * k + k * n + 2 * m * n), "flops": 2 * m * n * k}


class Mm3(Family):
    """G = (A B) (C D) in native FP64."""

    def inputs(self):
        c = self.case
        shapes = (("ni", "nk"), ("nk", "nj"), ("nj", "nm"), ("nm", "nl"))
        self.abcd = [self.uniform(c[r], c[k], lo=-1.0, hi=1.0) for r, k in shapes]

    def buffers(self):
        c = self.case
        self.efg = [zeros(c[r], c[k]) for r, k in (("ni", "nj"), ("nj", "nl"), ("ni", "nl"))]

    def call(self, s):
        c = self.case
        ok(self.lib.b200_polybench_3mm(*ptrs(*self.abcd, *self.efg), c["ni"], c["nj"], c["nk"],
                                       c["nl"], c["nm"], None, s))

    def outputs(self):
        return dict(zip("EFG", self.efg))

    def exact_values(self):
        a, b, c, d = self.abcd
        return {"E": a @ b, "F": c @ d, "G": (a @ b) @ (c @ d)}

    @staticmethod
    def work(c):
        ni, nj, nk, nl, nm = (c[k] for k in ("ni", "nj", "nk", "nl", "nm"))
        return {"bytes": 8 * (ni * nk + nk * nj + nj * nm + nm * nl + ni * nj + nj * nl +
                              ni * nl),
                "flops": 2 * (ni * nj * nk + nj * nl * nm + ni * nl * nj)}


FAMILIES = {"loops": Loops, "stream": Stream, "scan": Scan, "index": Index, "mesh2d": Mesh2D,
            "mesh3d": Mesh3D, "jacobi": Jacobi, "heat": Heat, "fdtd": Fdtd,
            "gemm_split": GemmSplit, "mm3": Mm3}


def prepare(case, seed):
    return FAMILIES[case["family"]](case, seed).ready()


def run(state):
    return state.run()


def work(case):
    return FAMILIES[case["family"]].work(case)


def exact(case, seed):
    return FAMILIES[case["family"]](case, seed).exact_values()
