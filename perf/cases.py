"""What a user of the mechanics library has it do, as measurable cases.

Every case goes through the public entry points (epi_b200.capi.Context, or
the C ABI where the binding has no method of its own). The kinds:

  steps    a burst of mechanics steps from given positions: positions in from
           host memory, n steps, positions back (a program that renews cell
           states, writes frames or analyses positions between bursts). One
           tissue or a batch of uneven ones, square or triangular membranes,
           cells of the simple states or every cell state, FP64 forces or the
           mixed path, one call for the burst or a call per step.
  host     one step of a batch that lives in host memory (epi_step_host).
  dropin   the calls of the C++ drop-in for each step of the reference's own
           loop: upload of the renewed cells (which connects), lists and
           dermis out, interaction and commit, positions out.
  adjoint  loss and gradient of a run with respect to the force constants.
  field    the reference's loop with its cell maps and stimulus diffusion
           after every mechanics step, then the grids out.
  noalloc  connection lists of one tissue in the caller's device memory.

Sizes and constants are those of the repository's own workloads (the 16 x 16,
64 x 64 and 256 x 256 tissues, the 512-tissue ensemble, its triangular form,
the all-states tissue, the 129 x 129 x 65 grid); tissues of a "ragged" batch
have any side from 16 to 64, odd ones among them.
"""
import ctypes
import math

import numpy as np
import torch

from epi_b200 import capi
from epi_b200 import tissue as T

FP64, MIXED = capi.EPI_PREC_FP64, capi.EPI_PREC_MIXED

_DEFAULTS = {
    "kind": "steps",      # see above
    "tissues": 1,         # tissues of the batch
    "side": 16,           # membrane side of a single tissue
    "layers": 2,          # cell layers of a single tissue
    "shapes": "single",   # single | ensemble (sides 16..64 of the ensemble) | ragged (any side)
    "lattice": "square",  # square | tri
    "states": "simple",   # simple | aged (simple states, ages 0..24) | all (every cell state)
    "precision": "mixed",
    "steps": 20,
    "mode": "graph",      # graph | eager: one call for all steps; each: one call per step
}


def _case(name=None, **kw):
    c = dict(_DEFAULTS, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest tissue, one call per step: a host loop that looks at
        # the tissue between steps; latency and launches are all there is
        _case("one_small_each", side=16, layers=2, precision="fp64", mode="each", steps=20),
        # the ordinary single tissue, a run of 100 steps
        _case("one_mid", side=64, layers=8, steps=100),
        # an odd-sided, thin tissue in FP64
        _case("one_odd_fp64", side=37, layers=3, precision="fp64", steps=100),
        # a tissue too large for 16-bit candidate rows
        _case("one_large", side=256, layers=16, steps=50),
        # the parameter study: the whole 512-tissue ensemble (the largest case)
        _case("ensemble", tissues=512, shapes="ensemble", steps=100),
        # a part of it with FP64 forces, the accuracy reference of such a study
        _case("ensemble_fp64", tissues=96, shapes="ensemble", precision="fp64", steps=50),
        # the reference's default lattice, ragged tissues
        _case("ragged_tri", tissues=128, shapes="ragged", lattice="tri", steps=50),
        # every cell state and law (dermis, stem cells, pairs): the general path
        _case("all_states_fp64", tissues=64, states="all", precision="fp64", steps=50),
        # state renewal on the host, positions in and out every step
        _case("host_step", kind="host", tissues=128, shapes="ensemble", steps=1),
        # calibration: gradient of a 200-step run on the 36,864-particle tissue
        _case("adjoint", kind="adjoint", side=64, layers=8, precision="fp64", steps=200),
        # mechanics, cell maps and stimulus, step by step
        _case("field_loop", kind="field", side=64, layers=8, states="aged", precision="fp64",
              steps=50),
        # connection lists for a caller whose device memory is its own
        _case("connect_noalloc", kind="noalloc", side=64, layers=8, steps=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "batch", "batch", "all", "host", "dropin", "adjoint",
                       "field", "noalloc"])
    lattice = rng.choice(["square", "tri"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "single":
        side = _log(rng, 16, 220)
        layers = rng.randint(2, 8) if side < 48 else rng.randint(2, 14)
        return _case(side=side, layers=layers, lattice=lattice, precision=precision,
                     states=rng.choice(["simple", "simple", "aged"]),
                     mode=rng.choice(["graph", "graph", "eager", "each"]),
                     steps=_log(rng, 10, 100))
    if kind == "batch":
        return _case(tissues=_log(rng, 2, 256), shapes=rng.choice(["ensemble", "ragged"]),
                     lattice=lattice, precision=precision,
                     mode=rng.choice(["graph", "graph", "eager"]), steps=_log(rng, 10, 100))
    if kind == "all":
        return _case(tissues=_log(rng, 1, 128), states="all", lattice=lattice, precision="fp64",
                     mode=rng.choice(["graph", "eager"]), steps=_log(rng, 10, 100))
    if kind == "host":
        return _case(kind="host", tissues=_log(rng, 4, 200),
                     shapes=rng.choice(["ensemble", "ragged"]), lattice=lattice,
                     precision=precision, steps=1)
    if kind == "dropin":
        return _case(kind="dropin", side=_log(rng, 16, 80), layers=rng.randint(2, 8),
                     lattice=lattice, precision="fp64", steps=rng.randint(2, 6))
    if kind == "adjoint":
        return _case(kind="adjoint", side=_log(rng, 16, 64), layers=rng.randint(2, 8),
                     lattice=lattice, precision="fp64", steps=_log(rng, 20, 200))
    if kind == "field":
        return _case(kind="field", side=_log(rng, 16, 72), layers=rng.randint(2, 8),
                     lattice=lattice, states="aged", precision="fp64",
                     steps=_log(rng, 10, 60))
    side = _log(rng, 16, 64)
    return _case(kind="noalloc", side=side, layers=rng.randint(2, 8), steps=1)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
_TARGET = 0.05   # adjoint targets: observed positions within this of the start


def _layered(case, side, layers, seed, params=None):
    if case["lattice"] == "tri":
        return T.tri_layered_tissue(side, T.tri_rows(side), layers, seed, params=params)
    return T.layered_tissue(side, layers, seed, params=params)


def _shapes(case):
    """(side, layers, params) of every tissue of a batch: the case's own, so
    inputs of every seed have the same sizes."""
    if case["shapes"] == "ensemble":
        return T.config4_specs(n_tissues=case["tissues"])
    r = np.random.default_rng(case["tissues"])
    out = []
    for _ in range(case["tissues"]):
        s = np.exp(r.uniform(math.log(0.5), math.log(2.0), 3))
        out.append((int(r.integers(16, 65)), int(r.integers(2, 9)),
                    T.Params().scaled(float(s[0]), float(s[1]), float(s[2]))))
    return out


def _tissues(case, seed):
    if case["states"] == "all":
        lat = T.TRIANGULAR if case["lattice"] == "tri" else T.SQUARE
        return [T.mixed_state_tissue(T.mix_seed(seed, t), lat) for t in range(case["tissues"])]
    if case["shapes"] == "single":
        ts = [_layered(case, case["side"], case["layers"], T.mix_seed(seed, 0))]
    else:
        ts = [_layered(case, side, layers, T.mix_seed(seed, t), p)
              for t, (side, layers, p) in enumerate(_shapes(case))]
    if case["states"] == "aged":
        for k, t in enumerate(ts):
            r = np.random.default_rng(T.mix_seed(seed, k, 13))
            t.agek[t.nmemb:] = r.uniform(0.0, 24.0, t.n - t.nmemb)
    return ts


def _target(t, seed):
    r = np.random.default_rng(T.mix_seed(seed, 14))
    return tuple(a + r.uniform(-_TARGET, _TARGET, t.n) for a in (t.x, t.y, t.z))


def _grid(t):
    """Grid points per axis at the reference's half-unit spacing."""
    return int(round(2 * t.lx)), int(round(2 * t.ly)), int(round(2 * t.lz))


def _stimulus(dims, seed):
    r = np.random.default_rng(T.mix_seed(seed, 15))
    return r.uniform(0.0, 1.0, (dims[0] + 1, dims[1] + 1, dims[2] + 1))


def _pinned(a):
    p = torch.empty(a.shape[0], dtype=torch.float64, pin_memory=True)
    p.numpy()[:] = a
    return p


def prepare(case, seed):
    ts = _tissues(case, seed)
    kind = case["kind"]
    if kind == "noalloc":
        t = ts[0]
        dev = torch.device("cuda")
        s = {"case": case, "tissue": t, "max_conn": 64,
             "inputs": [torch.tensor(a, dtype=torch.float64, device=dev)
                        for a in (t.x, t.y, t.z, t.radius)],
             "conn": torch.full((t.n, 64), -1, dtype=torch.int32, device=dev),
             "count": torch.zeros(t.n, dtype=torch.int32, device=dev)}
        f = capi.lib().epi_connect_noalloc
        f.argtypes = ([ctypes.c_void_p] * 4 + [ctypes.c_int32] * 4 + [ctypes.c_double] * 4 +
                      [ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p])
        f.restype = ctypes.c_int
        s["entry"] = f
        return s
    cap = dict(max_conn=96, max_cand=192) if case["states"] == "all" else {}
    ctx = capi.Context(precision=FP64 if case["precision"] == "fp64" else MIXED, **cap)
    ctx.upload(ts)
    cat = tuple(np.concatenate([getattr(t, k) for t in ts]) for k in "xyz")
    keep = [_pinned(a) for a in cat] + [_pinned(a) for a in cat]
    s = {"case": case, "ctx": ctx, "tissues": ts, "keep": keep,
         "start": tuple(k.numpy() for k in keep[:3]), "end": tuple(k.numpy() for k in keep[3:])}
    if kind == "adjoint":
        s["target"] = _target(ts[0], seed)
    if kind == "field":
        dims = _grid(ts[0])
        ctx.field_init(*dims)
        ctx.field_set_ext(0, _stimulus(dims, seed))
    if kind == "dropin":
        s["rows"] = np.full(32 * ts[0].n, -1, np.int32)
    return s


def run(s):
    case = s["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "noalloc":
        t = s["tissue"]
        x, y, z, r = s["inputs"]
        rc = s["entry"](x.data_ptr(), y.data_ptr(), z.data_ptr(), r.data_ptr(), t.n, t.nmemb,
                        t.nmx, t.nmy, t.lx, t.ly, t.lz, t.params.lj_thresh, s["max_conn"],
                        s["conn"].data_ptr(), s["count"].data_ptr(),
                        torch.cuda.current_stream().cuda_stream)
        if rc != capi.EPI_OK:
            raise RuntimeError(capi.strerror(rc))
        return {"conn": s["conn"], "count": s["count"]}
    ctx = s["ctx"]
    if kind == "host":
        return ctx.step_host(s["start"], s["end"])
    if kind == "dropin":
        t = s["tissues"][0].copy()
        t.x, t.y, t.z = s["start"]
        for _ in range(steps):
            ctx.upload([t])
            off, idx = ctx.connections()
            s["rows"][:idx.size] = idx  # the program's own copy of the lists
            s["rows"][idx.size:] = -1
            dermis = ctx.dermis()
            ctx.interact_commit()
            t.x, t.y, t.z = ctx.positions(s["end"])
        return {"pos": s["end"], "off": off, "idx": s["rows"], "dermis": dermis}
    ctx.set_positions(*s["start"])
    if kind == "adjoint":
        loss, grad = ctx.adjoint(steps, s["target"])
        return {"loss": loss, "grad": grad, "pos": ctx.positions(s["end"])}
    if kind == "field":
        for _ in range(steps):
            ctx.step(1)
            ctx.field_step(1)
        cmap1, cmap2, ext, zzmax = ctx.field(0)
        return {"cmap1": cmap1, "cmap2": cmap2, "ext": ext, "zzmax": zzmax,
                "pos": ctx.positions(s["end"])}
    if case["mode"] == "each":
        for _ in range(steps):
            ctx.step(1)
    else:
        ctx.step(steps, case["mode"])
    return ctx.positions(s["end"])


def _particles(case):
    """Particles of the case (batches: the mean of their shapes)."""
    if case["states"] == "all":
        return 1100 * case["tissues"]
    if case["shapes"] == "single":
        rows = T.tri_rows(case["side"]) if case["lattice"] == "tri" else case["side"]
        return case["side"] * rows * (case["layers"] + 1)
    return sum(side * (T.tri_rows(side) if case["lattice"] == "tri" else side) * (layers + 1)
               for side, layers, _ in _shapes(case))


def work(case):
    """Per particle and step: position in and out and the cell's state (52
    bytes), and about seven connections of some 40 operations. A gradient
    reads and writes its adjoints as well; a grid point's stimulus is read and
    written with its two map entries; the lists are written once."""
    n, steps = _particles(case), case["steps"]
    w = {"bytes": 52.0 * n * steps, "flops": 7 * 40.0 * n * steps}
    if case["kind"] == "adjoint":
        w = {"bytes": 3 * w["bytes"], "flops": 4 * w["flops"]}
    elif case["kind"] == "field":
        side = case["side"]
        rows = T.tri_rows(side) * math.sqrt(0.75) if case["lattice"] == "tri" else side
        points = (2 * side + 1) * (2 * rows + 1) * 65
        w = {"bytes": w["bytes"] + 21.0 * points * steps, "flops": w["flops"] + 20.0 * points * steps}
    elif case["kind"] in ("noalloc", "dropin"):
        w["bytes"] += 4.0 * 8 * n * steps
    return w


# --------------------------------------------------------------------------
# the same results in 64 bits, with torch alone
# --------------------------------------------------------------------------
_ALIVE, _DEAD, _FIX, _DER, _MUSUME, _AIR, _MEMB = 0, 1, 4, 6, 7, 8, 9
_SKIN = 0.3  # margin of the pair list, rebuilt once a particle has moved half of it


class _Model:
    """epi5_MT's mechanics step (cell_connection.cpp, cell_interaction.cpp) of
    a batch of tissues as plain FP64 tensor operations: every pair once, i the
    higher index."""

    def __init__(self, tissues, device):
        self.dev = device
        cat = lambda f, dt: torch.tensor(np.concatenate([np.asarray(f(t)) for t in tissues]),
                                         dtype=dt, device=device)
        f64, i64 = torch.float64, torch.int64
        self.n = sum(t.n for t in tissues)
        base = np.concatenate([[0], np.cumsum([t.n for t in tissues])])
        self.tid = cat(lambda t: np.zeros(t.n), i64)
        for k in range(len(tissues)):
            self.tid[base[k]:base[k + 1]] = k
        self.r = cat(lambda t: t.radius, f64)
        self.st = cat(lambda t: t.state, i64)
        self.old = cat(lambda t: t.agek > t.params.thresh_sp, torch.bool)
        self.agek = cat(lambda t: t.agek, f64)
        per = lambda f: torch.tensor([float(f(t)) for t in tissues], dtype=f64, device=device)
        self.lx_t, self.ly_t, self.lz_t = per(lambda t: t.lx), per(lambda t: t.ly), per(lambda t: t.lz)
        self.lx, self.ly = self.lx_t[self.tid], self.ly_t[self.tid]
        self.par = {k: per(lambda t, k=k: getattr(t.params, k)) for k in (
            "dt", "eps_m", "p_memb", "der_der_const", "k_total", "k_desmosome", "kspring",
            "kspring_d", "kbend", "delta_r", "para_ljp2", "kspring_division", "lj_thresh")}
        # multipliers of the spring constants, eps_m and kbend (the gradient's variables)
        self.s = None
        self.memb = self.st == _MEMB
        self.simple = bool(((self.st == _MEMB) | (self.st == _ALIVE) | (self.st == _DEAD) |
                            (self.st == _AIR)).all())
        pair = np.concatenate([np.where(t.pair >= 0, t.pair + b, -1)
                               for t, b in zip(tissues, base[:-1])])
        self.pair = torch.tensor(pair, dtype=i64, device=device)
        self.spr = cat(lambda t: t.spr_nat_len, f64)
        rest = cat(lambda t: t.rest_div_times, i64)
        mate = self.st[self.pair.clamp(min=0)]
        self.sfm = torch.where((self.pair >= 0) & (mate == _FIX), 1, torch.where(rest > 0, 2, 0))
        rmax = max(float(t.radius.max()) for t in tissues)
        rcell = max(float(t.radius[t.nmemb:].max()) for t in tissues)
        self.reach = max(t.params.lj_thresh for t in tissues) * (rmax + rcell) + _SKIN
        self._lattice(tissues, base)
        self._cells(tissues)

    def _lattice(self, tissues, base):
        """Membrane lattice sites: global indices of every stencil site."""
        rows = {"square": [], "tri": []}
        for t, b in zip(tissues, base[:-1]):
            j = np.arange(t.nmemb)
            c, w = j % t.nmx, j // t.nmx
            site = lambda c, w: b + (w % t.nmy) * t.nmx + c % t.nmx
            if t.lattice == T.TRIANGULAR:
                def step(c, w, k):
                    even = w % 2 == 0
                    if k in (0, 3):
                        return c + (1 if k == 0 else -1), w
                    up = -1 if k in (1, 2) else 1
                    right = k in (1, 5)
                    return c + np.where(even, 0 if right else -1, 1 if right else 0), w + up
                nb = [site(*step(c, w, k)) for k in range(6)]
                ring = []
                for k in range(6):
                    c1, w1 = step(c, w, (k + 1) % 6)
                    ring.append(site(*step(c1 % t.nmx, w1 % t.nmy, k)))
                rows["tri"].append(np.stack([b + j] + nb + ring))
            else:
                off = [(0, 0), (1, 0), (2, 0), (-1, 0), (-2, 0), (0, 1), (0, 2), (0, -1), (0, -2),
                       (1, -2), (2, -2)]
                rows["square"].append(np.stack([site(c + a, w + d) for a, d in off]))
        to = lambda v: torch.tensor(np.concatenate(v, axis=1), device=self.dev) if v else None
        self.square, self.tri = to(rows["square"]), to(rows["tri"])

    def _cells(self, tissues):
        """Search cells at least as wide as the reach, three or more per axis."""
        dims, start, total = [], [], 0
        for t in tissues:
            d = [max(3, int(t.lx / self.reach)), max(3, int(t.ly / self.reach)),
                 int(t.lz / self.reach) + 2]
            assert t.lx / d[0] >= self.reach and t.ly / d[1] >= self.reach
            dims.append(d)
            start.append(total)
            total += d[0] * d[1] * d[2]
        self.dims = torch.tensor(dims, device=self.dev)
        self.cell0 = torch.tensor(start, device=self.dev)
        self.ncells = total

    def _min(self, d, L):
        return d - L * torch.round(d / L)

    def build(self, X):
        """Pairs (i > j) within the reach, membrane pairs left out."""
        with torch.no_grad():
            X = [x.detach() for x in X]
            d = self.dims[self.tid]
            q = [torch.remainder((X[0] / self.lx * d[:, 0]).floor().long(), d[:, 0]),
                 torch.remainder((X[1] / self.ly * d[:, 1]).floor().long(), d[:, 1]),
                 (X[2] / self.reach).floor().long().clamp(min=0)]
            q[2] = torch.minimum(q[2], d[:, 2] - 1)
            cid = self.cell0[self.tid] + (q[0] * d[:, 1] + q[1]) * d[:, 2] + q[2]
            order = torch.argsort(cid, stable=True)
            counts = torch.bincount(cid, minlength=self.ncells)
            first = torch.cumsum(counts, 0) - counts
            most = int(counts.max())
            me = torch.arange(self.n, device=self.dev)
            out = []
            for ax in (-1, 0, 1):
                for ay in (-1, 0, 1):
                    nx, ny = torch.remainder(q[0] + ax, d[:, 0]), torch.remainder(q[1] + ay, d[:, 1])
                    for az in (-1, 0, 1):
                        nz = q[2] + az
                        ok = (nz >= 0) & (nz < d[:, 2])
                        c = torch.where(ok, self.cell0[self.tid] + (nx * d[:, 1] + ny) * d[:, 2] + nz, 0)
                        cnt, f0 = torch.where(ok, counts[c], 0), first[c]
                        for k in range(most):
                            i = me[cnt > k]
                            if i.numel() == 0:
                                break
                            j = order[f0[i] + k]
                            keep = (j < i) & ~(self.memb[i] & self.memb[j])
                            i, j = i[keep], j[keep]
                            dx = self._min(X[0][i] - X[0][j], self.lx[i])
                            dy = self._min(X[1][i] - X[1][j], self.ly[i])
                            dz = X[2][i] - X[2][j]
                            near = dx * dx + dy * dy + dz * dz <= (
                                1.2 * (self.r[i] + self.r[j]) + _SKIN) ** 2
                            out.append(torch.stack([i[near], j[near]]))
            ij = torch.cat(out, 1)
            self.at = X
            self.i, self.j = ij[0], ij[1]
            self.ptid = self.tid[self.i]
            self.rs = self.r[self.i] + self.r[self.j]
            self.both_old = self.old[self.i] & self.old[self.j]
        self._constants()

    def _p(self, k, t):
        v = self.par[k][t] if len(self.par[k]) > 1 else self.par[k][0]
        if self.s is not None:
            if k in ("der_der_const", "k_total", "k_desmosome", "kspring", "kspring_d",
                     "kspring_division"):
                v = v * self.s[0]
            elif k == "eps_m":
                v = v * self.s[1]
            elif k == "kbend":
                v = v * self.s[2]
        return v

    def _constants(self):
        t = self.ptid
        self.c_dt, self.c_lt = self._p("dt", t), self._p("lj_thresh", t)
        self.plx, self.ply = self.lx[self.i], self.ly[self.i]

    def _lj(self, e4, d2, rs):
        u = rs ** 6 / d2 ** 3
        return e4 * u * (u - 1) / d2

    def _adhesion(self, k, d, rs, lt):
        m = d / rs - 1
        c = -(k / d) * m * (1 - m * m / ((lt - 1) * (lt - 1)))
        return torch.where(m + 1 > lt, torch.zeros_like(c), c)

    def _pair_coef(self, d2, conn):
        t = self.ptid
        rs, d = self.rs, torch.sqrt(d2)
        e4 = 4 * self._p("eps_m", t)
        lt = self.c_lt
        near = d2 < rs * rs
        lj = self._lj(e4, d2, rs)
        ad = self._adhesion(torch.where(self.both_old, self._p("k_total", t),
                                        self._p("k_desmosome", t)), d, rs, lt)
        aad = torch.where(near, lj, ad)
        if self.simple:
            return torch.where(conn, aad, torch.zeros_like(aad))
        zero = torch.zeros_like(lj)
        fixmu = torch.where(near, lj, self._adhesion(self._p("k_desmosome", t), d, rs, lt))
        fix_memb = torch.where(near, lj, -(self._p("kspring", t) / d) * (d / rs - 1))
        dd = d + self._p("delta_r", t)
        u = rs ** 6 / dd ** 6
        h, para = e4 * u * (u - 1), self._p("para_ljp2", t)
        der = torch.where(dd < rs, h / (d * dd) + para, torch.where(near, para + zero, h / (d * d) + para))
        dermis = self._dermis(d2, conn)
        total = zero
        # what c applies while it iterates its connection o (cell_interaction.cpp:549-634)
        for c, o, higher in ((self.i, self.j, True), (self.j, self.i, False)):
            sc, so = self.st[c], self.st[o]
            aad_c = (sc == _ALIVE) | (sc == _AIR) | (sc == _DEAD)
            aad_o = (so == _ALIVE) | (so == _AIR) | (so == _DEAD)
            sfm = self.sfm[c]
            k = torch.where(sfm == 1, self._p("kspring", t),
                            torch.where(sfm == 2, self._p("kspring_d", t), zero))
            mu_memb = torch.where(near, lj, self._adhesion(k, d, rs, lt))
            apart = self.pair[c] != o
            is_d = (sc == _DER)
            total = total + torch.where(is_d, torch.where((so == _DER) & higher, der, lj), zero)
            total = total + torch.where(aad_c & ((aad_o & higher) | (~aad_o & (so != _DER))), aad, zero)
            fm = ((sc == _FIX) & apart & (((so == _FIX) & higher) | (so == _MUSUME))) | (
                (sc == _MUSUME) & apart & (so == _MUSUME) & higher)
            total = total + torch.where(fm, fixmu, zero)
            mine = dermis[c] == o
            total = total + torch.where((sc == _FIX) & (so == _MEMB), torch.where(mine, fix_memb, lj), zero)
            total = total + torch.where((sc == _MUSUME) & (so == _MEMB), torch.where(mine, mu_memb, lj), zero)
        return torch.where(conn, total, zero)

    def _dermis(self, d2, conn):
        """Nearest connected membrane particle of each FIX / MUSUME cell."""
        best = torch.full((self.n,), math.inf, dtype=torch.float64, device=self.dev)
        who = torch.full((self.n,), -1, dtype=torch.int64, device=self.dev)
        st_i = self.st[self.i]
        m = conn & ((st_i == _FIX) | (st_i == _MUSUME)) & self.memb[self.j]
        i, j, v = self.i[m], self.j[m], d2[m].detach()
        best.scatter_reduce_(0, i, v, "amin")
        hit = v == best[i]
        who[i[hit]] = j[hit]
        return who

    def _offsets(self, X, sites):
        c = sites[0]
        out = []
        for k in range(1, sites.shape[0]):
            q = sites[k]
            out.append(torch.stack([self._min(X[0][q] - X[0][c], self.lx[c]),
                                    self._min(X[1][q] - X[1][c], self.ly[c]), X[2][q] - X[2][c]]))
        return out

    def _bend(self, c):
        below = 1 + torch.where(c >= 0, torch.zeros_like(c), c)
        return torch.where(c >= 0, 1 - c, 1 / (below * below))

    def _membrane(self, X, D):
        for sites, tri in ((self.square, False), (self.tri, True)):
            if sites is None:
                continue
            c = sites[0]
            t = self.tid[c]
            o = self._offsets(X, sites)
            dt = self._p("dt", t)
            unit = lambda v: v / torch.sqrt((v * v).sum(0))
            dot = lambda a, b: (a * b).sum(0)
            cross = lambda a, b: torch.linalg.cross(a, b, dim=0)
            if tri:
                n, ring = o[:6], o[6:]
                f = 0
                for k in range(6):
                    a, b, e = n[k], n[(k + 1) % 6], n[(k + 2) % 6]
                    ab, be = a - b, b - e
                    n1, n2 = unit(cross(-b, ab)), unit(cross(ab, ring[k] - b))
                    p = dot(n1, n2)
                    f = f + self._bend(p) * cross(ab, n2 - p * n1)
                    n1, n2 = unit(cross(-e, be)), unit(cross(-b, ab))
                    p = dot(n1, n2)
                    f = f + self._bend(p) * (cross(be, n2 - p * n1) + cross(ab, n1 - p * n2))
                links = o[:6]
            else:
                r, rr, l, ll, u, uu, b, bb, bbr, bbrr = o
                size = lambda v: torch.sqrt((v * v).sum(0))
                nv, nvr, nvl, nvll = unit(r), unit(rr - r), unit(-l), unit(l - ll)
                mv, mvu, mvb, mvbb = unit(u), unit(uu - u), unit(-b), unit(b - bb)
                ipn, ipnl, ipnll = dot(nv, nvr), dot(nvl, nv), dot(nvll, nvl)
                ipm, ipmb = dot(mv, mvu), dot(mvb, mv)
                ipmbb = dot(unit(bbr - bb), unit(bbrr - bbr))  # as the reference has it (:380)
                dn, dnl, dm, dmb = size(r), size(l), size(u), size(b)
                half = lambda v, vr, vl, vll, p, q, w, da, db: (
                    -self._bend(p) * (vr - p * v) / da +
                    self._bend(q) * ((v - q * vl) / db - (vl - q * v) / da) +
                    self._bend(w) * (vll - w * vl) / db)
                f = (half(nv, nvr, nvl, nvll, ipn, ipnl, ipnll, dn, dnl) +
                     half(mv, mvu, mvb, mvbb, ipm, ipmb, ipmbb, dm, dmb))
                links = [l, r, b, u]
            f = (dt * self._p("kbend", t)) * f
            # lattice springs (CI_memb_to_memb) and the wall
            P, e4, kd = self._p("p_memb", t), 4 * self._p("eps_m", t), self._p("der_der_const", t)
            where = {6: sites[1:7], 4: [sites[3], sites[1], sites[7], sites[5]]}[len(links)]
            for v, q in zip(links, where):
                d2 = (v * v).sum(0)
                d, rs = torch.sqrt(d2), self.r[c] + self.r[q]
                cr2 = (rs * P) ** 2
                lam = torch.where(d2 < rs * rs, 2 * rs, (1 + P) * rs - d)
                u3 = (rs * P) ** 6 / lam ** 6
                far = -(kd / rs) * ((1 - P) / P) - e4 * u3 * (u3 - 1) / (lam * d)
                mid = -(kd / d) * (d / (rs * P) - 1)
                u1 = cr2 ** 3 / d2 ** 3
                w = torch.where(d2 < cr2, e4 * u1 * (u1 - 1) / d2, torch.where(d2 < rs * rs, mid, far))
                f = f - dt * w * v
            D = [D[k].index_add(0, c, f[k]) for k in range(3)]
        return D

    def step(self, X):
        with torch.no_grad():
            if max(float(((X[0] - self.at[0] - self.lx * torch.round((X[0] - self.at[0]) / self.lx)) ** 2 +
                          (X[1] - self.at[1] - self.ly * torch.round((X[1] - self.at[1]) / self.ly)) ** 2 +
                          (X[2] - self.at[2]) ** 2).max()), 0.0) > (_SKIN / 2) ** 2:
                self.build(X)
        i, j = self.i, self.j
        dx = self._min(X[0][i] - X[0][j], self.plx)
        dy = self._min(X[1][i] - X[1][j], self.ply)
        dz = X[2][i] - X[2][j]
        d2 = dx * dx + dy * dy + dz * dz
        conn = d2 <= self.c_lt * self.c_lt * self.rs * self.rs
        c = self.c_dt * self._pair_coef(d2, conn)
        D = [torch.zeros_like(X[0]) for _ in range(3)]
        D = [D[k].index_add(0, i, c * v).index_add(0, j, -c * v)
             for k, v in enumerate((dx, dy, dz))]
        D = self._membrane(X, D)
        # the wall under membrane and dermis (wall_interaction)
        t = self.tid
        w = (self.memb | (self.st == _DER)) & (X[2] < self.r)
        z = torch.where(w, X[2], self.r)
        u = self.r ** 6 / z ** 6
        wall = self._p("dt", t) * 4 * self._p("eps_m", t) * u * (u - 1) / (4 * z * z) * 2 * z
        D[2] = D[2] + torch.where(w, wall, torch.zeros_like(wall))
        if bool((self.pair >= 0).any()):
            a = torch.nonzero(self.pair >= 0)[:, 0]
            b = self.pair[a]
            v = [self._min(X[0][a] - X[0][b], self.lx[a]), self._min(X[1][a] - X[1][b], self.ly[a]),
                 X[2][a] - X[2][b]]
            d = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            k = -self._p("kspring_division", self.tid[a]) * (d - self.spr[torch.maximum(a, b)]) / d
            k = self._p("dt", self.tid[a]) * k
            D = [D[m].index_add(0, a, k * v[m]) for m in range(3)]
        X = [X[k] + D[k] for k in range(3)]
        for k, L in ((0, self.lx), (1, self.ly)):
            X[k] = torch.where(X[k] > L, X[k] - L, torch.where(X[k] < 0, X[k] + L, X[k]))
        return X

    def start(self, tissues):
        X = [torch.tensor(np.concatenate([getattr(t, k) for t in tissues]), dtype=torch.float64,
                          device=self.dev) for k in "xyz"]
        self.build(X)
        return X


def _exact_adjoint(case, seed, t, model):
    """Loss and gradient by automatic differentiation, recomputing segments."""
    from torch.utils.checkpoint import checkpoint
    model.s = torch.ones(3, dtype=torch.float64, device=model.dev, requires_grad=True)
    X = model.start([t])
    done, cells = 0, t.nmemb
    target = [torch.tensor(a, dtype=torch.float64, device=model.dev) for a in _target(t, seed)]

    def segment(k):
        def go(x, y, z, s):
            model.s = s
            model.build([x, y, z])
            v = [x, y, z]
            for _ in range(k):
                v = model.step(v)
            return v[0], v[1], v[2]
        return go

    s = model.s
    while done < case["steps"]:
        k = min(10, case["steps"] - done)
        X = list(checkpoint(segment(k), X[0], X[1], X[2], s, use_reentrant=False))
        done += k
    d = [model._min(X[0] - target[0], model.lx), model._min(X[1] - target[1], model.ly),
         X[2] - target[2]]
    loss = sum((v[cells:] ** 2).sum() for v in d) / (t.n - cells)
    loss.backward()
    return {"loss": loss.detach().reshape(1), "grad": s.grad.reshape(1, 3),
            "pos": [x.detach() for x in X]}


def _exact_maps(model, t, X, dims):
    """setup_map_lat (map.cpp:24-167): (cell index + 1 or 0, mask, highest cell)."""
    nx, ny, nz = dims
    dev, f64 = model.dev, torch.float64
    dx, dy, dz = t.lx / nx, t.ly / ny, t.lz / nz
    inv = (nx / t.lx, ny / t.ly, nz / t.lz)
    ir = [int(1.4 * n / L) for n, L in ((nx, t.lx), (ny, t.ly), (nz, t.lz))]
    cmap = torch.zeros((nx + 1) * (ny + 1) * (nz + 1), dtype=torch.int64, device=dev)
    mask = torch.zeros_like(cmap)
    lat = [(X[0] * inv[0]).long() % nx, (X[1] * inv[1]).long() % ny, (X[2] * inv[2]).long() % nz]
    afm = (model.st == _ALIVE) | (model.st == _FIX) | (model.st == _MUSUME)
    half = lambda d, L: torch.where(d > 0.5 * L, d - L, torch.where(d <= -0.5 * L, d + L, d))
    mark = torch.arange(1, t.n + 1, device=dev)
    r2, c2 = model.r * model.r, (2.0 * model.r) * (2.0 * model.r)
    for a in range(-2 * ir[0], 2 * ir[0] + 1):
        ka = lat[0] + a
        ex = half(ka.to(f64) * dx - X[0], t.lx)
        for b in range(-2 * ir[1], 2 * ir[1] + 1):
            kb = lat[1] + b
            ey = half(kb.to(f64) * dy - X[1], t.ly)
            wide = (abs(a) > ir[0]) | (abs(b) > ir[1])
            for c in range(-2 * ir[2], 2 * ir[2] + 1):
                kc = lat[2] + c
                use = (kc >= 1) & (kc < nz)
                if wide or abs(c) > ir[2]:
                    use = use & afm
                ez = kc.to(f64) * dz - X[2]
                d2 = (ex * ex + ey * ey) + ez * ez
                v = ((ka + nx) % nx * (ny + 1) + (kb + ny) % ny) * (nz + 1) + kc
                m = use & (d2 < r2)
                cmap.scatter_reduce_(0, v[m], mark[m], "amax")
                m = use & afm & (d2 < c2)
                mask[v[m]] = 1
    cmap, mask = (g.reshape(nx + 1, ny + 1, nz + 1) for g in (cmap, mask))
    for g in (mask, cmap):
        g[:, ny, :nz] = g[:, 0, :nz]
        g[nx, :, :nz] = g[0, :, :nz]
    alive = (model.st == _DEAD) | afm
    return cmap, mask, max(0.0, float(X[2][alive].max()) if bool(alive.any()) else 0.0)


def _exact_field(case, seed, t, model):
    nx, ny, nz = dims = _grid(t)
    dev = model.dev
    cur = torch.tensor(_stimulus(dims, seed), device=dev)
    nxt = cur.clone()
    X = model.start([t])
    inv_dz = nz / t.lz
    for _ in range(case["steps"]):
        X = model.step(X)
        cmap, mask, zz = _exact_maps(model, t, X, dims)
        izb = min(int((zz + 2.0 * 1.4) * inv_dz), nz)
        c = cur[:nx, :ny, :izb]
        up = torch.arange(izb, device=dev)
        pz, nz_ = (up - 1).abs(), torch.where(up + 1 == nz, nz - 1, up + 1)
        total = 0
        for at in ((-1, 0), (0, -1), None, None, (0, 1), (1, 0)):
            if at is None:
                continue
            g, m = (torch.roll(v[:nx, :ny, :izb], (-at[0], -at[1]), (0, 1)) for v in (cur, mask))
            total = total + m * (g - c)
        for q in (pz, nz_):
            total = total + mask[:nx, :ny][:, :, q] * (cur[:nx, :ny][:, :, q] - c)
        cell = cmap[:nx, :ny, :izb] - 1
        st = torch.where(cell >= 0, model.st[cell.clamp(min=0)], -1)
        age = torch.where((st == _DEAD) | (st == _ALIVE), model.agek[cell.clamp(min=0)], 0.0)
        on = (age > 22.0 - 0.5) & (age <= 22.0 + 2.0)
        new = c + 0.01 * (0.0009 * total * inv_dz * inv_dz + (on.to(c.dtype) - 0.025 * c))
        nxt[:nx, :ny, :izb] = new
        nxt[:nx, ny, :izb] = nxt[:nx, 0, :izb]
        nxt[nx, :, :izb] = nxt[0, :, :izb]
        cur, nxt = nxt, cur
    return {"cmap1": None, "cmap2": None, "ext": cur, "zzmax": zz, "pos": X}


def exact(case, seed):
    if case["kind"] == "noalloc":
        return None  # whole numbers only
    ts = _tissues(case, seed)
    model = _Model(ts, torch.device("cuda" if torch.cuda.is_available() else "cpu"))
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, ts[0], model)
    if case["kind"] == "field":
        return _exact_field(case, seed, ts[0], model)
    with torch.no_grad():
        X = model.start(ts)
        for _ in range(case["steps"]):
            X = model.step(X)
    if case["kind"] == "dropin":
        return {"pos": X, "off": None, "idx": None, "dermis": None}
    return X
