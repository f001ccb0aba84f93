"""Performance cases of the T-mixer framework: the work that its users have it
do, through the public Python entry points (``Solver``, ``Batch``).

Three kinds of case:

  solve    one mixer advanced by a run of steps, then its mixing statistics or
           totals and all its macroscopic fields read, as a user does between
           two outputs of a solve;
  batch    many mixers of uneven size and parameters advanced together by one
           chunk of the request loop, then every mixer's outlet mixing index
           and health flag, and the fields of the mixers that retire;
  output   what is written about a solve that stands at an output step: the
           totals, the mixing rows, the pressure and power rows, all fields.

Sizes are those of the repository's own configurations and tests (the small
grid of the golden fixtures, the W-layout widths 4 to 64, the reference's
401 x 51 x 51 + 101 x 750 x 51 case) and ragged boxes in between.  Parameters
(velocity, relaxation times, rate, inlet concentrations) come from the seed,
in the ranges of the batched configuration.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tmixer_b200 as T

FORMS = ("fp64", "fp32", "fp16")
# bytes of one lattice update: 76 populations read and written (the FP16 form
# also reads and writes its 32-byte moment record)
LUP_BYTES = {"fp64": 1216, "fp32": 608, "fp16": 368}
LUP_FLOPS = 900  # sums, momentum, equilibria, collision and reaction of four fields


def _wbox(W: int) -> dict:
    return dict(inx=8 * W, iny=W, nz=W, mnx=2 * W, mny=4 * W, ia=3 * W + 1)


def _solve(name: str, form: str, steps: int, box: dict) -> dict:
    return dict(name=name, kind="solve", form=form, steps=steps, **box)


REFERENCE = dict(inx=401, iny=51, nz=51, mnx=101, mny=750, ia=151)
TINY = dict(inx=21, iny=7, nz=7, mnx=7, mny=14, ia=8)
# widths of the batched configuration (16, 24, 32, 48), 64 of them
BATCH64 = ",".join(str(w) for w in [16, 48, 24, 32, 32, 16, 48, 24] * 8)


def listed() -> list:
    return [
        # the smallest grid of the repository's fixtures: launch latency of
        # every kernel of a step
        _solve("fp64-tiny", "fp64", 100, TINY),
        # the single-mixer benchmark configuration in its bit-exact form
        _solve("fp64-w32", "fp64", 500, _wbox(32)),
        # the reference's own case, its largest (odd sizes, 4.9M nodes)
        _solve("fp64-reference", "fp64", 400, REFERENCE),
        # an ordinary mixer whose mixing box (48 wide) is no multiple of a warp
        _solve("fp32-w24", "fp32", 1000, _wbox(24)),
        # the precision configuration's width, FP32 storage
        _solve("fp32-w64", "fp32", 500, _wbox(64)),
        # a small mixer in the served form's storage, one at a time
        _solve("fp16-w8", "fp16", 500, _wbox(8)),
        # the single-mixer configuration, FP16 storage
        _solve("fp16-w32", "fp16", 1000, _wbox(32)),
        # the reference's case in FP16 storage
        _solve("fp16-reference", "fp16", 600, REFERENCE),
        # a few bit-exact mixers side by side (a small parameter study)
        dict(name="fp64-batch4", kind="batch", form="fp64", steps=100, widths="16,24,12,20", tune=False, retire=4),
        # a handful of small requests as a program serves them that did not tune
        dict(name="fp16-batch8", kind="batch", form="fp16", steps=100, widths="8,16,12,24,9,16,10,20", tune=False,
             retire=2),
        # the served form's working set: 64 mixers, tuned launch shape, one
        # convergence-check chunk, one mixer retiring
        dict(name="fp16-batch64", kind="batch", form="fp16", steps=100, widths=BATCH64, tune=True, retire=1),
        # everything that is written at an output step of a middling solve
        dict(name="fp64-output-w48", kind="output", form="fp64", steps=40, **_wbox(48)),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nodes(c: dict) -> int:
    return c["nz"] * (c["inx"] * c["iny"] + c["mnx"] * c["mny"])


def _ragged(rng) -> dict:
    """Boxes of any proportions, 5 thousand to 3 million nodes."""
    while True:
        nz, iny = _log_int(rng, 5, 70), _log_int(rng, 5, 70)
        mnx = _log_int(rng, 5, 130)
        inx = mnx + 2 + _log_int(rng, 4, 400)
        b = dict(inx=inx, iny=iny, nz=nz, mnx=mnx, mny=_log_int(rng, 5, 500), ia=rng.randint(2, inx - mnx))
        if 5000 <= _nodes(b) <= 3000000:
            return b


def draw(rng) -> dict:
    form = rng.choice(FORMS)
    kind = rng.choice(("solve", "solve", "solve", "batch", "batch", "output"))
    if kind == "batch":
        n = _log_int(rng, 2, 40)
        widths = [_log_int(rng, 5, 40) for _ in range(n)]
        lups = sum(16 * w ** 3 for w in widths)
        steps = max(20, min(300, int(1.5e9 / lups)))
        return dict(kind=kind, form=form, steps=steps, widths=",".join(map(str, widths)), tune=rng.random() < 0.5,
                    retire=min(2, n))
    box = _wbox(_log_int(rng, 4, 46)) if rng.random() < 0.5 else _ragged(rng)
    steps = 40 if kind == "output" else max(20, min(600, int(1.5e9 / _nodes(box))))
    return dict(kind=kind, form=form, steps=steps, **box)


# ---------------------------------------------------------------------------
# inputs: case constants from the seed
# ---------------------------------------------------------------------------
def _params(rng: np.random.Generator, box: dict) -> dict:
    """Parameters in the batched configuration's ranges: velocity maximum 0.02
    to 0.08 (a duct's mean is about half its maximum), tau_f 0.6 to 0.8, tau_c
    0.52 to 0.7, k 1e-4 to 1e-2, species A at inlet 1 and B at inlet 2."""
    tau_c = float(rng.uniform(0.52, 0.7))
    rho = float(rng.uniform(1.0, 3.0))
    ca, cb = float(rng.uniform(0.5, 1.0)), float(rng.uniform(0.5, 1.0))
    return dict(box, tau=float(rng.uniform(0.6, 0.8)), tau_a=tau_c, tau_b=tau_c, tau_c=tau_c, rho0=rho, rho_out=rho,
                c_in=[[ca, 0.0], [0.0, cb], [0.0, 0.0]], rateconst=float(10 ** rng.uniform(-4, -2)),
                umean=float(rng.uniform(0.01, 0.035)))


def _inputs(case: dict, seed: int) -> list:
    """The parameter sets of a case's mixers."""
    rng = np.random.default_rng([seed, 20261203])
    if case["kind"] == "batch":
        return [_params(rng, _wbox(int(w))) for w in case["widths"].split(",")]
    return [_params(rng, {k: case[k] for k in ("inx", "iny", "nz", "mnx", "mny", "ia")})]


# the macroscopic fields as a user keeps them: density, velocity and species of
# both boxes, each group one array (box by box, field by field)
GROUPS = {"density": ("rho",), "velocity": ("ux", "uy", "uz"), "species": ("cA", "cB", "cC")}


def _read_fields(read, groups=GROUPS):
    """The groups from a reader of one field of one box."""
    return {g: np.concatenate([read(b, f).ravel() for b in (0, 1) for f in names]) for g, names in groups.items()}


def _buffers(p: dict):
    """Host buffers of a mixer's groups, and each field's place in them."""
    shapes = ((p["inx"], p["iny"], p["nz"]), (p["mnx"], p["mny"], p["nz"]))
    sizes = [math.prod(s) for s in shapes]
    out, view = {}, {}
    for g, names in GROUPS.items():
        # (filled, as a program's buffers are after its first output)
        out[g] = np.zeros(len(names) * sum(sizes))
        at = 0
        for b in (0, 1):
            for f in names:
                view[b, f] = out[g][at: at + sizes[b]].reshape(shapes[b])
                at += sizes[b]
    return out, view


def prepare(case: dict, seed: int):
    """What a user's program has in hand: a started solve and the host buffers
    that it reads the fields into, or a batch with its mixers admitted (and
    tuned, where the program tunes)."""
    form = T.PRECISIONS[case["form"]]
    specs = [T.CaseSpec(precision=form, **p) for p in _inputs(case, seed)]
    if case["kind"] == "batch":
        B = T.Batch(form, budget=sum(T.Batch.footprint(s) for s in specs) + (1 << 20))
        slots = [B.add(s) for s in specs]
        if case["tune"]:
            B.tune(10)
        return case, B, slots
    S = T.Solver(specs[0]).init()
    if case["kind"] == "output":
        S.step(case["steps"])
        S.sync()
    return case, S, _buffers(_inputs(case, seed)[0])


def run(state):
    case, h, at = state
    if case["kind"] == "batch":
        h.step(case["steps"])
        im = h.outlet_im(at)
        bad = h.health(at)
        fields = [_read_fields(lambda b, f: h.field(at[m], b, f)) for m in range(case["retire"])]
        return dict(fields=fields, im=im, bad=np.array(bad))
    out = {}
    if case["kind"] == "output":
        rows, im = h.mixing()
        prow, px, pw, units = h.pressure_power()
        out.update(rows=rows, im=im, prow=prow, px=px, pw=pw, units=units, sums=h.sums())
    else:
        h.step(case["steps"])
        # the bit-exact form's user follows the mixing index, the reduced
        # forms' also watches their FP64 totals
        if case["form"] == "fp64":
            out["rows"], out["im"] = h.mixing()
        else:
            out["sums"] = h.sums()
    out["fields"], views = at
    for (b, f), v in views.items():
        h.field(b, f, out=v)
    return out


def work(case: dict) -> dict:
    if case["kind"] == "batch":
        ws = [int(w) for w in case["widths"].split(",")]
        n = sum(16 * w ** 3 for w in ws)
        out = sum(16 * w ** 3 for w in ws[: case["retire"]])
    else:
        n = out = _nodes(case)
    if case["kind"] == "output":  # the seven fields read and returned
        return {"bytes": 112 * n, "flops": 60 * n}
    return {"bytes": case["steps"] * n * LUP_BYTES[case["form"]] + 112 * out, "flops": case["steps"] * n * LUP_FLOPS}


def tolerance(case: dict):
    # FP64: the same operations in the same order as the reference, bit for
    # bit.  FP32 and FP16: the largest error against exact() over the listed
    # cases and 14 drawn ones was 1.5e-4 (velocity after 1000 steps; density
    # and species 2e-5 or less), times four.
    if case["form"] == "fp64":
        return "exact"
    return {"rel": 6e-4}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
E = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
     (-1, -1, 0), (1, -1, 0), (1, 0, 1), (-1, 0, 1), (-1, 0, -1), (1, 0, -1), (0, 1, 1), (0, -1, 1), (0, -1, -1),
     (0, 1, -1)]
IDX = {e: q for q, e in enumerate(E)}
OPP = [IDX[tuple(-c for c in e)] for e in E]


def _inlets(p: dict, dev):
    """Uin1[j, k] and Uin2[j, k], 0-based nodes: the rectangular-duct series
    scaled to its mean, shifted by one node in z."""
    ny, nz = p["iny"], p["nz"]
    d, w = (nz - 1.0) / 2.0, (ny - 1.0) / 2.0
    ar = w / d
    odd = torch.arange(1, 101, 2, dtype=torch.float64, device=dev)
    j = torch.arange(ny, dtype=torch.float64, device=dev)
    k = torch.arange(nz, dtype=torch.float64, device=dev)
    sm = torch.sin(odd[:, None] * math.pi / (2.0 * ar * d) * j[None, :])
    sn = torch.sin(odd[:, None] * math.pi / (2.0 * d) * k[None, :])
    den = odd[:, None] * odd[None, :] * (odd[:, None] ** 2 + ar * ar * odd[None, :] ** 2)
    raw = torch.einsum("mj,mn,nk->jk", sm, 4.0 / den, sn)
    raw = raw * (p["umean"] / raw.mean())
    u1, u2 = torch.zeros_like(raw), torch.zeros_like(raw)
    # the profile one node down in z for inlet 1 and one up, negated, for
    # inlet 2; nothing on the first (second) side's end plane
    u1[:, :-1] = raw[:, 1:]
    u1[:, 0] = 0.0
    u2[:, 1:] = -raw[:, :-1]
    u2[:, -1] = 0.0
    return u1, u2


class _Exact:
    """One mixer in 64 bits.  State: the post-collision populations fn[box]
    (4 fields, 19 directions, x, y, z) and the densities r[box] of the step
    before.  0-based node indices."""

    def __init__(self, p: dict, dev):
        self.p, self.dev = p, dev
        self.nx, self.ny, self.nz = (p["inx"], p["mnx"]), (p["iny"], p["mny"]), p["nz"]
        self.a = p["ia"] - 1  # first inlet column over the opening
        self.b = self.a + p["mnx"] - 1
        f64 = dict(dtype=torch.float64, device=dev)
        self.ev = torch.tensor(E, **f64)
        self.w = torch.tensor([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, **f64)
        self.tau = torch.tensor([p["tau"], p["tau_a"], p["tau_b"], p["tau_c"]], **f64)
        self.sgn = torch.tensor([0.0, -1.0, -1.0, 2.0], **f64)
        self.cin = p["c_in"]
        self.u1, self.u2 = _inlets(p, dev)
        self.zero = torch.tensor([p["rho_out"], 0.0, 0.0, 0.0], **f64)
        self.r, self.u, self.fn = [], [], []
        for bx in (0, 1):
            shape = (self.nx[bx], self.ny[bx], self.nz)
            r = torch.zeros((4,) + shape, **f64)
            r[0] = p["rho0"]
            self.r.append(r)
            self.u.append(torch.zeros((3,) + shape, **f64))
            f = torch.zeros((4, 19) + shape, **f64)
            f[0] = p["rho0"] * self.w[:, None, None, None]
            self.fn.append(f)
        # two post-collision sets: one holds the step's sources
        self.f = [torch.zeros_like(x) for x in self.fn]
        for bx in (0, 1):
            self.f[bx].copy_(self.fn[bx])
            self._collide(bx)

    def _collide(self, bx: int):
        r, u, f, fn = self.r[bx], self.u[bx], self.f[bx], self.fn[bx]
        u2 = 1.5 * (u * u).sum(0)
        rt = self.p["rateconst"] * r[1] * r[2]
        om = (1.0 / self.tau)[:, None, None, None]
        for q in range(19):
            eu = self.ev[q, 0] * u[0] + self.ev[q, 1] * u[1] + self.ev[q, 2] * u[2]
            g = self.w[q] * (1.0 + 3.0 * eu + 4.5 * eu * eu - u2)
            fn[:, q] = f[:, q] + om * (r * g - f[:, q]) + self.sgn[:, None, None, None] * (self.w[q] * rt)

    def _stream(self):
        """Pull: own box, then the two rows that meet at the opening."""
        a, b, nz = self.a, self.b, self.nz
        for bx in (0, 1):
            f, fn, n = self.f[bx], self.fn[bx], (self.nx[bx], self.ny[bx], nz)
            for q, e in enumerate(E):
                dst = tuple(slice(max(c, 0), m + min(c, 0)) for c, m in zip(e, n))
                src = tuple(slice(max(-c, 0), m + min(-c, 0)) for c, m in zip(e, n))
                f[(slice(None), q) + dst] = fn[(slice(None), q) + src]
        f0, f1, fn0, fn1 = self.f[0], self.f[1], self.fn[0], self.fn[1]
        m = self.nx[1]
        for q, (ex, ey, ez) in enumerate(E):
            zd = slice(max(ez, 0), nz + min(ez, 0))
            zs = slice(max(-ez, 0), nz + min(-ez, 0))
            if ey == 1:  # inlet row 0 over the opening, from the mixing box's last row
                f0[:, q, a + max(ex, 0): a + m + min(ex, 0), 0, zd] = \
                    fn1[:, q, max(-ex, 0): m + min(-ex, 0), -1, zs]
            elif ey == -1:  # the mixing box's last row, from inlet row 0
                f1[:, q, :, -1, zd] = fn0[:, q, a - ex: a - ex + m, 0, zs]

    # -- closures on a node set (box, x, y, z: ints or slices) ---------------
    def _v(self, s):
        return self.f[s[0]][(slice(None), slice(None)) + s[1:]]

    def _face(self, s, axis: int, n: int, nb=None, outlet=None):
        """A wall face with inward normal n along an axis: bounce back with the
        transverse correction for the flow; the species are those pulled by
        the interior neighbour nb.  outlet: the pinned density of the outlet."""
        v = self._v(s)[0]
        t1, t2 = [c for c in range(3) if c != axis]
        par = lambda t: sum(v[q] * E[q][t] for q in range(19) if E[q][axis] == 0 and E[q][t])  # noqa: E731
        # half the tangential momentum of the directions along the wall
        half = {t: 0.5 * par(t) for t in (t1, t2)}
        new = {}
        ru = 0.0
        if outlet is not None:
            ru = outlet - (sum(v[q] for q in range(19) if E[q][axis] == 0)
                           + 2.0 * sum(v[q] for q in range(19) if E[q][axis] == -n))
        for q in range(19):
            e = E[q]
            if e[axis] != n:
                continue
            o = v[OPP[q]]
            if e[t1] == 0 and e[t2] == 0:
                new[q] = o + ru / 3.0
            else:
                t = t1 if e[t1] else t2
                new[q] = o + ru / 6.0 - e[t] * half[t]
        for q, x in new.items():
            v[q] = x
        self._v(s)[1:] = self._v(nb)[1:]

    def _inlet(self, side: int):
        x = 0 if side == 0 else self.nx[0] - 1
        n = 1 if side == 0 else -1
        s = (0, x, slice(1, -1), slice(1, -1))
        v = self._v(s)
        U = (self.u1 if side == 0 else self.u2)[1:-1, 1:-1]
        rho = self._inlet_rho(side, slice(1, -1), slice(1, -1))
        new = {}
        for q in range(19):
            if E[q][0] != n:
                continue
            o, w = OPP[q], self.w[q]
            t = next((c for c in (1, 2) if E[q][c]), None)
            if t is None:
                flow = v[0, o] + n * rho * U / 3.0
            else:
                par = sum(v[0, p] * E[p][t] for p in range(19) if E[p][0] == 0 and E[p][t])
                flow = v[0, o] + n * rho * U / 6.0 - E[q][t] * 0.5 * par
            new[q] = [flow] + [2.0 * w * self.cin[c][side] - v[1 + c, o] for c in range(3)]
        for q, x in new.items():
            for fl in range(4):
                v[fl, q] = x[fl]

    def _inlet_rho(self, side: int, y, z):
        n = 1 if side == 0 else -1
        v = self.f[0][0, :, 0 if side == 0 else self.nx[0] - 1, y, z]
        U = (self.u1 if side == 0 else self.u2)[y, z]
        return (sum(v[q] for q in range(19) if E[q][0] == 0) + 2.0 * sum(v[q] for q in range(19) if E[q][0] == -n)) \
            / (1.0 - n * U)

    def _edge(self, s, ax1: int, n1: int, ax2: int, n2: int, dens=None):
        """An edge between walls with inward normals n1 along ax1 and n2 along
        ax2: bounce back of the directions that point inward, the momentum
        along the edge spread over the mixed ones, and the buried pair from a
        density (dens: a value per field) or the mean of its own two
        post-collision values."""
        v = self._v(s)
        t = 3 - ax1 - ax2
        corr = 0.25 * (v[:, IDX[self._unit(t, 1)]] - v[:, IDX[self._unit(t, -1)]]).clone()
        new = {}
        buried = []
        for q in range(1, 19):
            e = E[q]
            i1, i2 = e[ax1] * n1, e[ax2] * n2
            if i1 * i2 == -1:
                buried.append(q)
            elif i1 > 0 or i2 > 0:
                new[q] = v[:, OPP[q]] - (e[t] * corr if e[t] else 0.0)
        for q, x in new.items():
            v[:, q] = x
        self._pair(s, buried, dens)

    def _pair(self, s, pair, dens):
        v = self._v(s)
        if dens is None:
            own = self.fn[s[0]][(slice(None), slice(None)) + s[1:]]
            x = 0.5 * (own[:, pair[0]] + own[:, pair[1]])
        else:
            x = 0.5 * (dens - sum(v[:, q] for q in range(19) if q not in pair))
        v[:, pair[0]] = x
        v[:, pair[1]] = x

    @staticmethod
    def _unit(axis: int, n: int):
        e = [0, 0, 0]
        e[axis] = n
        return tuple(e)

    @staticmethod
    def _buried_yz(ny: int, nz: int):
        """The pair in the y-z plane that points along neither normal."""
        return IDX[(0, 1, -ny * nz)], IDX[(0, -1, ny * nz)]

    def _corner(self, s, n, closed=None, dens=None):
        """A corner with inward normals n: bounce back of the six directions
        that point inward, the buried pairs averaged from their own
        post-collision values, the closed pair (if any) from a density."""
        v = self._v(s)
        own = self.fn[s[0]][(slice(None), slice(None)) + s[1:]]
        new, pairs = {}, []
        for q in range(1, 19):
            c = [E[q][t] * n[t] for t in range(3) if E[q][t]]
            if all(x > 0 for x in c):
                new[q] = v[:, OPP[q]]
            elif min(c) < 0 < max(c) and q < OPP[q]:
                pairs.append((q, OPP[q]))
        for q, x in new.items():
            v[:, q] = x
        for q, o in pairs:
            if closed is None or q not in closed:
                x = 0.5 * (own[:, q] + own[:, o])
                v[:, q] = x
                v[:, o] = x
        if closed is not None:
            self._pair(s, closed, dens)

    def _junction(self, x: int, closed):
        """The edge where the opening's rim meets the inlet box's y wall."""
        s = (0, x, 0, slice(1, -1))
        v, own = self._v(s), self.fn[0][:, :, x, 0, 1:-1]
        for q in range(1, 19):
            if q < OPP[q] and q not in closed:
                m = 0.5 * (own[:, q] + own[:, OPP[q]])
                v[:, q] = m
                v[:, OPP[q]] = m
        self._pair(s, closed, self.r[0][:, x, 1, 1:-1])

    def _boundary(self):
        a, b, NX, NY, M, Y = self.a, self.b, self.nx[0] - 1, self.ny[0] - 1, self.nx[1] - 1, self.ny[1] - 1
        Z = self.nz - 1
        r0, r1, rout = self.r[0], self.r[1], self.p["rho_out"]
        i = slice(1, -1)
        lo, hi = slice(1, a), slice(b + 1, NX)  # inlet columns beside the opening
        op = slice(a + 1, b)  # and over it

        def flow_now(side, y, z, old):  # the inlets' flow density of this step
            d = old.clone()
            d[0] = self._inlet_rho(side, y, z)
            return d

        def pinned(old):
            d = old.clone()
            d[0].fill_(rout)
            return d

        # densities of this step that edges beside the inlets close with,
        # before the inlets change their populations (they do not depend on
        # the populations that the inlets set)
        dens = {}
        for side, x in ((0, 0), (1, NX)):
            dens[side, "z1"] = flow_now(side, i, 1, r0[:, x, 1:-1, 1])
            dens[side, "y1"] = flow_now(side, 1, i, r0[:, x, 1, 1:-1])
            dens[side, "yt"] = flow_now(side, NY - 1, i, r0[:, x, NY - 1, 1:-1])
            dens[side, "zt"] = r0[:, x, 1:-1, Z - 1]
        for xs in (lo, hi):  # edges along x at y = 0
            self._edge((0, xs, 0, Z), 1, 1, 2, -1)
            self._edge((0, xs, 0, 0), 1, 1, 2, 1)
        for z, n in ((Z, -1), (0, 1)):
            self._edge((0, i, NY, z), 1, -1, 2, n)
        for side, x, n in ((0, 0, 1), (1, NX, -1)):
            self._edge((0, x, i, 0), 0, n, 2, 1, dens[side, "z1"])
            # species C keeps one of its own two values at the first inlet's
            # upper edge (the reference's slip of a letter)
            self._edge((0, x, i, Z), 0, n, 2, -1, dens[side, "zt"])
            if side == 0:
                s = (0, 0, i, Z)
                v = self._v(s)
                q, o = IDX[(1, 0, 1)], IDX[(-1, 0, -1)]
                own = self.fn[0][3, o, 0, 1:-1, Z]
                rest = sum(v[3, p] for p in range(19) if p not in (q, o))
                v[3, q] = 0.5 * (dens[0, "zt"][3] - rest)
                v[3, o] = own
            self._edge((0, x, 0, i), 0, n, 1, 1, dens[side, "y1"])
            self._edge((0, x, NY, i), 0, n, 1, -1, dens[side, "yt"])
        # corners of the inlet box
        for x, nx in ((0, 1), (NX, -1)):
            for y, ny in ((NY, -1), (0, 1)):
                for z, nz in ((Z, -1), (0, 1)):
                    d = r0[:, x, y, Z - 1 if z == Z else 1]
                    self._corner((0, x, y, z), (nx, ny, nz), self._buried_yz(ny, nz), d)
        # corners of the mixing box at the outlet: species close with zero
        zero = self.zero
        for x, nx in ((0, 1), (M, -1)):
            for z, nz in ((0, 1), (Z, -1)):
                self._corner((1, x, 0, z), (nx, 1, nz), self._buried_yz(1, nz), zero)
        # corners of the opening's rim: the walls there are z and the rim;
        # six directions bounce back, the others average
        for x, sx in ((a, 1), (b, -1)):
            for z, nz in ((Z, -1), (0, 1)):
                self._rim((0, x, 0, z), sx, nz)
        # edges of the mixing box
        for z, n in ((0, 1), (Z, -1)):
            self._edge((1, i, 0, z), 1, 1, 2, n, pinned(r1[:, 1:-1, 1, z]))
            for x, nx in ((0, 1), (M, -1)):
                self._edge((1, x, slice(1, None), z), 0, nx, 2, n)
        for x, n in ((0, 1), (M, -1)):
            self._edge((1, x, 0, i), 0, n, 1, 1, pinned(r1[:, x, 1, 1:-1]))
        self._junction(a, (IDX[(1, 1, 0)], IDX[(-1, -1, 0)]))
        self._junction(b, (IDX[(-1, 1, 0)], IDX[(1, -1, 0)]))
        # faces
        self._inlet(0)
        self._inlet(1)
        self._face((0, i, NY, i), 1, -1, (0, i, NY - 1, i))
        for xs in (lo, hi):
            self._face((0, xs, 0, i), 1, 1, (0, xs, 1, i))
        self._face((1, i, 0, i), 1, 1, (1, i, 1, i), rout)
        up = slice(1, None)
        self._face((1, 0, up, i), 0, 1, (1, 1, up, i))
        self._face((1, M, up, i), 0, -1, (1, M - 1, up, i))
        for z, n, zn in ((Z, -1, Z - 1), (0, 1, 1)):
            self._face((0, i, i, z), 2, n, (0, i, i, zn))
            self._face((0, op, 0, z), 2, n, (0, op, 0, zn))
            self._face((1, i, up, z), 2, n, (1, i, up, zn))

    def _rim(self, s, sx: int, nz: int):
        """A corner of the opening's rim: the z direction, its four diagonals
        and the upward diagonal away from the rim bounce back, the other
        three pairs average their own post-collision values."""
        v = self._v(s)
        own = self.fn[0][(slice(None), slice(None)) + s[1:]]
        back = [IDX[(0, 0, nz)]] + [IDX[(x, 0, nz)] for x in (1, -1)] + [IDX[(0, y, nz)] for y in (1, -1)]
        back.append(IDX[(sx, 1, 0)])
        new = {q: v[:, OPP[q]] for q in back}
        used = set(back) | {OPP[q] for q in back}
        for q in range(1, 19):
            if q not in used:
                new[q] = 0.5 * (own[:, q] + own[:, OPP[q]])
        for q, x in new.items():
            v[:, q] = x.clone()

    def step(self):
        self._stream()
        self._boundary()
        for bx in (0, 1):
            f = self.f[bx]
            self.r[bx].copy_(f.sum(1))
            if bx == 1:
                self.r[1][0, :, 0, :].fill_(self.p["rho_out"])
            for c in range(3):
                m = sum(f[0, q] * E[q][c] for q in range(19) if E[q][c])
                self.u[bx][c] = m / self.r[bx][0]
            self._collide(bx)

    def advance(self, n: int):
        if self.dev == "cpu" or n < 8:
            for _ in range(n):
                self.step()
            return self
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            self.step()
            self.step()
        torch.cuda.current_stream().wait_stream(side)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self.step()
        for _ in range(n - 2):
            g.replay()
        torch.cuda.synchronize()
        return self

    # -- outputs ---------------------------------------------------------------
    def fields(self) -> dict:
        at = {"rho": (self.r, 0), "ux": (self.u, 0), "uy": (self.u, 1), "uz": (self.u, 2), "cA": (self.r, 1),
              "cB": (self.r, 2), "cC": (self.r, 3)}
        return _read_fields(lambda b, f: at[f][0][b][at[f][1]].cpu().numpy())

    def sums(self) -> np.ndarray:
        tot = [float(self.r[0][f].sum() + self.r[1][f].sum()) for f in range(4)]
        flux = float((self.r[1][0, :, 0] * self.u[1][1, :, 0]).sum())
        return np.array(tot + [sum(tot[1:]), flux, 0.0, float(_nodes(self.p))])

    def pressure_power(self):
        p, nz, mnx = self.p, self.nz, self.nx[1]
        top = slice(self.a, self.b + 1)
        rows = torch.cat([self.r[1][0].sum((0, 2)), self.r[0][0, top].sum((0, 2))]) / (nz * mnx) / 3.0
        prow = np.empty((rows.numel(), 3))
        prow[:, 0] = np.arange(1, rows.numel() + 1)
        prow[:, 1] = rows.cpu().numpy()
        prow[:, 2] = prow[:, 1] - prow[-1, 1]
        px = np.empty((self.nx[0], 2))
        px[:, 0] = np.arange(1, self.nx[0] + 1)
        px[:, 1] = (self.r[0][0].mean((1, 2)) / 3.0).cpu().numpy()
        i = slice(1, -1)
        u = self.u[1]
        dx = 0.5 * (u[:, 2:, i, i] - u[:, :-2, i, i])
        dy = 0.5 * (u[:, i, 2:, i] - u[:, i, :-2, i])
        dz = 0.5 * (u[:, i, i, 2:] - u[:, i, i, :-2])
        xz, xy, yz = dz[0] + dx[2], dx[1] + dy[0], dz[1] + dy[2]
        sec = dx[0] ** 2 + dz[2] ** 2 + 0.5 * xz ** 2
        tot = dx[0] ** 2 + dy[1] ** 2 + dz[2] ** 2 + 0.5 * (xy ** 2 + xz ** 2 + yz ** 2)
        k = 2.0 * (2.0 * p["tau"] - 1.0) / 6.0 / ((nz - 2) * (mnx - 2))
        pw = np.empty((self.ny[1] - 2, 5))
        pw[:, 0] = np.arange(2, self.ny[1])
        for c, x in enumerate((sec[-1].sum(1), tot[-1].sum(1), sec.sum((0, 2)), tot.sum((0, 2)))):
            pw[:, 1 + c] = (k * x).cpu().numpy()
        return prow, px, pw


# steps x nodes (and steps x mixers, each a graph of its own) that take the
# plain torch form under 20 seconds
EXACT_LUPS, EXACT_STEPS = 3.5e9, 8000


def exact(case: dict, seed: int):
    inputs = _inputs(case, seed)
    keep = case["retire"] if case["kind"] == "batch" else 1
    if case["steps"] * sum(_nodes(p) for p in inputs[:keep]) > EXACT_LUPS or case["steps"] * keep > EXACT_STEPS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        # (the outlet index is undefined until all species reach the outlet)
        return dict(fields=[_Exact(p, dev).advance(case["steps"]).fields() for p in inputs[:keep]], im=None, bad=None)
    x = _Exact(inputs[0], dev).advance(case["steps"])
    if case["kind"] == "output":
        prow, px, pw = x.pressure_power()
        # the mixing rows of a field that has not spread yet are differences
        # of nearly equal numbers
        return dict(rows=None, im=None, prow=prow, px=px, pw=pw, units=None, sums=x.sums(), fields=x.fields())
    out = dict(fields=x.fields())
    out.update(dict(rows=None, im=None) if case["form"] == "fp64" else dict(sums=x.sums()))
    return out
