"""The FP16 form's tiled interior kernels (TMX_SHAPE_SWEEP8 / SWEEP4: tiles of
32 x 8 or 32 x 4 nodes walked through z, the writers' moment records staged in
shared memory) give the flat kernel's results bit for bit: every population,
moment-derived field and mixing row, on geometries whose boxes are not
multiples of the tile (ragged x and y tiles), with the opening next to the
inlet faces, and with z-chunks of one plane up to the whole box."""
import numpy as np
import pytest

import tmixer_b200 as T
from tests.cases import GOLDEN_CASES, ORACLE_CASES, ref_like, to_spec

pytestmark = pytest.mark.gpu


def _case(name):
    if name in GOLDEN_CASES:
        return to_spec(GOLDEN_CASES[name][0])
    return to_spec(ORACLE_CASES[name])


def _state(spec, shape, zchunk, steps):
    with T.Solver(spec) as s:
        if shape is not None:  # None: the handle's default shape
            s.set_shape(shape, zchunk)
        s.init()
        s.step(steps)
        fields = [s.field(b, f) for b in (0, 1) for f in T.FIELDS]
        pops = [s.populations(b, fld) for b in (0, 1) for fld in range(4)]
        rows, _ = s.mixing()
    return fields + pops + [rows]


def _same(a, b):
    return all(np.array_equal(x.view(np.uint64), y.view(np.uint64)) for x, y in zip(a, b))


CASES = [("w24", None), ("tiny_species", None), ("wide_opening", None), ("odd_ia", None), ("w8", None),
         ("col33", None), ("col3", None)]

# boxes whose last column would be alone in its tile (65 and 33 columns: an x
# wall's species come from its neighbour in the same warp), and a mixing box
# whose two x walls share their neighbour
EXTRA = {
    "col33": dict(ref_like(65, 6, 5, 33, 7, tau=0.65, k=2.0, rho0=1.5, rho_out=1.4, umean=0.05,
                           cin=[[0.9, 0.2], [0.1, 1.1], [0.05, 0.02]]), ia=9),
    "col3": ref_like(9, 5, 4, 3, 5, umean=0.03, cin=[[1.0, 0.25], [0.3, 1.0], [0.1, 0.05]]),
}


def _spec(name):
    if name.startswith("w") and name[1:].isdigit():
        return T.w_layout(int(name[1:]), u_max=0.05, tau_f=0.6, tau_c=0.6, k=1e-3, rho=1.0, precision=T.TMX_FP16)
    s = to_spec(EXTRA[name]) if name in EXTRA else _case(name)
    s.precision = T.TMX_FP16
    return s


@pytest.mark.parametrize("name", [c[0] for c in CASES])
def test_sweep_equals_flat(gpu, name):
    spec = _spec(name)
    steps = 25
    want = _state(spec, T.SHAPE_FLAT, 8, steps)
    for shape, zchunk in ((None, 0), (T.SHAPE_SWEEP8, 8), (T.SHAPE_SWEEP4, 3), (T.SHAPE_SWEEP8, 1),
                          (T.SHAPE_SWEEP4, 1000)):
        got = _state(spec, shape, zchunk, steps)
        assert _same(got, want), (name, shape, zchunk)


# boxes whose columns take 32-, 16- and 8-wide tiles of a batch (sweep_tiles):
# one group and less, each remainder, and a last column that is never alone
GROUP_BOXES = [(16, 5, 5, 8, 9, 4), (20, 9, 4, 9, 17, 5), (44, 6, 5, 18, 35, 9), (50, 11, 5, 24, 20, 3),
               (73, 7, 4, 33, 9, 20), (97, 18, 5, 41, 34, 30)]


@pytest.mark.parametrize("kind,zchunk", [(T.SHAPE_SWEEP4, 4), (T.SHAPE_SWEEP8, 2), (T.SHAPE_SWEEP4, 1)])
def test_batch_groups_equal_flat(gpu, kind, zchunk):
    specs = []
    for n, (inx, iny, nz, mnx, mny, ia) in enumerate(GROUP_BOXES):
        s = to_spec(dict(ref_like(inx, iny, nz, mnx, mny, umean=0.02 + 0.01 * n, k=0.5), ia=ia))
        s.precision = T.TMX_FP16
        specs.append(s)
    with T.Batch(T.TMX_FP16, budget=sum(T.Batch.footprint(s) for s in specs) + (1 << 20)) as B:
        slots = [B.add(s) for s in specs]
        B.set_sweep(kind, zchunk)
        B.step(12)
        for s, m in zip(specs, slots):
            with T.Solver(s) as one:
                one.set_shape(T.SHAPE_FLAT, 8)
                one.init()
                one.step(12)
                for b in (0, 1):
                    assert _same([B.field(m, b, f) for f in T.FIELDS], [one.field(b, f) for f in T.FIELDS])


def test_sweep_shape_rejected_outside_fp16(gpu):
    spec = T.w_layout(4, u_max=0.05, tau_f=0.6, tau_c=0.6, k=1e-3, rho=1.0, precision=T.TMX_FP32)
    with T.Solver(spec) as s:
        with pytest.raises(T.TmxError):
            s.set_shape(T.SHAPE_SWEEP8, 8)
        s.set_shape(T.SHAPE_FLAT, 8)
