"""Batches with more work than the grid has blocks: tiles and runs handed out by
the steps' counters, from one mixer's to another's, and the kernels changed
between steps.  Every mixer's fields equal a handle's alone, bit for bit."""
import dataclasses

import pytest

import tmixer_b200 as T
from tests.cases import ref_like, to_spec, w_like
from tests.conftest import bit_equal, first_mismatch

pytestmark = pytest.mark.gpu


def _spec(case, precision):
    return dataclasses.replace(to_spec(case), precision=precision)


def _check(B, slot, spec, steps):
    with T.Solver(spec) as one:
        one.init().step(steps)
        for b in (0, 1):
            for f in T.FIELDS:
                got, want = B.field(slot, b, f), one.field(b, f)
                assert bit_equal(got, want), (slot, b, f, first_mismatch(got, want))


# two W=32 mixers: 7,680 tiles of one plane, and at most 592 blocks
WIDE = [w_like(32, umean=0.03, tau=0.6, tau_c=0.6, k=1e-3, rho=1.0),
        w_like(32, umean=0.02, tau=0.7, tau_c=0.55, k=1e-2, rho=1.4)]


@pytest.mark.parametrize("flat", [1, 2, 3])
def test_kernel_changed_between_steps(gpu, flat):
    """Steps by tiles, by the flat kernel (which leaves the tile counters as they
    are), and by tiles again."""
    specs = [_spec(c, T.TMX_FP16) for c in WIDE]
    with T.Batch(T.TMX_FP16, budget=sum(map(T.Batch.footprint, specs)) + (1 << 20)) as B:
        slots = [B.add(s) for s in specs]
        B.set_sweep(T.SHAPE_SWEEP4, 1)
        B.step(3)
        B.set_shape(256, 4096)
        B.step(flat)
        B.set_sweep(T.SHAPE_SWEEP4, 1)
        B.step(1)
        for slot, spec in zip(slots, specs):
            _check(B, slot, spec, 4 + flat)


# uneven mixers, together some thousand runs and tiles
UNEVEN = [w_like(20, umean=0.03, tau=0.6, tau_c=0.6, k=1e-3, rho=1.0),
          dict(ref_like(97, 18, 25, 41, 34, umean=0.05, k=0.5), ia=30),
          w_like(5, umean=0.02, tau=0.7, tau_c=0.55, k=1e-2, rho=1.4),
          dict(ref_like(241, 9, 31, 33, 120, umean=0.03, k=0.5, rho0=1.5, rho_out=1.45), ia=9)]


@pytest.mark.parametrize("precision", [T.TMX_FP64, T.TMX_FP32, T.TMX_FP16])
def test_more_work_than_blocks(gpu, precision):
    """Blocks take run after run (tile after tile) of mixers of other sizes; a
    mixer joins at an odd step, another leaves; 16 steps to a graph and single
    ones."""
    specs = [_spec(c, precision) for c in UNEVEN]
    with T.Batch(precision, budget=2 * sum(map(T.Batch.footprint, specs)) + (1 << 20)) as B:
        if precision == T.TMX_FP16:
            B.set_sweep(T.SHAPE_SWEEP4, 1)
        slots = [B.add(s) for s in specs[1:]]
        B.step(3)
        first = B.add(specs[0])
        B.step(87)
        for slot, spec in zip(slots, specs[1:]):
            _check(B, slot, spec, 90)
        _check(B, first, specs[0], 87)
        B.remove(slots[0])
        B.step(1)
        _check(B, slots[1], specs[2], 91)
        _check(B, first, specs[0], 88)


@pytest.mark.parametrize("threads,cells", [(128, 1024), (256, 2048), (512, 8192)])
def test_flat_shapes_agree(gpu, threads, cells):
    """The flat kernels of the FP16 form and its face kernel, whose persistent
    blocks take several cell blocks and list chunks."""
    specs = [_spec(c, T.TMX_FP16) for c in UNEVEN]
    with T.Batch(T.TMX_FP16, budget=sum(map(T.Batch.footprint, specs)) + (1 << 20)) as B:
        B.set_shape(threads, cells)
        B.set_boundary(1, True)
        slots = [B.add(s) for s in specs]
        B.step(21)
        for slot, spec in zip(slots, specs):
            _check(B, slot, spec, 21)


def test_shape_before_the_first_step(gpu):
    """An untuned batch reports the planes that its next step will take, whatever
    came or went since the last one."""
    spec = _spec(WIDE[0], T.TMX_FP16)
    with T.Batch(T.TMX_FP16, budget=5 * T.Batch.footprint(spec) + (1 << 20)) as B:
        slots = [B.add(spec) for _ in range(5)]  # 2,560 tiles of 8 planes, four rounds of 592
        before = B.shape()
        B.step(1)
        assert before == B.shape() and before["zchunk"] == 8
        B.remove(slots[0])
        before = B.shape()
        B.step(1)
        assert before == B.shape() and before["zchunk"] == 4
