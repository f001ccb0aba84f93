"""The bits of the reduced-precision forms, single and batched: digests of every
field of both boxes, and a batch's outlet indices, equal to those that the
kernels of commit b8a3c24 gave (tests/golden/reduced_bits.json).  In the W=17
mixer species C has densities of a few of FP32's smallest denormals ahead of its
front, where a closure's product rounded once or twice shows in the outlet index's
first digits."""
import dataclasses
import json
import os

import pytest

import tmixer_b200 as T
from tests.cases import ORACLE_CASES, to_spec, w_like
from tests.golden.make_golden import digest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reduced_bits.json")
CASES = {
    "odd_ia": (ORACLE_CASES["odd_ia"], 151),
    "w9_species": (dict(w_like(9, umean=0.03, tau=0.71, tau_c=0.63, k=0.0031, rho=1.3), rho_out=1.25,
                        cin=[[0.77, 0.13], [0.21, 0.61], [0.05, 0.07]]), 150),
    "w17": (w_like(17, umean=0.023, tau=0.71, tau_c=0.63, k=0.0031, rho=1.7), 301),
}


def run(name, form):
    """Digests of the case's fields, alone and in a batch, and the batch's outlet indices."""
    case, steps = CASES[name]
    spec = dataclasses.replace(to_spec(case), precision=T.PRECISIONS[form])
    with T.Solver(spec) as s:
        s.init().step(steps)
        alone = {"b%d_%s" % (b, f): digest(s.field(b, f)) for b in (0, 1) for f in T.FIELDS}
    with T.Batch(spec.precision, budget=T.Batch.footprint(spec) + (1 << 20)) as B:
        m = B.add(spec)
        B.step(steps)
        batch = {"b%d_%s" % (b, f): digest(B.field(m, b, f)) for b in (0, 1) for f in T.FIELDS}
        im = [float(x).hex() for x in B.outlet_im([m])[0]]
    return alone, batch, im


@pytest.mark.parametrize("form", ["fp32", "fp16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_bits(gpu, name, form):
    with open(GOLDEN) as fh:
        want = json.load(fh)[form][name]
    alone, batch, im = run(name, form)
    assert alone == want["fields"]
    assert batch == want["fields"]
    assert im == want["outlet_im"]
