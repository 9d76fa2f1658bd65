"""A mixed HEATF step that ends at its iteration limit gives what it has given
all along, to the roundings of a few GMRES scalars.

The discontinuity capturing divides by the temperature gradient, and the step
stops unconverged after ten iterations, so single roundings of the element and of
the FP32 sums travel into the result (by up to 1e-7 at a node on finer meshes).
golden/heatf_mixed_step.npy holds A of this step as the colour launches and the
FP32 sums of one lane per row gave it.  Mesh and state use no transcendental
function, so that every machine makes the same numbers.

Tolerance: the element and the FP32 sums keep their bits; the rotations of a
GMRES column are FP64 numbers of another rounding (1e-16), which reach FP32 values
only where they decide one: 1e-12 in norm.
"""
import dataclasses
from pathlib import Path

import numpy as np
import pytest

from svfsi_gb300 import fsils, meshgen, problems

pytestmark = pytest.mark.gpu

GOLD = Path(__file__).parent / "golden" / "heatf_mixed_step.npy"


def step():
    x, ien = meshgen.kuhn_box(7, 6, 31, 1.0, 1.0, 5.0)
    rp, cp = meshgen.csr_from_ien(x.shape[0], ien)
    base = problems.heatf_cylinder(h=0.5)
    p = dataclasses.replace(base, x=x, ien=ien, rowPtr=rp, colPtr=cp, Y0=None,
                            dirichlet=[problems.DirBC(meshgen.nodes_on_plane(x, 2, 0.0), 1.0)])
    A, Y, D = p.initial_state()
    a, b, c = x.T
    Y[:, 0] = 2.0 * (a - 0.5) * (b - 0.25) * (c - 2.0)
    Y[:, 1] = -1.5 * a * (b - 0.5) * (c - 1.0)
    Y[:, 2] = 480.0 * a * (1.0 - a) * b * (1.0 - b)
    Y[:, 4] = 1.0 - c / 5.0 + 0.1 * (a - 0.4) * (b * b - 0.3) + 0.02 * c * (5.0 - c) * a
    lhs, mesh, eq = problems.build_equation(p, fsils.PREC_MIXED)
    eq.set_state(A, Y, D)
    info = eq.step()
    assert info.newton_itr == 10
    out = eq.get_state()[0][:, 4].copy()
    del eq
    mesh.free()
    lhs.free()
    return out


def test_unconverged_mixed_step_keeps_its_bits(gsls):
    want, got = np.load(GOLD), step()
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
