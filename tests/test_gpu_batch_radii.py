"""A batch whose designs' filter radii need both filter kernels (up to 8 elements,
and beyond): a design gives the same bits alone and in the mix, and its first
compliance is the single-design solver's, to the PCG tolerance."""

import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

from toptimization_b200.batch import Batch, random_designs  # noqa: E402
from toptimization_b200.optimizer.simp import SimpDesign  # noqa: E402

RADII = (3.0, 8.0, 8.5, 12.0)


def _run(problems):
    b = Batch(len(problems))
    slots = [b.add(p) for p in problems]
    b.run()
    out = [b.result(s) for s in slots]
    b.close()
    return out


def test_radii_of_both_kernels_in_one_batch(tpo_built):
    ps = [dataclasses.replace(p, rmin=r)
          for p, r in zip(random_designs(4, seed=31, nelx_range=(64, 110), max_iter=3), RADII)]
    mix = _run(ps)
    for p, (rho, hist) in zip(ps, mix):
        alone, hist1 = _run([p])[0]
        assert np.array_equal(alone, rho)
        assert np.array_equal(hist1["compliance"], hist["compliance"])
        d = SimpDesign(p, precision="mixed", preconditioner=p.preconditioner)
        c = d.step().compliance
        assert abs(hist["compliance"][0] - c) < 1e-7 * c
