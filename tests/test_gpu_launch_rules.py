"""GPU tests that the launch rules change no result: the order of the stage segments in calls
of many regions, on both sides of the sizes where it changes."""
import numpy as np
import pytest

from common import eos9, gpu_zeros, oracle, params_for, to_cpu, to_gpu
from particleclem_b200 import abi, hydro, workloads as wl

pytestmark = pytest.mark.gpu
FORMS = [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED]


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("nspec,edges,count", [
    (1, (7, 5, 6), 3), (1, (35, 34, 33), 6), (1, (35, 34, 33), 7), (1, (35, 35, 34), 2),
    (9, (7, 5, 6), 5), (9, (27, 28, 26), 2), (9, (27, 28, 27), 2), (9, (59, 58, 58), 2), (9, (59, 59, 58), 2)])
def test_boxes_of_one_call_equal_calls_of_one_box(prec, nspec, edges, count):
    """Around 40000 cells per region and 2^18 per call with one species, 20000 and 200000
    per region for mixtures."""
    eos = wl.GammaLaw() if nspec == 1 else eos9()
    hydro.init(0)
    hydro.set_eos(eos)
    oracle().set_eos(eos)
    boxes, many, one = [], [], []
    for m in range(count):
        p = wl.random_patch(edges, 40 + m, eos if nspec > 1 else None, shock=False)
        uin = to_gpu(p.fab)
        dt = 0.3 * oracle().estdt(p.lo, p.hi, p.fab, p.dx)
        many.append(gpu_zeros(abi.nvar(nspec), p.lo, p.hi))
        one.append(gpu_zeros(abi.nvar(nspec), p.lo, p.hi))
        boxes.append(hydro.make_box(p.lo, p.hi, uin, many[-1], p.dx, dt))
        hydro.hydro_box(params_for(p, dt, prec=prec, nspec=nspec), p.lo, p.hi, uin, one[-1])
    hydro.hydro_boxes(params_for(p, 0.0, prec=prec, nspec=nspec), boxes)
    for a, b in zip(many, one):
        a = to_cpu(a)
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, to_cpu(b))
