"""GPU tests that the launch rules change no result: the order of the stage segments in calls
of many regions and the register caps of few species, on both sides of the sizes where they
change."""
import numpy as np
import pytest

from common import eos9, gpu_zeros, oracle, params_for, to_cpu, to_gpu
from particleclem_b200 import abi, hydro, native, thermo, workloads as wl

pytestmark = pytest.mark.gpu
FORMS = [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED]


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("nspec,edges,count", [
    (1, (7, 5, 6), 3), (1, (35, 34, 33), 6), (1, (35, 34, 33), 7), (1, (35, 35, 34), 2),
    (9, (7, 5, 6), 5), (9, (27, 28, 26), 2), (9, (27, 28, 27), 2), (9, (35, 34, 33), 2), (9, (35, 35, 34), 2),
    (9, (59, 58, 58), 2), (9, (59, 59, 58), 2)])
def test_boxes_of_one_call_equal_calls_of_one_box(prec, nspec, edges, count):
    """Around 40000 cells per region and 2^18 per call with one species, 20000, 40000 and
    200000 per region for mixtures."""
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


@pytest.mark.parametrize("nspec", [2, 3])
@pytest.mark.parametrize("edges", [(35, 34, 33), (52, 47, 45)])
def test_few_species_equal_oracle_where_every_stage_changes_its_caps(nspec, edges):
    """The second Riemann stage, whose marches of two y- or z-faces per thread make the fewest
    blocks, launches 1755 blocks of the larger box (876 + 439 + 440)."""
    if nspec not in hydro.species_counts():
        pytest.skip(f"library built without {nspec} species")
    nx, ny, nz = edges
    cells, march = nx * ny * nz, 1 if nx * ny * nz <= 60000 else 2
    threads = ((nx + 1) * ny * nz, nx * nz * -(-(ny + 1) // march), nx * ny * -(-(nz + 1) // march))
    blocks = sum(-(-t // 128) for t in threads)
    assert cells <= 120000 and (blocks > 1184) == (edges[0] == 52)
    lib = native.load()
    assert lib.pcg_launch_variant_for(abi.PREC_FP64, nspec, 5, blocks) == (2 if blocks > 1184 else 0)
    eos = thermo.standin_mixture(nspec)
    hydro.init(0)
    hydro.set_eos(eos)
    oracle().set_eos(eos)
    p = wl.random_patch(edges, 18, eos)
    prm = params_for(p, 0.3 * oracle().estdt(p.lo, p.hi, p.fab, p.dx), prec=abi.PREC_FP64, nspec=nspec)
    ref, _ = oracle().hydro_box(prm, p.lo, p.hi, p.fab)
    out = gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
    hydro.hydro_box(prm, p.lo, p.hi, to_gpu(p.fab), out)
    np.testing.assert_array_equal(to_cpu(out), ref.data)


@pytest.mark.parametrize("prec", FORMS)
def test_steps_overlapping_on_two_streams_equal_steps_waited_for(prec):
    """Patches stepped on two streams at once, each call's launches overlapping, against the
    same steps with a wait after each."""
    import torch

    eos = eos9()
    hydro.init(0)
    hydro.set_eos(eos)
    sets = [[wl.flame_patch(e, 60 + k, eos) for k, e in enumerate(edges)]
            for edges in ([(8, 12, 6), (12, 9, 11)], [(16, 8, 8), (5, 7, 11), (9, 10, 12)])]
    prm = abi.make_params((1, 1, 1), 0.0, 9, (0, 0, 0), (0, 0, 0), (0, 0, 0), (0, 0, 0), precision_mode=prec)
    bc = (abi.BC_OUTFLOW,) * 3

    def start(patches):
        states = [to_gpu(p.fab) for p in patches]
        boxes = [hydro.make_box(p.lo, p.hi, s, None, p.dx, 0.0, p.lo, p.hi, bc, bc) for p, s in zip(patches, states)]
        dt = torch.full((len(patches),), 1e-9, dtype=torch.float64, device="cuda")
        return states, boxes, dt, torch.empty_like(dt)

    results = []
    for wait in (True, False):
        runs = [start(p) for p in sets]
        streams = [torch.cuda.Stream() for _ in sets]
        torch.cuda.synchronize()
        for _ in range(6):
            for m, (_, boxes, dt, dt_next) in enumerate(runs):
                # no copies on the streams: successive steps swap the two timestep arrays
                hydro.step_boxes(prm, boxes, 0.3, dt, dt_next, stream=streams[m])
                runs[m] = (runs[m][0], boxes, dt_next, dt)
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        results.append([to_cpu(s) for r in runs for s in r[0]] + [r[2].cpu().numpy() for r in runs])
    for a, b in zip(*results):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
