"""Grids at the limits of the row padding: a length of 1 to 3 voxels is no row where another axis
can be, and the 2^31 limit counts voxels, not the padded positions."""
import numpy as np
import pytest

from conftest import has_gpu


def box(synth, shape, h, nspecies=5):
    """One domain, no boundaries; shape in geometry voxels of size h."""
    spec = synth.tiny((12, 12, 16), serca=False, pryr=False)
    spec["voxels"] = np.zeros(shape, dtype=np.uint8)
    spec["h"], spec["global_size"] = h, [h * n for n in shape]
    spec["boundaries"] = []
    spec.pop("ryr", None)
    spec["species"] = spec["species"][:nspecies]
    spec["domain_species"] = {
        d: dict(v, diffusive=[s for s in v["diffusive"] if s < nspecies], sigma=v["sigma"][:nspecies],
                init=v["init"][:nspecies], buffers=[b for b in v["buffers"] if b["species"][0] < nspecies])
        for d, v in spec["domain_species"].items()}
    return spec


@pytest.mark.parametrize("S,refused", [(215, False), (216, True)])
def test_limit_counts_voxels(pkg, synth, S, refused):
    """1290^3 voxels are below 2^31, 1290 x 1290 x 1292 positions above; 1296^3 voxels are above.
    Without a GPU a grid that is not refused fails at the device instead."""
    if has_gpu():
        pytest.skip("would take 20 GB of device memory and as much time")
    with pytest.raises(pkg.CspError) as e:
        pkg.Simulation(box(synth, (6, 6, 6), 6.0 * S, 1), dict(h=6.0, tstop=1.0, seed=1))
    assert ("grid too large" in str(e.value)) == refused
    assert (e.value.code == -1) == refused


FLAT = [(21, 50, 3), (50, 3, 21), (3, 21, 50), (33, 35, 1), (7, 1, 1), (5, 6, 3), (1, 37, 41)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", FLAT)
def test_flat_grids_bitwise(pkg, synth, shape):
    spec = box(synth, shape, 6.0)
    u0 = np.random.default_rng(3).uniform(0.5, 1.0, (5,) + shape)
    got = []
    for kernel in (0, 1):
        sim = pkg.Simulation(spec, dict(h=6.0, tstop=1.0, seed=1))
        sim.set_state(u0 * sim.state())
        sim.set_kernel(kernel)
        sim.advance(23)
        got.append(sim.state())
        sim.close()
    assert np.isfinite(got[0]).all()
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2001, 1001, 1), (1001, 3, 601)])
def test_flat_grids_take_no_padding(pkg, synth, shape):
    """Two FP32 buffers of five species, domain byte and group code: 41.25 bytes per voxel, and
    what the planes are rounded up to."""
    import torch
    torch.cuda.init()
    pkg.Simulation(box(synth, (9, 9, 9), 6.0), dict(h=6.0, tstop=1.0, seed=1)).close()
    before = torch.cuda.mem_get_info()[0]
    sim = pkg.Simulation(box(synth, shape, 6.0), dict(h=6.0, tstop=1.0, seed=1))
    used = before - torch.cuda.mem_get_info()[0]
    sim.close()
    assert used < 1.25 * 41.25 * np.prod(shape) + (8 << 20)
