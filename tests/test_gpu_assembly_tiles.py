"""The tiled Rankine assembly and the narrower wave tiles at the edges of
their tiles: panel counts around the 128-row tile, below and above the size
where a tile takes four columns (with a remainder of one to three), every
combination of terms, direct and indirect, against the CPU oracle.

Bound: both sides evaluate the same closed forms in FP64 with different
orders of a few dozen operations, so entries agree to a few 1e-15 of the
largest one; 1e-12 is asked, as for the assembly elsewhere."""
import numpy as np
import pytest

MASKS = {
    "rankine": lambda mh: (mh.Rankine(),),
    "reflected": lambda mh: (mh.RankineReflected(),),
    "negative": lambda mh: (mh.Rankine(), mh.RankineReflectedNegative()),
    "cancelling": lambda mh: (mh.Rankine(), mh.RankineReflected(), mh.RankineReflectedNegative(), mh.GFWu()),
    "wu": lambda mh: (mh.Rankine(), mh.RankineReflected(), mh.GFWu()),
    "wu only": lambda mh: (mh.GFWu(),),
}


def _close(a, b):
    return np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("terms", list(MASKS))
@pytest.mark.parametrize("resolution,direct", [((2, 5), True), ((2, 31), False), ((10, 25), True), ((8, 32), False),
                                              ((6, 43), True), ((16, 99), False), ((26, 63), True)])
def test_assembly_tiles(mh, gpu, oracle, terms, resolution, direct):
    mesh = mh.mesh_hemisphere(1.3, (0.2, -0.1, 0.0), resolution)
    gfs = MASKS[terms](mh)
    S, D = mh.assemble_matrices(gfs, mesh, 0.7, direct=direct, ctx=gpu)
    So, Do = oracle.assemble(mesh, 0.7, mh.gf_mask(gfs), direct)
    assert _close(S, So) and _close(D, Do)


@pytest.mark.gpu
@pytest.mark.parametrize("resolution,nw", [((2, 31), 7), ((10, 25), 9), ((6, 43), 6), ((16, 99), 6), ((36, 71), 6)])
def test_batched_wave_tiles(mh, series_fp64, resolution, nw):
    """The frequency-batched pass (its columns per tile follow the mesh) against
    the same call a few frequencies at a time, which uses the other kernel."""
    gpu = series_fp64
    mesh = mh.mesh_hemisphere(1.3, (0.2, -0.1, 0.0), resolution)
    om = np.linspace(0.5, 2.9, nw)
    dofs = [mh.translational_dofs(mesh, "Heave"), mh.translational_dofs(mesh, "Surge")]
    kw = dict(green_functions=(mh.Rankine(), mh.RankineReflected(), mh.ExactGuevelDelhommeau()), tol=1e-12, ctx=gpu)
    A, B, F, _, _ = mh.hydro_batch(mesh, om, dofs, [0.3], **kw)
    for z in range(0, nw, 3):
        a, b, f, _, _ = mh.hydro_batch(mesh, om[z:z + 3], dofs, [0.3], **kw)
        for x, y in ((A[:, :, z:z + 3], a), (B[:, :, z:z + 3], b), (F[:, z:z + 3], f)):
            assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))
