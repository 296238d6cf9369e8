"""The FP64 products and the residual control of the mixed refinement at the
edges of their tiles: panel counts around the 32-row tiles, few and many
matrices (one or two rows per lane, 8 or 16 warps), every group of
right-hand-side counts, the direct and conjugate-transposed products.

Bound: the refinement runs to a relative residual of 1e-12 and the matrices'
condition is below 10, so phi, and the forces that are sums of it, are within
1e-11 of the FP64 LU's; 1e-10 of the largest output is asked.  The gradients
add the adjoint solve's own 1e-11 to the forward's through sums with
cancellation of at most two digits here: 1e-8."""
import numpy as np
import pytest


def _dofs(mh, mesh, nd, seed):
    rng = np.random.default_rng(seed)
    return [np.ascontiguousarray(rng.standard_normal((mesh.nfaces, 3))) for _ in range(nd)]


@pytest.mark.gpu
@pytest.mark.parametrize("resolution,nw,nd,nb,direct", [
    ((2, 31), 1, 1, 0, True),      # less than one tile
    ((2, 33), 2, 2, 0, False),     # one row past a tile
    ((10, 13), 3, 2, 1, True),     # 65 panels
    ((8, 16), 90, 1, 1, True),     # 64 panels, two tiles in many matrices
    ((16, 32), 150, 2, 2, False),  # 256 panels: two rows per lane
    ((17, 27), 2, 4, 1, True),     # 243 panels, five right-hand sides
    ((17, 27), 2, 6, 1, False),    # seven
    ((10, 13), 3, 6, 3, True),     # nine
    ((10, 13), 3, 8, 5, True),     # thirteen
    ((10, 13), 3, 10, 6, False),   # sixteen, the most
])
def test_products_and_refinement(mh, gpu, resolution, nw, nd, nb, direct):
    mesh = mh.mesh_hemisphere(1.0, (0.1, 0.2, 0.0), resolution)
    om = np.linspace(0.6, 2.0, nw)
    betas = np.linspace(0.0, 2.0, nb)
    dofs = _dofs(mh, mesh, nd, 3)
    kw = dict(direct=direct, ctx=gpu)
    want = mh.hydro_batch(mesh, om, dofs, betas, precision="fp64_batched", **kw)
    got = mh.hydro_batch(mesh, om, dofs, betas, precision="mixed", tol=1e-12, **kw)
    assert got[4].n_fallback == 0 and got[4].max_rel_residual <= 1e-12
    for a, b in zip(got[:4], want[:4]):
        if b.size:
            assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("resolution,nw,nd,nb,direct", [
    ((2, 33), 1, 1, 0, True), ((17, 27), 2, 2, 1, False), ((10, 13), 3, 4, 1, True), ((10, 13), 2, 6, 3, False),
    ((16, 32), 40, 2, 1, True)])
def test_conjugate_products(mh, gpu, resolution, nw, nd, nb, direct):
    mesh = mh.mesh_hemisphere(1.0, (0.1, 0.2, 0.0), resolution)
    om = np.linspace(0.6, 2.0, nw)
    betas = np.linspace(0.0, 2.0, nb)
    dofs = _dofs(mh, mesh, nd, 4)
    rng = np.random.default_rng(5)
    bars = [rng.standard_normal((nd, nd, nw)), rng.standard_normal((nd, nd, nw)),
            rng.standard_normal((nd, nw, nb)) + 1j * rng.standard_normal((nd, nw, nb)), None]
    kw = dict(direct=direct, ctx=gpu)
    want = mh.hydro_batch_vjp(mesh, om, dofs, betas, *bars, precision="fp64_batched", **kw)
    got = mh.hydro_batch_vjp(mesh, om, dofs, betas, *bars, precision="mixed", tol=1e-12, **kw)
    assert got.info.n_fallback == 0
    for a, b in zip([got.mesh.vertices, got.mesh.centers, got.mesh.normals, got.mesh.areas, got.omegas, *got.dofs],
                    [want.mesh.vertices, want.mesh.centers, want.mesh.normals, want.mesh.areas, want.omegas, *want.dofs]):
        assert np.max(np.abs(a - b)) <= 1e-8 * np.max(np.abs(b))
