"""Ring matrices whose tiles evaluate each line once per control point (Mesh.induction_matrix3,
pvl_induction_normal_tiled), against the kernel that evaluates every ring's own lines
(pvl_induction_normal), at the edges of the tiles: control points around a block of eight and odd
numbers of them, rings around a tile of 128, rings of three to seven lines, a ring of more lines than
a tile's shared memory holds; points that are mesh nodes (inside the cut-off of the lines that meet
there), near the lines (the arctangent form) and far from them (each length of the series)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(n_rings, sides):
    """`sides`-gons in a row, neighbours sharing an edge, slightly out of plane."""
    pos = [(0.0, 0.0, 0.0), (0.0, 1.0, 0.1)]
    elements = []
    low, up = 0, 1
    for k in range(n_rings):
        n = len(pos)
        x = 0.9 * (k + 1)
        if sides == 3:
            pos.append((0.45 * (k + 1), 0.8 if k % 2 == 0 else 0.0, 0.02 * (k % 5)))
            elements.append([low, up, n] if k % 2 == 0 else [up, low, n])
            low, up = up, n
            continue
        pos += [(x - 0.9 + 0.9 * (i + 1) / (sides - 2), -0.2 - 0.05 * i, 0.03 * k % 0.4) for i in range(sides - 4)]
        pos += [(x, 0.05, 0.02 * (k % 7)), (x, 1.0, 0.1 + 0.01 * (k % 3))]
        elements.append([low, *range(n, n + sides - 2), up])
        low, up = n + sides - 4, n + sides - 3
    return np.array(pos, float), elements


def _points(pos, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = pos.min(0) - 0.5, pos.max(0) + 0.5
    p = rng.uniform(lo, hi, (n, 3))
    p[:, 2] = np.where(rng.random(n) < 0.5, rng.choice([-1.0, 1.0], n) * rng.uniform(0.3, 0.6, n),
                       rng.uniform(0.5, 40.0, n))  # 0.05 and more off every line
    p[::5] = pos[rng.integers(0, len(pos), len(p[::5]))]
    return p, rng.normal(size=(n, 3))


@pytest.mark.parametrize("sides,n_rings,n_cp", [
    (4, 1, 1), (4, 127, 7), (4, 128, 8), (4, 129, 9), (4, 300, 1023), (3, 255, 17), (3, 384, 64), (5, 130, 33),
    (7, 129, 12), (3300, 2, 9), (4, 5, 0),
])
@pytest.mark.parametrize("on_device", [False, True])
def test_tiled_matrix_matches_per_ring_kernel(sides, n_rings, n_cp, on_device):
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.cvl import Mesh
    from pyvl_b200.device import Workspace, ptr, stream_ptr

    pos, elements = _fan(n_rings, sides)
    mesh = Mesh(len(pos), elements)
    assert mesh.n_surfaces == n_rings
    cps, nrm = _points(pos, n_cp, sides + n_cp)
    tol = 1e-6
    dev = [torch.as_tensor(a, device="cuda") for a in (pos, cps, nrm)]
    got = mesh.induction_matrix3(tol, *(dev if on_device else (pos, cps, nrm)))
    got = got.cpu().numpy() if on_device else got
    assert got.shape == (n_cp, n_rings)
    d = mesh.device_arrays()
    assert (d["tile_max"] > Mesh.TILE_LINES_MAX) == (sides == 3300)
    want = torch.zeros((n_cp, n_rings), dtype=torch.float64, device="cuda")
    ws, nb = Workspace.get(_lib.query("pvl_segments_workspace", mesh.n_lines, _lib.PVL_F64))
    _lib.call("pvl_induction_normal", _lib.PVL_F64, mesh.n_points, mesh.n_lines, ptr(d["lines"]), ptr(dev[0]),
              n_rings, ptr(d["offsets"]), ptr(d["surface_lines"]), n_cp, ptr(dev[1]), ptr(dev[2]), tol, ptr(want),
              n_rings, ws, nb, stream_ptr())
    want = want.cpu().numpy()
    assert np.isfinite(got).all()
    if n_cp:
        # about twenty roundings of values that share one conditioning, |p - r| / h <= 1e2 at these points
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
        assert np.abs(want).max() > 0


def test_too_many_points_are_refused():
    import torch

    from pyvl_b200.cvl import Mesh

    pos, elements = _fan(1, 4)
    n = 65535 * 8 + 1
    z = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    with pytest.raises(ValueError):
        Mesh(len(pos), elements).induction_matrix3(1e-6, torch.as_tensor(pos, device="cuda"), z, z)


@pytest.mark.parametrize("tol", [1e-6, 0.3, 1e3])  # no line, some and all of them below the cut-off
def test_normals_that_are_not_finite(tol):
    """A NaN or infinite normal (a degenerate ring's) makes its row's entries NaN or infinite also where
    every line of a ring is inside the cut-off: the same entries as in the per-ring kernel."""
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.cvl import Mesh
    from pyvl_b200.device import Workspace, ptr, stream_ptr

    pos, elements = _fan(40, 4)
    mesh = Mesh(len(pos), elements)
    cps, nrm = _points(pos, 24, 3)
    nrm[1], nrm[6, 2], nrm[11, 0] = np.nan, np.nan, np.inf
    dev = [torch.as_tensor(a, device="cuda") for a in (pos, cps, nrm)]
    got = mesh.induction_matrix3(tol, *dev).cpu().numpy()
    d = mesh.device_arrays()
    want = torch.zeros(got.shape, dtype=torch.float64, device="cuda")
    ws, nb = Workspace.get(_lib.query("pvl_segments_workspace", mesh.n_lines, _lib.PVL_F64))
    _lib.call("pvl_induction_normal", _lib.PVL_F64, mesh.n_points, mesh.n_lines, ptr(d["lines"]), ptr(dev[0]),
              mesh.n_surfaces, ptr(d["offsets"]), ptr(d["surface_lines"]), len(cps), ptr(dev[1]), ptr(dev[2]), tol,
              ptr(want), mesh.n_surfaces, ws, nb, stream_ptr())
    want = want.cpu().numpy()
    assert np.isnan(want[[1, 6]]).all()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    # as in the test above; 1e-12 of the largest finite entry
    assert np.abs(got[ok] - want[ok]).max() <= 1e-12 * np.abs(want[ok]).max()


@pytest.mark.parametrize("sides,n_rings,n_cp", [(14, 128, 9), (15, 129, 8), (16, 130, 9), (25, 200, 17)])
def test_tiles_that_fill_half_the_shared_memory(sides, n_rings, n_cp):
    """Tiles of 1665 to 3073 lines: up to 1791 two CTAs share an SM, above one has it alone and takes more
    threads."""
    test_tiled_matrix_matches_per_ring_kernel(sides, n_rings, n_cp, True)
