"""Hierarchies of very many levels: the number is the caller's (p_max_coarse_levels), and a mesh of
several parts never gets below one cell a part."""
import dataclasses

import numpy as np
import pytest

from matlab_ufvm_b200 import case, meshgen

pytestmark = pytest.mark.gpu


def copies(spec, k):
    """k copies of a case side by side, as one case."""
    m = spec.mesh
    npt, nc, fi = len(m.points), m.n_cells, m.n_interior
    order = [(c, np.arange(fi)) for c in range(k)]
    patches, at = [], k * fi
    for p in m.patches:
        order += [(c, np.arange(p.start, p.start + p.n)) for c in range(k)]
        patches.append(meshgen.Patch(p.name, p.type, at, k * p.n))
        at += k * p.n
    nodes = [m.face_nodes[m.face_start[f]:m.face_start[f + 1]] + c * npt for c, fs in order for f in fs]
    mesh = meshgen.PolyMesh(points=np.concatenate([m.points + [10.0 * c, 0, 0] for c in range(k)]),
                            face_start=np.concatenate([[0], np.cumsum([len(q) for q in nodes])]).astype(np.int32),
                            face_nodes=np.concatenate(nodes).astype(np.int32),
                            owner=np.concatenate([m.owner[fs] + c * nc for c, fs in order]).astype(np.int32),
                            neighbour=np.concatenate([m.neighbour + c * nc for c in range(k)]).astype(np.int32),
                            patches=patches)
    b = np.concatenate([fs - fi for _, fs in order[k:]])
    return dataclasses.replace(spec, mesh=mesh, val_u=spec.val_u[b], val_p=spec.val_p[b])


@pytest.mark.parametrize("smoother", ["ILU", "SOR"])
@pytest.mark.parametrize("levels", [10, 158, 159, 160, 161, 400])
def test_more_levels_than_operations_in_a_launch(ufvm_mod, oracle_mod, smoother, levels):
    spec = copies(case.channel_case(nx=3, ny=2, nz=2), 7)
    spec = dataclasses.replace(spec, p_smoother=smoother, p_max_coarse_levels=levels, p_max_cycles=2)
    g, o = ufvm_mod.GpuCase(spec), oracle_mod.OracleCase(spec)
    for _ in range(2):
        g.iterate()
        o.iterate()
    assert o.nlevels() == levels + 1 and len(g.level_array(levels, "ac")) == 7
    for name in ("U", "p", "mdot"):
        a, b = g.get(name), o.get(name)
        assert np.isfinite(b).all() and np.array_equal(a, b), name
