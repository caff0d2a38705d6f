"""Momentum assembly at the edges of the per-cell face list."""
import dataclasses

import numpy as np
import pytest

from matlab_ufvm_b200 import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gaps", [(0,), (0, 1, 2), (7, 20)])
def test_cell_numbers_without_faces(ufvm_mod, oracle_mod, gaps):
    """A mesh may leave cell numbers unused (the number of cells is the largest one in owner and
    neighbour plus one): such a cell has an empty face list, and nothing is read through it. Its zero
    diagonal is reported; the other cells' rows are those of the mesh without the gaps."""
    spec = case.cavity_case(5, nu=0.01, quirks=case.QUIRKS_CONVERGING)
    n = spec.mesh.n_cells
    keep = np.setdiff1d(np.arange(n + len(gaps)), gaps)[:n].astype(np.int32)
    mesh = dataclasses.replace(spec.mesh, owner=keep[spec.mesh.owner], neighbour=keep[spec.mesh.neighbour])
    o = oracle_mod.OracleCase(spec)
    g = ufvm_mod.GpuCase(dataclasses.replace(spec, mesh=mesh, fixed_element=int(keep[0])))
    g.cfdUpdateFields()
    o.update_fields()
    for c in range(3):
        with pytest.raises(ufvm_mod.UfvmError) as e:
            g.cfdAssembleEquation("U", c + 1)
        assert e.value.code == 5  # UFVM_E_ZERO_DIAG
        o.assemble_u(c)
        assert np.array_equal(g.get("ac")[keep], o.get("ac")) and np.array_equal(g.get("bc")[keep], o.get("bc"))
        assert np.array_equal(g.get("anb"), o.get("anb"))


@pytest.mark.parametrize("spec,most", [
    (lambda: case.cavity_case(128, nu=0.01, quirks=case.QUIRKS_CONVERGING), 42057120),
    (lambda: case.cavity_case(32, nu=0.01, dim=3, quirks=case.QUIRKS_CONVERGING), 61932816),
])
def test_a_resident_case_takes_no_more_memory_than_with_separate_geometry_arrays(ufvm_mod, spec, most):
    """most: what the allocation counter said with one array per face value and 21 staged terms a face."""
    spec = spec()
    svc = ufvm_mod.Service(ufvm_mod.fast_settings(spec))
    svc.submit(spec, 100)
    svc.step()
    assert 0 < svc.stats()["resident_bytes"] <= most
    svc.close()
