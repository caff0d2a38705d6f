"""The service's wide paths: kernels on rows wider than any cavity's against plain loops, and schedules
in which a case's small levels exceed the shared memory of the coarse V-cycle."""
import os
import subprocess

import numpy as np
import pytest

from matlab_ufvm_b200 import build, case

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_kernels_against_plain_loops(ufvm_mod, tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run([build.NVCC, *build.ARCH, "-O1", "-std=c++17", "--fmad=false", "-Xcompiler", "-ffp-contract=off",
                    "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"),
                    os.path.join(HERE, "service_kernels_check.cu"), "-o", exe, ufvm_mod.LIB_PATH,
                    "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(ufvm_mod.LIB_PATH)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("OK\n"), r.stdout + r.stderr


def test_levels_beyond_shared_memory_give_the_same_bits(ufvm_mod):
    """One block runs all levels below the finest (2 x rows + the largest level: 29,000 floats for the
    40^3 cavity and 50,000 for the 250 x 250 one, against 16,384), packed or not, or the larger ones run as grid launches: same bits."""
    specs = [case.cavity_case(40, nu=0.01, dim=3, quirks=case.QUIRKS_CONVERGING),
             case.channel_case(nx=24, ny=12, nz=12, quirks=case.QUIRKS_CONVERGING),
             case.cavity_case(250, nu=0.005, quirks=case.QUIRKS_CONVERGING),
             case.cavity_case(20, nu=0.01, quirks=case.QUIRKS_CONVERGING)]
    out = []
    for cta_rows, packed in ((1, 0), (1 << 20, 0), (1 << 20, 1), (2000, 1)):
        svc = ufvm_mod.Service(ufvm_mod.fast_settings(specs[0]))
        svc.set_schedule(cta_rows, packed)
        ts = [svc.submit(s, 100) for s in specs]
        for _ in range(4):
            svc.step()
        out.append([svc.field(t, f) for t in ts for f in ("U", "p", "mdot")])
        svc.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.isfinite(a).all() and np.array_equal(a, b)
