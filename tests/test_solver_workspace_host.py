"""nbg_solver_solve where the memory for the slice form's plan is not there (host/solve.c
against stand-ins of the device calls, tests/c/solver_workspace.c).  CPU only."""
import os
import subprocess

from conftest import ROOT


def test_solves_without_the_plan_where_it_does_not_fit(tmp_path):
    from nbots_gb300 import _lib as L
    L.lib()  # built
    pkg, exe = os.path.dirname(L.GPU_SO), tmp_path / "solver_workspace"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "nbots_gb300", "host"),
                    os.path.join(ROOT, "tests", "c", "solver_workspace.c"), "-o", str(exe),
                    "-L" + pkg, "-lnbots_gpu", "-lnbots_host", "-Wl,-rpath," + pkg], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.returncode
