"""The package where accusim cannot be imported: the C-ABI bindings and the engine import and answer, what needs accusim
says so when it is made."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import importlib.abc, os, sys
class Hide(importlib.abc.MetaPathFinder):
    def find_spec(self, name, path=None, target=None):
        if name.split(".")[0] == "accusim":
            raise ModuleNotFoundError("No module named 'accusim'", name=name)
sys.meta_path.insert(0, Hide())
isdir = os.path.isdir
os.path.isdir = lambda p: False if os.fspath(p).endswith(os.path.join("_ref", "accusim")) else isdir(p)

import devinproj_b200 as b200
from devinproj_b200 import _accusim, ewald, learned, units
from devinproj_b200.engine import Engine, ForceField, LEN
from oracle import accusim_port as port
assert _accusim.accusim is None
for name in b200.__all__:
    assert hasattr(b200, name), name
assert not hasattr(b200, "no_such_name")
assert (units.k_B, units.k_e, units.amu, units.e_charge, units.N_A) == (port.K_B, port.K_E, port.AMU, port.E_CHARGE, port.N_A)
assert ewald._bind() and learned._bind()
makes = [lambda: b200.LennardJones({"Ar": (1.0, 1.0)}), lambda: b200.DampedShiftedCoulomb(1.0), b200.Ewald,
         lambda: b200.GpuSystem(3, box=1.0, periodic=True), b200.VelocityVerlet, lambda: b200.Langevin(1.0, 1.0),
         lambda: b200.NoseHoover(1.0, 1.0), lambda: b200.GpuSimulation(None, []), lambda: units.si(1.0, "s")]
for make in makes:
    try:
        make()
    except ImportError as e:
        assert str(e) == _accusim.MISSING, e
    else:
        raise AssertionError("made without accusim")
print("done")
"""


def test_package_without_accusim():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stderr[-2000:]
