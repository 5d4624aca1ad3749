"""The host framework these plug-ins plug into: the `accusim` package (erezbz/DevinProj).

The GPU classes of this package subclass accusim's own `Force` and `Integrator` classes, so that accusim's
`Simulation.run`, `AccuracyReport`, `calibrate_dt` and `timescales` accept them and their `isinstance` checks
(accusim/accuracy.py:149, accusim/advisor.py:36) see the reference classes. accusim is pure Python; it is
imported from the environment, or else from the repository's own offline install under `baseline/_ref`
(made by `baseline/install_reference.sh`).

Without accusim `accusim` is None here. The build script, the C-ABI bindings and the engine below the plug-ins need
nothing of it, so every module still imports; a class of accusim, or one derived from it, raises ImportError when an
object of it is made.
"""
from __future__ import annotations

import os
import sys

_REPO_INSTALL = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "baseline", "_ref")
MISSING = ("devinproj_b200 plugs into the accusim package, which is not importable: install it "
           "(pip install <accusim checkout>, or baseline/install_reference.sh)")

try:
    import accusim
except ImportError:
    accusim = None
    if os.path.isdir(os.path.join(_REPO_INSTALL, "accusim")):
        sys.path.append(_REPO_INSTALL)
        import accusim

if accusim is not None:
    import accusim.accuracy as accuracy
    import accusim.forces as forces
    import accusim.integrators as integrators
    import accusim.simulation as simulation
    import accusim.system as system
    import accusim.units as units
else:
    def _refuse(cls, *args, **kwargs):
        raise ImportError(MISSING)

    class _Absent:
        """A module of accusim that is not there: its names are classes that can be derived from, but not made."""

        def __getattr__(self, name):
            if name.startswith("__"):
                raise AttributeError(name)
            made = type(name, (), {"__new__": _refuse})
            setattr(self, name, made)
            return made

    accuracy, forces, integrators, simulation, system, units = (_Absent() for _ in range(6))

__all__ = ["accusim", "accuracy", "forces", "integrators", "simulation", "system", "units"]
