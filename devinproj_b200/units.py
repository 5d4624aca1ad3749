"""SI values of accusim's physical constants (accusim/units.py:226-233) as plain floats for the host code and the
engine's unit conversion, and accusim's own `si()` for arguments given as quantities."""
from __future__ import annotations

from ._accusim import accusim, units as _u

si = _u.si
if accusim is not None:
    k_B = float(_u.k_B.value)                         # J/K
    N_A = float(_u.N_A.value)                         # 1/mol
    e_charge = float(_u.e_charge.value)               # C
    k_e = float(_u.k_e.value)                         # J m / C^2
    amu = float(_u.parse_unit("u").value)             # kg
    c_light = float(_u.c.value)                       # m/s
else:   # the same numbers (SI of 2019, CODATA 2018), for the engine's units
    k_B, N_A, e_charge = 1.380649e-23, 6.02214076e23, 1.602176634e-19
    k_e, amu, c_light = 8987551792.261171, 1.6605390666e-27, 299792458.0
