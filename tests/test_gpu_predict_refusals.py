"""What warmstart.predict_cases refuses."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_case_without_cells():
    from fvdbm_jax_gb300 import cases as CS
    from fvdbm_jax_gb300 import warmstart as WS
    real = CS.porous_square(20, 6000, 0.003, rho_in=1.01, rho_out=0.99, porosity=0.8, fv_dt=1.0, seed=700, mesher=True)
    z = lambda *s: np.zeros(s)  # noqa: E731
    empty = (None, NS(face_indices=z(0, 3), face_normals=z(0, 3)),
             NS(stencil_cells_index=z(0, 2), stencil_dists=z(0, 2), L=z(0), n=z(0, 2), nodes_index=z(0, 2)),
             NS(type=z(0), rho=z(0)), NS(cell_centers=z(0, 2), cell_areas=z(0), face_centers=z(0, 2)))
    net = WS.MPNN(layers=1, scales=(16,))
    with pytest.raises(ValueError):
        WS.predict_cases(net, [real, empty], [1.01, 1.01], [0.99, 0.99])
