"""What a garment is charged when a server packs it under a memory budget."""
import ctypes as C

import pytest

from vistio_b200 import _lib, api, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [24, 64, 128])
def test_host_factored_garment_is_charged_what_its_batch_holds(side):
    """The server's set-ups are factorized on the host. Such a garment holds its
    factor and its state; its charge is that and, for packing, at most a tenth more
    (not the workspace of a factorization on the device, which it never uses)."""
    mesh = scenarios.hanging_sheet(side, 1.0)
    cfg = api.drape_config(host_factorization=True)
    s = api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, api.SetupDesc(), pinned=mesh.pinned)
    need = C.c_uint64()
    _lib.check(_lib.lib().vistio_solver_device_bytes(s.h, 0, C.byref(need)))
    held = api.Batch([s]).info()["device_bytes"]
    print(side, need.value, held)
    assert held <= 1.1 * need.value and need.value <= 1.1 * held
