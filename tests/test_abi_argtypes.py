"""Every bound entry point declares its argument types: ctypes passes an
undeclared integer argument, an array's address among them, as 32 bits."""
from espins_gb300 import lib as L


def test_every_entry_point_declares_its_arguments():
    lib = L.load()
    assert [f for f in L.EXPORTED if f != "esp_lp_num_params" and not getattr(lib, f).argtypes] == []
