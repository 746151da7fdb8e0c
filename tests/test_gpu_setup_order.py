"""Engines made while another thread keeps the legacy default stream busy.

The engine's stream does not wait for that one, so a buffer's clearing that
was issued there could land after the kernel that fills the buffer (the packed
Cholesky vectors, the exchange operands).  Such an engine takes the same step
and the same measurement, to the bit, as one made while the GPU is idle."""
import threading

import numpy as np
import pytest
import torch

from afqmclab_b200 import capi, inputs
from tests.parity_common import hubbard

pytestmark = pytest.mark.gpu


def outputs(make, wf, lw, al):
    e = make()
    e.set_walkers_async(wf.ctypes.data, lw.ctypes.data, al.ctypes.data)
    e.upload_wait()
    e.step(1)
    e.reset_measurement()
    e.add_mixed_measurement()
    out = [*e.get_walkers(), np.array(e.measurement())]
    assert e.status() == 0
    e.close()
    return out


def busy(stop):
    """About a millisecond of waiting kernels at a time on the default stream."""
    while not stop.is_set():
        torch.cuda._sleep(2_000_000)
        torch.cuda.default_stream().synchronize()


@pytest.mark.parametrize("form", ["phaseless fp64", "phaseless mixed", "constrained fp64", "constrained mixed"])
def test_engine_made_beside_default_stream_work(form):
    prec = capi.AFQMC_MIXED if form.endswith("mixed") else capi.AFQMC_FP64
    if form.startswith("phaseless"):
        m = inputs.molecule_inputs(64, 16, 16, 64, dt=0.005, decay=20.0, seed=7)
        wf, lw, al = inputs.initial_walkers(m.phiTUp, 8, seed=3, noise=0.02)
        make = lambda: capi.pl_engine(m, 8, 5, 1000, 1000, precision=prec)  # noqa: E731
    else:
        m = hubbard("densitySpin", False, nx=4, ny=4, nup=5, ndn=4)
        wf, lw, al = inputs.initial_walkers(m.phiT, 8, seed=3, noise=0.02)
        make = lambda: capi.cp_engine(m, 8, 5, 1000, 1000, precision=prec)  # noqa: E731
    quiet = outputs(make, wf, lw, al)
    torch.cuda.init()
    stop = threading.Event()
    t = threading.Thread(target=busy, args=(stop,))
    t.start()
    try:
        for _ in range(5):
            for a, b in zip(outputs(make, wf, lw, al), quiet):
                np.testing.assert_array_equal(a, b)
    finally:
        stop.set()
        t.join()
