"""Lattices created on the device take the bytes that admission counts, and a
request that the server's budget holds only without the array for two-step
launches is served, as it is with a larger budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_lattices_take_the_bytes_admission_counts():
    import torch
    from bgk3d_gpu_b200.lattice import Lattice
    torch.zeros(1, device="cuda")
    specs = [("f32", "periodic", (256, 192, 160)), ("f64", "driven", (160, 128, 128)), ("f32", "inflow", (256, 160, 160)),
             ("f64", "channel", (199, 120, 100)), ("f32", "driven", (256, 192, 160)), ("f32_f64", "periodic", (40, 600, 256))]
    Lattice(32, 32, 32).close()                       # the pool, the module
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    lats = [Lattice(*s, kind=k, bcase=b, omega=1.0) for k, b, s in specs]
    taken = free0 - torch.cuda.mem_get_info()[0]
    assert all(lat.uses_two_steps for lat in lats)
    counted = sum(lat.device_bytes for lat in lats)
    extra = counted // 38                             # about 190 MB that were not counted
    assert taken < counted + extra // 2
    for lat in lats:
        lat.close()


def test_request_that_fits_only_without_the_extra_array():
    from bgk3d_gpu_b200.serve import Request, Server, _bytes
    trace = [Request(q, 0.0, "ldc", 128, 24, 0.6, "f32") for q in range(3)]
    full, least = _bytes(trace[0])
    assert full > least
    done, summary = Server(budget_bytes=(full + least) / 2).run(trace, keep_states=True)
    more, _ = Server(budget_bytes=10 * full).run(trace, keep_states=True)
    assert summary["requests"] == 3
    want = {d["rid"]: d["state"] for d in more}
    for d in done:
        assert np.array_equal(d["state"], want[d["rid"]])
    with pytest.raises(RuntimeError, match="more than the budget"):
        Server(budget_bytes=least - 1).run(trace)
