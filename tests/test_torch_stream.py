"""The torch derivative operators' stream ordering."""
import pytest

from css_b200 import problem
from css_b200.context import Simulation

pytestmark = pytest.mark.gpu


def test_default_stream_orders_with_torch(gpu_available):
    """On PyTorch's default stream (handle 0) the operator waits for the work
    that makes its input and its readers wait for it: the same values as with
    a synchronisation on both sides."""
    import torch
    from css_b200 import torch_ops
    p, prof, _, _, _ = problem.build((64, 64, 96), decomp=(2, 2, 3))
    sim = Simulation(p, prof)
    x0 = torch.randn(p.nr, p.nphi, p.nth, generator=torch.Generator().manual_seed(3), dtype=torch.float64).cuda()
    a = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    want = torch_ops.dbydt(x0 * 3.0, sim)
    torch.cuda.synchronize()
    want = want + 1.0
    for _ in range(10):
        for _ in range(4):
            b = a @ a  # keeps the default stream busy before the input is made
        x = x0 * 3.0
        got = torch_ops.dbydt(x, sim) + 1.0
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    del b
    sim.close()


@pytest.mark.parametrize("direction", [0, 1, 2])
def test_first_backward_on_a_side_stream(direction, gpu_available):
    """The first adjoint of a (direction, order, closure) makes its tables:
    they are on the device before the kernel that reads them, on any stream and
    with several threads calling first at once.  The same bits as a second
    call."""
    import threading
    import torch
    from css_b200 import torch_ops  # noqa: F401
    p, prof, _, _, _ = problem.build((32, 48, 60), decomp=(2, 2, 3))
    g = torch.randn(p.nr, p.nphi, p.nth, generator=torch.Generator().manual_seed(5), dtype=torch.float64).cuda()
    torch.cuda.synchronize()
    for order in (1, 2):
        for bdry in (range(5) if direction < 2 else (0,)):
            sim = Simulation(p, prof)
            first = [None] * 4

            def call(k):
                s = torch.cuda.Stream()
                with torch.cuda.stream(s):
                    first[k] = torch.ops.css.deriv_adjoint(g, sim.h.value, direction, order, bdry)
                s.synchronize()

            threads = [threading.Thread(target=call, args=(k,)) for k in range(4)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            again = torch.ops.css.deriv_adjoint(g, sim.h.value, direction, order, bdry)
            torch.cuda.synchronize()
            for a in first:
                assert torch.equal(a, again), (order, bdry)
            sim.close()


def test_host_data_is_in_place_before_the_first_kernel(gpu_available):
    """What a call sends up from host memory is there for the first kernel that
    reads it: the cyclic derivative right after a run is made, and the network's
    BF16 weights right after its parameters are set, each equal to a second
    call after the device has come to rest."""
    import ctypes
    import numpy as np
    import torch
    from css_b200 import _lib
    from css_b200 import closure as C
    p, prof, _, _, _ = problem.build((20, 32, 48), decomp=(2, 2, 3))
    x = torch.randn(p.nr, p.nphi, p.nth, generator=torch.Generator().manual_seed(7), dtype=torch.float64).cuda()
    net = C.Mlp(135, 128, 12, max_rows=64, seed=3)
    net.set_forward("gemm")
    xr = torch.randn(64, 144, generator=torch.Generator().manual_seed(8)).to(torch.bfloat16).cuda()
    rng = np.random.default_rng(2)
    torch.cuda.synchronize()
    for k in range(8):
        sim, out = Simulation(p, prof), [torch.empty_like(x) for _ in range(2)]
        s = torch.cuda.Stream()
        for o in out:
            _lib.check(_lib.lib().css_dbydp_cyclic_dev(sim.h, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(o.data_ptr()),
                                                       2, ctypes.c_void_p(s.cuda_stream)))
            torch.cuda.synchronize()
        assert torch.equal(out[0], out[1]), k
        sim.close()
        for l in range(4):
            kk, m = net.dims[l], net.dims[l + 1]
            net.set_params(l, rng.standard_normal((kk, m)) * 0.1, rng.standard_normal(m) * 0.1)
        a = net.forward(xr, 64)
        torch.cuda.synchronize()
        assert torch.equal(a, net.forward(xr, 64)), k
    net.close()
