"""Steps whose kernels start while their predecessor drains (launch_chained):
the no-allocation entry point captured in a CUDA graph, after a device copy, a
host copy or nothing, and followed by a kernel of the caller's, gives the eager
call's fields on every replay; a run of single-step calls gives those of one
call (FP64, the fused form and FP32; both models)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [(2, 2, 2), (24, 20, 28), (40, 33, 37)])
@pytest.mark.parametrize("source", ["device", "host", "none"])
def test_captured_steps_equal_eager(sides, source):
    torch = pytest.importorskip("torch")
    from axions_gb300 import lattice
    from axions_gb300.params import ENERGY_EVOLUTION, make_params
    L = lattice.load_library()
    nx, ny, nz = sides
    p = make_params(0, nx=nx, ny=ny, nz=nz, d=0.5, dt=0.1, lam=2.0, g=1.0, damped_nt=0, alpha=3.0, energy_form=ENERGY_EVOLUTION)
    gen = torch.Generator(device="cuda").manual_seed(3)
    initial = torch.randn(5, 2, p.N, device="cuda", dtype=torch.float64, generator=gen)
    src = initial.cpu().pin_memory() if source == "host" else initial
    fields = torch.empty_like(initial)

    def steps():
        if source != "none":
            fields.copy_(src, non_blocking=True)
        assert L.lat_ah_step_f64_noalloc(ctypes.byref(p), ctypes.c_void_p(fields.data_ptr()), 0, 3,
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        fields.neg_()

    fields.copy_(src)
    steps()
    torch.cuda.synchronize()
    want = fields.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        steps()
    for _ in range(3):
        fields.copy_(src)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(fields, want)


@pytest.mark.parametrize("model,precision", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 1)])
@pytest.mark.parametrize("n", [4, 30])
def test_single_steps_equal_one_call(model, precision, n):
    from axions_gb300 import lattice
    from axions_gb300.params import ENERGY_EVOLUTION, make_params
    p = make_params(model, n=n, d=0.5, dt=0.1, lam=2.0, g=1.0, damped_nt=0, alpha=3.0, energy_form=ENERGY_EVOLUTION,
                    precision=precision, **({"lambda2": 2.0, "q1": 1.0, "q2": 2.0} if model else {}))
    res = []
    for single in (True, False):
        with lattice.Lattice(p) as lat:
            lat.random_phase_ic_device(4)
            if single:
                diags = []
                for _ in range(12):
                    diags += list(lat.advance(1, diag_every=3))
                    lat.get_slots()
            else:
                diags = list(lat.advance(12, diag_every=3))
            res.append((lat.get_slots(), diags))
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1] == res[1][1]
