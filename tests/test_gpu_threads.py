"""Handles of different meshes used by several host threads at once, each on a
stream of its own: the row kernels' shared memory follows the mesh, and one
thread's launch does not depend on what another one launches."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def navier_stokes(F, M, vertex_map):
    xyz2, el2 = F.structured_mesh(M, 2, seed=51)
    xyz1, el1 = F.structured_mesh(M, 1, seed=51)
    if not vertex_map:
        el1 = np.ascontiguousarray(el1[:, [1, 0, 2, 3]])
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=xyz1.shape[0], viscosity=0.01)
    return a, 0.5 * F.fourier_field(xyz2, seed=51), F.uniform_field(51, xyz1.shape[0])


CASES = {"velocity rows": lambda F: [navier_stokes(F, 1, True), navier_stokes(F, 6, True)],
         "pressure rows": lambda F: [navier_stokes(F, 1, False), navier_stokes(F, 4, False)]}


@pytest.mark.parametrize("case", list(CASES))
def test_two_threads(case):
    import torch
    import feddlib_gb300 as F
    handles = CASES[case](F)
    failures = []

    def work(a, u, p):
        try:
            want, ru, _ = a.assemble(u=u, p=p)
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                du, dp = (None if x is None else torch.from_numpy(x).cuda() for x in (u, p))
                bufs = [torch.empty(w.size, dtype=torch.float64, device="cuda") for w in want]
                dru = torch.empty(a.n_u, dtype=torch.float64, device="cuda")
                drp = torch.empty(max(a.n_p, 1), dtype=torch.float64, device="cuda")
            stream.synchronize()
            args = (None if du is None else du.data_ptr(), None if dp is None else dp.data_ptr(),
                    [b.data_ptr() for b in bufs], dru.data_ptr(), drp.data_ptr())
            start.wait()
            for _ in range(3000):
                a.assemble_device(*args, stream=stream.cuda_stream)
            stream.synchronize()
            assert all(np.array_equal(b.cpu().numpy(), w) for b, w in zip(bufs, want))
            assert np.array_equal(dru.cpu().numpy(), ru)
        except BaseException as e:
            failures.append(e)
            start.abort()

    start = threading.Barrier(len(handles))
    threads = [threading.Thread(target=work, args=h) for h in handles]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
        assert not t.is_alive()
    assert not failures, failures
