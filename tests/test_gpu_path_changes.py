"""Changed contacts make new chain lists: not at the cost of other threads'
captures, nor of the host's time."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(type_id=(17, 0), num_unitcells=300, num_modes=4, contact_mu=(0.0, -0.4), contact_T=(300.0, 300.0),
          eq_integration_pts=(48, 48, 96), noneq_integration_pts=(400,), E_zPlus_imag=1e-3)


def _tube():
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    t = CNT(**KW)
    U = site_potential(t.site_positions(), 5)
    t.set_potential(U, (U[0], U[-1]))
    return t


def test_contacts_change_while_another_thread_captures():
    """40 changes of the contacts (each retires a list), made by a second thread
    between the begin and the end of a capture of this one: the graph is whole and
    gives the plan's charge, and every charge of the second thread is the one of its
    contacts."""
    import torch
    from electrostatic_b200.negf import ChargePlan, compute_charge
    planned, changed = _tube(), _tube()
    Q = torch.zeros(planned.num_field_sites, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(Q)
    plan = ChargePlan([planned], Q)
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    mus = [(0.0, -0.4), (0.01, -0.39)]
    ref = []
    for mu in mus:  # buffers of both sizes exist before the capture
        changed.set_contact_mu(mu)
        compute_charge([changed], out=out, stream=other)
        other.synchronize()
        ref.append(out.cpu().numpy())
    with torch.cuda.stream(s):
        plan.launch(stream=s)
    s.synchronize()
    want = Q.cpu().numpy().copy()
    begun, done, errors, events = threading.Event(), threading.Event(), [], []
    outs = [torch.zeros_like(out) for _ in range(40)]
    torch.cuda.synchronize()

    def work():
        try:
            begun.wait(30)
            for i, o in enumerate(outs):
                changed.set_contact_mu(mus[i % 2])
                compute_charge([changed], out=o, stream=other)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)
        finally:
            done.set()

    th = threading.Thread(target=work)
    th.start()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="global"):
        plan.launch(stream=s)
        begun.set()
        done.wait(30)
        plan.launch(stream=s)
    th.join()
    assert not errors, errors
    Q.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(Q.cpu().numpy(), want)
    for i, o in enumerate(outs):
        assert np.array_equal(o.cpu().numpy(), ref[i % 2]), i
    del graph
    plan.close()


def test_a_path_change_does_not_wait_for_the_stream():
    """A call with a device result returns while earlier work of its stream still
    runs, also after the contacts changed."""
    import torch
    from electrostatic_b200.negf import compute_charge
    t = _tube()
    s = torch.cuda.Stream()
    out = torch.zeros(t.num_field_sites, dtype=torch.float64, device="cuda")
    for mu in ((0.0, -0.4), (0.01, -0.39)):
        t.set_contact_mu(mu)
        compute_charge([t], out=out, stream=s)
    ref = t.Solve_NEGF()
    torch.cuda.synchronize()
    t.set_contact_mu((0.0, -0.4))
    end = torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(400_000_000)  # 0.2 s and more
    t0 = time.perf_counter()
    compute_charge([t], out=out, stream=s)
    t.set_contact_mu((0.01, -0.39))
    compute_charge([t], out=out, stream=s)
    dt = time.perf_counter() - t0
    end.record(s)
    assert not end.query() and dt < 0.1, dt
    s.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)


def test_retired_lists_are_freed(negf_lib):
    """The memory of replaced lists is bounded, and release_scratch hands it back."""
    import torch
    from electrostatic_b200.negf import compute_charge, release_scratch
    t = _tube()
    out = torch.zeros(t.num_field_sites, dtype=torch.float64, device="cuda")
    compute_charge([t], out=out)
    release_scratch()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for i in range(1500):  # 50 KB each
        t.set_contact_mu((1e-5 * i, -0.4))
        compute_charge([t], out=out)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20
    release_scratch()
    assert free0 - torch.cuda.mem_get_info()[0] <= 8 << 20
