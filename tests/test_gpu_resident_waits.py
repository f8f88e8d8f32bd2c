"""Halo waits of the resident loops that give up, as the calls report them.

With SWIT_RES_WAIT_POLLS=0 a wait gives up at its first miss and goes on without
waiting; a loop whose shots lie in one band each (100 column tiles per band, at
these sizes) has no halo and waits for nothing, so one engine can have a loop that
fails beside one that cannot.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from swit_gb300 import Engine, MultiEngine, SwitError, _lib, survey

pytestmark = pytest.mark.gpu


def problem():
    s = survey.small(nx=37, nz=28, npml=9, nt=140, ns=2, zs=20.0)
    pb = O.Problem(s.nx, s.nz, s.npml, s.nt, s.dx, s.dt, s.src_xz, s.rec_xz, free_surface=1)
    return s, pb, s.source(), s.rho(s.vp_true)


def bands(monkeypatch, fwd, bwd):
    """Column tiles per band; 0 polls: with 1 the loop fails, with 100 it does not."""
    monkeypatch.setenv("SWIT_RES_WAIT_POLLS", "0")
    monkeypatch.setenv("SWIT_RES_FWD_TILES", str(fwd))
    monkeypatch.setenv("SWIT_RES_BWD_TILES", str(bwd))


def ptr(a):
    return a.ctypes.data


def timeout():
    return pytest.raises(SwitError, match="SWIT_E_TIMEOUT")


@pytest.mark.parametrize("call", ["gradient_l2", "gradient_l2 misfit", "backward", "backward_exact", "export_snapshot",
                                  "misfit_l2"])
def test_every_call_with_host_buffers_reports(call, monkeypatch):
    import torch
    s, pb, src, rho = problem()
    forward_fails = call not in ("backward", "backward_exact")
    bands(monkeypatch, 1 if forward_fails else 100, 100 if forward_fails else 1)
    adj = np.ones((s.ns, s.ng, s.nt), np.float32)
    with Engine(**s.engine_args(), adjoint="exact" if call == "backward_exact" else "fd2dmpi") as e:
        e.set_model(s.vp_true, rho)
        if call == "gradient_l2":  # without the misfit, the only output that waits by itself
            grad = np.zeros((s.nx, s.nz), np.float32)
            with timeout():
                _lib.check(e._lib.swit_gradient_l2(e._h, ptr(src), ptr(adj), ptr(grad), None, None, None, None, 0, None))
        elif call == "gradient_l2 misfit":
            with timeout():
                e.gradient_l2(src, adj)
        elif call == "misfit_l2":
            with timeout():
                e.misfit_l2(src, adj)
        elif call == "export_snapshot":
            e.forward(torch.from_numpy(src).cuda(), save_boundary=True)  # device buffers: no report
            with timeout():
                e.export_snapshot()
        else:
            e.forward(src, save_boundary=True)
            with timeout():
                e.backward_exact(adj) if call == "backward_exact" else e.backward(adj)
        with timeout():
            e.check()
        e.check()


def test_multi_engine_without_misfits_reports_every_instance(monkeypatch):
    s, pb, src, rho = problem()
    bands(monkeypatch, 1, 100)
    obs = np.ones((s.ns, s.ng, s.nt), np.float32)
    grads = [np.zeros((s.nx, s.nz), np.float32) for _ in range(2)]

    def array(xs):
        return (C.c_void_p * 2)(*xs)
    with MultiEngine([s.engine_args()] * 2) as m:
        for e in m.engines:
            e.set_model(s.vp_true, rho)
        with timeout():
            _lib.check(m._lib.swit_multi_gradient_l2(m._h, array([ptr(src)] * 2), array([ptr(obs)] * 2),
                                                     array(map(ptr, grads)), None, None, None, 0, None))
        for e in m.engines:
            with timeout():
                e.check()
            e.check()


def test_a_reported_wait_leaves_later_calls_alone(monkeypatch):
    """After the report the forward run counts as not made, and calls whose own waits are in order
    succeed without a swit_check between."""
    s, pb, src, rho = problem()
    ref = O.forward(pb, s.vp_true, rho, src, store=True)
    adj = (ref["seis"] * 0.5).astype(np.float32)
    want = O.adjoint(pb, s.vp_true, rho, src, adj, ref)
    bands(monkeypatch, 1, 100)
    with Engine(**s.engine_args()) as e:
        e.set_model(s.vp_true, rho)
        with timeout():
            e.forward(src, save_boundary=True)
        with pytest.raises(SwitError, match="SWIT_E_STATE"):
            e.backward(adj)
        e.import_snapshot(src, *[ref[k] for k in ("boundary", "p_end", "u_end", "w_end")])
        for a, k in zip(e.backward(adj), ("g", "fw", "bk")):
            np.testing.assert_array_equal(a, want[k], err_msg=k)
        with timeout():
            e.check()  # still reports the forward, once
        e.check()
