"""Resident time loops (csrc/kernels_resident.cuh): the default kernels of FP32
engines, against the FP32 oracle.

The loops evaluate the oracle's expressions in its order without FMA, so every
result is expected bit for bit: seismograms, strips, end states, gradient and
illuminations.  The sizes sit where a split can go wrong: bands of one, two and
three 4-column tiles and a shot in one band, grids whose last tile has 1 to 4
columns, every alignment of the free surface and of the bottom row to the 4-row
tiles, the smallest grid, columns of several warps, scattered and coinciding
receivers.  SWIT_RES_FWD_TILES / SWIT_RES_BWD_TILES set the band width,
SWIT_RES_FWD_COLS the forward's columns per thread (4 or 8).
"""
import numpy as np
import pytest

from oracle import oracle as O
from swit_gb300 import Engine, SwitError, survey

pytestmark = pytest.mark.gpu


def problem(nx=37, nz=28, npml=9, nt=140, ns=2, zs=20.0, zr=10.0, free_surface=1, comp="p", scattered=False):
    s = survey.small(nx=nx, nz=nz, npml=npml, nt=nt, ns=ns, zs=zs, zr=zr)
    s.free_surface = free_surface
    if scattered:  # two nodes with several receivers, one receiver off the line
        rec = s.rec_xz.copy()
        rec[:, 5] = rec[:, 4] + np.array([3.0, 0.0], np.float32)
        rec[:, 9] = rec[:, 4]
        rec[:, 7, 1] += 20.0
        s.rec_xz = rec
    pb = O.Problem(s.nx, s.nz, s.npml, s.nt, s.dx, s.dt, s.src_xz, s.rec_xz, free_surface=free_surface, comp=comp)
    return s, pb


def split(monkeypatch, tiles):
    for k in ("SWIT_RES_FWD_TILES", "SWIT_RES_BWD_TILES"):
        monkeypatch.setenv(k, str(tiles))


SHAPES = ([(dict(nx=37, nz=28, npml=n), t) for n in (8, 9, 10, 11) for t in (1, 2)] +
          [(dict(nx=nx, nz=30, npml=7), 3) for nx in (34, 35, 36, 37)] +
          [(dict(nx=36, nz=nz, npml=8, zs=70.0, zr=0.0), 2) for nz in (27, 28, 29, 30)] +
          [(dict(nx=8, nz=8, npml=2, ns=1, nt=60), 3), (dict(nx=8, nz=8, npml=2, ns=1, nt=60), 1),
           (dict(nx=40, nz=36, npml=8, zs=120.0, free_surface=0), 2), (dict(nx=40, nz=36, npml=9, scattered=True), 15),
           (dict(nx=40, nz=36, npml=9, zr=60.0, zs=120.0, scattered=True), 1), (dict(nx=61, nz=210, npml=12, nt=90), 2),
           (dict(comp="vx"), 2), (dict(comp="vz"), 2)])


@pytest.mark.parametrize("cols", [4, 8])
@pytest.mark.parametrize("shape,tiles", SHAPES)
def test_forward_matches_oracle(shape, tiles, cols, monkeypatch):
    s, pb = problem(**shape)
    src, rho = s.source(), s.rho(s.vp_true)
    ref = O.forward(pb, s.vp_true, rho, src, store=True)
    split(monkeypatch, tiles)
    monkeypatch.setenv("SWIT_RES_FWD_COLS", str(cols))
    with Engine(**s.engine_args(), receiver_component=shape.get("comp", "p")) as e:
        e.set_model(s.vp_true, rho)
        plain = e.forward(src, save_boundary=False)
        seis = e.forward(src, save_boundary=True)
        snap = e.export_snapshot()
        e.check()
    np.testing.assert_array_equal(seis, ref["seis"])
    np.testing.assert_array_equal(plain, ref["seis"])
    for k in ("boundary", "p_end", "u_end", "w_end"):
        np.testing.assert_array_equal(snap[k], ref[k], err_msg=k)


@pytest.mark.parametrize("shape,tiles", [(a, t) for a, t in SHAPES if a.get("comp") != "vx"])
def test_reverse_matches_oracle(shape, tiles, monkeypatch):
    s, pb = problem(**shape)
    src, rho = s.source(), s.rho(s.vp_true)
    ref = O.forward(pb, s.vp_true, rho, src, store=True)
    adj = (np.random.default_rng(tiles).standard_normal(ref["seis"].shape) * 1e-3).astype(np.float32)
    want = O.adjoint(pb, s.vp_true, rho, src, adj, ref)
    split(monkeypatch, tiles)
    with Engine(**s.engine_args(), receiver_component=shape.get("comp", "p")) as e:
        assert e.query()["kernel"] == "resident"
        e.set_model(s.vp_true, rho)
        e.forward(src, save_boundary=True)
        first = e.backward(adj)
        again = e.backward(adj)
        e.check()
    for got in (first, again):
        for a, k in zip(got, ("g", "fw", "bk")):
            np.testing.assert_array_equal(a, want[k], err_msg=k)


@pytest.mark.parametrize("every", [16, 32, 50, 139, 140])
def test_checkpointed_segments_match_oracle(every, monkeypatch):
    """Segments of a checkpointed run start and end in the fields the loop before left in memory."""
    s, pb = problem()
    src, rho = s.source(), s.rho(s.vp_true)
    ref = O.forward(pb, s.vp_true, rho, src, store=True)
    adj = (ref["seis"] * 0.5).astype(np.float32)
    want = O.adjoint(pb, s.vp_true, rho, src, adj, ref)
    split(monkeypatch, 2)
    with Engine(**s.engine_args(), checkpoint_every=every) as e:
        assert e.query()["kernel"] == "resident"
        e.set_model(s.vp_true, rho)
        np.testing.assert_array_equal(e.forward(src, save_boundary=True), ref["seis"])
        for a, k in zip(e.backward(adj), ("g", "fw", "bk")):
            np.testing.assert_array_equal(a, want[k], err_msg=k)


@pytest.mark.parametrize("cols", [4, 8])
@pytest.mark.parametrize("shape,tiles,every", [(a, t, 0) for a, t in SHAPES if "comp" not in a] +
                         [(dict(), 2, k) for k in (16, 50, 139, 140)])
def test_exact_adjoint_matches_oracle(shape, tiles, every, cols, monkeypatch):
    s, pb = problem(**shape)
    src, rho = s.source(), s.rho(s.vp_true)
    adj = np.random.default_rng(tiles).standard_normal((pb.ns, pb.ngmax, s.nt)).astype(np.float32)
    want = O.exact(pb, s.vp_true, rho, src, adj)
    split(monkeypatch, tiles)
    monkeypatch.setenv("SWIT_RES_FWD_COLS", str(cols))
    with Engine(**s.engine_args(), adjoint="exact", checkpoint_every=every) as e:
        assert e.query()["kernel"] == "resident"
        e.set_model(s.vp_true, rho)
        seis = e.forward(src, save_boundary=True)
        first = e.backward_exact(adj)
        again = e.backward_exact(adj)
        e.check()
    np.testing.assert_array_equal(seis, want["seis"])
    for got in (first, again):
        np.testing.assert_array_equal(got[0], want["g"])
        np.testing.assert_array_equal(got[1], want["gsrc"])


def test_routes():
    """What the resident loops do not take stays on the step kernels."""
    s, _ = problem()
    for opts, kernel in ((dict(), "resident"), (dict(kernel="vec"), "vec"), (dict(shots_per_batch=1), "vec"),
                         (dict(precision="fp64"), "vec"), (dict(path="plain"), "vec"), (dict(graph_branches=2), "vec"),
                         (dict(block_x=8), "vec"), (dict(checkpoint_every=15), "vec"),
                         (dict(receiver_component="vx"), "vec"), (dict(adjoint="exact"), "resident"),
                         (dict(adjoint="exact", receiver_component="vz"), "vec")):
        with Engine(**s.engine_args(), **opts) as e:
            assert e.query()["kernel"] == kernel, opts


@pytest.mark.parametrize("bad", [np.inf, np.nan, np.finfo(np.float32).max])
def test_values_that_are_not_finite_spread_as_in_the_step_kernels(bad, monkeypatch):
    """What a tile computes beyond the update ranges never reaches a value inside them."""
    s, pb = problem(ns=3)
    src = s.source().copy()
    src[1, 40] = bad
    rho, out = s.rho(s.vp_true), []
    split(monkeypatch, 2)
    for kernel in ("auto", "vec"):
        with Engine(**s.engine_args(), kernel=kernel) as e:
            e.set_model(s.vp_true, rho)
            seis = e.forward(src, save_boundary=True)
            adj = seis.copy()
            adj[2, 3, 90] = bad
            out.append([seis, *e.backward(adj)])
        with Engine(**s.engine_args(), kernel=kernel, adjoint="exact") as e:
            e.set_model(s.vp_true, rho)
            e.forward(src, save_boundary=True)
            out[-1] += e.backward_exact(adj)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert np.isfinite(out[0][0][[0, 2]]).all()


def test_halo_timeout_is_reported_and_the_context_stays_usable(monkeypatch):
    """With a poll limit of 0 every halo wait gives up at its first miss, records
    it in the engine's error word and goes on without waiting: the call with host
    buffers raises, check() clears the word, and an engine created afterwards
    computes the oracle's seismograms."""
    s, pb = problem()
    src, rho = s.source(), s.rho(s.vp_true)
    ref = O.forward(pb, s.vp_true, rho, src, store=False)
    split(monkeypatch, 1)
    monkeypatch.setenv("SWIT_RES_WAIT_POLLS", "0")
    with Engine(**s.engine_args()) as e:
        e.set_model(s.vp_true, rho)
        with pytest.raises(SwitError, match="SWIT_E_TIMEOUT"):
            e.forward(src, save_boundary=False)
        with pytest.raises(SwitError, match="SWIT_E_TIMEOUT"):
            e.check()
        e.check()  # the word was cleared
    monkeypatch.delenv("SWIT_RES_WAIT_POLLS")
    with Engine(**s.engine_args()) as e:
        e.set_model(s.vp_true, rho)
        np.testing.assert_array_equal(e.forward(src, save_boundary=False), ref["seis"])
        e.check()


@pytest.mark.parametrize("kernels,env", [(("auto", "vec", "auto"), {}), (("vec", "vec", "vec"), {}),
                                         (("vec", "vec", "vec"), {"SWIT_MULTI_WAVE_BYTES": "1"}),
                                         (("vec", "auto", "vec"), {"SWIT_MULTI_WAVE_BYTES": "5e5",
                                                                   "SWIT_MULTI_GRAPH_NODES": "0"}),
                                         (("vec", "vec", "vec"), {"SWIT_MULTI_WAVE_BYTES": "1",
                                                                  "SWIT_MULTI_GRAPH_NODES": "300"})])
def test_multi_engine_resident_and_wave_instances(kernels, env, monkeypatch):
    """Instances with resident loops run beside instances in waves of the step
    kernels (kernel="vec"), in every wave layout; every result equals the
    instance's own engine's."""
    import torch
    from swit_gb300 import MultiEngine
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    shapes = [dict(nx=37, nz=28, npml=9, nt=120, ns=2), dict(nx=61, nz=41, npml=12, nt=150, ns=3),
              dict(nx=30, nz=26, npml=8, nt=100, ns=1)]
    probs, args = [problem(**k)[0] for k in shapes], []
    for s, kernel in zip(probs, kernels):
        args.append(dict(s.engine_args(), kernel=kernel))
    srcs = [torch.from_numpy(s.source()).cuda() for s in probs]
    obss = [torch.rand((s.ns, s.ng, s.nt), device="cuda", generator=torch.Generator("cuda").manual_seed(i)) * 1e-3
            for i, s in enumerate(probs)]
    want = []
    for a, s, x, o in zip(args, probs, srcs, obss):
        with Engine(**a) as e:
            e.set_model(s.vp_true, s.rho(s.vp_true))
            want.append((e.gradient_l2(x, o), e.misfit_l2(x, o)))
    with MultiEngine(args) as m:
        for e, s in zip(m.engines, probs):
            e.set_model(s.vp_true, s.rho(s.vp_true))
        got = m.gradient_l2(srcs, obss)
        some = m.misfit_l2(srcs, obss, active=[True, False, True])
        every = m.misfit_l2(srcs, obss)
    for g, (w, v) in zip(got, want):
        for k in ("grad", "illum_fw", "illum_bk"):
            torch.testing.assert_close(g[k], w[k], rtol=0, atol=0)
        assert g["misfit"] == w["misfit"]
    assert every == [v for _, v in want]
    assert some == [want[0][1], 0.0, want[2][1]]
