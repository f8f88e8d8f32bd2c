"""Resident reverse loops of more than 384 threads per block: an instance of its own (128 registers a thread),
against the FP32 oracle, bit for bit.  The band widths below give 416 to 512 threads, with one, two and six
bands."""
import numpy as np
import pytest

from oracle import oracle as O
from swit_gb300 import Engine, survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,tiles,threads,opts", [
    (dict(nx=36, nz=45, npml=11), 15, 416, {}), (dict(nx=59, nz=57, npml=11), 11, 416, {}),
    (dict(nx=36, nz=53, npml=11), 15, 480, {}), (dict(nx=38, nz=56, npml=11), 15, 512, {}),
    (dict(nx=61, nz=210, npml=12, nt=90), 4, 480, {}),
    (dict(nx=59, nz=57, npml=11), 11, 416, dict(free_surface=0)),
    (dict(nx=59, nz=57, npml=11), 11, 416, dict(comp="vz")),
    (dict(nx=61, nz=210, npml=12, nt=90), 4, 480, dict(scattered=True)),
    (dict(nx=59, nz=57, npml=11), 11, 416, dict(every=30))])
def test_wide_blocks_match_oracle(shape, tiles, threads, opts, monkeypatch):
    s = survey.small(**dict(dict(nt=140, ns=2, zs=20.0), **shape))
    s.free_surface = opts.get("free_surface", 1)
    comp = opts.get("comp", "p")
    if opts.get("scattered"):  # two nodes with several receivers, one receiver off the line
        rec = s.rec_xz.copy()
        rec[:, 5] = rec[:, 4] + np.array([3.0, 0.0], np.float32)
        rec[:, 9] = rec[:, 4]
        rec[:, 7, 1] += 20.0
        s.rec_xz = rec
    pb = O.Problem(s.nx, s.nz, s.npml, s.nt, s.dx, s.dt, s.src_xz, s.rec_xz, free_surface=s.free_surface, comp=comp)
    src, rho = s.source(), s.rho(s.vp_true)
    ref = O.forward(pb, s.vp_true, rho, src, store=True)
    adj = (np.random.default_rng(tiles).standard_normal(ref["seis"].shape) * 1e-3).astype(np.float32)
    want = O.adjoint(pb, s.vp_true, rho, src, adj, ref)
    monkeypatch.setenv("SWIT_RES_BWD_TILES", str(tiles))
    with Engine(**s.engine_args(), receiver_component=comp, checkpoint_every=opts.get("every", 0)) as e:
        loop = e.query_loop("reverse")
        assert loop["kernel"] == "resident" and loop["threads"] == threads
        e.set_model(s.vp_true, rho)
        e.forward(src, save_boundary=True)
        got = e.backward(adj)
        e.check()
    for a, k in zip(got, ("g", "fw", "bk")):
        np.testing.assert_array_equal(a, want[k], err_msg=k)
