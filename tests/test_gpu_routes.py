"""Which kernels, batches and branches an engine's time loops take by themselves."""
import numpy as np
import pytest

from swit_gb300 import Engine, survey

pytestmark = pytest.mark.gpu


def problem(nx, nz, npml, ns, nt):
    s = survey.small(nx=nx, nz=nz, npml=npml, nt=nt, ns=ns)
    return s, s.source(), s.rho(s.vp_true)


@pytest.mark.parametrize("opts,shape,forward,reverse", [
    # every shot's state counts against the L2 for the FP32 step kernels of fd2dmpi's adjoint only, forward and
    # reverse each by its own
    (dict(kernel="vec"), (481, 141, 40, 5), 3, 3),
    (dict(kernel="vec"), (1460, 716, 50, 9), 3, 2),
    (dict(kernel="vec"), (1131, 1141, 23, 4), 2, 2),
    (dict(kernel="vec"), (1273, 1104, 24, 10), 2, 2),
    (dict(kernel="vec"), (2001, 601, 60, 3), 3, 2),
    (dict(kernel="vec"), (1884, 896, 57, 7), 2, 1),
    (dict(kernel="vec"), (1915, 2337, 22, 3), 1, 3),
    (dict(kernel="vec", graph_branches=3), (1884, 896, 57, 4), 3, 3),
    (dict(kernel="vec", precision="fp64"), (1700, 800, 40, 3), 3, 3),
    (dict(kernel="walk"), (1700, 800, 40, 3), 3, 3),
    (dict(kernel="vec", adjoint="exact"), (1739, 1192, 33, 2), 2, 2)])
def test_branches(opts, shape, forward, reverse):
    s, _, _ = problem(*shape, nt=4)
    with Engine(**s.engine_args(), **opts) as e:
        for loop, n in (("forward", forward), ("saving", forward), ("reverse", reverse)):
            assert e.query_loop(loop) == dict(kernel=opts["kernel"], shots=1 if s.nx > 500 else e.query()["shots_per_batch"],
                                              threads=0, branches=n), loop
        assert e.query()["graph_branches"] == reverse


def test_loops_on_different_branches_match_one_branch():
    s, src, rho = problem(1460, 716, 50, 4, 9)
    adj = np.random.default_rng(1).standard_normal((s.ns, s.ng, s.nt)).astype(np.float32)
    out = []
    for br in (0, 1):
        with Engine(**s.engine_args(), kernel="vec", graph_branches=br) as e:
            e.set_model(s.vp_true, rho)
            out.append((e.forward(src, save_boundary=False), e.forward(src, save_boundary=True), *e.backward(adj)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
