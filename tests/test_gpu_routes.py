"""Which kernels, batches and branches an engine's time loops take by themselves."""
import numpy as np
import pytest

from swit_gb300 import Engine, SwitError, survey

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


@pytest.mark.parametrize("shape,kernel", [((481, 141, 40, 30), "resident"), ((587, 238, 48, 23), "vec")])
def test_launch_counts_are_those_of_the_loops_that_run(shape, kernel):
    s, _, _ = problem(*shape, nt=400)
    with Engine(**s.engine_args()) as e:
        q, rev, sav = e.query(), e.query_loop("reverse"), e.query_loop("saving")
    assert q["kernel"] == rev["kernel"] == kernel and sav["kernel"] == "resident"
    assert rev["branches"] == (1 if kernel == "resident" else 3)
    per_launch = 1 if kernel == "resident" else 2 * (s.nt - 1)
    assert q["kernels_per_backward"] == per_launch * -(-s.ns // rev["shots"])
    assert q["kernels_per_forward"] == -(-s.ns // sav["shots"])


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


def test_multi_engine_runs_waves_for_all_where_one_instance_needs_them(monkeypatch):
    """With 0 polls any resident loop with a halo fails: beside an instance on the step kernels nothing runs
    resident, and every result is the instance's own."""
    from swit_gb300 import MultiEngine
    probs = [problem(*shape, nt=nt) for shape, nt in (((60, 40, 12, 2), 60), ((52, 36, 10, 3), 80), ((40, 30, 8, 1), 50))]
    obss = [np.random.default_rng(i).standard_normal((s.ns, s.ng, s.nt)).astype(np.float32) * np.float32(1e-3)
            for i, (s, _, _) in enumerate(probs)]
    want = []
    for (s, src, rho), o in zip(probs, obss):
        with Engine(**s.engine_args()) as e:
            e.set_model(s.vp_true, rho)
            want.append((e.gradient_l2(src, o), e.misfit_l2(src, o)))
    for k, v in (("SWIT_RES_WAIT_POLLS", "0"), ("SWIT_RES_FWD_TILES", "1"), ("SWIT_RES_BWD_TILES", "1")):
        monkeypatch.setenv(k, v)
    srcs = [src for _, src, _ in probs]
    with MultiEngine([dict(s.engine_args(), kernel=k) for (s, _, _), k in zip(probs, ("auto", "vec", "auto"))]) as m:
        for e, (s, _, rho) in zip(m.engines, probs):
            e.set_model(s.vp_true, rho)
        got = m.gradient_l2(srcs, obss)
        every = m.misfit_l2(srcs, obss)
        with pytest.raises(SwitError, match="SWIT_E_TIMEOUT"):  # the two others run resident
            m.misfit_l2(srcs, obss, active=[True, False, True])
    for g, (w, _) in zip(got, want):
        for k in ("grad", "illum_fw", "illum_bk"):
            np.testing.assert_array_equal(g[k], w[k])
        assert g["misfit"] == w["misfit"]
    assert every == [v for _, v in want]


@pytest.mark.parametrize("env", [{}, {"SWIT_MULTI_WAVE_BYTES": "1"}, {"SWIT_MULTI_WAVE_BYTES": "5e5"},
                                 {"SWIT_MULTI_WAVE_BYTES": "1", "SWIT_MULTI_GRAPH_NODES": "0"},
                                 {"SWIT_MULTI_WAVE_BYTES": "5e5", "SWIT_MULTI_GRAPH_NODES": "0"},
                                 {"SWIT_MULTI_WAVE_BYTES": "1", "SWIT_MULTI_GRAPH_NODES": "700"}])
def test_multi_engine_waves_of_step_kernels_match_resident_engines(env, monkeypatch):
    """Every wave layout on the step kernels (kernel="vec": nothing resident), also after a partial call, against
    the problems' own engines on the default kernels."""
    import torch
    from swit_gb300 import MultiEngine
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    probs = [survey.small(nx=nx, nz=nz, npml=npml, nt=nt, dx=dx, ns=ns, seed=seed) for nx, nz, npml, nt, dx, ns, seed in
             ((52, 30, 10, 260, 10.0, 3, 3), (40, 36, 8, 180, 12.0, 2, 4), (64, 24, 9, 320, 10.0, 4, 5))]
    srcs, obss, want = [s.source() for s in probs], [], []
    for s, x in zip(probs, srcs):
        with Engine(**s.engine_args()) as e:
            assert e.query()["kernel"] == "resident"
            e.set_model(s.vp_true, s.rho(s.vp_true))
            obss.append(e.forward(x, save_boundary=False))
            e.set_model(s.vp_init, s.rho(s.vp_true))
            want.append(e.gradient_l2(x, obss[-1]))
    with MultiEngine([dict(s.engine_args(), kernel="vec") for s in probs]) as m:
        for e, s in zip(m.engines, probs):
            assert e.query()["kernel"] == "vec"
            e.set_model(s.vp_init, s.rho(s.vp_true))
        outs = [m.gradient_l2(srcs, obss), m.gradient_l2(srcs, obss)]
        assert m.misfit_l2(srcs, obss) == [w["misfit"] for w in want]
        assert m.misfit_l2(srcs, obss, active=[False, True, False]) == [0.0, want[1]["misfit"], 0.0]
        outs.append(m.gradient_l2(srcs, obss))
        outs.append([{k: v.cpu().numpy() if torch.is_tensor(v) else v for k, v in o.items()} for o in
                     m.gradient_l2([torch.from_numpy(x).cuda() for x in srcs], [torch.from_numpy(x).cuda() for x in obss])])
    for out in outs:
        for g, w in zip(out, want):
            for k in ("grad", "illum_fw", "illum_bk"):
                np.testing.assert_array_equal(g[k], w[k])
            assert g["misfit"] == w["misfit"]


@pytest.mark.parametrize("shape,resident", [
    # where both fit, the faster one by a wide margin (us per step of forward, saving forward and reverse, resident
    # and vec): 1.4, 1.8, 2.3 and 5.0, 5.4, 8.6
    ((101, 51, 20, 1), (1, 1, 1)),
    ((481, 141, 40, 10), (1, 1, 1)),   # 2.5, 3.0, 9.0 and 8.5, 9.0, 16
    ((2001, 601, 60, 1), (1, 1, 0)),   # 5.2, 5.7 and 8.5, 8.9; no reverse split fits
    ((1350, 660, 30, 1), (1, 1, 0)),   # 5.5, 5.9 and 7.8, 8.2
    ((1350, 660, 30, 3), (0, 0, 0)),   # 16.5, 18.6 and 13.4, 13.6
    ((691, 780, 16, 3), (0, 0, 0)),    # 12.4, 14.9 and 9.3, 9.6
    ((587, 238, 48, 23), (1, 1, 0)),   # 10.1, 11.6, 67.6 and 24.9, 27.6, 51.1
    ((338, 311, 51, 14), (1, 1, 0))])  # 6.7, 8.0, 40.7 and 12.0, 12.2, 23.0
def test_resident_loops_run_where_they_are_faster(shape, resident):
    s, _, _ = problem(*shape, nt=400)
    with Engine(**s.engine_args()) as e:
        got = tuple(int(e.query_loop(k)["kernel"] == "resident") for k in ("forward", "saving", "reverse"))
        assert got == resident
        assert e.query()["kernel"] == ("resident" if resident[1] and resident[2] else "vec")


def test_exact_adjoint_keeps_both_loops_on_one_path():
    """Its saving forward and its reverse loop share the layout of the stored divergence."""
    for shape in ((241, 121, 20, 4), (687, 820, 38, 3)):
        s, _, _ = problem(*shape, nt=40)
        with Engine(**s.engine_args(), adjoint="exact") as e:
            assert e.query_loop("saving")["kernel"] == e.query_loop("reverse")["kernel"] == \
                ("resident" if s.nx == 241 else "vec")


def test_forward_and_reverse_on_different_kernels_match_the_step_kernels():
    s, src, rho = problem(338, 311, 51, 14, 90)
    adj = np.random.default_rng(2).standard_normal((s.ns, s.ng, s.nt)).astype(np.float32)
    out = []
    for kernel in ("auto", "vec"):
        with Engine(**s.engine_args(), kernel=kernel) as e:
            assert [e.query_loop(k)["kernel"] for k in ("saving", "reverse")] == \
                (["resident", "vec"] if kernel == "auto" else ["vec", "vec"])
            e.set_model(s.vp_true, rho)
            out.append((e.forward(src, save_boundary=True), *e.backward(adj)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_checkpointed_forward_and_reverse_on_different_kernels_match_the_step_kernels():
    """The forward pass leaves checkpoints that the other kernels' reverse pass starts from."""
    s, src, rho = problem(643, 225, 53, 17, 64)
    adj = np.random.default_rng(3).standard_normal((s.ns, s.ng, s.nt)).astype(np.float32)
    out = []
    for kernel in ("auto", "vec"):
        with Engine(**s.engine_args(), kernel=kernel, checkpoint_every=21) as e:
            assert [e.query_loop(k)["kernel"] for k in ("forward", "saving", "reverse")] == \
                (["resident", "vec", "vec"] if kernel == "auto" else ["vec"] * 3)
            e.set_model(s.vp_true, rho)
            out.append((e.forward(src, save_boundary=True), *e.backward(adj)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("every", [0, 30])
def test_capture_beyond_the_node_bound_takes_the_resident_loops_that_fit(every, monkeypatch):
    """The reverse loop (with checkpoints also the forward) runs on the step kernels here; captured into a graph it
    would exceed the bound, and the same results come from resident loops."""
    import torch
    s, src, rho = problem(338, 311, 51, 14, 90)
    monkeypatch.setenv("SWIT_GRAPH_NODES", "300")
    src = torch.from_numpy(src).cuda()
    adj = torch.randn(s.ns, s.ng, s.nt, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    with Engine(**s.engine_args(), checkpoint_every=every) as e:
        assert e.query_loop("reverse")["kernel"] == "vec"
        e.set_model(s.vp_true, rho)
        seis = torch.zeros(s.ns, s.ng, s.nt, device="cuda")
        outs = [torch.zeros(s.nx, s.nz, device="cuda") for _ in range(3)]

        def step():
            e.forward(src, save_boundary=True, seis=seis)
            e.backward(adj, *outs)
        step()
        torch.cuda.synchronize()
        want = [x.clone() for x in (seis, *outs)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            step()
        for x in (seis, *outs):
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        e.check()
    for a, b in zip((seis, *outs), want):
        torch.testing.assert_close(a, b, rtol=0, atol=0)
