"""The graph path's wide kernels (sbx_wide.cu) where they can go wrong: rows past their fixed
slots, chain neighbours that do not point back, and scenes of another layout, which keep the
per-system sequence. The reference of each is the per-system path of the same scene
(bit-identical to the oracle: tests/test_gpu_parity.py)."""
import copy

import numpy as np
import pytest

from helpers import assert_same, compare_scenes, oracle_dense_run, small_dense

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from softbox_b200 import device as D  # noqa: E402


@pytest.fixture(scope="module")
def warm(orc_dm):
    sc = small_dense(0.05)
    oracle_dense_run(orc_dm, sc, 0, 300)
    return sc


def _run(sc, mode, steps=40, caps=None):
    from softbox_b200.engine import DenseNetwork
    net = DenseNetwork(copy.deepcopy(sc))
    if caps is not None:
        net.test_caps(**caps)
    net.run(300, steps, mode=mode)
    net.status()
    stats, n = net.fused_stats(), net.kernels_per_step
    out = D.to_host(net.dev)
    net.close()
    return out, stats, n


@pytest.mark.parametrize("caps", [dict(cell_slots=0), dict(row_slots=0), dict(cell_slots=1, row_slots=1)],
                         ids=["cells", "rows", "both"])
def test_rows_past_their_slots(warm, caps):
    ref, _, _ = _run(warm, "unfused")
    got, stats, _ = _run(warm, "graph", caps=caps)
    assert stats["cell_list"] > 0 if "cell_slots" in caps else stats["link_list"] > 0 and stats["motor_list"] > 0
    assert len(compare_scenes(ref, got)) > 80


@pytest.mark.parametrize("heads,links", [(2, 4), (4, 5), (5, 8), (15, 9), (16, 16), (17, 17), (40, 33)])
def test_long_rows(warm, heads, links):
    # one rod with many bound heads and both ends of many links, around the sizes of a row's parts
    sc = copy.deepcopy(warm)
    rng = np.random.default_rng(heads)
    m = rng.permutation(len(sc["mot"]["boundSeg"]))[:heads]
    sc["mot"]["boundSeg"][m] = 7
    sc["mot"]["bindArc"][m] = 0.0
    k = rng.permutation(len(sc["xl"]["linkFilA"]))
    sc["xl"]["linkFilA"][k[:links]] = 7
    sc["xl"]["linkFilB"][k[links:2 * links]] = 7
    ref, _, _ = _run(sc, "unfused", steps=2)
    got, stats, _ = _run(sc, "graph", steps=2)
    assert np.asarray(ref["xl"]["segCountA"])[7] >= links and np.asarray(ref["xl"]["segCountB"])[7] >= links
    assert (stats["link_list"] > 0) == (links > 16) and (stats["motor_list"] > 0) == (heads > 16)
    assert len(compare_scenes(ref, got)) > 80


def test_neighbours_that_do_not_point_back(warm):
    sc = copy.deepcopy(warm)
    f = sc["fil"]
    for k in (3, 4, 57, 200):                      # rod k + 1 forgets rod k, which keeps its joint
        assert f["end2NbrSlot"][k] == k + 1
        f["end1NbrSlot"][k + 1] = -1
    for k in (21, 121):                            # and the other way round
        assert f["end2NbrSlot"][k] == k + 1
        f["end2NbrSlot"][k] = -1
    ref, _, _ = _run(sc, "unfused")
    got, _, _ = _run(sc, "graph")
    assert len(compare_scenes(ref, got)) > 80


def test_other_layouts_keep_the_per_system_sequence(warm):
    sc = copy.deepcopy(warm)
    a, b = sc["dim"]["motorA"].copy(), sc["dim"]["motorB"].copy()
    sc["dim"]["motorA"][0], sc["dim"]["motorB"][0] = b[0], a[0]
    ref, _, n_wide = _run(warm, "graph", steps=1)
    ref, _, _ = _run(sc, "unfused")
    got, _, n = _run(sc, "graph")
    assert n > 40 > n_wide
    assert len(compare_scenes(ref, got)) > 80


@pytest.mark.parametrize("rods", [75_770, 75_780])
def test_rods_kernel_on_both_sides_of_its_rule(rods):
    # above 148 x 4 x 128 rods the kernel with more blocks an SM
    from softbox_b200 import scenes
    from softbox_b200.engine import DenseNetwork
    sc = scenes.dense_contractile(scenes.dense_scaled(rods))
    n = len(sc["fil"]["end1NbrSlot"])
    out = []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(sc), fp64_coords=True)
        net.run(0, 6, mode=mode)
        assert net.status() == 0
        out.append(D.to_host(net.dev))
        net.close()
    assert len(compare_scenes(*out)) > 80 and n == rods


def test_graph_and_fused_steps_alternate(warm):
    from softbox_b200.engine import DenseNetwork
    ref, _, _ = _run(warm, "unfused", steps=12)
    net = DenseNetwork(copy.deepcopy(warm))
    t = 300
    for mode, k in (("graph", 1), ("fused", 3), ("graph", 2), ("unfused", 1), ("graph", 1), ("fused", 1), ("graph", 3)):
        net.run(t, k, mode=mode)
        t += k
    assert t == 312 and net.status() == 0
    assert len(compare_scenes(ref, D.to_host(net.dev))) > 80
    assert_same(np.asarray(ref["mot"]["boundSeg"]), net.pull("mot", "boundSeg"), "boundSeg")
    net.close()


@pytest.mark.parametrize("runs", [((300, 3), (303, 4), (307, 5), (312, 1)), ((300, 9), (400, 2), (402, 8), (0, 1))],
                         ids=["on", "jumps"])
def test_runs_of_any_length(warm, runs):
    # runs around the steps of a graph, each going on from the last one or from another step index
    from softbox_b200.engine import DenseNetwork
    out = []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(warm))
        for t, n in runs:
            net.run(t, n, mode=mode)
        if mode == "graph":                            # the fused kernel moves the step index as well
            net.run(20, 2, mode="fused")
            net.run(22, 5, mode="graph")
        else:
            net.run(20, 7, mode=mode)
        assert net.status() == 0
        out.append(D.to_host(net.dev))
        net.close()
    assert len(compare_scenes(*out)) > 80


@pytest.mark.parametrize("refresh", [False, True])
def test_step_index_beside_a_captured_run(warm, refresh):
    # a captured run (the fused kernel) moves the step index at its replay, not at its capture;
    # after a refresh the per-system kernels are captured, as the topology cannot be read there
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import LIB
    ref = DenseNetwork(copy.deepcopy(warm))
    for t, n in ((300, 3), (303, 5), (303, 2), (308, 4), (312, 1)):
        ref.run(t, n, mode="unfused")
    net = DenseNetwork(copy.deepcopy(warm))
    net.run(300, 3, mode="graph")
    if refresh:
        assert LIB.sbx_dense_plan_refresh(net.plan) == 0
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(LIB.sbx_ctx_stream(net.ctx.h))):
        net.run(303, 2)
    net.run(303, 5, mode="graph")
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    net.run(308, 4, mode="graph")
    net.run(312, 1, mode="graph")
    assert net.status() == 0 and ref.status() == 0
    assert len(compare_scenes(D.to_host(ref.dev), D.to_host(net.dev))) > 80
    del g
    ref.close()
    net.close()


def test_auto_takes_the_graph_and_fused_runs_after_a_refresh(warm):
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import LIB
    ref, _, _ = _run(warm, "unfused", steps=6)
    net = DenseNetwork(copy.deepcopy(warm))
    k = net.kernels_per_step
    n0 = net.ctx.launches()
    net.run(300, 2)
    assert net.ctx.launches() - n0 >= 2 * k                # (one launch for both steps on the fused path)
    assert LIB.sbx_dense_plan_refresh(net.plan) == 0
    net.run(302, 2, mode="fused")
    net.run(304, 2)
    assert net.fused_available and net.status() == 0
    assert len(compare_scenes(ref, D.to_host(net.dev))) > 80
    net.close()


def _with_bodies(sc, extra, counted):
    # `extra` bodies of the caller's after the heads in the body view, owned by no store
    sc = copy.deepcopy(sc)
    g = sc["grid"]
    cap, rng = g["cap"], np.random.default_rng(extra)
    head = np.asarray(sc["mot"]["body"]["coord"]).reshape(3, -1)[:, :extra]
    center = np.zeros((3, cap + extra), np.float32)
    center[:, cap:] = head + rng.normal(scale=0.02, size=head.shape).astype(np.float32)
    g["center"] = center.reshape(-1)
    for k, v in (("boundingRadius", 0.05), ("ownerStore", -1), ("ownerSlot", -1), ("bodyCell", -1),
                 ("gridCellContents", -1)):
        g[k] = np.concatenate([g[k], np.full(extra, v, g[k].dtype)])
    g["cap"] = cap + extra
    g["gridCounts"][1] = cap + (extra if counted else 0)
    return sc


@pytest.mark.parametrize("counted", [True, False], ids=["before", "after"])
def test_bodies_past_the_published_ones(warm, counted):
    # counted into the view before the plan is made, or on the device afterwards
    from softbox_b200.engine import DenseNetwork
    sc, out = _with_bodies(warm, 40, counted), []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(sc))
        if not counted:
            net.dev["grid"]["gridCounts"][1] = sc["grid"]["cap"]
        net.run(300, 9, mode=mode)
        assert net.status() == 0
        net.ctx.sync()
        out.append(D.to_host(net.dev))
        net.close()
    assert (np.asarray(out[0]["grid"]["bodyCell"])[-40:] >= 0).all()
    assert len(compare_scenes(*out)) > 80


def test_a_moved_body_view_is_reported(warm):
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import SbxError
    net = DenseNetwork(copy.deepcopy(warm))
    net.dev["mot"]["publishParams"][0] = 0
    net.run(300, 1, mode="graph")
    with pytest.raises(SbxError, match="publishParams"):
        net.ctx.sync()
    net.close()


@pytest.mark.parametrize("change", ["sides", "partners", "backbones", "tethers"])
def test_dimer_tables_changed_on_the_device(warm, change):
    # the graph path takes the dimer tables as they are at each step: changed after the plan was
    # made, and changed back
    from softbox_b200.engine import DenseNetwork
    out = []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(warm))
        dim, mini = net.dev["dim"], net.dev["mini"]
        keep = [x.clone() for x in (dim["motorA"], dim["motorB"], mini["headBackboneSlot"], mini["motorA"])]
        n, far = dim["motorA"].numel(), dim["motorA"].numel() - 1
        net.run(300, 5, mode=mode)
        if change == "sides":
            dim["motorA"][3], dim["motorB"][3] = keep[1][3], keep[0][3]
        elif change == "partners":
            dim["motorB"][1], dim["motorB"][far] = keep[1][far], keep[1][1]
        elif change == "backbones":
            rows = torch.randint(0, n, (n,), generator=torch.Generator().manual_seed(4)).cuda()
            mini["headBackboneSlot"].copy_(keep[2][rows])           # of unequal lengths, some empty
        else:
            mini["motorA"][0], mini["motorA"][far] = keep[3][far], keep[3][0]
        net.run(305, 6, mode=mode)
        mid = D.to_host(net.dev)
        for x, k in zip((dim["motorA"], dim["motorB"], mini["headBackboneSlot"], mini["motorA"]), keep):
            x.copy_(k)
        net.run(311, 5, mode=mode)
        assert net.status() == 0
        out.append((mid, D.to_host(net.dev)))
        net.close()
    for ref, got in zip(*out):
        assert len(compare_scenes(ref, got)) > 80


@pytest.mark.parametrize("mode", ["fused", "auto"])
def test_captured_fused_run_after_a_refresh(warm, mode):
    # the topology of a refresh is read behind the change while the context's stream is captured
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import LIB
    sc = copy.deepcopy(warm)
    ref, _, _ = _run(sc, "unfused", steps=6)
    net = DenseNetwork(sc)
    net.run(300, 2)
    assert LIB.sbx_dense_plan_refresh(net.plan) == 0
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    n0 = net.ctx.launches()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(LIB.sbx_ctx_stream(net.ctx.h))):
        assert net.fused_available
        net.run(302, 2, mode=mode)
    assert net.ctx.launches() - n0 == 1                # one launch for both steps
    g.replay()
    torch.cuda.synchronize()
    net.run(304, 2)
    assert net.status() == 0
    assert len(compare_scenes(ref, D.to_host(net.dev))) > 80
    del g
    net.close()


def test_a_refresh_inside_a_capture_keeps_the_capture(warm):
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import LIB, SbxError
    ref, _, _ = _run(warm, "unfused", steps=5)
    net = DenseNetwork(copy.deepcopy(warm))
    net.run(300, 2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(LIB.sbx_ctx_stream(net.ctx.h))):
        assert LIB.sbx_dense_plan_refresh(net.plan) == 0
        assert net.fused_available
        with pytest.raises(SbxError, match="capture"):
            net.run(302, 2, mode="fused")
        net.run(302, 2)
    g.replay()
    torch.cuda.synchronize()
    net.run(304, 1, mode="fused")
    assert net.status() == 0
    assert len(compare_scenes(ref, D.to_host(net.dev))) > 80
    del g
    net.close()


def test_fused_run_between_a_first_capture_and_its_replay(warm):
    # the plan's first fused run is a captured one: another may come before the replay
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import LIB
    ref, _, _ = _run(warm, "unfused", steps=5)
    net = DenseNetwork(copy.deepcopy(warm))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(LIB.sbx_ctx_stream(net.ctx.h))):
        net.run(302, 2)
    net.run(300, 2, mode="fused")
    g.replay()
    torch.cuda.synchronize()
    net.run(304, 1, mode="fused")
    assert net.status() == 0
    assert len(compare_scenes(ref, D.to_host(net.dev))) > 80
    del g
    net.close()


def test_noise_in_chunks(warm):
    # noise set anew between runs, on and off, without new graphs
    from softbox_b200.engine import DenseNetwork
    out = []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(warm))
        d, t = net.dev, 300
        sizes = (d["fil"]["body"]["n"], d["mot"]["body"]["n"], d["mini"]["backbone"]["n"])
        rng = torch.Generator("cuda").manual_seed(9)
        for steps in (1, 6, 0, 5, 4):
            if steps:
                net.set_noise(*(torch.randn(steps, 6, n, device="cuda", generator=rng) for n in sizes), t)
            else:
                net.set_noise(None, None, None, 0)
            net.run(t, steps or 3, mode=mode)
            t += steps or 3
        assert net.status() == 0
        out.append(D.to_host(net.dev))
        net.close()
    assert len(compare_scenes(*out)) > 80


@pytest.mark.parametrize("runs,reported", [(("graph",), False), (("auto",), True), (("graph", "auto"), True),
                                           (("auto", "graph"), True), (("graph", "unfused"), False)])
def test_a_reach_overflow_is_its_runs(runs, reported):
    # reported for the runs of fused size, whatever ran before or after them; not for the graph's
    import physics_gates as G
    from softbox_b200.engine import DenseNetwork
    from softbox_b200.runtime import SbxError
    net = DenseNetwork(G.crowded_dense())
    assert net.fused_available
    t = 0
    for first in (("auto",), ()):                      # once after an auto run whose report was taken
        for mode in first:
            net.run(t, 1, mode=mode)
            t += 1
            with pytest.raises(SbxError):
                net.status()
            assert net.status() == 0
        for mode in runs:
            net.run(t, 1, mode=mode)
            t += 1
        if reported:
            with pytest.raises(SbxError) as e:
                net.status()
            assert e.value.code == -3
        assert net.status() == 0
    net.close()


def test_more_rods_than_graphs_of_several_steps_take():
    # above 2^17 rods a graph holds one step: the largest size's rule, on more than one scan tile a row
    from softbox_b200 import scenes
    from softbox_b200.engine import DenseNetwork
    sc, out = scenes.dense_contractile(scenes.dense_scaled(131_080)), []
    for mode in ("unfused", "graph"):
        net = DenseNetwork(copy.deepcopy(sc), fp64_coords=True)
        net.run(0, 5, mode=mode)
        net.run(5, 1, mode=mode)
        assert net.status() == 0
        out.append(D.to_host(net.dev))
        net.close()
    assert len(sc["fil"]["end1NbrSlot"]) > 1 << 17 and len(compare_scenes(*out)) > 80
