"""Free rods in many steps of one call (drawing warps ahead of the stepping warp) against one
call a step (one thread a rod): part-filled blocks and chunks, every noise source, both centre
precisions; bit for bit."""
import copy

import numpy as np
import pytest

from helpers import assert_same
from softbox_b200 import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,steps", [(1, 65), (7, 33), (9, 32), (33, 31), (257, 40), (4099, 12)])
@pytest.mark.parametrize("mode,fp64", [("wang", True), ("philox", False), ("supplied", True)])
def test_many_steps_equal_single_steps(n, steps, mode, fp64):
    from softbox_b200.engine import FreeRods
    f = scenes.free_rods_box(n=n, seed=n)
    f["body"]["forceSum"][:] = np.random.default_rng(n).normal(scale=1e-14, size=3 * n).astype(np.float32)
    noise = None
    if mode == "supplied":
        noise = torch.randn((steps, 6, n), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    a, b = (FreeRods(copy.deepcopy(f), fp64_coords=fp64) for _ in range(2))
    a.run(5, steps, noise=mode, philox_seed=77, supplied=noise)
    for s in range(steps):
        b.run(5 + s, 1, noise=mode, philox_seed=77, supplied=noise[s:s + 1].contiguous() if noise is not None else None)
    torch.cuda.synchronize()
    keys = ("coord", "uVec", "yVec", "zVec", "end1", "end2", "randForce", "randTorque") + (("coord64",) if fp64 else ())
    for k in keys:
        assert_same(b.pull(k), a.pull(k), k)
    assert a.dev["counts"].tolist() == b.dev["counts"].tolist()


@pytest.mark.parametrize("n,steps", [(40, 33), (2401, 20), (4739, 20), (9475, 16), (14210, 24), (18944, 24)])
@pytest.mark.parametrize("mode", ["wang", "philox", "supplied"])
def test_rods_with_and_without_forces(n, steps, mode):
    # every number of rods a block, and blocks in which some rods have a force or torque and others none
    from softbox_b200.engine import FreeRods
    rng = np.random.default_rng(n)
    f = scenes.free_rods_box(n=n, seed=n)
    for key in ("forceSum", "torqueSum"):
        some = (rng.random(n) < 0.3).astype(np.float32)
        f["body"][key][:] = (rng.normal(scale=1e-14, size=(3, n)) * some).astype(np.float32).reshape(-1)
    assert (f["body"]["forceSum"] == 0).any() and (f["body"]["torqueSum"] != 0).any()
    noise = None
    if mode == "supplied":
        noise = torch.randn((steps, 6, n), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    a, b = (FreeRods(copy.deepcopy(f), fp64_coords=True) for _ in range(2))
    a.run(5, steps, noise=mode, philox_seed=77, supplied=noise)
    for s in range(steps):
        b.run(5 + s, 1, noise=mode, philox_seed=77, supplied=noise[s:s + 1].contiguous() if noise is not None else None)
    torch.cuda.synchronize()
    for k in ("coord", "coord64", "uVec", "yVec", "zVec", "end1", "end2", "randForce", "randTorque"):
        assert_same(b.pull(k), a.pull(k), k)
