"""The broad phase where its lanes can go wrong: body counts off the block and lane-group
sizes, padding slots, lists past MAX_CAND, a grid one cell wide in each direction; bit for bit
against the oracle (order included)."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cap,S,box,dims", [(1, 1, 1.0, (3, 3, 3)), (37, 33, 1.0, (4, 3, 2)), (1003, 1003, 2.0, (9, 8, 1)),
                                            (1500, 1400, 0.6, (2, 2, 2)), (700, 700, 0.3, (1, 1, 1)),
                                            (2051, 2049, 3.0, (1, 13, 12))])
def test_broad_phase_bitwise(orc_dm, cap, S, box, dims):
    from softbox_b200.systems import SpatialGrid
    rng = np.random.default_rng(cap)
    nX, nY, nZ = dims
    C_ = nX * nY * nZ
    cell = 0.25
    g = {"center": rng.uniform(0, box, 3 * cap).astype(np.float32),
         "boundingRadius": rng.uniform(0.02, 0.06, cap).astype(np.float32),
         "gridParams": np.array([0, 0, 0, cell, 1 / cell, 0.07], np.float32),
         "gridDims": np.array([nX, nY, nZ, C_], np.int32), "gridCounts": np.array([0, S, 0, 0], np.int32),
         "bodyCell": np.full(cap, -1, np.int32), "cellCount": np.zeros(C_, np.int32),
         "chunkSum": np.zeros((C_ + 511) // 512 + 1, np.int32), "gridCellOffsets": np.zeros(C_ + 1, np.int32),
         "gridCellContents": np.full(cap, -1, np.int32)}
    d = {k: torch.from_numpy(v).cuda() for k, v in g.items()}
    SpatialGrid.bodyCell(d["center"], d["gridParams"], d["gridDims"], d["gridCounts"], d["bodyCell"])
    SpatialGrid.build(d["bodyCell"], d["gridCounts"], d["gridDims"], d["cellCount"], d["chunkSum"],
                      d["gridCellOffsets"], d["gridCellContents"])
    cand = torch.full((cap * 256,), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((cap,), -7, dtype=torch.int32, device="cuda")
    SpatialGrid.broadPhase(d["center"], d["boundingRadius"], d["bodyCell"], d["gridCellOffsets"],
                           d["gridCellContents"], d["gridDims"], d["gridParams"], d["gridCounts"], cand, cnt)
    h = {k: d[k].cpu().numpy() for k in ("bodyCell", "gridCellOffsets", "gridCellContents")}
    ocand, ocnt = np.full(cap * 256, -1, np.int32), np.zeros(cap, np.int32)
    orc_dm.broad_phase(cap, g["center"], g["boundingRadius"], h["bodyCell"], h["gridCellOffsets"],
                       h["gridCellContents"], g["gridDims"], g["gridParams"], S, ocand, ocnt)
    assert_same(ocnt, cnt.cpu().numpy(), "candCount")
    assert_same(ocand, cand.cpu().numpy(), "candPartner")
    if dims == (1, 1, 1):
        assert ocnt.max() > 256
