"""The batch's list of new voxel cells where its buffers turn over: batches so
large that a warp claims more cells than its buffer holds, and of one point, one
warp and one block; the tree, its grids and voxels equal the oracle's."""
import numpy as np
import pytest

from gpu_helpers import build_gpu, build_oracle, compare_grids, compare_nodes, compare_stats, compare_voxels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,batch", [(1, 1), (33, 32), (700, 257), (2_097_152, 2_097_152), (2_097_152, 1_900_001)])
def test_new_cells_of_any_batch_size(c1_cloud, points, batch):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::len(cloud) // points][:points])
    ctx, _ = build_gpu(cloud, bmin, bmax, batch)
    tree = build_oracle(cloud, bmin, bmax, batch)
    nodes = compare_nodes(ctx, tree)
    compare_stats(ctx, tree)
    compare_voxels(ctx, tree, nodes)
    compare_grids(ctx, tree, nodes)
    ctx.close()
    tree.close()
