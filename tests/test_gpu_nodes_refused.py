"""The node radiosity's neighbour lists built and exported while the scratch is refused on the host (vt_refuse): the same lists, the
same solution."""
import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu

NONE = 2 ** 64 - 1
SCRATCH = 2


@pytest.mark.parametrize("level,nbr_k", [(2, 16), (4, 5)])
def test_neighbour_lists_without_scratch(level, nbr_k):
    sc = dome.make_dome_scene(seed=1, width=16, height=16, level=level)
    runs = []
    for at_build, at_export in ((NONE, NONE), (0, NONE), (NONE, 0), (0, 0)):
        r = TwinRenderer.create(sc, nodes=False)
        r.lib.vt_refuse(r._ctx, SCRATCH, at_build)
        r.build_nodes(nbrK=nbr_k, gatherK=16)
        r.lib.vt_refuse(r._ctx, SCRATCH, NONE)
        r.set_pose_array(A.identity_poses(1))
        r.converge(5)
        if at_export != NONE:   # what is held already is given back when more is refused
            r.lib.vt_refuse(r._ctx, SCRATCH, 0)
            with pytest.raises(Exception, match="scratch"):
                r.solve_radiosity(np.zeros((3000, 3000), np.float32), np.zeros(3000, np.float32), np.ones((3000, 64), np.float32))
        export = r.nodes_export()
        runs.append((export["nbr"], export["active"], r.get_node_state()[0]))
        r.destroy()
    nbr = runs[0][0]
    assert (nbr[..., 1] != 0).any() and nbr.shape[1] == nbr_k
    for run in runs[1:]:
        for a, b in zip(run, runs[0]):
            assert np.array_equal(a, b)
