"""The drivers behind the resident BFS and CC (knob resident 0), which run
where those do not fit in memory or are switched off: the tests of the
graph-driven BFS (record modes, split pull, bitmap staging, kernel residency,
loop shapes, hand-over, learned choice), of the device-driven CC with and
without hooking and of the batch, which set those drivers' own knobs only,
collected here once more with `resident` 0."""
import numpy as np
import pytest

from graptor_b200 import gg
from oracle import oracle as O
from test_gpu_async import *  # noqa: F401,F403
from test_gpu_batch import (  # noqa: F401
    test_batch_bfs_cc_one_graph_launch, test_bfs_level_multi_single_root_matches_bfs_level, test_union_bfs_and_cc_per_part)
from test_gpu_parity import (  # noqa: F401
    test_graph_bfs_kernel_residency_exact, test_pull_first_record_modes_exact, test_pull_stage_and_fresh_exact,
    test_split_pull_exact)
from test_gpu_persistent import (  # noqa: F401
    fusion_knobs, test_cc_hooking_exact, test_cc_hooking_repeated_long_chains, test_graph_bfs_handoff_to_device_driven,
    test_graph_driven_bfs_equals_host_loop, test_graph_loop_shapes_exact)
from test_gpu_selector import (  # noqa: F401
    test_graph_keeps_its_copy_of_the_weights, test_learned_choice_never_changes_results)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def not_resident():
    old = gg.tuning_get("resident")
    gg.tuning_set("resident", 0)
    yield
    gg.tuning_set("resident", old)


@pytest.mark.parametrize("threshold", [gg.THRESH_DEFAULT, gg.THRESH_LEARNED])
def test_the_graph_driven_run_is_the_one_that_runs(ctx, threshold):
    """The kernels launched tell the drivers apart: two by the resident run, the
    graph's chain of kernels per step, one and more per step from the host."""
    og = O.rmat(14, 16 << 14, seed=23)
    g = ctx.upload(og.off, og.adj)
    opts, want = gg.default_opts(threshold), O.bfs_level(og, 0)
    kernels = []
    try:
        for resident, graph in ((1, 1), (0, 1), (0, 0)):
            gg.tuning_set("resident", resident)
            gg.tuning_set("graph", graph)
            st = gg.RunStats()
            assert np.array_equal(g.bfs_level(0, opts=opts, stats=st), want)
            kernels.append(st.kernels)
    finally:
        gg.tuning_set("graph", 1)
    assert kernels[0] == 2 and len(set(kernels)) == 3, kernels
    g.close()
