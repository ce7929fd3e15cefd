"""The tuner keeps the default of every field that the system's kernels do not read at its size:
the entry also serves larger sizes of the same power of two, where the field counts."""
import pytest

pytestmark = pytest.mark.gpu
ACC = dict(algorithm=1, box_mode=1, accuracy_parameter=1.0, relative_accuracy=0.006, relative_theta_floor=0.2,
           flags=0x170)
TREE = {"sort_keys_per_thread", "sort_lookback", "scan_lookback", "moment_blocks_per_sm"}
DIRECT = {"direct_targets", "direct_blocks_per_sm"}


# the largest systems below each bound (one-block direct sums and trees, small sort tiles,
# small moments launches), and REFERENCE math, which has one direct-sum shape
@pytest.mark.parametrize("prm,n,unused,candidates", [
    (dict(algorithm=0), 12288, DIRECT, 4), (dict(algorithm=0, math_mode=1), 20000, DIRECT, 4),
    (dict(algorithm=1), 8192, TREE, 7), (ACC, 3072, TREE, 9),
    (dict(algorithm=1), 131072, {"sort_keys_per_thread", "moment_blocks_per_sm"}, 7)])
def test_unused_fields_keep_their_defaults(gs, prm, n, unused, candidates):
    default = gs.shape_defaults().as_dict()
    for seed in range(4):
        r = gs.tune_shape(gs.default_params(**prm), n, generator=gs.GEN_UNIFORM_DISK, seed=seed, steps=3)
        assert r.candidates >= candidates and r.best_ms <= r.default_ms
        assert {k: r.best.as_dict()[k] for k in unused} == {k: default[k] for k in unused}
    gs.clear_shape_table()
