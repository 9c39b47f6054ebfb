"""Launch shapes of the prediction kernels at the sizes where they change: every output kind against
the CPU oracle."""
import pytest

from tests.helpers import random_forest_desc, random_rows
from tests.test_gpu_parity import _all_kinds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("storage", ["dense", "sparse"])
@pytest.mark.parametrize("kw", [dict(n_trees=3, postproc="sigmoid"),
                                dict(n_trees=67, n_outputs=3, postproc="softmax"),
                                dict(n_trees=130, n_outputs=5, vector=True, average=True),
                                dict(n_trees=40, categorical=True, n_features=37)])
def test_small_batches_split_over_clusters(kw, storage, precision):
    """Row counts around the edges of a tile and of every cluster size, forests with fewer trees
    than CTAs in a cluster and with a tree count no cluster size divides."""
    desc = random_forest_desc(90, max_depth=6, **kw)
    for n in (1, 33, 128, 481, 1057, 4737):
        X = random_rows(n, n, desc.n_features, "float64", nan_frac=0.03,
                        categories=22 if kw.get("categorical") else None)
        _all_kinds(desc, X, precision, "depth_first", storage)


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n_trees", [4, 7, 29, 30])
def test_one_output_per_tree_at_every_alignment(n_trees, precision):
    """Leaf ids and per-tree outputs leave as 16-byte stores, four lanes at a time or one by one,
    whatever the tree count and wherever the batch ends inside a group of four rows."""
    for storage, depth in (("dense", 4), ("dense", 7), ("sparse", 9)):
        desc = random_forest_desc(92, n_trees=n_trees, n_features=9, max_depth=depth, p_leaf=0.05)
        for n in (11_001, 11_002, 11_003):
            _all_kinds(desc, random_rows(n, n, 9, "float64", nan_frac=0.02), precision,
                       "depth_first", storage)


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n_features", [1, 2, 7, 28, 33, 61, 100])
def test_rank_prepass_over_ragged_feature_groups(n_features, precision):
    """Feature counts that make one wide group, narrow tails of several groups, and groups that are
    ranked several tiles at a time; row tiles of every size, a partial last tile, NaN in some tiles
    only, categories, thresholds that rows hit exactly, infinities."""
    import numpy as np

    desc = random_forest_desc(91, n_trees=61, n_features=n_features, max_depth=5, mixed_ops=True,
                              categorical=n_features == 33, postproc="sigmoid")
    thr = desc.threshold[desc.node_kind == 1]
    for n, chunk in ((70, 1), (1000, 2), (1000, 4), (5001, 8), (12_007, 4), (12_007, 8)):
        X = random_rows(n, n, n_features, np.float64, nan_frac=0.0,
                        categories=22 if n_features == 33 else None)
        X[: n // 3, 0] = np.resize(thr, n // 3)
        X[n // 2, -1] = np.nan
        X[-1, 0] = np.nan
        X[1, 0], X[2, 0] = np.inf, -np.inf
        _all_kinds(desc, X, precision, "depth_first", "dense", chunk_size=chunk)


@pytest.mark.parametrize("n_features,max_depth", [(32, 5), (96, 8)])
def test_rank_prepass_with_sixteen_ranks_per_thread(n_features, max_depth):
    """Batches large enough for it (256 rows and 32 features per SM, groups of 32 only): row tiles of every
    size, which are ranked 1 to 16 at a time, a partial last tile, few and many halvings, NaN in some tiles
    only, thresholds that rows hit exactly, infinities."""
    import numpy as np

    desc = random_forest_desc(97, n_trees=61, n_features=n_features, max_depth=max_depth, mixed_ops=True,
                              postproc="sigmoid")
    thr = desc.threshold[desc.node_kind == 1]
    n = 38_145
    X = random_rows(n, n, n_features, np.float64, nan_frac=0.0)
    X[: n // 3, 0] = np.resize(thr, n // 3)
    X[n // 2, -1] = np.nan
    X[-1, 0] = np.nan
    X[1, 0], X[2, 0] = np.inf, -np.inf
    from cuml_b200.fil import _lib

    for chunk in (1, 2, 4, 8, None):
        _all_kinds(desc, X, "single", "depth_first", "dense", chunk_size=chunk)
        assert "ranks=16" in _lib.last_variant(), _lib.last_variant()


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n_trees,n_features", [(3, 5), (61, 9), (190, 40)])
def test_deep_trees_at_batch_sizes_where_the_launch_shape_changes(n_trees, n_features, precision):
    """Blocks of four nodes below the heaps: trees deep enough for several blocks on a walk, values
    that hit thresholds (open tests), unaligned rows, and row counts around the edges of tiles,
    clusters and rounds of CTAs."""
    import numpy as np

    desc = random_forest_desc(93, n_trees=n_trees, n_features=n_features, max_depth=15, p_leaf=0.2,
                              mixed_ops=True)
    thr = desc.threshold[desc.node_kind == 1]
    for n in (1, 129, 1025, 4750, 9473, 19_001):
        X = random_rows(n, n, n_features, np.float64, nan_frac=0.02)
        X[::3, 0] = np.resize(thr, len(X[::3]))
        _all_kinds(desc, X, precision, "depth_first", "sparse")


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n_features", [1, 3, 4, 6, 50, 132])
def test_row_tiles_of_every_alignment(n_features, precision):
    """Rows that start on 16-byte boundaries and rows that do not, fewer columns than one load and
    more than the warps of a CTA bring at once, full and partial tiles, and one missing value in the
    batch, in its last row and column: the kernels that stage rows themselves must see it."""
    desc = random_forest_desc(93, n_trees=33, n_features=n_features, max_depth=7)
    for storage, kw in (("dense", dict(quantize_rows=False)), ("sparse", {}),
                        ("sparse", dict(compact_nodes=False))):
        for n in (1, 31, 33, 600, 30_001):
            X = random_rows(n, n, n_features, "float64", nan_frac=0.0)
            X[-1, -1] = float("nan")
            _all_kinds(desc, X, precision, "depth_first", storage, **kw)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_deep_forest_beyond_the_caches_repeats_itself(dtype):
    """Leaf ids of a forest whose nodes come from HBM, predicted again and again, against the kernel
    that stages no trees: the loads of a heap are held up behind node fetches for longer than it takes
    to refill the heap's stage, so a stage that is given back before they have arrived shows here (one
    call in sixty of this fp64 forest)."""
    import torch

    from cuml_b200.fil import ForestInference
    from perf import cases

    case = dict(cases.BASE, forest="regressor", trees=200, depth=20, leaves=60_000, features=64,
                dtype=dtype, rows=200_000, call="apply")
    g = torch.Generator(device="cuda:0")
    g.manual_seed(5)
    desc = cases._bagged_forest(case, g, "cuda:0")
    X = cases._rows(case, g, "cuda:0")
    kw = dict(precision="double" if dtype == "float64" else "single", storage="sparse")
    want = ForestInference.load_from_treelite_model(desc, compact_nodes=False, **kw).apply(X)
    fi = ForestInference.load_from_treelite_model(desc, **kw)
    assert fi.describe()["compact_image"] == 1
    differing = [int((fi.apply(X) != want).sum()) for _ in range(400)]
    assert max(differing) == 0, f"{sum(d > 0 for d in differing)} of 400 calls, up to {max(differing)} ids"


@pytest.mark.parametrize("kw", [dict(storage="dense", quantize_rows=False), dict(storage="dense"),
                                dict(storage="sparse"), dict(storage="sparse", compact_nodes=False)])
def test_any_chunk_size_of_the_c_interface(kw):
    """The C interface takes every chunk_size (the Python layer only powers of two): row tiles are
    rounded down to a power of two, and results do not depend on them."""
    import numpy as np
    import torch

    from cuml_b200.fil import ForestInference, _lib
    from cuml_b200.fil._desc import INFER_LEAF_ID
    from oracle import oracle

    desc = random_forest_desc(94, n_trees=40, n_features=18, max_depth=7)
    X = random_rows(5, 20_001, 18, np.float32, nan_frac=0.02)
    want = oracle.predict(desc, X, INFER_LEAF_ID, "single")
    Xd = torch.as_tensor(X, device="cuda:0")
    fi = ForestInference.load_from_treelite_model(desc, **kw)
    for n in (97, 20_001):
        for chunk in (3, 5, 6, 7, 9, 2**26, 2**31 - 1):
            out = torch.full((n, 40), -1, dtype=torch.int32, device="cuda:0")
            _lib.check(_lib.load().b2fil_predict(
                fi.forest.handle, INFER_LEAF_ID, Xd.data_ptr(), n, 18, out.data_ptr(), chunk, 0.5,
                torch.cuda.current_stream().cuda_stream))
            assert np.array_equal(out.cpu().numpy().astype(np.uint32), want[:n]), (n, chunk)


@pytest.mark.parametrize("precision", ["single", "double"])
def test_pinned_inputs_of_every_length_are_fetched_to_their_end(precision):
    """Pinned rows that a kernel fetches from the caller's array itself: lengths that are no multiple of
    the 16 bytes of a load, the last values counting."""
    import torch

    for n_features in (1, 3, 5, 7, 8):
        desc = random_forest_desc(95, n_trees=12, n_features=n_features, max_depth=6)
        for n in (16_385 // (4 * n_features) + 1, 1001 * 8 // n_features + 13, 30_003):
            X = random_rows(n, n, n_features, "float64", nan_frac=0.02)
            dt = torch.float32 if precision == "single" else torch.float64
            pinned = torch.empty(X.shape, dtype=dt, pin_memory=True)
            pinned.copy_(torch.from_numpy(X))
            _all_kinds(desc, pinned.numpy(), precision, "depth_first", "auto", host=True)


def test_launch_shape_does_not_depend_on_what_ran_before():
    """A plain and a categorical forest of the same size, predicted in both orders by fresh threads
    (each has its own table of recent launch shapes): the same kernels and shapes every time."""
    import threading

    import torch

    from cuml_b200.fil import ForestInference, _lib, synthetic_complete_forest

    plain, cat = (ForestInference.load_from_treelite_model(
        synthetic_complete_forest(300, 6, 40, 7, n_categorical=c, n_categories=20)) for c in (0, 8))
    seen = {}
    for n in (64, 700, 3000, 6000, 12_000):
        X = torch.zeros((n, 40), device="cuda:0")
        for order in ((plain, cat), (cat, plain)):
            def run():
                for fi in order:
                    fi.predict_proba(X)
                    seen.setdefault((n, fi is cat), set()).add(_lib.last_variant().replace(",CAT", ""))

            t = threading.Thread(target=run)
            t.start()
            t.join()
    assert all(len(v) == 1 for v in seen.values()), seen
    # (the sizes are such that the two have shapes of their own)
    assert any(seen[n, False] != seen[n, True] for n in (64, 700, 3000, 6000, 12_000)), seen


def test_tensor_without_memory_is_an_error():
    """A fake CUDA tensor has shapes and no data: every call with it raises, the first one (ctypes)
    and later ones (compiled call path), and the forest goes on predicting."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cuml_b200.fil import ForestInference, synthetic_complete_forest

    fi = ForestInference.load_from_treelite_model(synthetic_complete_forest(20, 4, 6, 1))
    X = torch.zeros((7, 6), device="cuda:0")
    with FakeTensorMode():
        fake = torch.empty((7, 6), device="cuda:0")
    for _ in range(3):
        with pytest.raises(RuntimeError):
            fi.apply(fake)
        assert fi.apply(X).shape == (7, 20)


def test_missing_values_come_and_go_between_overlapped_calls():
    """Batches with and without missing values in turn, never waited for: kernels of neighbouring calls
    share SMs (small forests leave room) and scratch addresses, and every call has to see its own flags."""
    import torch

    from cuml_b200.fil import ForestInference

    desc = random_forest_desc(96, n_trees=150, n_features=10, max_depth=4, postproc="sigmoid")
    fi = ForestInference.load_from_treelite_model(desc, storage="dense")
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    X = [torch.randn((60_000, 10), generator=g, device="cuda:0") for _ in range(2)]
    X[1][torch.rand(X[1].shape, generator=g, device="cuda:0") < 0.1] = float("nan")
    want = [fi.apply(x) for x in X]
    proba = [fi.predict_proba(x) for x in X]
    torch.cuda.synchronize()
    got = [(fi.apply(X[i % 2]), fi.predict_proba(X[i % 2])) for i in range(40)]
    for i, (ids, p) in enumerate(got):
        assert torch.equal(ids, want[i % 2]) and torch.equal(p, proba[i % 2]), i


def test_the_variants_that_these_tests_are_about_are_launched():
    """Trees split over a cluster, row tiles with doubled columns, two row-tile buffers: at the shapes that
    the tests above take them to run at."""
    import numpy as np
    import torch

    from cuml_b200.fil import ForestInference, _lib, synthetic_complete_forest
    from cuml_b200.fil._desc import INFER_DEFAULT, INFER_LEAF_ID
    from oracle import oracle

    small = random_forest_desc(90, max_depth=6, n_trees=130, n_features=9)
    for storage, kernel in (("dense", "dense_kernel"), ("sparse", "sparse_compact_kernel")):
        fi = ForestInference.load_from_treelite_model(small, storage=storage)
        fi._run(torch.zeros((481, 9), device="cuda:0"), INFER_DEFAULT, None)
        assert kernel in _lib.last_variant() and "forest_splits=" in _lib.last_variant()
    desc = synthetic_complete_forest(300, 6, 60, 11)
    assert desc.default_left.any()
    fi = ForestInference.load_from_treelite_model(desc)
    X = random_rows(9, 60_001, 60, np.float32, nan_frac=0.03)
    x = torch.as_tensor(X, device="cuda:0")
    p = fi.predict_proba(x).cpu().numpy()
    assert "nan_columns" in _lib.last_variant() and "tiles=2" in _lib.last_variant()
    np.testing.assert_allclose(p[:, 1:], oracle.predict(desc, X, INFER_DEFAULT, "single"), rtol=1e-5,
                               atol=1e-6)
    assert np.array_equal(fi.apply(x).cpu().numpy().astype(np.uint32),
                          oracle.predict(desc, X, INFER_LEAF_ID, "single"))
    assert "nan_columns" not in _lib.last_variant()


@pytest.mark.parametrize("n_trees,max_depth,kw", [(250, 4, {}), (251, 5, {}), (173, 6, dict(vector=True, n_outputs=3)),
                                                  (109, 10, {}), (321, 4, {})])
def test_outputs_of_eight_trees_leave_together(n_trees, max_depth, kw):
    """One output per row and tree from a tile per SM and 1000 visits per row on: tree counts with and without
    rows on 16-byte boundaries, a partial last group of eight, a batch that ends inside four rows, missing
    values; top nodes in the small parameter block and (321 trees) the large one."""
    import numpy as np
    import torch

    from cuml_b200.fil import ForestInference, _lib
    from cuml_b200.fil._desc import INFER_LEAF_ID, INFER_PER_TREE
    from oracle import oracle

    desc = random_forest_desc(98, n_trees=n_trees, n_features=9, max_depth=max_depth, p_leaf=0.05, **kw)
    X = random_rows(3, 37_891, 9, np.float32, nan_frac=0.01)
    X[5000:30_000] = np.nan_to_num(X[5000:30_000])  # most tiles hold none
    fi = ForestInference.load_from_treelite_model(desc, storage="dense")
    x = torch.as_tensor(X, device="cuda:0")
    ids = fi.apply(x).cpu().numpy()
    # (eight trees of depth 10 do not fit three times beside a tile of 256 rows; four do)
    assert f"NT={4 if max_depth == 10 else 8},DEPTH={max_depth}" in _lib.last_variant(), _lib.last_variant()
    assert np.array_equal(ids.astype(np.uint32), oracle.predict(desc, X, INFER_LEAF_ID, "single"))
    per = fi.predict_per_tree(x).cpu().numpy()
    assert np.array_equal(per.reshape(len(X), -1),
                          oracle.predict(desc, X, INFER_PER_TREE, "single").reshape(len(X), -1))


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("max_depth,n_features,kw", [(4, 500, {}), (7, 480, {}), (8, 400, dict(vector=True, n_outputs=2)),
                                                     (9, 440, {}), (10, 300, dict(vector=True, n_outputs=3)),
                                                     (10, 512, {})])
def test_few_trees_in_flight(max_depth, n_features, kw, precision):
    """Row tiles that leave room for few trees, as they are chosen: one to six trees in flight, payloads in global
    memory, every output kind, partial groups of trees, missing values."""
    import numpy as np

    desc = random_forest_desc(99, n_trees=19, n_features=n_features, max_depth=max_depth, p_leaf=0.02, **kw)
    X = random_rows(4, 2_500, n_features, np.float64, nan_frac=0.002)
    for chunk in (4, 8):
        _all_kinds(desc, X, precision, "depth_first", "dense", chunk_size=chunk)


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("max_depth,n_features,n_trees", [(3, 11, 70), (8, 11, 61), (10, 300, 21)])
def test_missing_values_that_all_go_right(max_depth, n_features, n_trees, precision):
    """Forests that send every missing value right, with tests that nothing and that everything passes: in the
    images for ranks the former send missing values to the left of exchanged children."""
    import numpy as np

    desc = random_forest_desc(100, n_trees=n_trees, n_features=n_features, max_depth=max_depth, p_leaf=0.02)
    inner = np.flatnonzero(desc.node_kind == 1)
    desc.threshold[inner[::5]] = np.nan
    desc.threshold[inner[2::5]] = np.inf
    desc.default_left[:] = 0
    X = random_rows(6, 21_003, n_features, np.float64, nan_frac=0.02)
    _all_kinds(desc, X, precision, "depth_first", "dense")


@pytest.mark.parametrize("max_depth,n_features,n_rows,shape", [
    (10, 400, 38_001, "NT=3,DEPTH=10> R=128 G=5"),   # 256 rows leave room for 3 trees, 128 for 15
    (10, 300, 38_001, "NT=3,DEPTH=10> R=256 G=3"),   # 9 and 18: as many walks
    (9, 860, 9_001, "NT=4,DEPTH=9> R=64"),           # the same of 128 rows
    (9, 30, 20_001, "NT=4,DEPTH=9> R=128 G=4 S=2 K=1 tiles=2")])  # vector leaves: 16 trees and two tiles, or 18 trees
def test_row_tiles_that_leave_room_for_few_trees(max_depth, n_features, n_rows, shape):
    """Depth 9 and 10: row tiles are halved where that at least doubles the walks in flight, and small tiles of
    forests with few visits come in two buffers where that costs few walks."""
    import numpy as np

    from cuml_b200.fil import _lib
    from cuml_b200.fil._desc import INFER_DEFAULT

    kw = dict(vector=True, n_outputs=2) if n_features == 30 else {}
    desc = random_forest_desc(101, n_trees=103, n_features=n_features, max_depth=max_depth, p_leaf=0.02, **kw)
    X = random_rows(7, n_rows, n_features, np.float32, nan_frac=0.001)
    fi = _all_kinds(desc, X[:3001], "single", "depth_first", "dense")
    import torch

    from oracle import oracle
    from tests.test_gpu_parity import _tol

    raw = fi._run(torch.as_tensor(X, device="cuda:0"), INFER_DEFAULT, None).cpu().numpy()
    assert shape in _lib.last_variant(), _lib.last_variant()
    np.testing.assert_allclose(raw, oracle.predict(desc, X, INFER_DEFAULT, "single"), **_tol(desc, "single"))


def test_fixed_scratch_takes_the_largest_batch_of_large_tiles():
    """434 features: 38,656 rows of ranks leave 1,024 bytes of the array, enough for the flags of tiles of 256 rows
    and not for those of 128."""
    import numpy as np
    import torch

    from cuml_b200.fil import ForestInference, _lib
    from cuml_b200.fil._desc import INFER_DEFAULT

    desc = random_forest_desc(102, n_trees=30, n_features=434, max_depth=9, p_leaf=0.02)
    fi = ForestInference.load_from_treelite_model(desc, storage="dense")
    g = torch.Generator(device="cuda:0")
    g.manual_seed(2)
    x = torch.randn((38_657, 434), generator=g, device="cuda:0")
    out = torch.zeros((38_656, 1), device="cuda:0")
    call = _lib.load().b2fil_predict_fixed_scratch
    args = (434, out.data_ptr(), 0, 0.5, torch.cuda.current_stream().cuda_stream)
    _lib.check(call(fi.forest.handle, INFER_DEFAULT, x.data_ptr(), 38_656, *args))
    assert "R=256" in _lib.last_variant()
    np.testing.assert_allclose(out.cpu().numpy(), fi._run(x[:-1], INFER_DEFAULT, None).cpu().numpy(), rtol=1e-5,
                               atol=1e-5)
    assert "R=128" in _lib.last_variant()
    assert call(fi.forest.handle, INFER_DEFAULT, x.data_ptr(), 38_657, *args) != 0


def _force(lib, shape, leafg=0):
    for key, v in zip((b"q_R", b"q_G", b"q_NT", b"q_S", b"q_K"), shape):
        lib.b2fil_set_tuning(key, v)
    lib.b2fil_set_tuning(b"q_leafg", leafg)


def test_forced_shapes_are_refused_where_there_is_no_such_kernel():
    """Six trees in flight exist for sums and eight for one output per row and tree: a forced shape that asks for
    the other is not taken, and the record names the kernel that ran."""
    import torch

    from cuml_b200.fil import ForestInference, _lib, synthetic_complete_forest

    fi = ForestInference.load_from_treelite_model(synthetic_complete_forest(60, 6, 20, 3))
    x = torch.zeros((9000, 20), device="cuda:0")
    lib = _lib.load()
    try:
        for nt, taken, call in ((6, "float,scalar,NT=6", fi.predict_proba), (8, "float,leaf_id,NT=8", fi.apply)):
            _force(lib, (128, 2, nt, 2, 1))
            call(x, chunk_size=4)
            assert taken in _lib.last_variant() and "G=2 S=2 K=1" in _lib.last_variant(), _lib.last_variant()
            other = fi.apply if nt == 6 else fi.predict_proba
            other(x, chunk_size=4)
            assert f"NT={nt}" not in _lib.last_variant(), _lib.last_variant()
    finally:
        _force(lib, (0, 0, 0, 0, 0), -1)


def test_ranks_per_thread():
    """Sixteen for large batches of whole groups of 32 features, eight where a group is ragged, the batch is smaller
    or values are fp64, four for a few small tiles."""
    import torch

    from cuml_b200.fil import ForestInference, _lib, synthetic_complete_forest

    for n_features, rows, chunk, precision, ranks in ((96, 13_000, 8, "single", 16), (96, 12_000, 8, "single", 8),
                                                      (100, 13_000, 8, "single", 8), (96, 13_000, 8, "double", 8),
                                                      (96, 5_000, 4, "single", 4)):
        fi = ForestInference.load_from_treelite_model(synthetic_complete_forest(40, 5, n_features, 3),
                                                      precision=precision)
        dt = torch.float64 if precision == "double" else torch.float32
        fi.predict_proba(torch.zeros((rows, n_features), device="cuda:0", dtype=dt), chunk_size=chunk)
        # (256 rows and 32 features per SM are 37,888 on 148 SMs: 12,630 rows of three groups)
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        want = 8 if ranks == 16 and rows * 3 < 256 * sms else ranks
        assert f"ranks={want}" in _lib.last_variant(), (n_features, rows, _lib.last_variant())


@pytest.mark.parametrize("max_depth", [4, 5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("kw", [dict(), dict(vector=True, n_outputs=2), dict(vector=True, n_outputs=3),
                                dict(vector=True, n_outputs=6)])
def test_bodies_for_one_and_two_trees_in_flight(max_depth, kw):
    """Every depth and output kind of the bodies that wide forests take, forced (they are chosen where shared memory
    holds few trees beside the row tile): partial groups of trees, missing values, tests that nothing passes."""
    import numpy as np
    import torch

    from cuml_b200.fil import ForestInference, _lib
    from cuml_b200.fil._desc import INFER_DEFAULT, INFER_LEAF_ID, INFER_PER_TREE
    from oracle import oracle
    from tests.test_gpu_parity import _tol

    desc = random_forest_desc(103, n_trees=23, n_features=9, max_depth=max_depth, p_leaf=0.03, **kw)
    desc.threshold[np.flatnonzero(desc.node_kind == 1)[::11]] = np.nan
    X = random_rows(8, 1_003, 9, np.float32, nan_frac=0.0)
    X[500:] = random_rows(9, 503, 9, np.float32, nan_frac=0.1)
    x = torch.as_tensor(X, device="cuda:0")
    fi = ForestInference.load_from_treelite_model(desc, storage="dense")
    lib = _lib.load()
    mode = "vector" if kw else "scalar"
    try:
        for shape in ((128, 2, 1, 2, 2), (64, 3, 2, 2, 1), (32, 1, 2, 3, 1)):
            _force(lib, shape)
            for kind, name in ((INFER_DEFAULT, mode), (INFER_PER_TREE, None), (INFER_LEAF_ID, "leaf_id")):
                got = fi._run(x, kind, 4).cpu().numpy()
                v = _lib.last_variant()
                assert f"NT={shape[2]},DEPTH={max_depth}" in v and (name is None or name in v), v
                want = oracle.predict(desc, X, kind, "single")
                if kind == INFER_DEFAULT:
                    np.testing.assert_allclose(got, want, **_tol(desc, "single"))
                else:
                    assert np.array_equal(got.reshape(len(X), -1).astype(want.dtype), want.reshape(len(X), -1))
    finally:
        _force(lib, (0, 0, 0, 0, 0), -1)


@pytest.mark.parametrize("precision,max_depth", [("single", 1), ("single", 2), ("single", 3), ("single", 11),
                                                 ("single", 12), ("double", 1), ("double", 3), ("double", 6),
                                                 ("double", 9), ("double", 11)])
def test_forests_in_heap_order(precision, max_depth):
    """Forests that are walked with the depth read at run time: every output kind, one and several classes, vector
    leaves, missing values that all go right and that go either way, tests that nothing passes."""
    import numpy as np

    from cuml_b200.fil import _lib

    for i, kw in enumerate((dict(), dict(n_outputs=3), dict(vector=True, n_outputs=2), dict(vector=True, n_outputs=6))):
        desc = random_forest_desc(104, n_trees=25, n_features=7, max_depth=max_depth, p_leaf=0.02, **kw)
        desc.threshold[np.flatnonzero(desc.node_kind == 1)[::9]] = np.nan
        if i % 2:
            desc.default_left[:] = 0
        X = random_rows(10, 2_003, 7, np.float64, nan_frac=0.03)
        _all_kinds(desc, X, precision, "depth_first", "dense", chunk_size=8)
        assert "dense_q_kernel" in _lib.last_variant() and "DEPTH=runtime" in _lib.last_variant(), _lib.last_variant()


def test_leaf_ids_of_more_trees_than_the_parameter_block_holds():
    import torch

    from cuml_b200.fil import _lib

    for max_depth in (4, 6, 9, 10):
        desc = random_forest_desc(105, n_trees=2_051, n_features=9, max_depth=max_depth, p_leaf=0.3)
        fi = _all_kinds(desc, random_rows(11, 700, 9, "float64", nan_frac=0.02), "single", "depth_first", "dense",
                        chunk_size=8)
        fi.apply(torch.zeros((700, 9), device="cuda:0"), chunk_size=8)
        assert "dense_q_kernel<float,leaf_id,NT=4,DEPTH=" in _lib.last_variant(), _lib.last_variant()
        assert "runtime" not in _lib.last_variant()
