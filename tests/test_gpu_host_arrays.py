"""Predictions on host arrays: the three ways they take by size (in place, fetched in parts, in
blocks), at the sizes where one ends and the next begins, against the CPU oracle."""
import threading

import numpy as np
import pytest

from cuml_b200.fil import ForestInference, _lib
from cuml_b200.fil._desc import INFER_DEFAULT, INFER_LEAF_ID
from oracle import oracle
from tests.helpers import random_forest_desc, random_rows

pytestmark = pytest.mark.gpu


def _model(n_features, n_trees=9, precision="single", seed=70):
    desc = random_forest_desc(seed, n_trees=n_trees, n_features=n_features, max_depth=5,
                              postproc="sigmoid")
    return desc, ForestInference.load_from_treelite_model(desc, precision=precision)


def _check(desc, fi, X, precision="single"):
    X = np.ascontiguousarray(X, np.float32 if precision == "single" else np.float64)
    assert np.array_equal(fi.apply(X).astype(np.uint32), oracle.predict(desc, X, INFER_LEAF_ID, precision))
    np.testing.assert_allclose(fi._run(X, INFER_DEFAULT, None),
                               oracle.predict(desc, X, INFER_DEFAULT, precision), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n_features", [1, 3, 4, 7, 50])
def test_sizes_around_every_border(n_features):
    """Inputs of 16 KiB (in place / in parts), of one and several parts of 256 KiB, and of 16 MiB (in
    parts / in blocks), with rows that start on 16-byte boundaries and rows that do not; leaf ids, whose
    results have borders of their own (2 KiB, 256 KiB)."""
    desc, fi = _model(n_features)
    row = 4 * n_features
    for size in (1, 2 << 10, 16 << 10, 256 << 10, 700 << 10, 3 << 20, 16 << 20):
        n = max(1, size // row)
        for rows in {n, n + 1, n + 5} if size < 16 << 20 else {n, n + 1}:
            _check(desc, fi, random_rows(rows, rows, n_features, nan_frac=0.02))


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n_rows", [20, 3000, 60_000, 400_000])
def test_rows_with_a_stride(n_rows, precision):
    """The C interface takes rows that are parts of longer ones."""
    desc, fi = _model(13, precision=precision)
    dt = np.float32 if precision == "single" else np.float64
    whole = random_rows(n_rows, n_rows, 17, dt, nan_frac=0.02)
    out = np.full((n_rows, 9), -1, np.int32)
    _lib.check(_lib.load().b2fil_predict_host(fi.forest.handle, INFER_LEAF_ID, whole.ctypes.data, n_rows,
                                              17, out.ctypes.data, 0, 0.5))
    want = oracle.predict(desc, np.ascontiguousarray(whole[:, :13]), INFER_LEAF_ID, precision)
    assert np.array_equal(out.astype(np.uint32), want)


@pytest.mark.parametrize("n_rows", [10, 2000, 50_000, 900_000])
def test_pinned_inputs_and_results(n_rows):
    """Pinned arrays on either side are read and written where they are."""
    import torch

    desc, fi = _model(6)
    X = random_rows(n_rows, n_rows, 6, nan_frac=0.02)
    want = oracle.predict(desc, X, INFER_LEAF_ID, "single")
    pinned = torch.from_numpy(X).pin_memory().numpy()
    out = torch.empty((n_rows, 9), dtype=torch.int32, pin_memory=True).numpy()
    for x in (X, pinned):
        for preds in (None, out, np.empty((n_rows, 9), np.int32)):
            if preds is not None:
                preds[:] = -1
            assert np.array_equal(fi.apply(x, preds=preds).astype(np.uint32), want)


def test_batches_that_grow_and_shrink():
    desc, fi = _model(11)
    X = random_rows(4, 600_000, 11, nan_frac=0.02)
    want = oracle.predict(desc, X, INFER_LEAF_ID, "single")
    for n in (1, 900, 20_000, 21_000, 500, 35_000, 380_000, 3, 400_000, 600_000, 20_000):
        assert np.array_equal(fi.apply(X[:n]).astype(np.uint32), want[:n]), n


def test_threads_share_the_staging_memory():
    """Several models, two threads each, arrays of different sizes at the same time; models come and go
    meanwhile, which gives memory back."""
    models = [_model(f, seed=70 + f) for f in (5, 8, 12)]
    errors = []

    def work(desc, fi, seed):
        try:
            for i in range(6):
                n = (17, 4000, 90_000, 500_000)[(seed + i) % 4]
                X = random_rows(seed + i, n, desc.n_features, nan_frac=0.02)
                assert np.array_equal(fi.apply(X).astype(np.uint32),
                                      oracle.predict(desc, X, INFER_LEAF_ID, "single")), n
                d2, f2 = _model(4, n_trees=3, seed=seed)
                _check(d2, f2, random_rows(i, 5000, 4))
                del f2
        except Exception as e:  # noqa: BLE001  (reported by the test's thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(*m, k)) for k, m in enumerate(models * 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:2]


def test_scratch_of_a_freed_model_goes_back_to_the_device():
    """The scratch pool of a device outlives its models: freeing one that needed much returns what the
    others do not need."""
    import torch

    desc, small = _model(6, n_trees=200)
    x = torch.zeros((20_000, 6), device="cuda:0")
    small.predict_proba(x)
    wide, big = _model(200, n_trees=200)
    X = torch.zeros((1_000_000, 200), device="cuda:0")
    big.predict_proba(X)
    torch.cuda.synchronize()
    scratch = big.describe()["scratch_pool_bytes"]
    assert scratch > 100 << 20
    before = torch.cuda.mem_get_info()[0]
    big.forest.close()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] - before > scratch * 0.8
    assert torch.equal(small.predict_proba(x), small.predict_proba(x))
