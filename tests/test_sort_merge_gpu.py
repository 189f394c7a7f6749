"""The merge sort of small arrays (sort_merge.cu) and the radix sort, each forced,
against numpy's stable argsort: keys and values equal, at the edges of tiles and
of merge passes, with equal keys, sorted and reversed keys, and the greatest key
(which also fills up a tile's end)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 4, 5, 31, 2047, 2048, 2049, 4095, 4097, 6144, 8193, 30001, 262144, 262145, 270337]


def _keys(kind, n, rng):
    if kind == "random":
        return rng.integers(0, 1 << 63, n, dtype=np.uint64)
    if kind == "few":
        return rng.integers(0, 5, n).astype(np.uint64)
    if kind == "greatest":
        k = rng.integers(0, 1 << 63, n, dtype=np.uint64)
        k[rng.random(n) < 0.3] = np.uint64(2**64 - 1)
        return k
    k = np.sort(rng.integers(0, 1 << 40, n, dtype=np.uint64))
    return np.ascontiguousarray(k[::-1]) if kind == "reversed" else k


@pytest.mark.parametrize("form", ["merge", "radix", None])
@pytest.mark.parametrize("n", SIZES)
def test_sort_forms_are_stable(nb, cuda, monkeypatch, form, n):
    torch = cuda
    if form:
        monkeypatch.setenv("NBODY_SORT", form)
    rng = np.random.default_rng(n)
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode="bh")
    solver.set_stream(torch.cuda.current_stream().cuda_stream)
    for kind in ("random", "few", "greatest", "sorted", "reversed"):
        keys, vals = _keys(kind, n, rng), rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        order = np.argsort(keys, kind="stable")
        k = torch.from_numpy(keys.view(np.int64).copy()).cuda()
        v = torch.from_numpy(vals.view(np.int32).copy()).cuda()
        solver.sort_pairs_device(k, v, n)
        solver.sync()
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys[order])
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])
    solver.close()


@pytest.mark.parametrize("n", [4096, 6145, 8192, 14337, 16384, 16385, 32768, 32769, 65537, 131073, 262143])
def test_sort_by_searched_places(nb, cuda, monkeypatch, n):
    """Groups of four and of eight runs, whole and cut short, in one to three passes."""
    test_sort_forms_are_stable(nb, cuda, monkeypatch, "merge", n)
