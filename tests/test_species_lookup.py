"""Host species lookup: the array path for integer labels agrees with the label-by-label
lookup for every label container, and unknown labels raise as before."""
import numpy as np
import pytest

from aok_b200 import AOKError
from aok_b200.basis import species_indices


@pytest.mark.parametrize("zlist", [(1, 6, 7, 8), (8, 1, 7, 6), (3,), (-5, 2, 9), (2**40, 1)])
@pytest.mark.parametrize("wrap", [np.asarray, list, tuple, lambda a: np.asarray(a, dtype=np.int32),
                                  lambda a: np.asarray(a)[::-1][::-1], lambda a: [np.int64(x) for x in a],
                                  lambda a: [float(x) for x in a], lambda a: np.asarray(a, dtype=np.uint64)])
def test_array_path_equals_the_lookup(zlist, wrap):
    pick = np.random.default_rng(3).integers(0, len(zlist), 57)
    labels = [zlist[i] for i in pick]
    if wrap is not list and max(map(abs, zlist)) > 2**31 and getattr(wrap(labels[:1]), "dtype", None) == np.int32:
        pytest.skip("label does not fit")
    if min(zlist) < 0 and getattr(wrap([1]), "dtype", None) == np.uint64:
        pytest.skip("label does not fit")
    got = species_indices(zlist, wrap(labels))
    assert got.dtype == np.int64 and np.array_equal(got, pick + 1)


def test_other_labels():
    assert species_indices(("a", "b"), ["b", "a"]).tolist() == [2, 1]
    assert species_indices((2, 2), [2, 2]).tolist() == [2, 2]  # the last of equal labels, as the lookup
    assert species_indices((1,), []).tolist() == []
    for bad in ([1, 9, 6], np.array([1, 9]), ["x"]):
        with pytest.raises(AOKError, match="not in basis species list"):
            species_indices((1, 6), bad)
