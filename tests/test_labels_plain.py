"""An Index is an object with a tag and nothing else: no tuple, neither equal
to one nor unpacked like one, and the label algebra of the operations tells
labels apart as Index does."""
import random

import numpy as np
import pytest
import torch

from muscle_gb300.ops import _desc_args, _modes_for, _same_labels, binary_inds_c
from muscle_gb300.tensor import Index, Tensor, empty_colmajor, intersect, setdiff, union


def test_index_is_no_tuple():
    i = Index("x")
    assert i != ("Index", "x") and ("Index", "x") != i and not isinstance(i, tuple)
    assert "%s" % i == "index<x>" and "{}".format(i) == "index<x>"
    a = np.array([i, Index("y")], dtype=object)
    assert a.shape == (2,) and a[1] == Index("y")
    with pytest.raises(TypeError):
        len(i)
    with pytest.raises(TypeError):
        i < Index("y")
    i.tag = "z"
    assert i == Index("z") and repr(i) == "index<z>"


@pytest.mark.parametrize("kind", [str, int, tuple])
def test_binary_inds_c_is_the_label_algebra(kind):
    """The sum labels are dims (default: the shared ones) within both operands."""
    rng = random.Random(1)
    for _ in range(300):
        make = {str: str, int: int, tuple: lambda v: ("s", v)}[kind]
        ia, ib, dims = ([Index(make(rng.randrange(6))) for _ in range(rng.randrange(5))] for _ in range(3))
        for d in (None, dims):
            want = setdiff(union(ia, ib), intersect(intersect(ia, ib) if d is None else d, ia, ib))
            assert binary_inds_c(ia, ib, dims=d) == want


def test_labels_that_are_no_index_stay_apart():
    assert binary_inds_c(["i", "k"], ["k", "j"]) == ["i", "j"]
    modes = _modes_for([Index("i"), "i"], ["i", Index("j")])
    assert len(modes) == 3
    x = Tensor(np.zeros((2, 3)), ["i", "j"])
    assert _desc_args(x.data, x.inds, modes)[1] == (0, 2) and _desc_args(x.data, ["i", Index("i")], modes)[1] == (1, 0)


@pytest.mark.parametrize("tags", [[1.0, 2], [True, 2], ["1", "2"]])
def test_permutation_by_labels_of_another_type_is_refused(tags):
    assert _same_labels([Index(2), Index(1)], [Index(1), Index(2)])
    assert not _same_labels([Index(t) for t in tags], [Index(1), Index(2)]) or tags == ["1", "2"]


def test_empty_colmajor_takes_any_iterable():
    for shape in (iter([2, 0, 3]), (n for n in (2, 0, 3)), np.array([2, 0, 3])):
        t = empty_colmajor(shape, torch.float64, "cpu")
        assert tuple(t.shape) == (2, 0, 3) and t.stride() == (1, 2, 2)
    with pytest.raises(RuntimeError):
        empty_colmajor([2, -1], torch.float64, "cpu")
