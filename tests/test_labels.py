"""Labels and column-major arrays behind the small calls: an Index compares and
hashes by its tag, is no sequence, and survives copies; empty_colmajor has the
strides of a reversed contiguous array."""
import copy
import pickle

import pytest
import torch

from muscle_gb300.ops import _same_labels
from muscle_gb300.tensor import Index, Tensor, empty_colmajor


@pytest.mark.parametrize("tag", ["i", 3, ("Index", "i"), ("s", 1, 2), None])
def test_index_is_its_tag(tag):
    i = Index(tag)
    assert i.tag == tag and Index(i) == i and Index(Index(i)).tag == tag and hash(i) == hash(Index(tag))
    assert i != Index("other") and not i == tag and repr(i) == f"index<{tag}>"
    for j in (copy.copy(i), copy.deepcopy(i), pickle.loads(pickle.dumps(i))):
        assert type(j) is Index and j == i and j.tag == tag
    with pytest.raises(TypeError):
        list(i)
    with pytest.raises(TypeError):
        Tensor(torch.zeros(2, 2), i)


def test_index_tags_may_not_hash():
    i = Index(["a"])
    assert i == Index(["a"]) and i != Index(["b"])
    with pytest.raises(TypeError):
        hash(i)


@pytest.mark.parametrize("shape", [(), (3,), (2, 3, 4), (1, 5, 1), (0, 3), (3, 0, 2), (2, 1, 0)])
def test_empty_colmajor_strides(shape):
    t = empty_colmajor(list(shape), torch.float64, "cpu")
    want = torch.empty(list(reversed(shape)), dtype=torch.float64).permute(*reversed(range(len(shape)))) if shape \
        else torch.empty((), dtype=torch.float64)
    assert t.shape == want.shape and t.stride() == want.stride()


@pytest.mark.parametrize("xs,ys,same", [("ab", "ba", True), ("ab", "ac", False), ("aab", "aba", True),
                                        ("aab", "abb", False), ("ab", "aa", False), ("aa", "ab", False),
                                        ("a", "ab", False), ("", "", True)])
def test_same_labels(xs, ys, same):
    assert _same_labels([Index(x) for x in xs], [Index(y) for y in ys]) == same
