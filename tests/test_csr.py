"""Sequences as the Python mirror flattens them: every form as when each
sequence is assigned to its place, refused where that is, and arrays as a
whole, not word by word."""
import warnings

import numpy as np
import pytest
import torch

from m6502.engine import _csr


def _one_by_one(seqs):
    offs = np.zeros(len(seqs) + 1, dtype=np.uint32)
    for i, s in enumerate(seqs):
        offs[i + 1] = offs[i] + len(s)
    flat = np.zeros(max(int(offs[-1]), 1), dtype=np.uint16)
    for i, s in enumerate(seqs):
        flat[int(offs[i]):int(offs[i + 1])] = s
    return flat.tolist(), offs.tolist()


FORMS = {
    "none": [], "empty": [[], [1]], "all empty": [[], ()], "lists": [[1, 2], [3]], "tuples": ((1, 2), (3,)), "mixed": [[1, 2], (3,), np.array([4])],
    "uint16": [np.array([1, 2], dtype=np.uint16)], "int64 out of range": [np.array([1, 70000, -1])], "rows": np.array([[1, 2], [3, 4]]),
    "scalars out of range": [[np.int64(70000), np.int32(-1)]], "too large": [[70000]], "negative": [[-1]], "floats": [[1.5, 2.0]],
    "float array": [np.array([1.5])], "bools": [[True]], "tensor": [torch.tensor([1, 2])], "range": [range(3)], "objects": [np.array([1, 2], dtype=object)],
    "number strings": [["1", "2"]], "None": [[None]], "column": [np.array([[1], [2]])], "row of rows": [np.array([[1, 2]])], "string": ["12"],
    "bytes": [b"\x01\x02"], "set": [{1}], "dict": [{1: 2}], "nested": [[[1], [2]]], "array in a list": [[np.array([3])]],
    "arrays in lists": [[np.array([3])], [np.array([4])]], "long array in a list": [[np.array([3, 4])]], "0-d in a list": [[np.array(5)]],
    "not a sequence": [5], "complex": [[1 + 0j]],
}


def _result(f, seqs):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        try:
            flat, offs = f(seqs)
        except Exception:
            return "refused"
    return (flat, offs) if isinstance(flat, list) else (flat.tolist(), offs.tolist())


@pytest.mark.parametrize("form", FORMS)
def test_forms(form):
    assert _result(_csr, FORMS[form]) == _result(_one_by_one, FORMS[form])


def test_arrays_are_copied_whole():
    class Words(np.ndarray):
        def __iter__(self):
            raise AssertionError("walked word by word")

    a = np.arange(1000, dtype=np.uint16).view(Words)
    flat, offs = _csr([a, a[:10]])
    assert flat.dtype == np.uint16 and offs.dtype == np.uint32
    assert flat.tolist() == list(range(1000)) + list(range(10)) and offs.tolist() == [0, 1000, 1010]
