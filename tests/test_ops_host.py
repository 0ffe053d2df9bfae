"""Host side of the library calls (no GPU): what a call costs before it reaches the library."""
import ctypes as C

import pytest
import torch

from warpsph_b200 import _capi, ops


def test_structures_are_passed_by_address():
    """An int address, not a pointer object: building and casting one costs more than the rest of the
    argument list, a dozen times per right-hand side."""
    p = _capi.SphParams()
    assert ops._p(p) == C.addressof(p) and isinstance(ops._p(p), int)


def test_scratch_sizes_are_asked_once_per_dimension(monkeypatch):
    ops._floats_of.cache_clear()
    asked = []

    class Lib:
        @staticmethod
        def sph_compsph_prep_floats(dim):
            asked.append(dim)
            return {1: 8, 2: 8, 3: 9}[dim]

    monkeypatch.setattr(_capi, "lib", lambda: Lib)
    try:
        assert [ops._floats_of("sph_compsph_prep_floats", d) for d in (2, 3, 2, 3, 1)] == [8, 9, 8, 9, 8]
        assert asked == [2, 3, 1]
    finally:
        ops._floats_of.cache_clear()


@pytest.mark.parametrize("shape", [7, (7, 4), (3, 2, 2), 0, (0, 4)])
def test_empty_keeps_shape_type_and_device(shape):
    t = ops._empty(shape, torch.zeros(2), torch.int32)
    assert tuple(t.shape) == (shape if isinstance(shape, tuple) else (shape,)) and t.dtype == torch.int32 and t.is_contiguous()


def test_untimed_calls_share_one_context(monkeypatch):
    monkeypatch.setattr(ops, "TIMER", None)
    assert ops._timed("a") is ops._timed("b")
    monkeypatch.setattr(ops, "TIMER", ops.KernelTimer(names={"a"}))
    assert ops._timed("b") is ops._UNTIMED and ops._timed("a") is not ops._UNTIMED


@pytest.mark.parametrize("fn,good", [(_capi.fptr, torch.float32), (_capi.iptr, torch.int32)])
def test_pointer_checks_refuse_what_they_refused(fn, good):
    assert fn(None) is None
    with pytest.raises(RuntimeError, match="expected"):
        fn(torch.zeros(4, dtype=torch.float64))
    with pytest.raises(RuntimeError, match="CUDA"):
        fn(torch.zeros(4, dtype=good))
