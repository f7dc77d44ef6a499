"""The Python layer's native module without a GPU: what it refuses, it refuses
before any launch, with the exception types of the layer's contract."""
import pytest
import torch

from singa_b200 import _lib, singa_wrap as sw


@pytest.mark.parametrize("call", [
    lambda t: sw.ReLU(t), lambda t: sw.ReLUBackward(t, t), lambda t: sw.binary("add", t, t), lambda t: sw.SumRows(t),
    lambda t: sw.SoftMax(t), lambda t: sw.sgd_update_multi([t], [t], None, 0.1), lambda t: sw.pack([t], t)])
def test_cpu_tensors_are_refused(call):
    with pytest.raises(ValueError, match="no CPU path"):
        call(torch.zeros(4, 4))


@pytest.mark.parametrize("calls, error", [
    ([("sgb_no_such_call", (), False)], ValueError),
    ([("sgb_set_f32", (0.0, None), False)], TypeError),                    # wrong number of arguments
    ([("sgb_set_f32", (0.0, None, 0, "NO_SUCH_SLOT"), False)], ValueError),
    ([("sgb_set_f32", ("x", None, 0, "STREAM"), False)], ValueError),
    ([("sgb_set_f32", (0.0, None, 0), 1, 2, 3)], TypeError)])
def test_malformed_programs_are_refused(calls, error):
    with pytest.raises(error):
        _lib.native.program(calls, None)


def test_statuses_become_errors():
    with pytest.raises(TypeError):
        _lib.native.binary(0)
    assert _lib.native.program([("sgb_set_f32", (0.0, None, 0, "STREAM"), False)], None) is not None
