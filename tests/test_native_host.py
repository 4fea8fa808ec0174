"""The native host module on a machine without a GPU: it loads beside
libgbsv.so and leaves every call without plain CUDA tensors to the Python
functions, whose errors stay theirs."""
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300 import _native


@pytest.fixture(scope="module")
def mod(lib_built):
    return _native.load()


def test_leaves_other_calls_to_python(mod):
    s = torch.ones(4, dtype=torch.complex64)
    m = torch.eye(2, dtype=torch.complex64)
    assert mod.apply_operator(m, [0], s) is None
    assert mod.apply_operator(m, [0]) is None
    assert mod.apply_operator(None, "x", 3) is None
    assert mod.apply_layer(m, s, False) is None
    assert mod.apply_phase(torch.ones(4), s) is None
    assert mod.norm_squared(s) is None
    assert mod.abs_squared("state") is None
    assert mod.inner_product(s, s) is None
    assert mod.diag_expectation_value(torch.ones(4), s) is None


def test_errors_are_the_python_functions(mod):
    m = torch.eye(2, dtype=torch.complex64)
    with pytest.raises(ug.StateShapeError):
        ug.apply_operator(m, [0], torch.ones(3, dtype=torch.complex64))
    with pytest.raises(ValueError):
        ug.apply_operator(m, [2], torch.ones(4, dtype=torch.complex64))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ug.apply_operator(m, [0], torch.ones(4, dtype=torch.complex64))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ug.norm_squared(torch.ones(4, dtype=torch.complex64))
