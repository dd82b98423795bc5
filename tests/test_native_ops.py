"""The native half of neoml_b200/ops.py declines what it does not take, so that the Python code raises as it always did."""
import pytest
import torch

from neoml_b200 import ops


def test_native_calls_decline_other_tensors():
    native = ops._native()
    a, f = torch.zeros(2, 3, 4), torch.zeros(1, 3, 3, 4)
    assert native.batch_multiply_by_transposed(a, a, None, 0, True) is None                  # not on a GPU
    assert native.multiply_by_matrix(a, a, None, 0) is None
    assert native.transpose(1, a, 2, 1, 3, 4, None) is None
    assert native.vector_op(0, a, None, None, 0.0, None, None) is None
    assert native.vector_op(0, None, None, None, 0.0, None, None) is None
    assert native.blob_convolution(torch.zeros(1, 5, 5, 4), f, None, None, 0, 0, 1, 1, 1, 1, None, 0, 0.0, 0, True) is None
    with pytest.raises(TypeError):
        native.transpose(1, a)


def test_first_error_of_a_process_has_its_text(monkeypatch):
    """A native call does not go through capi.load(); an error that it answers is spelled out all the same."""
    monkeypatch.setattr(ops.capi, "_lib", None)
    with pytest.raises(ops.capi.Nb200Error, match=r"BlobConvolution failed: .*launch.*: .*\(-3\)") as e:
        ops._checked("BlobConvolution", ops.capi.ELAUNCH)
    assert e.value.code == ops.capi.ELAUNCH


def test_calls_without_the_native_half(monkeypatch):
    """Where it has not been built for this torch the Python code behind each call serves (and checks its arguments)."""
    a = torch.zeros(4, 8)
    monkeypatch.setattr(torch, "__version__", "0.0")
    monkeypatch.setattr(ops, "_native_module", None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    with pytest.warns(UserWarning, match="torch0.0"):
        assert ops._native().transpose(1, a, 2, 1, 2, 8, None) is None
    with pytest.raises(AssertionError, match="device-resident"):
        ops.MultiplyMatrixByTransposedMatrix(a, a)


@pytest.mark.gpu
def test_same_results_without_the_native_half(monkeypatch):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    a, f = torch.empty(3, 20, 36, device="cuda").normal_(generator=g), torch.empty(5, 3, 3, 36, device="cuda").normal_(generator=g)
    calls = [lambda: ops.BlobConvolution(a.view(1, 6, 10, 36), f), lambda: ops.MultiplyMatrixByTransposedMatrix(a[0], a[1]),
             lambda: ops.BatchMultiplyMatrixByTransposedMatrix(a, a), lambda: ops.MultiplyMatrixByMatrix(a[:, :, :20].contiguous(), a),
             lambda: ops.TransposeMatrix(3, a, 20, 1, 36, 1), lambda: ops.vector_op("EXP", a)]
    native = [call() for call in calls]
    monkeypatch.setattr(ops, "_native_module", ops._DeclinesAll())
    for call, want in zip(calls, native):
        got = call()
        assert got.shape == want.shape and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_products_where_work_space_does_not_fit(monkeypatch, native):
    """Odd depths want copies of both operands; without room for them the product is gathered, as it is without work space."""
    if not native:
        monkeypatch.setattr(ops, "_native_module", ops._DeclinesAll())
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    a, b = torch.empty(1, 20000, 1001, device="cuda").normal_(generator=g), torch.empty(1, 300, 1001, device="cuda").normal_(generator=g)
    want, batched = torch.empty(20000, 300, device="cuda"), torch.empty(1, 20000, 300, device="cuda")
    got = torch.empty_like(want)
    ops.MultiplyMatrixByTransposedMatrix(a[0], b[0], want, use_scratch=False)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        # half of what the copies take
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (40 << 20)) / total)
        ops.MultiplyMatrixByTransposedMatrix(a[0], b[0], got)
        ops.BatchMultiplyMatrixByTransposedMatrix(a, b, batched)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want) and torch.equal(batched[0], want)


@pytest.mark.gpu
def test_errors_are_the_python_codes():
    x, f = torch.zeros(1, 5, 5, 4, device="cuda"), torch.zeros(2, 3, 3, 4, device="cuda")
    y = ops.BlobConvolution(x, f)
    assert y.shape == (1, 3, 3, 2) and y.device == x.device and y.dtype == torch.float32
    with pytest.raises(AssertionError):
        ops.BlobConvolution(x.permute(0, 2, 1, 3), f)                # not contiguous
    with pytest.raises(AssertionError):
        ops.BlobConvolution(x.double(), f)
    with pytest.raises(AssertionError):
        ops.BlobConvolution(x, torch.zeros(2, 3, 3, 5, device="cuda"))
    with pytest.raises(ops.capi.Nb200Error):
        ops.MultiplyMatrixByTransposedMatrix(x.view(25, 4), f.view(18, 4), first_row_size=3)
    out = torch.empty(1, 3, 3, 2, device="cuda")
    assert ops.BlobConvolution(x, f, result=out) is not None and torch.equal(out, y)
