"""What the operator wrappers accept as `out` and `residual`: whole rows of the right width, and no fewer rows than the
input has.  The kernels take pointers and strides only, so this is where a mis-sized buffer has to be refused.  The
checks are host code and run on CPU tensors here (no launch)."""
import pytest
import torch

from tnn_b200 import ops


@pytest.fixture
def cpu_tensors(monkeypatch):
    monkeypatch.setattr(ops, "_require_cuda", lambda *ts: None)


def _half(*shape):
    return torch.zeros(shape, dtype=torch.float16)


def _linear(residual=None, out=None):
    epi = ops.EPI_BIAS if residual is None else ops.EPI_BIAS_RESIDUAL
    return ops._linear_desc(_half(41, 768), _half(768, 768), None, residual, epi, None, out, 0)[0]


def _layernorm(residual=None, out=None):
    g = torch.ones(768)
    return ops._layernorm_desc(_half(41, 768), g, g, 1e-12, residual, None, out)[0]


@pytest.mark.parametrize("desc", [_linear, _layernorm])
@pytest.mark.parametrize("which", ["residual", "out"])
@pytest.mark.parametrize("shape", [(41, 776), (1,), (7,), (100,), (5, 760), (41, 768 - 8)])
def test_widths_that_do_not_divide_into_rows_are_refused(cpu_tensors, desc, which, shape):
    with pytest.raises(RuntimeError):
        desc(**{which: _half(*shape)})


@pytest.mark.parametrize("desc", [_linear, _layernorm])
@pytest.mark.parametrize("which", ["residual", "out"])
@pytest.mark.parametrize("t", [_half(40, 768), _half(768), _half(0, 768), _half(40, 776)[:, :768]])
def test_fewer_rows_than_the_input_are_refused(cpu_tensors, desc, which, t):
    with pytest.raises(AssertionError):
        desc(**{which: t})


@pytest.mark.parametrize("desc", [_linear, _layernorm])
@pytest.mark.parametrize("t,ld", [(_half(41, 768), 768), (_half(41 * 768), 768), (_half(41, 1, 768), 768),
                                  (_half(64, 768), 768), (_half(41, 776)[:, :768], 776)])
def test_row_strides_of_what_is_accepted(cpu_tensors, desc, t, ld):
    d = desc(residual=t, out=t)
    assert (d.residual, d.y, d.ldr, d.ldy) == (t.data_ptr(), t.data_ptr(), ld, ld)


def test_no_columns_are_refused_as_a_reshape_refuses_them(cpu_tensors):
    with pytest.raises(RuntimeError):
        ops._linear_desc(_half(4, 8), _half(0, 8), None, None, ops.EPI_BIAS, None, None, 0)
