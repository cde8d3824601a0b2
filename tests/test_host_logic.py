"""Bookkeeping of the GPTQ handle that needs no device (src/gptq.py:22-136)."""
import math

import pytest
import torch
import torch.nn as nn

from moe_quant_b200 import GPTQ, QuantizationOrder, gptq, model_utils, ops, quant_utils
from moe_quant_b200._lib import MoeQuantError


def _layer(R=8, C=16, dtype=torch.bfloat16):
    return nn.Linear(C, R, bias=False, dtype=dtype)


def test_constructor_matches_reference_positional_order():
    layer = _layer()
    h = GPTQ(layer, 8, True, 0.05, 128, "activation", "absmax", is_distributed=True)
    assert (h.d_row, h.d_col) == (8, 16)
    assert h.group_size == 8 and h.sym and h.rel_damp == 0.05 and h.block_size == 128
    assert h.quantization_order is QuantizationOrder.ACTIVATION and h.is_distributed
    assert h.W_dtype == torch.bfloat16 and h.W_shape == (8, 16)
    assert h.H is None and h.tokens_collected == 0 and not h.has_hessian_issues()
    assert GPTQ(_layer(), None).block_size == 16      # block defaults to d_col (src/gptq.py:45)


def test_rejects_other_modules():
    with pytest.raises(AssertionError):
        GPTQ(nn.LayerNorm(4))


def test_tied_handle_reference_counting():
    gate = GPTQ(_layer(), 8, True)
    up = GPTQ(_layer(), 8, True, tied_gptq_handle=gate)
    assert gate.num_tied_handles == 1 and up.num_tied_handles == 0
    gate.H = torch.eye(16)
    gate.reset()
    assert gate.H is not None               # still needed by `up`
    up.quantization_pre_step()
    assert up.H is gate.H and not up.issue_zero_samples
    up.reset()
    assert gate.H is None and gate.num_tied_handles == 0


def test_zero_samples_falls_back_to_identity():
    h = GPTQ(_layer(), 8, True)
    h.quantization_pre_step()
    assert h.issue_zero_samples and torch.equal(h.H, torch.eye(16))


def test_update_on_cpu_raises():
    h = GPTQ(_layer(), 8, True)
    with pytest.raises(MoeQuantError):
        h.update(torch.zeros(4, 16, dtype=torch.bfloat16))


@pytest.mark.parametrize("error", [MoeQuantError, KeyboardInterrupt])
def test_failed_first_batch_leaves_an_empty_hessian(monkeypatch, error):
    def fail(H, *a):
        H.fill_(float("nan"))
        raise error("stop")
    monkeypatch.setattr(ops, "hessian_accum", fail)
    h = GPTQ(_layer(), 8, True)
    with pytest.raises(error):
        h.update(torch.zeros(4, 16, dtype=torch.bfloat16))
    assert torch.equal(h.H, torch.zeros(16, 16)) and h.tokens_collected == 0


class _On:
    """What the checks in front of a launch look at, on a GPU that need not be there."""
    is_cuda, dtype = True, torch.float32

    def __init__(self, index, *shape, dtype=torch.float32):
        self.device, self.shape, self.dtype = torch.device("cuda", index), shape, dtype

    def dim(self):
        return len(self.shape)

    def numel(self):
        return math.prod(self.shape)

    def stride(self, d):
        return math.prod(self.shape[d + 1:])

    def float(self):
        return self

    contiguous = float


@pytest.fixture
def no_launch(monkeypatch):
    def reached(*a, **k):
        raise AssertionError("went on to the library")
    for name in ("lib", "check"):
        monkeypatch.setattr(ops, name, reached)
    monkeypatch.setattr(torch, "empty", reached)


@pytest.mark.parametrize("devices", [(0, 1, 0), (1, 0, 0), (0, 0, 1)])
def test_error_metric_refuses_tensors_of_several_gpus(no_launch, devices):
    q, w, H = _On(devices[0], 4, 8), _On(devices[1], 4, 8), _On(devices[2], 8, 8)
    for call in (lambda: quant_utils.get_relative_mse_error(q, w, H), lambda: ops.error_forms(q, w, H)):
        with pytest.raises(MoeQuantError, match="one device"):
            call()
    if devices[0] != devices[2]:
        with pytest.raises(MoeQuantError, match="one device"):
            ops.quadratic_form(q, H)


@pytest.mark.parametrize("devices", [(0, 1, 0), (1, 0, 0), (0, 0, 1), (0, 1, None)])
def test_permutation_refuses_indices_of_another_gpu(no_launch, devices):
    src, cols, rows = (None if d is None else _On(d, *shape, dtype=dtype) for d, shape, dtype in
                       zip(devices, [(4, 8), (8,), (4,)], [torch.float32, torch.int32, torch.int32]))
    with pytest.raises(MoeQuantError, match="one device"):
        ops.permute_columns(src, cols, rows=rows)


def test_few_tokens_ask_for_all_products():
    """Below half as many tokens as columns; a tied handle goes by the handle that owns the Hessian; what the caller chose
    otherwise stays."""
    gate = GPTQ(_layer(C=1024), 8, True)
    up = GPTQ(_layer(C=1024), 8, True, tied_gptq_handle=gate)
    for tokens, split in ((0, 4), (511, 4), (512, 3), (5000, 3)):
        gate.num_samples = tokens
        assert gate._layer_precision().split_hinv == up._layer_precision().split_hinv == split
        assert gate._layer_precision().split_sweep == 3
    gate.num_samples = 10
    for p in (ops.Precision(split_hinv=2), ops.Precision(math=ops.MATH_FP32)):
        gate.precision = p
        assert gate._layer_precision() == p
    gate.precision = ops.Precision(compact=True)
    assert gate._layer_precision() == ops.Precision(split_hinv=4, compact=True)


def test_deep_updates_only_from_as_many_tokens_as_columns():
    """Nobody but a handle that has counted them says many_tokens, and only where three products are taken."""
    assert not ops.DEFAULT_PRECISION.many_tokens and ops.Precision().layer_math == ops.Precision().factor_math == ops.MATH_TENSOR
    gate = GPTQ(_layer(C=1024), 8, True)
    up = GPTQ(_layer(C=1024), 8, True, tied_gptq_handle=gate)
    for tokens, many in ((10, False), (512, False), (1023, False), (1024, True), (5000, True)):
        gate.num_samples = tokens
        for p in (gate._layer_precision(), up._layer_precision()):
            assert p.many_tokens == many
            assert p.layer_math == p.factor_math == ops.MATH_TENSOR | (0x200 if many else 0) and p.sweep_math == ops.MATH_TENSOR
    gate.precision = ops.Precision(compact=True)
    assert gate._layer_precision() == ops.Precision(compact=True, many_tokens=True) and gate._layer_precision().layer_math == ops.MATH_TENSOR | 0x300
    for p in (ops.Precision(split_hinv=4), ops.Precision(split_hinv=2), ops.Precision(math=ops.MATH_FP32)):
        gate.precision = p
        assert gate._layer_precision() == p


def test_few_tokens_are_counted_over_all_ranks(monkeypatch):
    """A rank that holds a third of the tokens decides by all of them, as a single process with the same tokens would."""
    h = GPTQ(_layer(C=1024), 8, True, is_distributed=True)
    h.H, h.num_samples = torch.eye(1024), 200
    assert h._layer_precision().split_hinv == 4
    monkeypatch.setattr(gptq.dist_utils, "is_dist_available_and_initialized", lambda: True)
    monkeypatch.setattr(gptq.dist, "all_reduce", lambda t, op=None: t.mul_(3))
    h.quantization_pre_step()
    assert h.tokens_collected == 200 and h._layer_precision().split_hinv == 3
    torch.testing.assert_close(h.H, torch.eye(1024))
    h.reset()
    assert h._hessian_tokens == 0


def test_few_tokens_after_the_owner_was_reset():
    """gate_proj quantized and reset before up_proj: the Hessian is still that of its tokens; a new batch starts afresh."""
    gate = GPTQ(_layer(C=1024), 8, True)
    up = GPTQ(_layer(C=1024), 8, True, tied_gptq_handle=gate)
    gate.H, gate.num_samples = torch.eye(1024), 5000
    gate.reset()
    assert gate.H is not None and gate.tokens_collected == 0
    assert up._layer_precision().split_hinv == 3
    up.reset()
    assert gate.H is None and gate._layer_precision().split_hinv == 4


def test_no_token_at_all_has_nothing_to_cancel():
    h = GPTQ(_layer(C=1024), 8, True)
    h.quantization_pre_step()
    assert h.issue_zero_samples and h._layer_precision().split_hinv == 3 and not h._layer_precision().many_tokens


def test_asymmetric_is_refused():
    h = GPTQ(_layer(), 8, False)
    h.H = torch.eye(16)
    with pytest.raises(MoeQuantError, match="symmetric"):
        h.quantize(4)


def test_model_utils():
    conv = nn.Conv2d(3, 5, 3)
    assert model_utils.get_number_of_rows_and_cols(conv) == (5, 27)
    model = nn.Sequential(nn.Linear(4, 4), nn.ReLU(), nn.Sequential(nn.Linear(4, 2)))
    got = model_utils.select_layers(model, "", ".*", model_utils.LINEAR_LAYERS)
    assert sorted(got) == ["0", "2.0"]
    assert sorted(model_utils.select_layers(model, "2", ".*", nn.Linear)) == ["2.0"]


def test_expired_device_wait_is_reported_with_the_layer_flags(monkeypatch):
    """Reading a layer's status words is where an expired wait of the tensor-core kernels must
    surface: the codes of that layer are garbage and may not be saved as a result."""
    from moe_quant_b200 import _lib

    h = GPTQ(_layer(), 8, True)
    h._pending_flags = [torch.zeros(4, dtype=torch.int32)]
    monkeypatch.setattr(_lib, "engine_fault", lambda: 13)
    with pytest.raises(MoeQuantError, match="bounded wait"):
        h.has_hessian_issues()
    # once reported, the flags are consumed; a healthy device reads clean again
    monkeypatch.setattr(_lib, "engine_fault", lambda: 0)
    h._pending_flags = [torch.tensor([1, 0, 0, 5], dtype=torch.int32)]
    assert h.issue_nan_hessian and h.issue_non_invertible


def test_tied_groups_and_compact_launch_scope():
    """Host side of quantize_many: handles tied to one another form one group led by the owner of
    the Hessian (wherever they stand in the list), a tied handle whose owner is not in the list
    stands alone; inside `compact_launches` a handle asks for compact launch shapes and gets its
    own precision object back afterwards, also when the body raises."""
    from moe_quant_b200 import gptq, ops

    def lin():
        return nn.Linear(16, 8, bias=False)

    gate0, gate1 = GPTQ(lin(), 8, True, 1e-2, 128), GPTQ(lin(), 8, True, 1e-2, 128)
    up0 = GPTQ(lin(), 8, True, 1e-2, 128, tied_gptq_handle=gate0)
    up1 = GPTQ(lin(), 8, True, 1e-2, 128, tied_gptq_handle=gate1)
    down = GPTQ(lin(), 8, True, 1e-2, 128)
    outsider = GPTQ(lin(), 8, True, 1e-2, 128, tied_gptq_handle=GPTQ(lin(), 8, True, 1e-2, 128))
    handles = [up0, gate0, down, gate1, outsider, up1]
    assert gptq._tied_groups(handles) == [[1, 0], [2], [3, 5], [4]]

    assert down.precision is None
    with gptq.compact_launches(down):
        assert down.precision.compact and down.precision.sweep_math == ops.MATH_TENSOR | 0x100
    assert down.precision is None
    mine = ops.Precision(math=0)
    down.precision = mine
    with pytest.raises(RuntimeError):
        with gptq.compact_launches(down):
            assert down.precision.compact and down.precision.math == 0
            raise RuntimeError("body failed")
    assert down.precision is mine and not mine.compact
    with gptq.compact_launches(down, on=False):
        assert down.precision is mine
