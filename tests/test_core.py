import json
import os

import numpy as np
import pytest
import torch

import keras_b200 as keras
from keras_b200 import tree
from keras_b200.core import dtypes

HERE = os.path.dirname(__file__)


def test_result_type_matches_reference_table():
    # table generated once by running the reference's `keras.backend.result_type`
    golden = json.load(open(os.path.join(HERE, "golden_result_type.json")))
    conv = lambda s: int if s == "pyint" else float if s == "pyfloat" else s
    for key, expected in golden.items():
        parts = [conv(p) for p in key.split(",")]
        try:
            got = dtypes.result_type(*parts)
        except ValueError:
            got = "ERR"
        assert got == expected, (key, got, expected)


def test_float8_has_no_implicit_promotion():
    with pytest.raises(ValueError):
        dtypes.result_type("float8_e4m3fn", "float32")


def test_variable_basics():
    v = keras.Variable(np.ones((2, 3), "float32"), name="w")
    assert v.shape == (2, 3) and v.dtype == "float32" and v.path == "w"
    v.assign(np.full((2, 3), 2.0, "float32"))
    v.assign_add(np.ones((2, 3), "float32"))
    np.testing.assert_allclose(v.numpy(), 3.0)
    with pytest.raises(ValueError):
        v.assign(np.ones((3, 2), "float32"))
    assert (v + 1).shape == (2, 3)
    with keras.name_scope("outer"):
        w = keras.Variable(0.0, name="b")
    assert w.path == "outer/b"


def test_stateless_scope_defers_and_overrides():
    v = keras.Variable(np.zeros((2,), "float32"))
    with keras.StatelessScope(state_mapping=[(v, np.ones((2,), "float32"))]) as scope:
        np.testing.assert_allclose(v.value.numpy(), 1.0)
        v.assign(v.value + 1)
    np.testing.assert_allclose(scope.get_current_value(v).numpy(), 2.0)
    np.testing.assert_allclose(v.numpy(), 0.0)


def test_tree_roundtrip():
    s = {"b": [1, (2, 3)], "a": 4}
    flat = tree.flatten(s)
    assert flat == [4, 1, 2, 3]
    assert tree.pack_sequence_as(s, flat) == s
    assert tree.map_structure(lambda x: x * 2, s) == {"b": [2, (4, 6)], "a": 8}
    assert [p for p, _ in tree.flatten_with_path(s)] == [("a",), ("b", 0), ("b", 1, 0), ("b", 1, 1)]
    with pytest.raises(ValueError):
        tree.assert_same_structure(s, {"a": 1})


def test_autocast_scope():
    from keras_b200.core.variables import AutocastScope

    v = keras.Variable(np.ones((2,), "float32"))
    with AutocastScope("bfloat16"):
        assert v.value.dtype == torch.bfloat16
    assert v.value.dtype == torch.float32


def test_kernel_front_ends_import_without_gpu():
    import importlib

    for name in ("gemm", "ops", "dispatch", "conv", "attention", "microbench", "build", "loader"):
        importlib.import_module(f"keras_b200.kernels.{name}")


def test_convolution_tiling_choices_without_a_gpu():
    """The host-side planning of the tcgen05 convolution (which pixel tile, whether vertical taps share one TMA box) is plain
    C++ and can be asked without a device: the ResNet-50 3x3 layers with 64 and 128 channels share rows, the others do not."""
    import ctypes
    import os

    import keras_b200

    path = os.path.join(os.path.dirname(keras_b200.__file__), "kernels", "libkb200.so")
    if not os.path.exists(path):
        pytest.skip("kernel library not built")
    lib = ctypes.CDLL(path)
    shares = lib.kb200_conv_igemm_shares_rows
    assert shares(256, 56, 56, 64, 64, 3, 3, 1) == 1 and shares(256, 56, 56, 64, 64, 3, 3, -1) == 1
    assert shares(256, 28, 28, 128, 128, 3, 3, 1) == 1
    assert shares(256, 14, 14, 256, 256, 3, 3, 1) == 0      # would need a quarter more tiles
    assert shares(256, 7, 7, 512, 512, 3, 3, 1) == 0
    assert shares(256, 56, 56, 64, 256, 1, 1, 0) == 0       # nothing to share in a 1x1 filter
    assert shares(2, 20, 20, 64, 64, 3, 3, 2) == 0          # dilated rows are not adjacent
    plan = (ctypes.c_int * 3)()
    assert lib.kb200_conv_igemm_plan(256, 56, 56, 64, 64, 3, 3, 1, plan) == 0
    grid, n_tiles, bn = plan[0], plan[1], plan[2]
    assert bn == 64 and n_tiles == 1 and 0 < grid <= 148
    assert lib.kb200_conv_igemm_plan(256, 14, 14, 256, 1024, 1, 1, 0, plan) == 0
    assert plan[2] == 256 and plan[1] == 4 and plan[0] % 4 == 0


def test_the_kernels_switch_is_read_from_the_environment_in_force(monkeypatch):
    import os

    from keras_b200.core import config

    for environ in (dict(os.environ), os.environ):  # a program may put a mapping of its own in its place
        monkeypatch.setattr(os, "environ", environ)
        for value, on in (("1", False), ("0", True), ("", True)):
            monkeypatch.setitem(os.environ, "KERAS_B200_DISABLE_FUSED_KERNELS", value)
            assert config.fused_kernels_enabled() is on
        monkeypatch.delitem(os.environ, "KERAS_B200_DISABLE_FUSED_KERNELS")
        assert config.fused_kernels_enabled()


def test_kernels_take_tensors_of_the_current_device_alone(monkeypatch):
    """Launches go to the current device; what lies on another one is the library's."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    from keras_b200.kernels import dispatch

    with FakeTensorMode():
        tensors = [torch.empty(2, 8, device=f"cuda:{i}") for i in range(2)]
        labels = [torch.zeros(2, dtype=torch.long, device=f"cuda:{i}") for i in range(2)]
    for current in range(2):
        monkeypatch.setattr(dispatch, "_current_device", lambda: current)
        assert [dispatch.enabled(t) for t in tensors] == [current == 0, current == 1]
        assert dispatch.softmax_cross_entropy(tensors[current], labels[1 - current]) is None
        assert dispatch.dense(tensors[1 - current], None, None, None) is None


def test_hooks_on_a_parameter_see_its_gradient():
    """A kernel that adds its gradient in place sends none through autograd: not for parameters with hooks."""
    from keras_b200.kernels import shadow

    def parameter():
        p = torch.nn.Parameter(torch.zeros(4))
        p.grad = torch.zeros(4)
        return p

    def has_slot(p):
        return shadow.grad_slot(p, (4,)) is not None

    plain, hooked, after, observed = (parameter() for _ in range(4))
    handle = hooked.register_hook(lambda g: None)
    after.register_post_accumulate_grad_hook(lambda q: None)
    observed.register_post_accumulate_grad_hook(lambda q: None)
    assert not has_slot(plain)
    with shadow.arena_backward():
        assert has_slot(plain) and not has_slot(hooked) and not has_slot(after)
        handle.remove()
        assert has_slot(hooked)
        shadow.set_slot_observer(lambda q: None)
        try:
            assert has_slot(observed) and has_slot(plain)
            observed.register_post_accumulate_grad_hook(lambda q: None)
            assert not has_slot(observed)
        finally:
            shadow.set_slot_observer(None)


def test_slices_of_tall_weight_gradients_fill_the_chip(monkeypatch):
    """Few tiles over very many rows: one slice a streaming multiprocessor, or as many as K has blocks for."""
    from keras_b200.kernels import gemm

    monkeypatch.setattr(gemm, "_sm_count", lambda device: 148)
    for M, N, K, tiles in ((512, 64, 200704, 4), (160, 96, 100352, 2), (32, 24, 100352, 1), (1024, 64, 30000, 8), (256, 128, 8192, 2)):
        slices = gemm.split_k_for(M, N, K, None)
        assert 0.8 * min(148, K // 256) <= slices * tiles <= 148, (M, N, K, slices)
    for M, N, K in ((512, 512, 2047), (2048, 2560, 5000), (64, 64, 100)):
        assert gemm.split_k_for(M, N, K, None) == 1


def test_float32_kernels_ask_for_tf32_by_either_setting():
    """Code in a process of its own: the settings cannot be unset."""
    import subprocess
    import sys

    template = "import torch; {}; from keras_b200.kernels import sgemm; print(sgemm.takes_weight_gradient(6400, 256, 1024, True))"
    matmul = "torch.backends.cuda.matmul"
    settings = {"pass": "True", f"{matmul}.allow_tf32 = True": "False", f"{matmul}.fp32_precision = 'tf32'": "False", "torch.backends.fp32_precision = 'tf32'": "False",
                f"{matmul}.fp32_precision = 'ieee'": "True"}
    runs = {s: subprocess.Popen([sys.executable, "-c", template.format(s)], stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True) for s in settings}
    for setting, run in runs.items():
        out, err = run.communicate(timeout=300)
        assert out.strip() == settings[setting], (setting, out, err[-400:])
