"""Operands that the layer functions of the extension module refuse. The checks come before anything touches a GPU, so CPU
tensors show them: with operands that fit, the same calls get as far as asking for a CUDA device."""
import pytest
import torch


@pytest.fixture(scope="module")
def ext():
    from gcow_b200 import _native
    try:
        return _native.ext()
    except Exception as e:          # the CUDA runtime library or its host path is not loadable on this machine
        pytest.skip(f"extension module not loadable: {e}")


def t(*shape, dtype=torch.float32):
    return torch.zeros(*shape, dtype=dtype)


def nhwc(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype).to(memory_format=torch.channels_last)


X, IMG = t(64, 32, dtype=torch.bfloat16), nhwc(2, 64, 8, 8)
CASES = [
    ("linear", (X, t(16, 24), None, None), "weight"),
    ("linear", (X, t(16 * 32), None, None), "weight"),
    ("linear", (X, t(16, 32), t(8), None), "bias"),
    ("linear", (X, t(16, 32), t(16), t(64, 8)), "residual"),
    ("ffn_residual", (X, t(64, 24), t(64), t(32, 64), t(32)), "first weight"),
    ("ffn_residual", (X, t(64, 32), t(64), t(32, 32), t(32)), "second weight"),
    ("ffn_residual", (X, t(64, 32), t(32), t(32, 64), t(32)), "first bias"),
    ("ffn_residual", (X, t(64, 32), t(64), t(32, 64), t(16)), "second bias"),
    ("layernorm", (X, t(16), t(32), 1e-5), "gamma"),
    ("layernorm", (X, t(32), t(31), 1e-5), "beta"),
    ("fused_attention", (t(1, 128, 2, 1, 64, dtype=torch.bfloat16), 0.125), "positions, 3, heads"),
    ("fused_attention", (t(1, 128, 3, 64, dtype=torch.bfloat16), 0.125), "dimensions"),
    ("attention", (t(2, 8, 16, dtype=torch.bfloat16), t(2, 8, 16, dtype=torch.bfloat16), t(1, 8, 16, dtype=torch.bfloat16), 1.0), "one shape"),
    ("attention", (t(2, 8, 16), t(2, 8, 16), t(2, 8, 16), 1.0), "bf16"),
    ("conv", (IMG, nhwc(64, 32, 3, 3), None, 0, 1, 1, 15), "input channels"),
    ("conv", (IMG, t(64, 64), None, 0, 1, 1, 15), "dimensions"),
    ("conv", (IMG, nhwc(64, 64, 3, 3), t(32), 0, 1, 1, 15), "bias"),
    ("conv", (IMG, nhwc(64, 64, 3, 3), None, 1, 0, 0, 15), "1 x 1"),
    ("conv", (IMG, nhwc(64, 64, 1, 1), None, 2, 1, 1, 15), "3 x 3"),
    ("conv1x1", (IMG, nhwc(64, 32, 1, 1), None), "weight"),
    ("conv1x1", (IMG, nhwc(64, 64, 1, 1), t(32)), "bias"),
    ("batchnorm_act", (IMG, t(32), t(64), None, None, None, True, 0.1, 1e-5, False), "gamma"),
    ("batchnorm_act", (IMG, t(64), t(32), None, None, None, True, 0.1, 1e-5, False), "beta"),
    ("batchnorm_act", (IMG, t(64), t(64), t(32), t(64), None, True, 0.1, 1e-5, False), "running"),
    ("batchnorm_act", (IMG, t(64), t(64), t(64), t(64, dtype=torch.bfloat16), None, True, 0.1, 1e-5, False), "running"),
    ("batchnorm_act", (IMG, t(64), t(64), None, None, nhwc(2, 64, 8, 4), True, 0.1, 1e-5, False), "one shape"),
    ("batchnorm_act", (t(2, 64, 8, 8, dtype=torch.bfloat16), t(64), t(64), None, None, None, True, 0.1, 1e-5, False), "channels-last"),
]


@pytest.mark.parametrize("name,args,message", CASES, ids=[f"{n}-{m.replace(' ', '_')}-{i}" for i, (n, _, m) in enumerate(CASES)])
def test_operands_that_do_not_fit_are_refused(ext, name, args, message):
    with pytest.raises((RuntimeError, IndexError), match=message):
        getattr(ext, name)(*args)


@pytest.mark.parametrize("name,args", [
    ("linear", (X, t(16, 32), t(16), t(64, 16))),
    ("ffn_residual", (X, t(64, 32), t(64), t(32, 64), t(32))),
    ("layernorm", (X, t(32), t(32), 1e-5)),
    ("fused_attention", (t(1, 128, 3, 1, 64, dtype=torch.bfloat16), 0.125)),
    ("attention", (t(2, 8, 16, dtype=torch.bfloat16),) * 3 + (1.0,)),
    ("conv", (IMG, nhwc(64, 64, 3, 3), t(64), 0, 1, 1, 15)),
    ("conv1x1", (IMG, nhwc(64, 64, 1, 1), t(64))),
    ("conv1x1", (IMG, t(64, 64), None)),
    ("batchnorm_act", (IMG, t(64), t(64), t(64), t(64), IMG, True, 0.1, 1e-5, False)),
])
def test_operands_that_fit_get_as_far_as_the_device(ext, name, args):
    with pytest.raises(RuntimeError, match="(?i)cuda"):
        getattr(ext, name)(*args)


def test_tensors_without_memory_are_refused(ext):
    """A FakeTensor says it is on a GPU and has no address."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        x, w, f = (torch.empty(64, 128, device="cuda", dtype=d) for d in (torch.bfloat16, torch.float32, torch.float32))
        byte, index = torch.empty(512, device="cuda", dtype=torch.uint8), torch.empty(17, device="cuda", dtype=torch.int64)
    for call in (lambda: ext.linear(x, w, None, None), lambda: ext.layernorm(x, f[0], f[0], 1e-5),
                 lambda: ext.compress(f.view(-1), 32, 32, 64, -1074, 1, False), lambda: ext.compress(f, 1, 16658, 64, -10, 2, False),
                 lambda: ext.decompress(byte, None, 32, 32, 64, -1074, (64,), None, 0),
                 lambda: ext.decompress(torch.zeros(512, dtype=torch.uint8), None, 32, 32, 64, -1074, (64,), f.view(-1)[:64], 0),
                 lambda: ext.ar_launch(f, f, None, 0, 64, None, *[0] * 6, 1.0, *[0] * 7)):
        with pytest.raises(RuntimeError, match="FakeTensor"):
            call()


@pytest.mark.parametrize("rows,cols,ld,at,launches", [(64, 6144, 6144, 0, 1), (64, 6152, 6152, 0, 2), (64, 30528, 30528, 0, 2), (4096, 3072, 3072, 0, 1),
                                                      (4097, 3072, 3072, 0, 2), (64, 60, 64, 0, 2), (64, 64, 68, 0, 2), (64, 64, 64, 8, 2)])
def test_column_sums_take_one_launch_where_that_is_faster(ext, rows, cols, ld, at, launches):
    """Both sides of each line: rows, columns (whose clusters have to be resident together), multiples of eight, alignment."""
    import ctypes as C
    from gcow_b200 import _native
    f = _native.cuda().gcow_colsum_launches
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_int, C.c_int]
    assert f(4096 + at, rows, cols, ld) == launches
