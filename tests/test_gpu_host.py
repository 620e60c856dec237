"""The native host calls (minit_b200._host) against the Python wrappers they shorten: same bits on the plain case, None (and
thus the wrapper's own errors) on everything else, and the caller's stream."""
import pytest
import torch

from oracle import qlinear_oracle as O
from tests.gpu_util import to_dev

DEV = "cuda:0"


def test_refuses_cpu_tensors_and_other_objects(lib_built):
    from minit_b200 import _lib
    x = torch.zeros((1, 64), dtype=torch.float16)
    q = torch.zeros((8, 64), dtype=torch.int32)
    s = torch.ones((1, 64), dtype=torch.float16)
    for bad in (x, None, 3, "x", q.numpy()):
        assert _lib._host.qgemm(bad, q, None, s, None, None, 4, 0) is None
        assert _lib._host.rms_norm(bad, s[0], 1e-5) is None
    assert _lib._host.attention_decode(x, x, x, 0) is None
    with pytest.raises(TypeError):
        _lib._host.qgemm(x, q)


def case(m, bits=4, dtype=torch.float16, act=False, n=512):
    c = O.make_gptq_case(1024, n, m, bits=bits, dtype=dtype, seed=m + bits, bias=True, act_order=act)
    return to_dev(c, DEV)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,dtype", [(4, torch.float16), (8, torch.bfloat16)])
@pytest.mark.parametrize("m", [1, 2, 3, 40, 300])
def test_linears_same_bits_as_the_wrappers(lib_built, m, bits, dtype):
    import minit_b200 as M
    from minit_b200 import _lib, feedforward as F
    d = case(m, bits, dtype)
    x, qw, qz, s, b = d["x"].view(1, m, -1), d["qweight"], d["qzeros"], d["scales"], d["bias"]
    out = torch.empty((1, m, 512), dtype=dtype, device=DEV)
    M.quantized_matrix_multiply(x, qw, qz, s, None, bits=bits, bias=b, out=out)          # sizes the workspace
    y = _lib._host.qgemm(x, qw, qz, s, None, b, bits, 0)
    assert y.shape == out.shape and torch.equal(y, out)
    r = torch.randn_like(out)
    F.quantized_matrix_multiply_residual(x, qw, qz, s, None, r, bits=bits, bias=b, out=out)
    assert torch.equal(_lib._host.qgemm_residual(x, qw, qz, s, None, r, b, bits, 0), out)
    half = torch.empty((1, m, 256), dtype=dtype, device=DEV)
    F.quantized_gate_up_swiglu(x, qw, qz, s, bits=bits, bias=b, out=half)
    assert torch.equal(_lib._host.qgemm_swiglu(x, qw, qz, s, b, bits, 0), half)
    a = case(m, bits, dtype, act=True)
    sq, perm = M.sort_act_order(a["qweight"], a["g_idx"], a["scales"].shape[0], bits)
    M.quantized_matrix_multiply_ordered(a["x"], sq, a["qzeros"], a["scales"], perm, bits=bits, out=out.view(m, -1))
    assert torch.equal(_lib._host.qgemm_ordered(a["x"], sq, a["qzeros"], a["scales"], perm, None, bits, 0), out.view(m, -1))


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 3])
def test_decoder_calls_same_bits(lib_built, m):
    from minit_b200 import _lib, decoder as D
    hq, hkv = 6, 1
    d = case(m, n=(hq + 2 * hkv) * 128)
    x, qw, qz, s = d["x"], d["qweight"], d["qzeros"], d["scales"]
    w = torch.rand(1024, device=DEV).half()
    assert torch.equal(_lib._host.rms_norm(x, w, 1e-5), D.rms_norm(x, w, 1e-5, out=torch.empty_like(x)))
    cos, sin = D.rope_tables(128, 64)
    zero = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = []
    for native in (True, False):
        torch.manual_seed(1)
        cache = D.KVCache(64, hkv, 128)
        cache.k.normal_(); cache.v.normal_()
        if native:
            D.qkv_rope_append(x, qw, qz, s, cos, sin, cache, hq, 9, bits=4)
            q = _lib._host.qkv_rope(x, qw, qz, s, None, cos, sin, cache.k, cache.v, hq, 9, 4, 0)
            D.attention_decode(q, cache, 9)
            y = _lib._host.attention_decode(q, cache.k, cache.v, 9)
        else:
            q = D.qkv_rope_append(x, qw, qz, s, cos, sin, cache, hq, 0, bits=4, offset_dev=zero + 9)
            y = D.attention_decode(q, cache, 9, out=torch.empty((m, hq * 128), dtype=q.dtype, device=DEV))
        got.append((q, cache.k, cache.v, y))
    for a, b in zip(*got):
        assert a is not None and torch.equal(a, b)


@pytest.mark.gpu
def test_everything_else_is_left_to_the_wrapper(lib_built):
    import minit_b200 as M
    from minit_b200 import _lib
    d = case(1)
    x, qw, qz, s = d["x"], d["qweight"], d["qzeros"], d["scales"]
    M.quantized_matrix_multiply(x, qw, qz, s, None, bits=4)
    f = _lib._host.qgemm
    assert f(x, qw, qz, s, None, None, 4, 0) is not None
    for args in ((x, qw, qz, s, None, None, 3, 0), (x[:, :512], qw, qz, s, None, None, 4, 0), (x.float(), qw, qz, s, None, None, 4, 0),
                 (x, qw, qz[:, :-1].contiguous(), s, None, None, 4, 0), (x, qw, qz, s.bfloat16(), None, None, 4, 0), (x[:0], qw, qz, s, None, None, 4, 0),
                 (x, qw, qz, s, qw[0], None, 4, 0), (x, qw, qz, s, None, s, 4, 0), (x, qw.t(), qz, s, None, None, 4, 0), (x, qw.cpu(), qz, s, None, None, 4, 0),
                 (x, qw, qz, s, None, None, 4.0, 0), (x, qw, qz, s, None, None, 4, 16 + 2 ** 40)):
        assert f(*args) is None
    with pytest.raises(ValueError):
        M.quantized_matrix_multiply(x, qw, qz, s.bfloat16(), None, bits=4)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert f(x, qw, qz, s, None, None, 4, 0) is None or (0, side.cuda_stream) in _lib._workspaces      # no workspace on a new stream yet
        a = M.quantized_matrix_multiply(x, qw, qz, s, None, bits=4)
        assert (0, side.cuda_stream) in _lib._workspaces
        b = f(x, qw, qz, s, None, None, 4, 0)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
    from torch.overrides import TorchFunctionMode
    with TorchFunctionMode():
        assert f(x, qw, qz, s, None, None, 4, 0) is None
    assert torch.func.vmap(lambda t: t * 2)(x) is not None and f(x, qw, qz, s, None, None, 4, 0) is not None


@pytest.mark.gpu
def test_graph_capture(lib_built):
    import minit_b200 as M
    d = case(1)
    args = (d["x"], d["qweight"], d["qzeros"], d["scales"], None)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ref = M.quantized_matrix_multiply(*args, bits=4)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            y = M.quantized_matrix_multiply(*args, bits=4)
        y.zero_()
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,hq,hkv,d", [(1, 8, 2, 128), (2, 4, 4, 64), (40, 8, 2, 128), (3, 4, 2, 96)])
def test_attention_same_bits_as_the_wrapper(lib_built, dtype, m, hq, hkv, d):
    from minit_b200 import _lib, decoder as D
    q = torch.randn((3, m, hq, d), device=DEV).to(dtype)
    k, v = (torch.randn((3, 200, hkv, d), device=DEV).to(dtype) for _ in range(2))
    offs = torch.tensor([150, 0, 64], dtype=torch.int32, device=DEV)
    f = _lib._host.attention
    for args, kw in (((q, k, v, 0, offs), dict(offsets=offs)), ((q, k, v, 100, None), dict(offset=100))):
        ref = D.attention(q, k, v, out=torch.empty((3, m, hq * d), dtype=dtype, device=DEV), **kw)
        y = f(*args)
        assert y.shape == ref.shape and torch.equal(y, ref) and torch.equal(D.attention(q, k, v, **kw), ref)
    for bad in ((q[0], k, v, 0, None), (q, k[:2], v[:2], 0, None), (q, k, v[:, :100], 0, None), (q, k.float(), v, 0, None), (q, k, v, 0, offs.long()),
                (q, k, v, 0, offs[:2]), (q, k, v, 200, None), (q, k, v, -1, None), (q, k, v, 0.0, None), (q[:, :0], k, v, 0, None), (q.cpu(), k, v, 0, None),
                (q, k.transpose(0, 1).contiguous().transpose(0, 1), v, 0, None)):
        assert f(*bad) is None
    with pytest.raises(Exception):
        D.attention(q, k, v, 200)
