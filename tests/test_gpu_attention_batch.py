"""decoder.attention beyond plain calls: captured graphs, large batches, calls without a workspace, values at the ends of the
types' ranges.  Reference: the expression in 64 bits (examples/llama3_70b.py:103-115)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def D(lib_built):
    from minit_b200 import decoder
    return decoder


def inputs(b, m, hq, hkv, d, offs, dtype=torch.float16, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed + d + m)
    cap = max(offs) + m
    make = lambda *shape: torch.randn(shape, device=DEV, generator=gen).to(dtype)
    return make(b, m, hq, d), make(b, cap, hkv, d), make(b, cap, hkv, d), torch.tensor(offs, dtype=torch.int32, device=DEV)


def exact(q, k, v, offs, scale=None):
    """The whole batch in fp64: [B, M, hq * d]; masked keys take no part, whatever they hold."""
    b, m, hq, d = q.shape
    group = hq // k.shape[2]
    scale = 1.0 / math.sqrt(d) if scale is None else scale
    out = torch.empty((b, m, hq, d), dtype=torch.float64, device=q.device)
    for s in range(b):
        for i in range(m):
            n = int(offs[s]) + i + 1
            kk, vv = (t[s, :n].double().repeat_interleave(group, dim=1) for t in (k, v))
            p = torch.softmax(torch.einsum("hd,thd->ht", q[s, i].double(), kk) * scale, dim=-1)
            out[s, i] = torch.einsum("ht,thd->hd", p, vv)
    return out.reshape(b, m, hq * d)


def test_graphs_on_one_stream_share_nothing(D):
    """Graphs captured on one stream hold no scratch of another call: replayed in reverse order, behind calls of other sizes whose
    scratch is freed and handed out again, and on two streams at once, they repeat the eager bits and write nowhere else."""
    a, b = inputs(3, 1, 8, 2, 64, [300, 1500, 40]), inputs(2, 2, 16, 2, 128, [2000, 700])
    side = torch.cuda.Stream()
    graphs, outs, refs = [], [], []
    with torch.cuda.stream(side):
        for x in (a, b):
            refs.append(D.attention(*x[:3], offsets=x[3]))
        torch.cuda.synchronize()
        for x in (a, b):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                outs.append(D.attention(*x[:3], offsets=x[3]))
            graphs.append(g)
        assert torch.equal(D.attention(*b[:3], offsets=b[3]), refs[1])
        filler = [torch.ones(n, dtype=torch.uint8, device=DEV) for n in (1 << 20, 1400000, 1400000, 2 << 20, 2600000, 2600000, 3 << 20)]
        for i in (1, 0):
            outs[i].zero_()
            graphs[i].replay()
    torch.cuda.synchronize()
    assert torch.equal(outs[0], refs[0]) and torch.equal(outs[1], refs[1])
    assert all(bool((f == 1).all()) for f in filler)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[0], refs[0]) and torch.equal(outs[1], refs[1])


def test_first_call_of_a_stream_inside_a_capture(D):
    """A capture that no call on its stream preceded leaves nothing behind that an eager call or another graph depends on."""
    x = inputs(4, 1, 8, 2, 128, [900, 20, 63, 1300], seed=3)
    ref = D.attention(*x[:3], offsets=x[3])
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    graphs, outs = [], []
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            outs.append(D.attention(*x[:3], offsets=x[3]))
        graphs.append(g)
    with torch.cuda.stream(side):
        assert torch.equal(D.attention(*x[:3], offsets=x[3]), ref)
        for i in (1, 0):
            outs[i].zero_()
            graphs[i].replay()
    torch.cuda.synchronize()
    assert torch.equal(outs[0], ref) and torch.equal(outs[1], ref)


@pytest.mark.parametrize("d,m,hq,hkv", [(64, 1, 8, 2), (128, 2, 16, 2)])
def test_scratch_may_hold_anything(D, d, m, hq, hkv):
    """The C call with a workspace full of ones, twice: the call clears what it counts in."""
    from minit_b200 import _lib
    q, k, v, offs = inputs(3, m, hq, hkv, d, [700, 5, 1200], seed=9)
    ref = D.attention(q, k, v, offsets=offs)
    need = _lib.lib.mt_attention_batch_workspace_bytes(m, hq, hkv, d)
    ws = torch.full((need,), 1, dtype=torch.uint8, device=DEV)
    for _ in range(2):
        out = torch.zeros_like(ref)
        rc = _lib.lib.mt_attention_batch(_lib.current_stream(q.device), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), offs.data_ptr(),
                                         3, m, hq, hkv, d, 0, k.shape[1], 1.0 / math.sqrt(d), ws.data_ptr(), need, 0)
        assert rc == 0 and torch.equal(out, ref)
