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


# ---- precision: probabilities and sums are fp32 -------------------------------------------------------------------------
def half_ulp(v, dtype):
    bits = 10 if dtype == torch.float16 else 7
    return torch.exp2(torch.floor(torch.log2(v.abs().clamp_min(2.0 ** -14 if dtype == torch.float16 else 2.0 ** -126))) - bits - 1)


@pytest.mark.parametrize("m", [1, 17])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("dtype,gap", [(torch.float16, 22.3), (torch.float16, 24.3), (torch.bfloat16, 24.3), (torch.bfloat16, 60.0)])
def test_long_tails_of_small_probabilities(D, m, d, dtype, gap):
    """One key takes nearly all of the probability and has no value; tens of thousands of keys `gap` powers of two below it make
    the result.  Their probabilities keep 2^-13 of themselves (fp16: 2^-40 / 2^-24.3 at most, 65 000 equal errors add up), and the
    divisor the sums of whole tiles: beside half an ulp 2^-12 of the result is left."""
    n = 65536 - m if gap < 30 else 9000
    q = torch.zeros((1, m, 2, d), device=DEV); k = torch.zeros((1, n + m, 2, d), device=DEV)
    q[..., 0] = 16.0
    k[:, 3, :, 0] = gap * math.log(2.0) * math.sqrt(d) / 16.0
    v = torch.full((1, n + m, 2, d), 1.0 if gap < 30 else 3e12, device=DEV)
    v[:, 3] = 0.0
    q, k, v = (t.to(dtype) for t in (q, k, v))
    out = D.attention(q, k, v, n).double()
    s = 16.0 * k[0, 3, 0, 0].double() / math.sqrt(d)
    for i in range(m):
        tail = n + i
        ref = tail * v[0, 0, 0, 0].double() / (tail + torch.exp(s))
        assert ((out[0, i] - ref).abs() <= 1.02 * half_ulp(ref, dtype) + 2.0 ** -12 * ref).all(), (out[0, i, 0].item(), ref.item())


@pytest.mark.parametrize("m", [1, 17])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sums_that_cancel_keep_fp32_probabilities(D, dtype, d, m):
    """Values chosen so that the weighted sum nearly vanishes: what is left is the error of the probabilities and the sums.  fp32
    evaluation: exp2 and the scores within 2^-22 of p each, so an rms below 2^-21 of sum p |v| (two terms of bf16 alone: 2^-20.3)."""
    b, h, n = 32, 8, 8
    gen = torch.Generator().manual_seed(d + m)
    total = n + m
    q = (0.3 * torch.randn((b, m, h, d), generator=gen)).to(dtype)
    k = torch.randn((b, total, h, d), generator=gen).to(dtype)
    v = torch.randn((b, total, h, d), generator=gen).to(dtype).double().permute(0, 2, 1, 3).contiguous()
    p = torch.softmax(torch.einsum("bhd,bthd->bht", q[:, -1].double(), k.double()) / math.sqrt(d), dim=-1)
    order = p.argsort(dim=-1, descending=True)
    for j in (0, 1, 2, total // 2):                      # each takes away what is left, to the precision of the type
        t = order[..., j]
        pt = p.gather(-1, t[..., None])
        at = t[..., None, None].expand(-1, -1, 1, d)
        rest = torch.einsum("bht,bhtd->bhd", p, v) - pt * v.gather(2, at)[:, :, 0]
        v.scatter_(2, at, (-rest / pt).clamp(-200, 200).to(dtype).double()[:, :, None])
    exact_sum, size = torch.einsum("bht,bhtd->bhd", p, v), torch.einsum("bht,bhtd->bhd", p, v.abs())
    out = D.attention(q.to(DEV), k.to(DEV), v.permute(0, 2, 1, 3).contiguous().to(dtype).to(DEV), n).cpu().double().view(b, m, h, d)[:, -1]
    err = (out - exact_sum - 0.0).pow(2).mean().sqrt() / size.pow(2).mean().sqrt()
    assert err <= 2.0 ** -21, f"{err.item():.3g}"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("m", [1, 17])
def test_long_sums_do_not_drift(D, dtype, d, m):
    """8000 values of one sign, taken back by the last key: running sums that are rounded towards zero on every step lose 2^-15 of
    sum p |v|; sums of at most 128 keys, added in fp32, lose 2^-20 (a key tile's steps at 2^-23 each) plus 2^-21 for the scores of
    a key whose score is 9."""
    b, h, n = 2, 4, 8000
    gen = torch.Generator().manual_seed(d)
    total = n + m
    q = torch.randn((b, m, h, d), generator=gen).to(dtype).to(DEV)
    k = torch.randn((b, total, h, d), generator=gen).to(dtype).to(DEV)
    v = (0.5 + torch.rand((b, total, h, d), generator=gen)).to(dtype).to(DEV)
    q64 = q[:, -1].double()
    scores = lambda: torch.einsum("bhd,bthd->bht", q64, k.double()) / math.sqrt(d)
    lse = torch.logsumexp(scores()[..., :-1], dim=-1)
    k[:, -1] = (q64 * (lse * math.sqrt(d) / q64.pow(2).sum(dim=-1))[..., None]).to(dtype)      # half of the probability
    p = torch.softmax(scores(), dim=-1)
    v64 = v.double()
    for t in (total - 1, total - 2, total - 3):
        rest = torch.einsum("bht,bthd->bhd", p, v64) - p[..., t, None] * v64[:, t]
        v64[:, t] = (-rest / p[..., t, None]).clamp(-3000, 3000).to(dtype).double()
    exact_sum, size = torch.einsum("bht,bthd->bhd", p, v64), torch.einsum("bht,bthd->bhd", p, v64.abs())
    out = D.attention(q, k, v64.to(dtype), n).double().view(b, m, h, d)[:, -1]
    err = (out - exact_sum).pow(2).mean().sqrt() / size.pow(2).mean().sqrt()
    assert err <= 2.0 ** -20 + 2.0 ** -19, f"{err.item():.3g}"


# ---- infinities and NaN -------------------------------------------------------------------------------------------------
def same(out, ref, dtype):
    """Infinities and NaN where the reference has them; elsewhere half an ulp and 2^-12 of the largest finite value."""
    out = out.double()
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(out[torch.isinf(ref)], ref[torch.isinf(ref)])
    size = ref[fin].abs().max()
    assert ((out - ref)[fin].abs() <= 1.02 * half_ulp(ref[fin], dtype) + 2.0 ** -12 * size).all()


@pytest.mark.parametrize("m,hq,hkv,offs", [(2, 8, 2, [300, 63, 0]), (40, 8, 2, [100, 0]), (150, 4, 4, [7])])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_infinities_and_nan_reach_the_rows_that_see_them(D, dtype, d, m, hq, hkv, offs):
    """An infinite value under a positive probability is the result; a value or key that is not a number makes the rows that see it
    so, and no other: rows before it, in the same tile of rows, are what they are without it."""
    q, k, v, dev_offs = inputs(len(offs), m, hq, hkv, d, offs, dtype, seed=5)
    last = offs[0] + m - 1
    for value, where, t in ((math.inf, "v", 0), (-math.inf, "v", last), (math.nan, "v", last - m // 2), (math.nan, "k", last), (math.inf, "k", last - 1)):
        kk, vv = k.clone(), v.clone()
        (vv if where == "v" else kk)[0, t, 0, 5] = value
        same(D.attention(q, kk, vv, offsets=dev_offs), exact(q, kk, vv, offs), dtype)
    vv = v.clone()
    vv[0, 0, 0, 5], vv[0, min(1, last), 0, 5], vv[0, 0, 0, 6] = math.inf, -math.inf, 65000.0
    same(D.attention(q, k, vv, offsets=dev_offs), exact(q, k, vv, offs), dtype)
    qq = q.clone()
    qq[0, m - 1, 1, 3] = math.nan                       # one query of one head
    same(D.attention(qq, k, v, offsets=dev_offs), exact(qq, k, v, offs), dtype)
    torch.testing.assert_close(D.attention(q, k, v, offsets=dev_offs).double(), exact(q, k, v, offs), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("m", [1, 40])
def test_result_in_the_place_of_the_queries(D, m):
    """out may be the queries' own memory, with infinities too (such rows are evaluated a second time from q)."""
    q, k, v, offs = inputs(2, m, 8, 2, 128, [200, 31], seed=11)
    v[0, 3, 1, 7] = math.inf
    buf = q.clone()
    same(D.attention(buf, k, v, offsets=offs, out=buf.view(2, m, -1)), exact(q, k, v, [200, 31]), torch.float16)


# ---- ends of the arguments' ranges --------------------------------------------------------------------------------------
@pytest.mark.parametrize("m", [1, 20])
@pytest.mark.parametrize("scale", [-0.2, 0.0, 1e-42])
def test_any_scale(D, m, scale):
    """The C call takes any scale: below zero the largest score is the smallest product, at zero all keys weigh the same."""
    from minit_b200 import _lib
    q, k, v, offs = inputs(2, m, 8, 2, 128, [150, 64], seed=21)
    need = _lib.lib.mt_attention_batch_workspace_bytes(m, 8, 2, 128)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    out = torch.empty((2, m, 8 * 128), dtype=torch.float16, device=DEV)
    rc = _lib.lib.mt_attention_batch(_lib.current_stream(q.device), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), offs.data_ptr(),
                                     2, m, 8, 2, 128, 0, k.shape[1], scale, ws.data_ptr(), need, 0)
    assert rc == 0
    same(out, exact(q, k, v, [150, 64], scale), torch.float16)


@pytest.mark.parametrize("m", [2, 20])
@pytest.mark.parametrize("d", [64, 128])
def test_offsets_past_the_capacity(D, m, d):
    """A device offset of the capacity or more: every query sees the whole cache, and nothing behind it."""
    q, k, v, _ = inputs(3, m, 8, 2, d, [101 - m] * 3, seed=31)
    offs = [101, 5000, 101 - m]
    out = D.attention(q, k - 3.0, v, offsets=torch.tensor(offs, dtype=torch.int32, device=DEV))
    clamped = torch.cat([exact(q[s:s + 1, i:i + 1], k[s:s + 1] - 3.0, v[s:s + 1], [min(offs[s] + i, 100)]) for s in range(3) for i in range(m)], dim=1)
    same(out.view(1, 3 * m, -1), clamped, torch.float16)


# ---- routes that plain calls do not take --------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,hq,hkv,d", [(1, 8, 2, 128), (2, 8, 1, 64), (4, 4, 4, 128)])
def test_call_without_a_workspace(D, dtype, m, hq, hkv, d):
    """mt_attention, and mt_attention_batch with less than it asks for: up to 16 rows on the tile kernel."""
    from minit_b200 import _lib
    q, k, v, offs = inputs(3, m, hq, hkv, d, [130, 0, 63], dtype, seed=41)
    ref = exact(q, k, v, [130, 0, 63])
    for name, extra in (("mt_attention", ()), ("mt_attention_batch", (None, 0)), ("mt_attention_batch", (torch.zeros(4096, dtype=torch.uint8, device=DEV).data_ptr(), 4096))):
        out = torch.empty((3, m, hq * d), dtype=dtype, device=DEV)
        rc = getattr(_lib.lib, name)(_lib.current_stream(q.device), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), offs.data_ptr(),
                                     3, m, hq, hkv, d, 0, k.shape[1], 1.0 / math.sqrt(d), *extra, _lib.dtype_code(dtype))
        assert rc == 0
        same(out, ref, dtype)


@pytest.mark.parametrize("m", [1, 3])
def test_more_pairs_than_counters(D, m):
    """2049 sequences of 8 kv heads: whole (sequence, head) pairs per CTA, none of them cut."""
    b, hq, hkv, d, cap = 2049, 16, 8, 64, 70
    gen = torch.Generator(device=DEV).manual_seed(m)
    make = lambda *shape: torch.randn(shape, device=DEV, generator=gen).half()
    q, k, v = make(b, m, hq, d), make(b, cap, hkv, d), make(b, cap, hkv, d)
    lengths = torch.randint(0, cap - m + 1, (b,), device=DEV, generator=gen, dtype=torch.int32)
    out = D.attention(q, k, v, offsets=lengths).view(b, m, hq, d)
    s = torch.einsum("bmhgd,bthd->bmhgt", q.double().view(b, m, hkv, 2, d), k.double()) / math.sqrt(d)
    t = torch.arange(cap, device=DEV)
    seen = t.view(1, 1, cap) <= (lengths.view(b, 1, 1) + torch.arange(m, device=DEV).view(1, m, 1))
    p = torch.softmax(s.masked_fill(~seen[:, :, None, None, :], -math.inf), dim=-1)
    same(out, torch.einsum("bmhgt,bthd->bmhgd", p, v.double()).reshape(b, m, hq, d), torch.float16)
