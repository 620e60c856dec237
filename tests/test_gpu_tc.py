"""The tcgen05 prefill kernel (forced with MT_FLAG_FORCE_TC) through the C ABI against the oracle."""
import pytest
import torch

from oracle import qlinear_oracle as O
from tests.gpu_util import assert_close, oracle_out, to_dev

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def M(lib_built):
    import minit_b200
    return minit_b200


def run(M, c, bits, bias=None, flags=2):
    from minit_b200 import _lib
    d = to_dev(c, DEV)
    out = M.quantized_matrix_multiply(d["x"], d["qweight"], d["qzeros"], d["scales"], None, bits=bits,
                                      bias=None if bias is None else bias.to(DEV), flags=flags)
    torch.cuda.synchronize()
    for ws in _lib._workspaces.values():
        assert _lib.workspace_error_word(ws) == 0, "a bounded wait inside the tcgen05 kernel expired"
    return out


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [64, 128, 256, 300, 1000])
def test_tc_matches_oracle(M, bits, dtype, m):
    c = O.make_gptq_case(1024, 512, m, bits=bits, dtype=dtype, seed=m)
    assert_close(run(M, c, bits), oracle_out(c, False), f"tc bits={bits} {dtype} M={m}")


@pytest.mark.parametrize("k,n", [(64, 128), (192, 136), (4096, 6144), (2048, 1000)])
def test_tc_shapes_edges_bias(M, k, n):
    c = O.make_gptq_case(k, n, 260, bits=4, group_size=64, seed=k + n, bias=True)
    assert_close(run(M, c, 4, bias=c["bias"]), oracle_out(c, False, c["bias"]), f"tc {k}x{n}")


def test_tc_many_tiles_per_cta_and_both_accumulators(M):
    """More tiles than SMs so every persistent CTA loops and alternates its two TMEM accumulators."""
    c = O.make_gptq_case(512, 128 * 40, 2048, bits=4, seed=9)
    assert_close(run(M, c, 4), oracle_out(c, False), "tc 320 tiles")


def test_tc_is_the_default_above_64_rows(M):
    c = O.make_gptq_case(1024, 256, 200, bits=4, seed=2)
    assert_close(run(M, c, 4, flags=0), oracle_out(c, False), "default dispatch M=200")


def test_tc_prefill_shape_4096(M):
    """Prefill config: (K,N) = (4096, 6144), M = 4096, bf16; oracle on 3 row blocks to bound CPU time."""
    c = O.make_gptq_case(4096, 6144, 4096, bits=4, dtype=torch.bfloat16, seed=1)
    out = run(M, c, 4).cpu()
    w = O.dequantize_packed(c["qweight"], None, c["qzeros"], c["scales"], 4)
    for r0 in (0, 2000, 3968):
        assert_close(out[r0:r0 + 128], O.qlinear(c["x"][r0:r0 + 128], w), f"prefill rows {r0}")


# The prefill config's other shapes at every batch size it names, in both dtypes.  One case per
# (shape, dtype) is built at the largest M and its leading rows serve the smaller ones; the oracle
# checks three 128-row blocks of each output to bound CPU time.
_PREFILL_CASES = {}


def _prefill_case(k, n, dtype):
    key = (k, n, dtype)
    if key not in _PREFILL_CASES:
        _PREFILL_CASES.clear()                      # one resident case at a time (hundreds of MB each)
        c = O.make_gptq_case(k, n, 8192, bits=4, dtype=dtype, seed=k + n)
        c.pop("q"); c.pop("z")
        c["w"] = O.dequantize_packed(c["qweight"], None, c["qzeros"], c["scales"], 4)
        _PREFILL_CASES[key] = c
    return _PREFILL_CASES[key]


@pytest.mark.parametrize("m", [2048, 4096, 8192])       # the top decorator varies fastest: a case is built once
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k,n", [(4096, 28672), (14336, 4096)])
def test_tc_prefill_config_shapes(M, k, n, dtype, m):
    c = _prefill_case(k, n, dtype)
    d = {key: val for key, val in c.items() if key != "w"}
    d["x"] = c["x"][:m].contiguous()
    out = run(M, d, 4, flags=0).cpu()                 # default dispatch: what a caller of this config gets
    assert tuple(out.shape) == (m, n)
    for r0 in (0, m // 2 - 64, m - 128):
        assert_close(out[r0:r0 + 128], O.qlinear(d["x"][r0:r0 + 128], c["w"]), f"prefill {k}x{n} M={m} {dtype} rows {r0}")


TMEM_A = 2 | 256          # MT_FLAG_FORCE_TC | MT_FLAG_TC_TMEM_A: the 256 x 192 tile with the dequantized weights in tensor memory


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [129, 192, 193, 256, 400, 1000])
def test_tensor_memory_operand_variant_matches_oracle(M, dtype, m):
    """Row counts on both sides of the 192-row tile; K = 1024 gives 16 k-blocks, so both converter groups and both
    slots of A in tensor memory are reused."""
    c = O.make_gptq_case(1024, 512, m, bits=4, dtype=dtype, seed=m + 1)
    assert_close(run(M, c, 4, flags=TMEM_A), oracle_out(c, False), f"tensor-memory A {dtype} M={m}")


@pytest.mark.parametrize("k,n", [(64, 256), (192, 264), (4096, 6144), (2048, 1000), (448, 512)])
def test_tensor_memory_operand_variant_shapes_edges_bias(M, k, n):
    """One k-block, an odd number of k-blocks (the groups swap slots from tile to tile), ragged N, bias."""
    c = O.make_gptq_case(k, n, 260, bits=4, group_size=64, seed=k + n + 1, bias=True)
    assert_close(run(M, c, 4, bias=c["bias"], flags=TMEM_A), oracle_out(c, False, c["bias"]), f"tensor-memory A {k}x{n}")


def test_tensor_memory_operand_variant_many_tiles_per_cta(M):
    c = O.make_gptq_case(512, 256 * 24, 2048, bits=4, seed=10)
    assert_close(run(M, c, 4, flags=TMEM_A), oracle_out(c, False), "tensor-memory A, 264 tiles")


@pytest.mark.parametrize("k,n,m,dtype,bias", [(2048, 4096, 1920, torch.float16, False),     # 160 tiles: the last 12 are cut in 2 along K
                                              (4096, 4096, 1900, torch.bfloat16, True),     # cut in 4, ragged last row tile, bias
                                              (1024, 4352, 1728, torch.float16, False)])    # 153 tiles, 16 k-blocks: too short to cut
def test_last_wave_of_tiles_cut_along_k(M, k, n, m, dtype, bias):
    """More tiles than SMs with a small remainder: the remaining tiles are split along K, their fp32 partial tiles are
    added in part order by whichever part arrives last, and the workspace counters return to zero."""
    from minit_b200 import _lib
    c = O.make_gptq_case(k, n, m, bits=4, dtype=dtype, seed=k + n + m, bias=bias)
    b = c["bias"] if bias else None
    out1 = run(M, c, 4, bias=b, flags=TMEM_A)
    out2 = run(M, c, 4, bias=b, flags=TMEM_A)
    assert torch.equal(out1, out2), "the split tiles must not depend on which part arrives last"
    assert_close(out1, oracle_out(c, False, b), f"split last wave {k}x{n} M={m}")
    torch.cuda.synchronize()
    for ws in _lib._workspaces.values():
        assert int(ws[:_lib.COUNTER_BYTES].view(torch.int32).abs().sum().item()) == 0


@pytest.mark.parametrize("k,n", [(2048, 512), (8192, 1024), (1024, 4352), (512, 264)])
@pytest.mark.parametrize("m,dtype", [(3, torch.float16), (33, torch.float16), (64, torch.bfloat16)])
def test_tensor_memory_operand_variant_with_64_row_tiles(M, k, n, m, dtype):
    """Up to 64 rows the same kernel runs with 64-row tiles, every tile cut along K into parts that are added in part
    order (deep K: up to 8 parts; K = 512: no cut); results repeat bit for bit and the counters return to zero."""
    from minit_b200 import _lib
    c = O.make_gptq_case(k, n, m, bits=4, dtype=dtype, seed=k + n + m + 5, bias=True)
    out1 = run(M, c, 4, bias=c["bias"], flags=TMEM_A)
    out2 = run(M, c, 4, bias=c["bias"], flags=TMEM_A)
    assert torch.equal(out1, out2)
    assert_close(out1, oracle_out(c, False, c["bias"]), f"64-row tiles {k}x{n} M={m}")
    torch.cuda.synchronize()
    for ws in _lib._workspaces.values():
        assert int(ws[:_lib.COUNTER_BYTES].view(torch.int32).abs().sum().item()) == 0


@pytest.mark.parametrize("k,n", [(2048, 1024), (8192, 512), (1024, 4352)])
@pytest.mark.parametrize("m", [33, 64, 65, 100, 160, 161, 192])
def test_default_dispatch_33_to_192_rows(M, k, n, m):
    """mt_qgemm with no flags: 33 to 192 rows on int4 weights with contiguous groups go to one row of tiles (64, 160 or 192
    rows) of the tensor-memory-A kernel, every tile cut along K where that fills the GPU better."""
    c = O.make_gptq_case(k, n, m, bits=4, seed=k + n + m + 9, bias=True)
    out = run(M, c, 4, bias=c["bias"], flags=0)
    assert_close(out, oracle_out(c, False, c["bias"]), f"default dispatch {k}x{n} M={m}")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k,n,gs,m", [(64, 256, 64, 193), (1024, 264, 128, 129), (4160, 512, 64, 33), (4096, 512, 4096, 100),
                                      (2048, 1000, 128, 191), (1088, 520, 64, 400), (11008, 512, 11008, 512)])
def test_8_bit_weights_in_tensor_memory(M, k, n, gs, m, dtype):
    """8-bit weights on the tensor-memory tile (rings of odd length): one k-block, odd numbers of k-blocks, one group for all of
    K, ragged columns and rows, tiles cut along K; same bits every time, counters back at zero."""
    from minit_b200 import _lib
    c = O.make_gptq_case(k, n, m, bits=8, group_size=gs, dtype=dtype, seed=k + n + m, bias=True)
    out1, out2 = (run(M, c, 8, bias=c["bias"], flags=0) for _ in range(2))
    assert torch.equal(out1, out2)
    assert_close(out1, oracle_out(c, False, c["bias"]), f"8-bit {k}x{n} M={m} {dtype}")
    for ws in _lib._workspaces.values():
        assert int(ws[:_lib.COUNTER_BYTES].view(torch.int32).abs().sum().item()) == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("k,n,m", [(2048, 256, 193), (4096, 1000, 700), (1984, 512, 257), (960, 1024, 384)])
def test_fewer_tiles_than_sms_cut_along_k(M, k, n, m, bits):
    """Parts of unequal length (k-blocks not divisible by the parts), too few k-blocks to cut (960), ragged edges."""
    c = O.make_gptq_case(k, n, m, bits=bits, group_size=64, seed=k + m, bias=True)
    out1, out2 = (run(M, c, bits, bias=c["bias"], flags=0) for _ in range(2))
    assert torch.equal(out1, out2)
    assert_close(out1, oracle_out(c, False, c["bias"]), f"few tiles int{bits} {k}x{n} M={m}")


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("k,n,gs,m", [(2048, 264, 128, 17), (2176, 512, 128, 32), (4224, 1000, 128, 48), (8448, 256, 128, 64), (2112, 512, 64, 30)])
def test_turns_of_128_k_and_their_parts(M, k, n, gs, m, bits):
    """64-row tiles with turns of 128 k (64 where the groups are that short), cut into parts of unequal length; 17 to 32 rows by
    default dispatch; same bits every time, counters back at zero."""
    from minit_b200 import _lib
    c = O.make_gptq_case(k, n, m, bits=bits, group_size=gs, seed=k + n + m, bias=True)
    outs = [run(M, c, bits, bias=c["bias"], flags=f) for f in (0, 0, TMEM_A, TMEM_A | (5 << 16))]
    assert torch.equal(outs[0], outs[1])
    for out in outs:
        assert_close(out, oracle_out(c, False, c["bias"]), f"128-k turns int{bits} {k}x{n} M={m}")
    for ws in _lib._workspaces.values():
        assert int(ws[:_lib.COUNTER_BYTES].view(torch.int32).abs().sum().item()) == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("gs,m", [(128, 64), (64, 64), (64, 200), (192, 300)])
def test_scales_of_the_right_group_every_time(M, gs, m, bits):
    """One scale group per turn (128 k, or 64 k with groups of 64): the next group of a converter group is two further on, and
    its scales are prefetched while the previous ones are in use.  Many tiles, repeated: any late copy would change bits."""
    c = O.make_gptq_case(7680, 4096, m, bits=bits, group_size=gs, seed=gs + m)
    ref = run(M, c, bits, flags=0)
    assert_close(ref[:, :512], oracle_out(c, False)[:, :512], f"groups of {gs}, M={m}")
    d = to_dev(c, DEV)
    for _ in range(20):
        assert torch.equal(M.quantized_matrix_multiply(d["x"], d["qweight"], d["qzeros"], d["scales"], None, bits=bits), ref)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("k,n,m", [(8192, 19 * 256, 32), (8192, 19 * 256, 150), (4096, 1024, 17), (14336, 4096, 1000), (4096, 28672, 400), (11008, 4096, 192)])
def test_the_workspace_that_is_asked_for_is_enough(M, k, n, m, bits):
    """A C caller that brings exactly mt_workspace_bytes gets the same bits as one that brings more: the parts per tile are counted
    the same way where the size is asked for and where the kernel is launched."""
    from minit_b200 import _lib
    d = to_dev(O.make_gptq_case(k, n, m, bits=bits, seed=k + n + m), DEV)
    outs = []
    for extra in (0, 64 << 20):
        ws = torch.zeros(_lib.lib.mt_workspace_bytes(m, n, k, bits) + extra, dtype=torch.uint8, device=DEV)
        out = torch.zeros((m, n), dtype=torch.float16, device=DEV)
        rc = _lib.lib.mt_qgemm(_lib.current_stream(out.device), d["x"].data_ptr(), d["qweight"].data_ptr(), None, d["qzeros"].data_ptr(), d["scales"].data_ptr(),
                               None, out.data_ptr(), m, n, k, k // 128, bits, 0, ws.data_ptr(), ws.numel(), 0)
        assert rc == 0
        torch.cuda.synchronize()
        assert int(ws[:_lib.COUNTER_BYTES].view(torch.int32).abs().sum().item()) == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
