// Standalone GPTQ dequantisation: packed int4/int8 -> W[K,N] in fp16/bf16, bit-exact with
// the reference formula (minit/quantize/dispatch.py:14-20):
//     W = (T(q) - (T(z) + 1)) * s        evaluated in T
// q, z+1 and their difference are small integers, exactly representable in T, so the only
// rounding is the final multiply.  (q - z - 1) * s is computed here in fp32, where the
// product of a <=9-bit integer and an 11-bit (8-bit for bf16) significand is exact, and is
// then rounded once to T with round-to-nearest-even -- the same value the T multiply gives.
//
// HBM-bound: 2 bytes written per weight.  A lane owns 8 adjacent columns (16-byte stores, a warp writes 512 contiguous bytes
// of a row) and walks down packed rows; the arithmetic is on pairs of adjacent columns, two values per instruction, so that
// it hides behind the stores: int4 4096 x 14336 with a g_idx in 28.9 us = 5.1 TB/s (one value at a time in fp32, four columns
// per lane, g_idx read by every lane: 34.7 us).
#include "common.cuh"

namespace mt {

namespace {

// a pair of adjacent columns, packed: scale and zero + 1 in the form that the arithmetic of the type wants
template <int BITS, typename T> struct PairConst { uint32_t s, za, zb; float sf[2]; float zf[2]; };

template <int BITS, typename T>
__device__ __forceinline__ void pair_const(PairConst<BITS, T>& c, uint32_t s2, uint32_t zp1_lo, uint32_t zp1_hi) {
    using H = F16x2<T>;
    if constexpr (BITS == 8 && H::kIsBf16) {                      // 128 + b does not fit 8 bits: fp32, one rounding
        c.sf[0] = __uint_as_float(s2 << 16); c.sf[1] = __uint_as_float(s2 & 0xffff0000u);
        c.zf[0] = 8388608.f + float(zp1_lo); c.zf[1] = 8388608.f + float(zp1_hi);
    } else {
        const uint32_t z2 = zp1_lo | (zp1_hi << 16);
        c.s = s2;
        c.za = (H::kIsBf16 ? 0x43004300u : 0x64006400u) | z2;    // 128 + (z + 1) / 1024 + (z + 1): exact
        if constexpr (BITS == 4 && !H::kIsBf16) c.zb = H::sub(0x64006400u, 0x64006400u + 0x00400040u + z2);     // -(64 + z + 1): exact
    }
}

// Words of two adjacent columns -> PACK rows of two values.  The words' 16-bit halves are joined first (prmt), so that one
// mask leaves the same k of both columns in place.
template <int BITS, typename T>
__device__ __forceinline__ void expand_pair(uint32_t w0, uint32_t w1, const PairConst<BITS, T>& c, uint32_t (&o)[32 / BITS]) {
    using H = F16x2<T>;
    if constexpr (BITS == 4) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t v = prmt(w0, w1, h == 0 ? 0x5410u : 0x7632u);        // k 4h .. 4h + 3 of both columns
            if constexpr (!H::kIsBf16) {
                const uint32_t v8 = v >> 8;
                o[4 * h + 0] = H::mul(H::sub(and_or(v, 0x000f000fu, 0x64006400u), c.za), c.s);
                o[4 * h + 1] = H::mul(H::fma(and_or(v, 0x00f000f0u, 0x64006400u), 0x2c002c00u, c.zb), c.s);     // (1024 + 16 q) / 16 - 64 - (z + 1)
                o[4 * h + 2] = H::mul(H::sub(and_or(v8, 0x000f000fu, 0x64006400u), c.za), c.s);
                o[4 * h + 3] = H::mul(H::fma(and_or(v8, 0x00f000f0u, 0x64006400u), 0x2c002c00u, c.zb), c.s);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) o[4 * h + j] = H::mul(H::sub(and_or(v >> (4 * j), 0x000f000fu, 0x43004300u), c.za), c.s);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t b = prmt(w0, w1, uint32_t(j) | (uint32_t(4 + j) << 4));      // the byte of both columns
            if constexpr (!H::kIsBf16) o[j] = H::mul(H::sub(prmt(b, 0x64646464u, 0x4140u), c.za), c.s);
            else
                o[j] = H::pack((__uint_as_float(prmt(b, 0x4B000000u, 0x7540u)) - c.zf[0]) * c.sf[0],
                               (__uint_as_float(prmt(b, 0x4B000000u, 0x7541u)) - c.zf[1]) * c.sf[1]);
        }
    }
}

// constants of the 8 columns c .. c + 7 of group g
template <int BITS, typename T>
__device__ __forceinline__ void load_consts(PairConst<BITS, T> (&pc)[4], const uint32_t* __restrict__ qzeros, const T* __restrict__ scales, int g, int n, int c) {
    constexpr int PACK = 32 / BITS;
    constexpr uint32_t MASK = (1u << BITS) - 1u;
    const uint4 sv = __ldg(reinterpret_cast<const uint4*>(scales + (size_t)g * n + c));
    const uint32_t s[4] = {sv.x, sv.y, sv.z, sv.w};
    uint32_t z[2] = {0u, 0u};
    if (qzeros) {
        const uint32_t* zp = qzeros + (size_t)g * (n / PACK) + c / PACK;
        z[0] = __ldg(zp);
        if constexpr (BITS == 8) z[1] = __ldg(zp + 1);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t zw = BITS == 4 ? z[0] >> (8 * i) : z[i >> 1] >> (16 * (i & 1));
        pair_const<BITS, T>(pc[i], s[i], qzeros ? (zw & MASK) + 1u : 1u << (BITS - 1), qzeros ? ((zw >> BITS) & MASK) + 1u : 1u << (BITS - 1));
    }
}

constexpr int DQ_WARPS = 4, DQ_ROWS = 8;         // packed rows per warp: 64 (32) values of k, inside one group of 128

}  // namespace

// grid: (256-column windows, runs of DQ_WARPS * DQ_ROWS packed rows); TALL: more runs than the grid's y holds, over y and z, in an
// instance of its own (in one kernel for both, a first pass on cold memory took 50.3 us where it takes 46.3: 4096 x 14336).
// `pitch` is n in an argument of its own: with row addresses formed from n the kernel takes 31.3 us, 29.3 as it is.  A packed row whose
// values of k all belong to one group (contiguous groups, or a g_idx that is) uses one set of constants per group; a mixed
// row (act-order) fetches the constants of every k: a block's window of scales and zeros (20 KB for 32 groups) stays in L1.
template <int BITS, typename T, bool TALL>
__global__ void __launch_bounds__(DQ_WARPS * 32)
dequant_kernel(const uint32_t* __restrict__ qweight, const int32_t* __restrict__ g_idx,
               const uint32_t* __restrict__ qzeros, const T* __restrict__ scales,
               T* __restrict__ w_out, int n, int k, int groups, long long pitch) {
    constexpr int PACK = 32 / BITS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool live = (blockIdx.x * 32 + lane) * 8 < n;           // lanes past the last column stay for the warp's shuffles
    const int c = live ? (blockIdx.x * 32 + lane) * 8 : 0;
    const int kp = k / PACK, gs = k / groups;
    const int r0 = ((TALL ? blockIdx.z * gridDim.y + blockIdx.y : blockIdx.y) * DQ_WARPS + warp) * DQ_ROWS;
    if (TALL && r0 >= kp) return;                                 // whole warps
    PairConst<BITS, T> pc[4];
    int g_have = -1;
#pragma unroll
    for (int rb = 0; rb < DQ_ROWS; rb += 4) {
        uint4 w[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (r0 + rb + i < kp) {
                const uint32_t* src = qweight + (size_t)(r0 + rb + i) * n + c;
                w[i][0] = ldg_stream(src); w[i][1] = ldg_stream(src + 4);
            }
        // the groups of the 4 packed rows: one value of k per lane
        int gl = 0;
        {
            const int kk = (r0 + rb) * PACK + lane;               // TALL: past 2^31 it must not come out below k
            if (lane < 4 * PACK && (TALL ? unsigned(kk) < unsigned(k) : kk < k)) gl = g_idx ? min(max(__ldg(g_idx + kk), 0), groups - 1) : kk / gs;
        }
        const unsigned mixed = __ballot_sync(0xffffffffu, gl != __shfl_sync(0xffffffffu, gl, lane & ~(PACK - 1)));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pr = r0 + rb + i;
            if (pr >= kp) return;
            const int g0 = __shfl_sync(0xffffffffu, gl, i * PACK);
            const bool one = ((mixed >> (i * PACK)) & ((1u << PACK) - 1u)) == 0u;
            const uint32_t wv[8] = {w[i][0].x, w[i][0].y, w[i][0].z, w[i][0].w, w[i][1].x, w[i][1].y, w[i][1].z, w[i][1].w};
            T* dst = w_out + (size_t)pr * PACK * pitch + c;
            if (one) {
                if (g0 != g_have) { g_have = g0; load_consts<BITS, T>(pc, qzeros, scales, g_have, n, c); }
                uint32_t o[4][PACK];
#pragma unroll
                for (int q = 0; q < 4; ++q) expand_pair<BITS, T>(wv[2 * q], wv[2 * q + 1], pc[q], o[q]);
#pragma unroll
                for (int j = 0; j < PACK; ++j)
                    if (live) *reinterpret_cast<uint4*>(dst + (size_t)j * pitch) = make_uint4(o[0][j], o[1][j], o[2][j], o[3][j]);
            } else {
                g_have = -1;
#pragma unroll
                for (int j = 0; j < PACK; ++j) {
                    load_consts<BITS, T>(pc, qzeros, scales, __shfl_sync(0xffffffffu, gl, i * PACK + j), n, c);
                    uint32_t v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t o[PACK];
                        expand_pair<BITS, T>(wv[2 * q], wv[2 * q + 1], pc[q], o);       // only o[j] is used: the rest is dead code
                        v[q] = o[j];
                    }
                    if (live) *reinterpret_cast<uint4*>(dst + (size_t)j * pitch) = make_uint4(v[0], v[1], v[2], v[3]);
                }
            }
        }
    }
}

// One element per byte -> W.  Serves QuantizedTensor.dequantize() when the caller holds the
// unpacked tensors the reference's QuantizedTensor is built from (minit/quantize/tensor.py:9-30).
template <typename T>
__global__ void __launch_bounds__(256)
dequant_unpacked_kernel(const uint8_t* __restrict__ q, const int32_t* __restrict__ g_idx, const uint8_t* __restrict__ z,
                        const T* __restrict__ scales, T* __restrict__ w_out, int n, int k, int groups) {
    const int gs = k / groups;
    const long long total = (long long)k * (n >> 2);
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int kk = int(idx / (n >> 2));
        const int c = int(idx - (long long)kk * (n >> 2)) << 2;
        const int g = g_idx ? min(max(__ldg(g_idx + kk), 0), groups - 1) : kk / gs;
        const uint32_t qv = __ldg(reinterpret_cast<const uint32_t*>(q + (size_t)kk * n + c));
        const uint32_t zv = __ldg(reinterpret_cast<const uint32_t*>(z + (size_t)g * n + c));
        const uint2 sv = __ldg(reinterpret_cast<const uint2*>(scales + (size_t)g * n + c));
        const uint16_t sh[4] = {uint16_t(sv.x & 0xffff), uint16_t(sv.x >> 16), uint16_t(sv.y & 0xffff), uint16_t(sv.y >> 16)};
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = float(int((qv >> (8 * i)) & 0xffu) - int((zv >> (8 * i)) & 0xffu) - 1) * F16x2<T>::to_float(sh[i]);
        uint2 o; o.x = F16x2<T>::pack(v[0], v[1]); o.y = F16x2<T>::pack(v[2], v[3]);
        *reinterpret_cast<uint2*>(w_out + (size_t)kk * n + c) = o;
    }
}

// int32-packed -> one element per byte (the reference's unpack(), examples/qwen1_5_int8.py:40-50,
// generalised to 4-bit with the accessor formula of examples/qwen1_5_int8.py:97-138).
// axis 0: [R/pack, C] -> [R, C];  axis 1: [R, C/pack] -> [R, C].
template <int BITS>
__global__ void __launch_bounds__(256)
unpack_kernel(const uint32_t* __restrict__ packed, uint8_t* __restrict__ out, int rows, int cols, int axis) {
    constexpr int PACK = 32 / BITS;
    constexpr uint32_t MASK = (1u << BITS) - 1u;
    const long long total = (long long)rows * cols;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int r = int(idx / cols), c = int(idx - (long long)r * cols);
        uint32_t w; int j;
        if (axis == 0) { w = __ldg(packed + (size_t)(r / PACK) * cols + c); j = r % PACK; }
        else { w = __ldg(packed + (size_t)r * (cols / PACK) + c / PACK); j = c % PACK; }
        out[idx] = uint8_t((w >> (j * BITS)) & MASK);
    }
}

static unsigned grid_for(long long total) {
    long long blocks = (total + 255) / 256;
    const long long cap = 148LL * 32;
    return (unsigned)(blocks > cap ? cap : blocks);
}

int launch_dequant_unpacked(cudaStream_t st, const uint8_t* q, const int32_t* g_idx, const uint8_t* z, const void* scales,
                            void* w_out, int n, int k, int groups, int dtype) {
    const long long total = (long long)k * (n / 4);
    if (total == 0) return MT_OK;
    if (dtype == MT_F16)
        dequant_unpacked_kernel<__half><<<grid_for(total), 256, 0, st>>>(q, g_idx, z, reinterpret_cast<const __half*>(scales),
                                                                          reinterpret_cast<__half*>(w_out), n, k, groups);
    else
        dequant_unpacked_kernel<__nv_bfloat16><<<grid_for(total), 256, 0, st>>>(q, g_idx, z, reinterpret_cast<const __nv_bfloat16*>(scales),
                                                                                 reinterpret_cast<__nv_bfloat16*>(w_out), n, k, groups);
    return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_CUDA;
}

int launch_unpack(cudaStream_t st, const uint32_t* packed, uint8_t* out, int rows, int cols, int bits, int axis) {
    const long long total = (long long)rows * cols;
    if (total == 0) return MT_OK;
    if (bits == 4) unpack_kernel<4><<<grid_for(total), 256, 0, st>>>(packed, out, rows, cols, axis);
    else unpack_kernel<8><<<grid_for(total), 256, 0, st>>>(packed, out, rows, cols, axis);
    return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_CUDA;
}

int launch_dequant(cudaStream_t st, const uint32_t* qweight, const int32_t* g_idx, const uint32_t* qzeros,
                   const void* scales, void* w_out, int n, int k, int groups, int bits, int dtype) {
    const int pack = 32 / bits;
    if (n == 0 || k == 0) return MT_OK;
    const unsigned runs = (unsigned)((k / pack + DQ_WARPS * DQ_ROWS - 1) / (DQ_WARPS * DQ_ROWS)), ny = runs < 65535u ? runs : 65535u;
    const dim3 grid((n + 255) / 256, ny, (runs + ny - 1) / ny);
    auto go = [&](auto kern, auto* sc, auto* out) { kern<<<grid, DQ_WARPS * 32, 0, st>>>(qweight, g_idx, qzeros, sc, out, n, k, groups, n); };
#define MT_DQ(B, TT) go(grid.z > 1 ? dequant_kernel<B, TT, true> : dequant_kernel<B, TT, false>, reinterpret_cast<const TT*>(scales), reinterpret_cast<TT*>(w_out))
    if (bits == 4) { if (dtype == MT_F16) MT_DQ(4, __half); else MT_DQ(4, __nv_bfloat16); }
    else           { if (dtype == MT_F16) MT_DQ(8, __half); else MT_DQ(8, __nv_bfloat16); }
#undef MT_DQ
    return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_CUDA;
}

}  // namespace mt
