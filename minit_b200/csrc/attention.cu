// Attention of new tokens against a key / value cache for batches of sequences:
//   out[b, i, n, :] = softmax_t(q[b, i, n, :] . k[b, t, n / G, :] * scale, t <= offset_b + i) @ v[b, :, n / G, :]
// (examples/llama3_70b.py:103-115: scores for every (query, key) pair, -inf above the diagonal shifted by the cached
// positions, softmax over the keys, weighted sum of the values).  G = query heads per kv head.
//
// Two kernels for heads of 64 and 128, chosen by how many query rows share a kv head (m new tokens x G heads); other head
// sizes stay on attention_rows_kernel (decode_ops.cu), one warp per four query rows on the CUDA cores:
//
//  * attention_stream_kernel, up to 16 rows: reading the cache once is all there is to do (R rows give R flops per byte),
//    so the key tiles of all (sequence, kv head) pairs form one line that is cut into equal runs, one per SM: sequences of
//    different lengths keep every SM busy to the end.  mma.sync with the KEYS as the 16 rows and the query rows as the 8
//    columns: no tensor work is spent on padding a few query rows to 16.  32 sequences of 512 to 2048 positions, 32 query and
//    8 kv heads of 128, one token each: 46 us for 172 MB (3.8 TB/s; attention_rows_kernel 1880 us).
//  * attention_tile_kernel, more rows: tcgen05 tiles of 128 query rows x 64 keys (heads of 64: 128 keys), scores and
//    probabilities in tensor memory.  One sequence of 2000 new tokens, 32 / 8 heads of 128: fp16 92 us, bf16 108 us
//    (attention_rows_kernel 3360 us); 4096 tokens, 64 / 8 heads: fp16 612 us = 449 TFLOP/s of causal flops, bf16 745 us (25.8 ms).
//    Two terms of both types and sums kept in tensor memory took 71 and 445 us.  The line between the two lies at 16 rows:
//    with 32 and more the mma.sync pipe (an eighth of the tcgen05 rate) is slower than HBM.
//
// Scores, softmax and sums are fp32.  The tensor cores take 16-bit probabilities, so each is split into 16-bit terms that are all
// multiplied with V (split_terms): three of bf16, which hold an fp32 value exactly, or two of fp16, which hold it to one unit
// of its last place (2^-23 of p), and to 2^-40 of the row's largest.  The tensor cores round their running sums towards zero: a
// sum over thousands of keys would drift (8000 keys of one sign: 2.7e-5), so at most 128 keys are summed there and these sums are
// added in fp32.  What is left of sums that cancel, relative to
// sum p |v| (rms over cases of 9 to 417 keys): bf16 8e-9 to 1.6e-7, fp16 2e-8 to 1.4e-7; attention_rows_kernel 2e-8 to 3e-7 and
// 3e-8 to 3e-7; with two bf16 terms 1.4e-7 to 9e-7.
#include "tma.cuh"
#include "tcgen05.cuh"

namespace mt {

namespace {

__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ bool bar_or(int id, int threads, bool mine) {       // the barrier, and whether any thread said yes
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %3, 0;\nbarrier.cta.red.or.pred q, %1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(any) : "r"(id), "r"(threads), "r"(uint32_t(mine)) : "memory");
    return any != 0u;
}
__device__ __forceinline__ uint32_t movmatrix(uint32_t a) {
    uint32_t d; asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a)); return d; }

// Two probabilities -> the packed 16-bit terms of both, largest first.  fp16 takes them times 2^15 (the sums are scaled
// back by kUnscale): below 2^-14 an fp16 value loses bits, below 2^-25 it is zero, and a long tail of small probabilities would
// go with it.
constexpr float kScale = 32768.f;       // probabilities are at most 1
template <typename T> constexpr float kUnscale = F16x2<T>::kIsBf16 ? 1.f : 1.f / kScale;
template <typename T> constexpr int kTerms = F16x2<T>::kIsBf16 ? 3 : 2;
template <typename T>
__device__ __forceinline__ void split_terms(float a, float b, uint32_t (&t)[kTerms<T>]) {
    using H = F16x2<T>;
    if constexpr (H::kIsBf16) {                                     // cut after 8 bits, twice: 8 are left at most, and all terms are exact
        t[0] = prmt(__float_as_uint(a), __float_as_uint(b), 0x7632u);
        a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u); b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
        t[1] = prmt(__float_as_uint(a), __float_as_uint(b), 0x7632u);
        a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u); b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
        t[2] = prmt(__float_as_uint(a), __float_as_uint(b), 0x7632u);
    } else {
        a *= kScale; b *= kScale;
        t[0] = H::pack(a, b);
        t[1] = H::pack(a - H::to_float(uint16_t(t[0] & 0xffff)), b - H::to_float(uint16_t(t[0] >> 16)));
    }
}

// Set to 8 by a kernel of this file whose wait ran out, read by mt_attention_error.  One word per device, in the module itself: calls
// without a workspace and calls whose scratch is gone by the time the host looks report here too.
__device__ unsigned g_attention_error;

// 32 lanes x 16 columns of tensor memory
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// One output row in fp32 on the CUDA cores, by a warp (the arithmetic of attention_rows_kernel for one query): lane i returns values
// D / 32 * i onwards.  For rows whose sums came out infinite or NaN: the tensor cores multiply every value of a key tile, so an
// infinity or NaN that a row does not see meets its zero probabilities, and one that it sees meets zero or negative small terms.
// Here masked keys take no part and a probability is one number: an infinity stays one, and reaches the rows that see it.
// Out of line: sound inputs never come here, and their sums are checked once per output value.
template <typename T, int D>
__device__ __noinline__ void attention_row(const uint16_t* q, const uint16_t* k, const uint16_t* v, size_t pitch, int keys, float scale, float (&o)[D / 32]) {
    using H = F16x2<T>;
    constexpr int E = D / 32;
    const int lane = threadIdx.x & 31;
    float mx = -INFINITY, l = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) o[e] = 0.f;
    for (int t0 = 0; t0 < keys; t0 += 32) {
        const int t = t0 + lane;
        float sc = -INFINITY;
        if (t < keys) {
            const uint16_t* kr = k + (size_t)t * pitch;
            sc = 0.f;
            for (int c = 0; c < D; ++c) sc = fmaf(H::to_float(q[c]) * scale, H::to_float(kr[c]), sc);
        }
        float bm = sc;
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, x));
        const float mn = fmaxf(mx, bm);
        const float corr = mn == -INFINITY ? 1.f : __expf(mx - mn), pr = t < keys ? __expf(sc - mn) : 0.f;
        float ps = pr;
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, x);
        l = l * corr + ps;
        mx = mn;
#pragma unroll
        for (int e = 0; e < E; ++e) o[e] *= corr;
        const int cnt = min(32, keys - t0);
        for (int j = 0; j < cnt; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pr, j);
            const uint16_t* vr = v + (size_t)(t0 + j) * pitch + lane * E;
#pragma unroll
            for (int e = 0; e < E; ++e) o[e] = fmaf(pj, H::to_float(vr[e]), o[e]);
        }
    }
    const float inv = 1.f / l;
#pragma unroll
    for (int e = 0; e < E; ++e) o[e] *= inv;
}

// On a wait that ran out: give the copies in flight time to land before the shared memory is given up.
__device__ __forceinline__ void drain_copies() { for (int i = 0; i < 1000; ++i) __nanosleep(1000); }

// ------------------------------------------------------------------------------------------------------------
// up to 16 query rows per kv head
// ------------------------------------------------------------------------------------------------------------
constexpr int AS_KEYS = 64;             // keys per tile
constexpr int AS_WARPS = 8;             // consuming warps: two groups of four take alternate tiles, a warp 16 keys of its tile
constexpr int AS_THREADS = (AS_WARPS + 2) * 32;
// Scratch of one call: word 0 is the error word, then an arrival counter per (sequence, kv head), then the runs' partial rows.
// Every call zeroes its counters (attention_zero_kernel): it relies on nothing that an earlier one left (a captured graph may
// be replayed in any order with others, and an aborted call may leave counts behind).
constexpr size_t AS_HEAD = 256;
constexpr int AS_MAX_SEGMENTS = 16384;                              // counters; more segments than that are never split
constexpr size_t AS_PART_OFF = AS_HEAD + (size_t)AS_MAX_SEGMENTS * 4;

struct StreamParams {
    const void *q, *k, *v; void* out;
    const int* offsets;         // [batch] or null: `offset` for all
    unsigned char* ws;
    int batch, m, hq, hkv, group, offset, capacity;
    int whole;                  // 1: a (sequence, kv head) pair is never cut (no workspace counters)
    float scale, c;             // c: scale * log2(e)
};

template <int D, int NT> struct StreamCfg {
    static constexpr int TILE_BYTES = AS_KEYS * D * 2;
    static constexpr int ROWS = NT * 8;
    static constexpr int PITCH = D + 4;                             // floats per merged row: D sums, max, sum, pad (16-byte rows)
    static constexpr int MERGE_BYTES = AS_WARPS * ROWS * PITCH * 4;
    // even, so that a stage always belongs to the same group of warps: a group that saw only every second phase of a
    // stage's barriers could pass a parity wait one phase early
    static constexpr int STAGES = NT == 1 ? 6 : 4;
    static_assert(STAGES % 2 == 0, "a consumer must walk every phase of the barriers it waits on");
    static constexpr int SMEM = STAGES * 2 * TILE_BYTES + MERGE_BYTES + 1024;
};

// keys of sequence b that any of its rows sees
__device__ __forceinline__ int stream_keys(const StreamParams& p, int b) {
    const int off = p.offsets ? __ldg(p.offsets + b) : p.offset;
    return max(1, min(off + p.m, p.capacity));
}
__device__ __forceinline__ int stream_tiles(const StreamParams& p, int b) { return (stream_keys(p, b) + AS_KEYS - 1) / AS_KEYS; }

// The stream kernel is launched programmatically behind this one and looks at the counters at the end of its first segment:
// 32 sequences of 512 to 2048 positions 0.2 us longer than with counters kept between calls, a memset 1.7.
__global__ void attention_zero_kernel(unsigned* counters, int n) {
    griddep_launch_dependents();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) counters[i] = 0u;
}

// all rows of pair (b, h) once more, spread over the consuming warps
template <typename T, int D>
__device__ __noinline__ void stream_rows(const StreamParams* p, int b, int h) {
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < p->m * p->group; r += AS_WARPS) {
        const int i = r / p->group;
        const size_t row = (((size_t)b * p->m + i) * p->hq + (size_t)h * p->group + (r - i * p->group)) * D;
        const size_t cache = ((size_t)b * p->capacity * p->hkv + h) * D;
        float o[D / 32];
        attention_row<T, D>(reinterpret_cast<const uint16_t*>(p->q) + row, reinterpret_cast<const uint16_t*>(p->k) + cache,
                            reinterpret_cast<const uint16_t*>(p->v) + cache, (size_t)p->hkv * D,
                            min((p->offsets ? __ldg(p->offsets + b) : p->offset) + i + 1, p->capacity), p->scale, o);
#pragma unroll
        for (int e = 0; e < D / 32; ++e) reinterpret_cast<uint16_t*>(p->out)[row + lane * (D / 32) + e] = F16x2<T>::from_float(o[e]);
    }
}

// Bound by HBM: one SM has to take 43 KB/us to keep up with its share, and holds six 32 KB stages in flight for that.
// Two warps issue the copies (one K, one V: one thread alone issues about four bulk copies per microsecond).
template <typename T, int D, int NT>
__global__ void __launch_bounds__(AS_THREADS, 1)
attention_stream_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv, const __grid_constant__ StreamParams p) {
    using H = F16x2<T>;
    using C = StreamCfg<D, NT>;
    constexpr int STAGES = C::STAGES, TB = C::TILE_BYTES;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[4 * STAGES];
    __shared__ int s_start[4];                                      // first sequence, head, tile of this CTA's run, number of units
    __shared__ long long s_span[2];                                 // first unit of the first segment, units per CTA
    __shared__ int s_abort, s_last, s_stop;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const uint32_t sbase = smem_u32(smem);
    float* merge = reinterpret_cast<float*>(smem + STAGES * 2 * TB);
    const uint32_t kfull = smem_u32(bars), vfull = kfull + 8 * STAGES, kempty = vfull + 8 * STAGES, vempty = kempty + 8 * STAGES;
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(kfull + 8 * i, 1); mbar_init(vfull + 8 * i, 1);
            mbar_init(kempty + 8 * i, 4); mbar_init(vempty + 8 * i, 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // ---- where this CTA's run starts: units are (sequence, kv head, tile) in that order ----
    if (warp == 0) {
        long long units = 0;
        if (p.offsets == nullptr) units = (long long)p.batch * stream_tiles(p, 0);
        else {
            for (int b = lane; b < p.batch; b += 32) units += stream_tiles(p, b);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) units += __shfl_xor_sync(0xffffffffu, units, o);
        }
        units *= p.hkv;
        long long per = (units + gridDim.x - 1) / gridDim.x, u0, seg0 = 0;
        int b0 = -1, h0 = 0, t0 = 0, count = 0;
        if (p.whole) {                                              // whole pairs: an equal number of them per CTA
            const long long segs = (long long)p.batch * p.hkv, sper = (segs + gridDim.x - 1) / gridDim.x;
            const long long sg0 = blockIdx.x * sper, sg1 = min(segs, sg0 + sper);
            for (long long sg = sg0 + lane; sg < sg1; sg += 32) count += stream_tiles(p, int(sg / p.hkv));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
            if (sg0 < sg1) { b0 = int(sg0 / p.hkv); h0 = int(sg0 % p.hkv); }
        } else {
            u0 = blockIdx.x * per;
            count = int(max(0LL, min(units, u0 + per) - u0));
            if (count > 0) {
                long long base = 0;
                for (int c0 = 0; c0 < p.batch && b0 < 0; c0 += 32) {
                    const int b = c0 + lane;
                    const long long n = b < p.batch ? (long long)stream_tiles(p, b) * p.hkv : 0;
                    long long incl = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { const long long v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
                    const unsigned hit = __ballot_sync(0xffffffffu, n > 0 && base + incl > u0);
                    if (hit) {
                        const int src = __ffs(hit) - 1;
                        const long long before = __shfl_sync(0xffffffffu, base + incl - n, src);
                        b0 = c0 + src;
                        const int tiles = stream_tiles(p, b0), rel = int(u0 - before);
                        h0 = rel / tiles; t0 = rel % tiles;
                        seg0 = before + (long long)h0 * tiles;
                    }
                    base += __shfl_sync(0xffffffffu, incl, 31);
                }
            }
        }
        if (lane == 0) { s_start[0] = b0; s_start[1] = h0; s_start[2] = t0; s_start[3] = count; s_span[0] = seg0; s_span[1] = per; }
    }
    __syncthreads();
    int b = s_start[0], h = s_start[1], t = s_start[2];
    const int count = s_start[3];

    if (warp >= AS_WARPS) {
        // ---- producers: warp 8 the keys, warp 9 the values ----
        if (lane == 0 && count > 0) {
            const bool keys = warp == AS_WARPS;
            const CUtensorMap* map = keys ? &mk : &mv;
            const uint32_t full = keys ? kfull : vfull, empty = keys ? kempty : vempty, dst = sbase + (keys ? 0 : TB);
            int tiles = stream_tiles(p, b), stage = 0;
            uint32_t phase = 1;                                     // the first turn finds every stage empty
            bool ok = true;
            for (int i = 0; i < count && ok; ++i) {
                ok = mbar_wait_sleep<32>(empty + 8 * stage, phase, abort_flag);
                if (!ok) break;
                mbar_expect_tx(full + 8 * stage, TB);
                tma_load_5d(dst + stage * 2 * TB, map, 0, t * AS_KEYS, 0, h, b, full + 8 * stage);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
                if (++t == tiles) { t = 0; if (++h == p.hkv) { h = 0; ++b; if (b < p.batch) tiles = stream_tiles(p, b); } }
            }
            if (!ok) drain_copies();
        }
        __syncwarp();
    } else if (count > 0) {
        const int grp = warp >> 2, wq = warp & 3, g = lane >> 2, tq = lane & 3;
        const int lm = lane >> 3, lr = lane & 7;
        const int R = p.m * p.group;
        // this lane's ldmatrix rows: keys as MMA rows (K) and values transposed (V)
        const int krow = 16 * wq + (lm & 1) * 8 + lr, vrow = 16 * wq + (lm >> 1) * 8 + lr;
        long long seg_first = s_span[0];
        const long long per = s_span[1];
        int stage = 0;
        uint32_t phase = 0;
        int i = 0;
        bool ok = true;
        while (i < count && ok) {
            // ---- one segment: the tiles of (b, h) that fall into this CTA's run ----
            const int keys = stream_keys(p, b), tiles = (keys + AS_KEYS - 1) / AS_KEYS;
            const int off = p.offsets ? __ldg(p.offsets + b) : p.offset;
            const int n = min(tiles - t, count - i);
            uint32_t qf[NT][D / 16][2];                             // B fragments of Q^T: (d = 16 ks + 2 tq, +1), (.. + 8) of row 8 nt + g
            int lim[NT][2];                                         // keys that this lane's two columns see
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int r = 8 * nt + g, mi = r / p.group;
                const uint32_t* q32 = reinterpret_cast<const uint32_t*>(p.q) +
                                      (((size_t)b * p.m + mi) * p.hq + (size_t)h * p.group + (r - mi * p.group)) * (D / 2);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    qf[nt][ks][0] = r < R ? __ldg(q32 + 8 * ks + tq) : 0u;
                    qf[nt][ks][1] = r < R ? __ldg(q32 + 8 * ks + 4 + tq) : 0u;
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) lim[nt][e] = min(off + min(8 * nt + 2 * tq + e, R - 1) / p.group + 1, keys);
            }
            float mx[NT][2], ls[NT][2], oc[NT][D / 16][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                mx[nt][0] = mx[nt][1] = -INFINITY; ls[nt][0] = ls[nt][1] = 0.f;
#pragma unroll
                for (int j = 0; j < D / 16; ++j) oc[nt][j][0] = oc[nt][j][1] = oc[nt][j][2] = oc[nt][j][3] = 0.f;
            }
            for (int u = 0; u < n; ++u, ++i, ++t) {
                const int st = stage; const uint32_t ph = phase;
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
                if ((i & 1) != grp) continue;                       // the other group's tile
                const uint32_t ka = sbase + st * 2 * TB, va = ka + TB;
                if (!mbar_wait(kfull + 8 * st, ph, abort_flag)) { ok = false; break; }
                float sc[NT][4];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    uint32_t a0, a1, a2, a3;
                    const int chunk = 2 * ks + (lm >> 1);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                                 : "r"(ka + (chunk >> 3) * (AS_KEYS * 128) + krow * 128 + (((chunk & 7) ^ (krow & 7)) << 4)));
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) mma16816<T>(sc[nt], a0, a1, a2, a3, qf[nt][ks][0], qf[nt][ks][1]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(kempty + 8 * st);
                const int key0 = t * AS_KEYS + 16 * wq + g;         // keys of this lane: key0 (registers 0, 1) and key0 + 8 (2, 3)
                uint32_t pt[NT][2][kTerms<T>];                      // B fragments of the probabilities
                if (t * AS_KEYS + AS_KEYS > min(off + 1, keys)) {   // a tile that some row does not see whole, or that ends behind the cache
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (key0 >= lim[nt][e]) sc[nt][e] = -INFINITY;
                            if (key0 + 8 >= lim[nt][e]) sc[nt][2 + e] = -INFINITY;
                        }
                }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float nm[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float v = fmaxf(sc[nt][e], sc[nt][2 + e]);
                        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
                        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
                        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
                        nm[e] = fmaxf(mx[nt][e], v);
                    }
                    if (__any_sync(0xffffffffu, nm[0] > mx[nt][0] || nm[1] > mx[nt][1])) {
                        float f[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            f[e] = mx[nt][e] == -INFINITY ? 0.f : ex2((mx[nt][e] - nm[e]) * p.c);
                            mx[nt][e] = nm[e];
                            ls[nt][e] *= f[e];
                        }
#pragma unroll
                        for (int j = 0; j < D / 16; ++j) { oc[nt][j][0] *= f[0]; oc[nt][j][1] *= f[1]; oc[nt][j][2] *= f[0]; oc[nt][j][3] *= f[1]; }
                    }
                    float pr[4];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float base = mx[nt][e] == -INFINITY ? 0.f : mx[nt][e] * p.c;      // nothing seen yet: every score is -inf
                        pr[e] = ex2(fmaf(sc[nt][e], p.c, -base));
                        pr[2 + e] = ex2(fmaf(sc[nt][2 + e], p.c, -base));
                        ls[nt][e] += pr[e] + pr[2 + e];
                    }
#pragma unroll
                    for (int k2 = 0; k2 < 2; ++k2) {
                        split_terms<T>(pr[2 * k2], pr[2 * k2 + 1], pt[nt][k2]);
#pragma unroll
                        for (int x = 0; x < kTerms<T>; ++x) pt[nt][k2][x] = movmatrix(pt[nt][k2][x]);      // (key, row) tile -> B fragment
                    }
                }
                if (!mbar_wait(vfull + 8 * st, ph, abort_flag)) { ok = false; break; }
                const bool tail = t * AS_KEYS + AS_KEYS > keys;
                if (tail) {
                    // rows behind the last key may hold anything (a NaN times a zero probability is a NaN): clear them
                    for (int r = 0; r < 16; ++r) {
                        const int key = 16 * wq + r;
                        if (t * AS_KEYS + key >= keys)
                            for (int c = lane; c < D / 8; c += 32)
                                asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(va + (c >> 3) * (AS_KEYS * 128) + key * 128 + ((c & 7) << 4)), "r"(0u) : "memory");
                    }
                    fence_proxy_async();
                    __syncwarp();
                }
#pragma unroll
                for (int j = 0; j < D / 16; ++j) {
                    uint32_t a0, a1, a2, a3;
                    const int chunk = 2 * j + (lm & 1);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                                 : "r"(va + (chunk >> 3) * (AS_KEYS * 128) + vrow * 128 + (((chunk & 7) ^ (vrow & 7)) << 4)));
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        float add[4] = {0.f, 0.f, 0.f, 0.f};        // small terms first, the running sum in fp32 outside the tensor core
#pragma unroll
                        for (int x = kTerms<T> - 1; x >= 0; --x) mma16816<T>(add, a0, a1, a2, a3, pt[nt][0][x], pt[nt][1][x]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) oc[nt][j][e] += add[e];
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(vempty + 8 * st);
            }
            // ---- merge the warps (in warp order), then the CTAs of the segment (in CTA order) ----
            if (!ok) *abort_flag = 1;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float v = ls[nt][e];
                    v += __shfl_xor_sync(0xffffffffu, v, 4);
                    v += __shfl_xor_sync(0xffffffffu, v, 8);
                    v += __shfl_xor_sync(0xffffffffu, v, 16);
                    float* row = merge + ((size_t)warp * C::ROWS + 8 * nt + 2 * tq + e) * C::PITCH;
                    if (g == 0) { row[D] = mx[nt][e]; row[D + 1] = v; }
#pragma unroll
                    for (int j = 0; j < D / 16; ++j) { row[16 * j + g] = oc[nt][j][e] * kUnscale<T>; row[16 * j + 8 + g] = oc[nt][j][2 + e] * kUnscale<T>; }
                }
            bar_sync(1, AS_WARPS * 32);
            const bool whole = n == tiles;
            const long long c_first = whole ? 0 : seg_first / per, c_last = whole ? 0 : (seg_first + tiles - 1) / per;
            auto slot = [&](long long cta) {                        // a CTA's partial of this segment: 0 when its run starts in it, else 1
                return reinterpret_cast<float*>(p.ws + AS_PART_OFF) + ((size_t)cta * 2 + (cta * per >= seg_first ? 0 : 1)) * C::ROWS * C::PITCH;
            };
            float zero = 0.f;                                       // stays so unless a stored value is infinite or NaN
            auto store = [&](int r, int d, float l, float a) {
                const int mi = r / p.group;
                const float v = a / l;
                zero = fmaf(v, 0.f, zero);
                reinterpret_cast<uint16_t*>(p.out)[(((size_t)b * p.m + mi) * p.hq + (size_t)h * p.group + (r - mi * p.group)) * D + d] = H::from_float(v);
            };
            for (int e = tid; e < R * D; e += AS_WARPS * 32) {
                const int r = e / D, d = e % D;
                float m_all = -INFINITY, l_all = 0.f, a_all = 0.f;
#pragma unroll
                for (int w = 0; w < AS_WARPS; ++w) m_all = fmaxf(m_all, merge[((size_t)w * C::ROWS + r) * C::PITCH + D]);
#pragma unroll
                for (int w = 0; w < AS_WARPS; ++w) {
                    const float* row = merge + ((size_t)w * C::ROWS + r) * C::PITCH;
                    const float f = row[D] == -INFINITY ? 0.f : ex2((row[D] - m_all) * p.c);
                    l_all = fmaf(row[D + 1], f, l_all);
                    a_all = fmaf(row[d], f, a_all);
                }
                if (whole) store(r, d, l_all, a_all);
                else {
                    float* dst = slot(blockIdx.x) + r * C::PITCH;
                    __stcg(dst + d, a_all);
                    if (d == 0) { __stcg(dst + D, m_all); __stcg(dst + D + 1, l_all); }
                }
            }
            if (!whole) {
                unsigned* counter = reinterpret_cast<unsigned*>(p.ws + AS_HEAD) + (size_t)b * p.hkv + h;
                griddep_wait();                                     // the counters are zeroed
                __threadfence();
                bar_sync(1, AS_WARPS * 32);
                if (tid == 0) s_last = atomicAdd(counter, 1u) == unsigned(c_last - c_first);
                bar_sync(1, AS_WARPS * 32);
                if (s_last) {
                    __threadfence();
                    for (int e = tid; e < R * D; e += AS_WARPS * 32) {
                        const int r = e / D, d = e % D;
                        float m_all = -INFINITY, l_all = 0.f, a_all = 0.f;
#pragma unroll 4
                        for (long long c = c_first; c <= c_last; ++c) m_all = fmaxf(m_all, __ldcg(slot(c) + r * C::PITCH + D));
#pragma unroll 4
                        for (long long c = c_first; c <= c_last; ++c) {
                            const float* row = slot(c) + r * C::PITCH;
                            const float mc = __ldcg(row + D);
                            const float f = mc == -INFINITY ? 0.f : ex2((mc - m_all) * p.c);
                            l_all = fmaf(__ldcg(row + D + 1), f, l_all);
                            a_all = fmaf(__ldcg(row + d), f, a_all);
                        }
                        store(r, d, l_all, a_all);
                    }
                }
            }
            if (tid == 0) s_stop = *abort_flag;                     // one answer for all warps: they leave the loop together
            if (bar_or(1, AS_WARPS * 32, !(zero == 0.f))) stream_rows<T, D>(&p, b, h);      // the merge rows are free again
            ok = s_stop == 0;
            seg_first += tiles;
            t = 0;
            if (++h == p.hkv) { h = 0; ++b; }
        }
    }
    griddep_wait();                                                 // in every CTA: this grid never ends before the zeroing one
    __syncthreads();
    if (tid == 0 && s_abort) {
        g_attention_error = 8u;
        *reinterpret_cast<unsigned*>(p.ws) = 8u;
    }
}

// ------------------------------------------------------------------------------------------------------------
// more rows: tcgen05 tiles
// ------------------------------------------------------------------------------------------------------------
constexpr int AT_THREADS = 384;

struct TileParams {
    const void *q, *k, *v;
    const int* offsets;
    unsigned* err;
    int batch, m, hq, hkv, group, offset, capacity;
    int pack;                   // query heads of one kv head that share a tile: row = position * pack + head
    int head_groups, pairs;     // hq / pack; pairs of 128-row tiles per (sequence, head group)
    float scale, c;             // c: scale * log2(e)
};

template <typename T, int D> struct TileCfg {
    // Tensor memory: 512 columns hold the scores and the sums of two tiles.  The probabilities lie over the scores, 16 columns per
    // term and 32 keys: three terms of 128 keys (192 columns) fit beside the sums of a 64-wide head, three of 64 keys (96) beside
    // those of a 128-wide one.  Registers give the same sizes: a thread holds KEYS scores and D sums.
    static constexpr int TERMS = kTerms<T>;
    static constexpr int KEYS = D == 128 ? 64 : 128;                // keys per tile
    static constexpr int S_COLS = 256 - D;                          // columns of a tile's scores / probabilities
    static_assert(KEYS <= S_COLS && KEYS / 32 * 16 * TERMS <= S_COLS, "tensor memory");
    static constexpr int QB = 128 * D * 2, KB = KEYS * D * 2;       // one tile of Q or the output; of K or V
    static constexpr int STAGES = 256 / KEYS;
    static constexpr int OFF_K = 2 * QB, OFF_V = OFF_K + STAGES * KB;
    static constexpr int SMEM = OFF_V + STAGES * KB + 1024;
    static constexpr int BARS = 4 * STAGES + 7;
};

// shared-memory descriptor of a [keys][64 d] tile as the MN-major operand (the d of V are the MMA's N): 128-byte rows,
// 8-key atoms 1024 bytes apart (stride byte offset), 64-column halves `half_bytes` apart (leading byte offset)
__device__ __forceinline__ uint64_t desc_sw128_mn(uint32_t saddr, uint32_t half_bytes) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(half_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// One CTA: two tiles of 128 query rows against the keys they see, KEYS keys at a time.  Warp 0 loads (TMA), warp 1 issues the
// MMAs, warpgroups 1 and 2 do the softmax of one tile each (a thread owns a row), so that one tile's softmax runs under
// the other's MMAs.  Tensor memory: S0 | S1 | O0 | O1; the probabilities overwrite the scores in place (per 32 keys: 16 columns
// of each term, largest first).  O is the sum over one tile of keys; the threads add it to the row's sums in registers when they
// have the next tile's scores (the MMAs complete in order), so that a new maximum rescales registers only.
template <typename T, int D>
__global__ void __launch_bounds__(AT_THREADS, 1)
attention_tile_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                      const __grid_constant__ CUtensorMap mo, const TileParams p) {
    using H = F16x2<T>;
    using C = TileCfg<T, D>;
    constexpr int KEYS = C::KEYS, STAGES = C::STAGES, QB = C::QB, KB = C::KB, TERMS = C::TERMS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[C::BARS];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t b0 = smem_u32(bars);
    const uint32_t qfull = b0, sfull = b0 + 8, pfull = b0 + 24, odone = b0 + 40;
    const uint32_t kfull = b0 + 56, kempty = kfull + 8 * STAGES, vfull = kempty + 8 * STAGES, vempty = vfull + 8 * STAGES;
    volatile int* abort_flag = &s_abort;

    // heavy tiles first: under the causal mask the last positions have the most keys
    const int per_pair = p.head_groups * p.batch;
    const int pair = p.pairs - 1 - int(blockIdx.x / per_pair), rest = int(blockIdx.x % per_pair);
    const int hg = rest % p.head_groups, b = rest / p.head_groups;
    const int kvh = hg * p.pack / p.group;
    const int off = p.offsets ? __ldg(p.offsets + b) : p.offset;
    const int ppt = 128 / p.pack;                                   // positions per tile
    int n[2], keys[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const int first = (2 * pair + w) * ppt, last = min(p.m, first + ppt) - 1;
        keys[w] = first < p.m ? max(1, min(off + last + 1, p.capacity)) : 0;
        n[w] = (keys[w] + KEYS - 1) / KEYS;
    }
    const int nmax = max(n[0], n[1]), kmax = max(keys[0], keys[1]);

    if (warp == 0) tc_alloc<512>(smem_u32(&s_tmem));
    if (tid == 0) {
        s_abort = 0;
        mbar_init(qfull, 1);
        for (int i = 0; i < STAGES; ++i) { mbar_init(kfull + 8 * i, 1); mbar_init(kempty + 8 * i, 1); mbar_init(vfull + 8 * i, 1); mbar_init(vempty + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(sfull + 8 * i, 1); mbar_init(pfull + 8 * i, 128); mbar_init(odone + 8 * i, 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            if (lane == 0) {
                mbar_expect_tx(qfull, (n[1] > 0 ? 2 : 1) * QB);
                tma_load_5d(sbase, &mq, 0, hg * p.pack, 2 * pair * ppt, 0, b, qfull);
                if (n[1] > 0) tma_load_5d(sbase + QB, &mq, 0, hg * p.pack, (2 * pair + 1) * ppt, 0, b, qfull);
                bool ok = true;
                for (int j = 0; j < nmax && ok; ++j) {
                    const int st = j % STAGES; const uint32_t ph = ((j / STAGES) & 1) ^ 1;
                    ok = mbar_wait_sleep<32>(kempty + 8 * st, ph, abort_flag);
                    if (ok) { mbar_expect_tx(kfull + 8 * st, KB); tma_load_5d(sbase + C::OFF_K + st * KB, &mk, 0, j * KEYS, 0, kvh, b, kfull + 8 * st); }
                    if (ok) ok = mbar_wait_sleep<32>(vempty + 8 * st, ph, abort_flag);
                    if (ok) { mbar_expect_tx(vfull + 8 * st, KB); tma_load_5d(sbase + C::OFF_V + st * KB, &mv, 0, j * KEYS, 0, kvh, b, vfull + 8 * st); }
                }
                if (!ok) drain_copies();
            }
            __syncwarp();
        } else if (warp == 1) {
            const uint32_t id_qk = tc_idesc_f16(H::kIsBf16, 128, KEYS);
            const uint32_t id_pv = tc_idesc_f16(H::kIsBf16, 128, D) | (1u << 16);       // B (V) MN-major
            auto qk = [&](int w, int j) {                            // S_w = Q_w K_j^T, announced on sfull[w]
                if (lane == 0) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) {
                        const uint32_t qo = (ks >> 2) * (128 * 128) + (ks & 3) * 32, ko = (ks >> 2) * (KEYS * 128) + (ks & 3) * 32;
                        tc_mma_ss(tmem + C::S_COLS * w, tc_desc_sw128(sbase + w * QB + qo), tc_desc_sw128(sbase + C::OFF_K + (j % STAGES) * KB + ko), id_qk, ks > 0);
                    }
                    tc_commit(sfull + 8 * w);
                }
                __syncwarp();
            };
            bool ok = mbar_wait(qfull, 0, abort_flag) && mbar_wait(kfull, 0, abort_flag);
            if (ok) {
                tc_fence_after();
                if (n[0] > 0) qk(0, 0);
                if (n[1] > 0) qk(1, 0);
                if (lane == 0) tc_commit(kempty);
                __syncwarp();
            }
            for (int j = 0; j < nmax && ok; ++j) {
                const int st = j % STAGES, sn = (j + 1) % STAGES;
                ok = mbar_wait(vfull + 8 * st, (j / STAGES) & 1, abort_flag);
                if (!ok) break;
                if (j == nmax - 1 && kmax < nmax * KEYS) {
                    // value rows behind the last key may hold anything (a NaN times a zero probability is a NaN): clear them
                    for (int key = kmax - j * KEYS; key < KEYS; ++key)
                        if (lane < D / 8)
                            asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};"
                                         ::"r"(sbase + C::OFF_V + st * KB + (lane >> 3) * (KEYS * 128) + key * 128 + ((lane & 7) << 4)), "r"(0u) : "memory");
                    fence_proxy_async();
                    __syncwarp();
                }
                bool knext = false;
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    if (j >= n[w]) continue;
                    ok = mbar_wait(pfull + 8 * w, j & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    if (lane == 0) {
#pragma unroll
                        for (int x = TERMS - 1; x >= 0; --x)         // the small terms first: their sums lose nothing
#pragma unroll
                            for (int ks = 0; ks < KEYS / 16; ++ks)
                                tc_mma_ts(tmem + 2 * C::S_COLS + D * w, tmem + C::S_COLS * w + (ks >> 1) * (16 * TERMS) + (ks & 1) * 8 + 16 * x,
                                          desc_sw128_mn(sbase + C::OFF_V + st * KB + ks * 2048, KEYS * 128), id_pv, ks > 0 || x < TERMS - 1);
                        if (j + 1 >= n[w]) tc_commit(odone + 8 * w);
                    }
                    __syncwarp();
                    if (j + 1 < n[w]) {
                        if (!knext) { ok = mbar_wait(kfull + 8 * sn, ((j + 1) / STAGES) & 1, abort_flag); knext = true; }
                        if (!ok) break;
                        qk(w, j + 1);
                    }
                }
                if (!ok) break;
                if (lane == 0) {
                    tc_commit(vempty + 8 * st);
                    if (knext) tc_commit(kempty + 8 * sn);
                }
                __syncwarp();
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const int w = (warp >> 2) - 1, row = tid & 127;
        if (n[w] > 0) {
            const uint32_t lane_base = (uint32_t)(warp & 3) << 21;  // 32 TMEM lanes per warp
            const uint32_t tS = tmem + C::S_COLS * w + lane_base, tO = tmem + 2 * C::S_COLS + D * w + lane_base;
            const int pos = min(p.m - 1, (2 * pair + w) * ppt + row / p.pack);
            const int lim = min(off + pos + 1, p.capacity);         // keys that this row sees
            const int first_lim = off + (2 * pair + w) * ppt + 1;   // ... and that every row of the tile sees
            float mrow = -INFINITY, l = 0.f;
            float acc[D], f = 0.f;                                  // sums of the tiles before the last; what to scale them by when it is added
#pragma unroll
            for (int e = 0; e < D; ++e) acc[e] = 0.f;
            auto add_tile = [&]() {
#pragma unroll
                for (int q = 0; q < D / 32; ++q) {
                    uint32_t o[32];
                    tc_ld32(tO + 32 * q, o);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[32 * q + e] = fmaf(acc[32 * q + e], f, __uint_as_float(o[e]));
                }
            };
            bool ok = true;
            for (int j = 0; j < n[w]; ++j) {
                ok = __all_sync(0xffffffffu, mbar_wait(sfull + 8 * w, j & 1, abort_flag));      // also says that P V of the tile before is complete
                if (!ok) break;
                tc_fence_after();
                constexpr int Q = KEYS / 32;
                uint32_t s[Q][32];
#pragma unroll
                for (int q = 0; q < Q; ++q) tc_ld32(tS + 32 * q, s[q]);
                tc_wait_ld();
                if (j * KEYS + KEYS > first_lim || j * KEYS + KEYS > p.capacity) {
                    const int left = lim - j * KEYS;
#pragma unroll
                    for (int q = 0; q < Q; ++q)
#pragma unroll
                        for (int e = 0; e < 32; ++e) if (32 * q + e >= left) s[q][e] = __float_as_uint(-INFINITY);
                }
                float x0 = -INFINITY, x1 = -INFINITY, x2 = -INFINITY, x3 = -INFINITY;
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int e = 0; e < 32; e += 4) {
                        x0 = fmaxf(x0, __uint_as_float(s[q][e])); x1 = fmaxf(x1, __uint_as_float(s[q][e + 1]));
                        x2 = fmaxf(x2, __uint_as_float(s[q][e + 2])); x3 = fmaxf(x3, __uint_as_float(s[q][e + 3]));
                    }
                const float mn = fmaxf(mrow, fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)));
                const float fn = mrow == -INFINITY ? 0.f : ex2((mrow - mn) * p.c);
                mrow = mn;
                float l0 = 0.f, l1 = 0.f;                           // the tile's own sum: added key by key to a long one, small terms are lost
                const float base = mrow == -INFINITY ? 0.f : mrow * p.c;
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    uint32_t r[TERMS][16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const float a = ex2(fmaf(__uint_as_float(s[q][2 * e]), p.c, -base)), d = ex2(fmaf(__uint_as_float(s[q][2 * e + 1]), p.c, -base));
                        l0 += a; l1 += d;
                        uint32_t t[TERMS];
                        split_terms<T>(a, d, t);
#pragma unroll
                        for (int x = 0; x < TERMS; ++x) r[x][e] = t[x];
                    }
#pragma unroll
                    for (int x = 0; x < TERMS; ++x) tc_st16(tS + 16 * (TERMS * q + x), r[x]);
                }
                l = fmaf(l, fn, l0 + l1);
                if (j > 0) add_tile();
                f = fn;
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(pfull + 8 * w);
            }
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(odone + 8 * w, 0, abort_flag));
            if (ok) {
                tc_fence_after();
                add_tile();
                const float inv = kUnscale<T> / l;
                const uint32_t so = sbase + w * QB;                 // the tile's Q is no longer needed
                float zero = 0.f;                                   // stays so unless a value is infinite or NaN
#pragma unroll
                for (int c = 0; c < D / 8; ++c) {
                    uint32_t v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float v0 = acc[8 * c + 2 * e] * inv, v1 = acc[8 * c + 2 * e + 1] * inv;
                        zero = fmaf(v0, 0.f, fmaf(v1, 0.f, zero));
                        v[e] = H::pack(v0, v1);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};"
                                 ::"r"(so + row * 128 + (c >> 3) * (128 * 128) + (((c & 7) ^ (row & 7)) << 4)), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
                }
                for (unsigned bad = __ballot_sync(0xffffffffu, !(zero == 0.f)); bad != 0u; bad &= bad - 1u) {
                    const int r = (warp & 3) * 32 + __ffs(bad) - 1, i = (2 * pair + w) * ppt + r / p.pack;
                    if (i >= p.m) continue;                         // behind the last token: never stored
                    float o[D / 32];
                    const size_t cache = ((size_t)b * p.capacity * p.hkv + kvh) * D;
                    attention_row<T, D>(reinterpret_cast<const uint16_t*>(p.q) + (((size_t)b * p.m + i) * p.hq + hg * p.pack + r % p.pack) * D,
                                        reinterpret_cast<const uint16_t*>(p.k) + cache, reinterpret_cast<const uint16_t*>(p.v) + cache, (size_t)p.hkv * D,
                                        min(off + i + 1, p.capacity), p.scale, o);
                    const int d0 = lane * (D / 32);
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < D / 32; e += 2)
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(so + r * 128 + (d0 >> 6) * (128 * 128) + ((((d0 >> 3) & 7) ^ (r & 7)) << 4) + ((d0 & 7) + e) * 2),
                                     "r"(H::pack(o[e], o[e + 1])) : "memory");
                }
                fence_proxy_async();
            }
            bar_sync(1 + w, 128);
            if (row == 0 && ok && !*abort_flag) {
                tma_store_5d(&mo, sbase + w * QB, 0, hg * p.pack, (2 * pair + w) * ppt, 0, b);          // rows past the last token are clipped
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc_fence_after(); tc_dealloc<512>(tmem); }
    if (tid == 0 && s_abort) {
        g_attention_error = 8u;
        if (p.err) *p.err = 8u;
    }
}

// q / out [batch, m, heads, d] (heads = hq) or a cache [batch, capacity, hkv, d] as (64 d, rows.., halves ..) boxes of a
// swizzled [half][row][64] shared-memory tile
bool encode_rows(CUtensorMap* map, const void* base, int dtype, int d, int heads, long long rows, long long batch, int box_heads, int box_rows, bool heads_inner) {
    EncodeTiledFn enc = get_tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t row_bytes = (cuuint64_t)heads * d * 2;
    cuuint64_t dims[5], strides[4]; cuuint32_t box[5], es[5] = {1, 1, 1, 1, 1};
    dims[0] = 64; box[0] = 64;
    dims[4] = (cuuint64_t)batch; box[4] = 1; strides[3] = row_bytes * (cuuint64_t)rows;
    if (heads_inner) {                                               // query tiles: (64, head, position, half, sequence)
        dims[1] = heads; strides[0] = (cuuint64_t)d * 2; box[1] = box_heads;
        dims[2] = (cuuint64_t)rows; strides[1] = row_bytes; box[2] = box_rows;
        dims[3] = d / 64; strides[2] = 128; box[3] = d / 64;
    } else {                                                         // key / value tiles: (64, position, half, head, sequence)
        dims[1] = (cuuint64_t)rows; strides[0] = row_bytes; box[1] = box_rows;
        dims[2] = d / 64; strides[1] = 128; box[2] = d / 64;
        dims[3] = heads; strides[2] = (cuuint64_t)d * 2; box[3] = 1;
    }
    return enc(map, dtype == MT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
bool set_smem(K kern, int bytes, bool (&done)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return false; }
    if (!done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) { cudaGetLastError(); return false; }
        done[dev] = true;
    }
    return true;
}

constexpr int AS_GRID = 148;            // one CTA per SM

template <typename T, int D, int NT>
int launch_stream_inst(cudaStream_t st, const CUtensorMap& mk, const CUtensorMap& mv, const StreamParams& p, int grid) {
    static bool done[64] = {};
    auto kern = attention_stream_kernel<T, D, NT>;
    if (!set_smem(kern, StreamCfg<D, NT>::SMEM, done)) return MT_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(AS_THREADS); cfg.dynamicSmemBytes = StreamCfg<D, NT>::SMEM; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = p.whole ? 0 : 1;               // behind attention_zero_kernel, which itself starts after everything before it
    if (cudaLaunchKernelEx(&cfg, kern, mk, mv, p) != cudaSuccess) { cudaGetLastError(); return MT_ERR_CUDA; }
    return MT_OK;
}
template <typename T, int D>
int launch_tile_inst(cudaStream_t st, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo, const TileParams& p, unsigned grid) {
    static bool done[64] = {};
    auto kern = attention_tile_kernel<T, D>;
    if (!set_smem(kern, TileCfg<T, D>::SMEM, done)) return MT_ERR_CUDA;
    kern<<<grid, AT_THREADS, TileCfg<T, D>::SMEM, st>>>(mq, mk, mv, mo, p);
    return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_CUDA;
}

}  // namespace

bool attention_batch_supported(int hq, int hkv, int d) { return (d == 64 || d == 128) && hkv >= 1 && hq % hkv == 0; }

size_t attention_batch_workspace_bytes(int m, int hq, int hkv, int d) {
    if (m < 1 || hq < 1 || !attention_batch_supported(hq, hkv, d) || (long long)m * (hq / hkv) > 16) return 0;      // no scratch
    return AS_PART_OFF + (size_t)AS_GRID * 2 * 16 * (d + 4) * 4;
}

int attention_error(unsigned* word, bool clear) {
    unsigned w = 0;
    const unsigned zero = 0;
    if (cudaMemcpyFromSymbol(&w, g_attention_error, 4) != cudaSuccess ||
        (w && clear && cudaMemcpyToSymbol(g_attention_error, &zero, 4) != cudaSuccess)) { cudaGetLastError(); return MT_ERR_CUDA; }
    *word = w;
    return MT_OK;
}

int launch_attention_batch(cudaStream_t st, const void* q, const void* k_cache, const void* v_cache, void* out, const int* offsets,
                           int batch, int m, int hq, int hkv, int d, int offset, int capacity, float scale,
                           void* workspace, size_t workspace_bytes, int dtype) {
    const int group = hq / hkv;
    const float c = scale * 1.4426950408889634f;
    CUtensorMap mk, mv;
    // rows that are evaluated a second time read q again behind the first store: with out in q's place the tile kernel, which
    // stores a row once, takes the call
    const size_t bytes = (size_t)batch * m * hq * d * 2;
    const bool apart = static_cast<const char*>(q) + bytes <= static_cast<const char*>(out) || static_cast<const char*>(out) + bytes <= static_cast<const char*>(q);
    if (workspace && apart && (long long)m * group <= 16 && workspace_bytes >= attention_batch_workspace_bytes(m, hq, hkv, d)) {
        StreamParams p;
        p.q = q; p.k = k_cache; p.v = v_cache; p.out = out; p.offsets = offsets; p.scale = scale; p.ws = static_cast<unsigned char*>(workspace);
        p.batch = batch; p.m = m; p.hq = hq; p.hkv = hkv; p.group = group; p.offset = offset; p.capacity = capacity; p.c = c;
        p.whole = (long long)batch * hkv > AS_MAX_SEGMENTS;
        if (!p.whole) {
            const int n = batch * hkv;
            attention_zero_kernel<<<(n + 1023) / 1024, 256, 0, st>>>(reinterpret_cast<unsigned*>(p.ws + AS_HEAD), n);
            if (cudaGetLastError() != cudaSuccess) return MT_ERR_CUDA;
        }
        if (!encode_rows(&mk, k_cache, dtype, d, hkv, capacity, batch, 1, AS_KEYS, false) ||
            !encode_rows(&mv, v_cache, dtype, d, hkv, capacity, batch, 1, AS_KEYS, false)) return MT_ERR_CUDA;
        const int nt = m * group <= 8 ? 1 : 2;
        const long long most = (long long)batch * hkv * ((capacity + AS_KEYS - 1) / AS_KEYS);
        const int grid = int(most < AS_GRID ? most : AS_GRID);
#define MT_STREAM(T_, D_) return nt == 1 ? launch_stream_inst<T_, D_, 1>(st, mk, mv, p, grid) : launch_stream_inst<T_, D_, 2>(st, mk, mv, p, grid)
        if (dtype == MT_F16) { if (d == 128) MT_STREAM(__half, 128); else MT_STREAM(__half, 64); }
        if (d == 128) MT_STREAM(__nv_bfloat16, 128); else MT_STREAM(__nv_bfloat16, 64);
#undef MT_STREAM
    }
    TileParams p;
    p.q = q; p.k = k_cache; p.v = v_cache; p.scale = scale;
    p.offsets = offsets; p.err = workspace_bytes >= 4 ? static_cast<unsigned*>(workspace) : nullptr;
    p.batch = batch; p.m = m; p.hq = hq; p.hkv = hkv; p.group = group; p.offset = offset; p.capacity = capacity; p.c = c;
    p.pack = 1;
    while (p.pack < 128 && group % (2 * p.pack) == 0) p.pack *= 2;
    p.head_groups = hq / p.pack;
    const int ppt = 128 / p.pack;
    p.pairs = (m + 2 * ppt - 1) / (2 * ppt);
    const long long grid = (long long)p.pairs * p.head_groups * batch;
    if (grid > 0x7fffffffLL) return MT_ERR_TOO_LARGE;
    CUtensorMap mq, mo;
    const int keys = d == 128 ? TileCfg<__half, 128>::KEYS : TileCfg<__half, 64>::KEYS;      // the same for bf16
    if (!encode_rows(&mk, k_cache, dtype, d, hkv, capacity, batch, 1, keys, false) || !encode_rows(&mv, v_cache, dtype, d, hkv, capacity, batch, 1, keys, false) ||
        !encode_rows(&mq, q, dtype, d, hq, m, batch, p.pack, ppt, true) || !encode_rows(&mo, out, dtype, d, hq, m, batch, p.pack, ppt, true)) return MT_ERR_CUDA;
    if (dtype == MT_F16)
        return d == 128 ? launch_tile_inst<__half, 128>(st, mq, mk, mv, mo, p, (unsigned)grid) : launch_tile_inst<__half, 64>(st, mq, mk, mv, mo, p, (unsigned)grid);
    return d == 128 ? launch_tile_inst<__nv_bfloat16, 128>(st, mq, mk, mv, mo, p, (unsigned)grid) : launch_tile_inst<__nv_bfloat16, 64>(st, mq, mk, mv, mo, p, (unsigned)grid);
}

}  // namespace mt
