// Backward of the gate -> grouped causal FIR -> gate operator on tcgen05 / TMEM (bf16 operands and filters, up to 128 taps
// shared by multiples of 16 channels): dx, dB, dC and dh in ONE pass over dy, x, B, C and y2 (vortex/ops/hyena_se/bwd.py:11,
// math ref_bwd.py:31-115).  With z = B * x, g2 = dy * C and the lag filter w[j] = h[g, K-1-j]:
//   dC = dy * y2,   dz[t] = sum_j w[j] g2[t + j],   dx = dz * B,   dB = dz * x,   dw[j] = sum_t,c g2[t, c] z[t - j, c].
//
// Both reductions are contractions of the same tiles.  A work item is one group of 16 channels and two independent
// streams (batch element x time segment).  A chunk of 128 samples is a [128 x 64] tile: head of both streams (32 columns),
// remainder of both streams (32 columns).
//   dz    blocked Toeplitz: the chunk's g2 is stored with time REVERSED, which turns the anti-causal filter into the causal
//         operand [T^ | T][i][j] = w[128 + i - j] of the forward kernel, here applied to (next chunk, this chunk).
//   dw    W[i][i'] += sum over the 32 columns of g2[i] z[i'] for the chunk's 128 rows of g2 against the 256 rows of z that
//         end with the chunk: an ordinary M128 x N256 contraction of K-major tiles, accumulated in TMEM over two chunks;
//         dw[j] is the sum along an anti-diagonal of W, kept in fp32 registers over the item.
//
// Precision.  g2 and z are products of two bf16 numbers: 16 significant bits, so head + remainder in bf16 hold them exactly
// between 2^-117 and 3.39e38 (the fp32 kernels of gcg_bwd.cu work on the same products; below, the remainder is cut to
// bf16's subnormals, above, the head is infinite).  Taps are bf16, accumulation is fp32, one rounding on
// the way out.  dw takes all four products of heads and remainders.
// A product that is infinite or NaN, or whose head is, would make dz NaN over the 256 rows of the contraction's window and dh
// at every lag; the sums it reaches are formed again under the taps alone (dz_under_taps, dw_under_taps).
//
// What bounds it: 10 bytes in and 6 bytes out per element (B=2, L=8192, D=4096: 1.07 GB = 164 us at 6.54 TB/s), i.e. 2900
// cycles per chunk and SM, of which the tensor pipe needs 16 x 85 (dz) + 8 x 128 (dw) and shared memory about as many.
// Measured: 326 us with the launch that clears the fp32 accumulator, the fp32 kernels 1290 us; B=4: 617 us = 3.5 TB/s.  A
// W that gathers all chunks of an item is 50 us faster and too inexact (WCHUNKS).
// Everything arrives by TMA: with 224 KB of the SM carved out as shared memory L1 holds some 220 lines, so plain loads of
// 32-byte row pieces kept 7 KB in flight (first version: 18000 cycles per chunk, 700 us).
//
// One persistent CTA per SM walks the items (strided by the launch width: concurrent CTAs read neighbouring groups of the
// same rows).  18 warps: 0-7 front end (staged rows -> products -> tiles; dC leaves from here), 8-11 epilogue (dz out of
// TMEM, gates, stores; the next item's Toeplitz operand), 12 MMA issue, 13 TMA issue, 14-17 the sums along W (as a part of
// the epilogue they cost 8 us more).  x and B stay in their stage until the epilogue, one to two chunks later, has used them.  TMEM:
// operand 128 columns, dz 2 x 64, W 256 -- all 512.  All waits are bounded.
#include "tma.cuh"
#include "umma.cuh"

namespace vtx {

VTX_DEFINE_STATUS_READER()

namespace gbt {

using namespace umma;

constexpr int NS = 2, CH = 16, CHUNK = 128;
constexpr int NFE = 8, W_EP = NFE, W_MMA = NFE + 4, W_TMA = NFE + 5, W_DW = NFE + 6, THREADS = 32 * 18;
constexpr int WROWS = CHUNK / NFE;                 // rows of a chunk per front-end warp
constexpr int TILE = CHUNK * 128;                  // [128 rows][64 columns] bf16, 128-byte swizzle
constexpr int BOX = CHUNK * CH * 2;                // staged box: 128 rows x 16 channels of one stream and tensor
constexpr int NG = 2, NZ = 3;                      // tile rings: g2 is consumed in its own step, z also in the next one
constexpr int NXS = 4, NDS = 3;                    // stages of (x, B), held until the epilogue is done, and of (dy, C, y2)
constexpr int X_STAGE = 2 * NS * BOX, D_STAGE = 3 * NS * BOX;
constexpr int OFF_Z = 0, OFF_G = OFF_Z + NZ * TILE, OFF_X = OFF_G + NG * TILE, OFF_D = OFF_X + NXS * X_STAGE;
// Chunks whose products meet in W before it is read out.  The tensor core truncates an accumulator at every step, so the
// error grows with them: dh of random operands against 64 bits, B=2, L=8192, D=4096, K=128 (L=131072, D=512): 1.6e-7
// (2.2e-7) with one, 2.8e-7 (3.0e-7) with two, 5.6e-7 with four, 2.3e-6 (8.4e-6) over whole items; the fp32 kernels 3.3e-7
// (5.0e-7).  Operands of one sign, whose truncations do not cancel: 8.8e-8 (1.1e-7), 2.2e-7 (2.3e-7), 5.4e-7 (5.3e-7),
// 2.6e-6 (1.1e-5); the fp32 kernels 1.2e-7 (3.3e-7).  Time: 400, 326, 304 and 288 us.
constexpr int WCHUNKS = 2;
constexpr int RUNS = 4, RUN = 40;                  // sums along the anti-diagonals of W: runs per warp, most columns per run
constexpr int RUN_LAGS = RUN + 32;                 // words of a run's sums
constexpr int OFF_TAPS = OFF_D + NDS * D_STAGE, OFF_RUNS = OFF_TAPS + 384 * 2, OFF_BARS = OFF_RUNS + 4 * RUNS * RUN_LAGS * 4;
constexpr int NBARS = 2 * (NG + NZ + NXS + NDS) + 4 + 4;
constexpr int SMEM_BYTES = OFF_BARS + NBARS * 8 + 16 + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
constexpr int A_COL = 0, DZ_COL = 128, W_COL = 256, TMEM_COLS = 512;

struct Args {
    const __nv_bfloat16* h;
    __nv_bfloat16 *dx, *dB, *dC;
    float* dh;
    int64_t B, L, D, G, K;       // G: groups of 16 channels
    int64_t dg;                  // channels that share a filter (a multiple of 16)
    int64_t nseg, seg_len, nstream, nset, nitems, item0, item1;
    // the operands, for the sums that are not contracted
    const __nv_bfloat16 *dy, *x, *Bg, *C;
    int64_t dy_sb, dy_sl, x_sb, x_sl, b_sb, b_sl, c_sb, c_sl;
};

struct Stream { int b, ts, te; bool active; };
__device__ __forceinline__ Stream stream_of(const Args& a, int set, int s) {
    Stream st;
    const int id = set * NS + s;
    st.active = id < (int)a.nstream;
    st.b = st.active ? id / (int)a.nseg : (int)a.B;          // a batch index outside the tensor: its boxes are zeros
    st.ts = (id % (int)a.nseg) * (int)a.seg_len;
    st.te = st.ts + a.seg_len < a.L ? st.ts + (int)a.seg_len : (int)a.L;
    return st;
}

// product of two packed bf16 pairs, exact in fp32, as bf16 head and bf16 remainder
__device__ __forceinline__ void split_mul(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
    const float p0 = bf_lo(a) * bf_lo(b), p1 = bf_hi(a) * bf_hi(b);
    hi = pack_bf16(p0, p1);
    lo = pack_bf16(p0 - bf_lo(hi), p1 - bf_hi(hi));
}
__device__ __forceinline__ uint4 ld_sh16(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void st_sh16(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// products of 8 channels into row r of a tile: head in 16-byte piece c, remainder in piece c + 4
__device__ __forceinline__ void split_tile(uint32_t tile, int r, int c, const uint4& a, const uint4& b) {
    uint32_t h[4], l[4];
    split_mul(a.x, b.x, h[0], l[0]); split_mul(a.y, b.y, h[1], l[1]);
    split_mul(a.z, b.z, h[2], l[2]); split_mul(a.w, b.w, h[3], l[3]);
    const uint32_t addr = tile + (uint32_t)(r * 128) + (uint32_t)((c ^ (r & 7)) << 4);
    st_sh16(addr, h);
    st_sh16(addr ^ 64u, l);
}
__device__ __forceinline__ uint32_t mul_pair(uint32_t a, uint32_t b) { return pack_bf16(bf_lo(a) * bf_lo(b), bf_hi(a) * bf_hi(b)); }

struct Maps { CUtensorMap dy, x, Bg, C, y2; };

// The sums under the filter's taps alone, in fp32 on the exact products: the contractions multiply every row of their
// windows, and a zero times infinity or NaN is NaN.  A warp whose sums are not all finite takes these instead.  (Among them
// finite products whose head rounds to infinity.)
__device__ __forceinline__ void mul_rows(const __nv_bfloat16* p, const __nv_bfloat16* q, float (&out)[CH]) {
    const uint4 a0 = reinterpret_cast<const uint4*>(p)[0], a1 = reinterpret_cast<const uint4*>(p)[1];
    const uint4 b0 = reinterpret_cast<const uint4*>(q)[0], b1 = reinterpret_cast<const uint4*>(q)[1];
    const uint32_t aw[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) { out[2 * j] = bf_lo(aw[j]) * bf_lo(bw[j]); out[2 * j + 1] = bf_hi(aw[j]) * bf_hi(bw[j]); }
}
// dz at row t of 16 channels from c0 on (rows past the end are not stored)
__device__ __noinline__ void dz_under_taps(const Args& a, int64_t b, int64_t c0, int64_t t, uint32_t* out) {
    const __nv_bfloat16* const w = a.h + (c0 / a.dg) * a.K + a.K - 1;
    float sum[CH] = {};
    for (int64_t j = 0; j < a.K; ++j) {
        bool done = true;
        if (t + j < a.L) {
            float g2[CH];
            mul_rows(a.dy + b * a.dy_sb + (t + j) * a.dy_sl + c0, a.C + b * a.c_sb + (t + j) * a.c_sl + c0, g2);
            const float wj = __bfloat162float(w[-j]);
#pragma unroll
            for (int c = 0; c < CH; ++c) { sum[c] = fmaf(wj, g2[c], sum[c]); done = done && isnan(sum[c]); }
        }
        if (__all_sync(0xffffffffu, done)) break;
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) out[c] = __float_as_uint(sum[c]);
}
// sum over rows ts .. te - 1 that are rows first .. first + 31 of their chunk, and 16 channels, of g2[t] z[t - lag]
__device__ __noinline__ float dw_under_taps(const Args& a, int64_t b, int64_t c0, int ts, int te, int first, int lag) {
    float total = 0.f;
    for (int t0 = ts + first; t0 < te; t0 += CHUNK) {
        float sum = 0.f;
#pragma unroll 4
        for (int t = t0; t < t0 + 32; ++t) {
            if (t >= te || t < lag || lag >= a.K) continue;
            float g2[CH], z[CH];
            mul_rows(a.dy + b * a.dy_sb + t * a.dy_sl + c0, a.C + b * a.c_sb + t * a.c_sl + c0, g2);
            mul_rows(a.x + b * a.x_sb + (t - lag) * a.x_sl + c0, a.Bg + b * a.b_sb + (t - lag) * a.b_sl + c0, z);
#pragma unroll
            for (int c = 0; c < CH; ++c) sum = fmaf(g2[c], z[c], sum);
        }
        total += sum;
        if (__all_sync(0xffffffffu, isnan(total) || lag >= a.K)) break;
    }
    return total;
}

__global__ void __launch_bounds__(THREADS, 1) gcg_bwd_tc_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Args a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sm_u = (smem_u32(smem_raw) + 1023u) & ~1023u;
    auto smp = [&](uint32_t off) { return reinterpret_cast<uint8_t*>(__cvta_shared_to_generic(sm_u + off)); };
    const uint32_t bar_u = sm_u + OFF_BARS;
    auto bar = [&](uint32_t first, uint32_t i) { return bar_u + 8u * (first + i); };
    constexpr uint32_t G_FULL = 0, G_FREE = G_FULL + NG, Z_FULL = G_FREE + NG, Z_FREE = Z_FULL + NZ, X_FULL = Z_FREE + NZ,
                       X_FREE = X_FULL + NXS, D_FULL = X_FREE + NXS, D_FREE = D_FULL + NDS, DZ_FULL = D_FREE + NDS, DZ_EMPTY = DZ_FULL + 2,
                       W_FULL = DZ_EMPTY + 2, W_EMPTY = W_FULL + 1, A_READY = W_EMPTY + 1, TAPS_READY = A_READY + 1;
    static_assert(TAPS_READY + 1 == NBARS, "barrier count");
    const uint32_t tslot = bar_u + 8u * NBARS;

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int ncta = (int)gridDim.x;
    const int nmine = (int)((a.item1 - a.item0 - (int64_t)blockIdx.x + ncta - 1) / ncta);
    const int K = (int)a.K;
    const int n = (int)(a.seg_len / CHUNK);            // chunks of an item; steps 0 (z halo), 1..n, n+1 (g2 halo)
    auto item_group = [&](int t) { return (int)((a.item0 + (int64_t)blockIdx.x + (int64_t)t * ncta) % a.G); };
    auto item_set = [&](int t) { return (int)((a.item0 + (int64_t)blockIdx.x + (int64_t)t * ncta) / a.G); };

    if (tid == 0) {
        for (int i = 0; i < NG; ++i) { mbar_init(bar(G_FULL, i), NFE); mbar_init(bar(G_FREE, i), 1); }
        for (int i = 0; i < NZ; ++i) { mbar_init(bar(Z_FULL, i), NFE); mbar_init(bar(Z_FREE, i), 1); }
        for (int i = 0; i < NXS; ++i) { mbar_init(bar(X_FULL, i), 1); mbar_init(bar(X_FREE, i), NFE + 4); }
        for (int i = 0; i < NDS; ++i) { mbar_init(bar(D_FULL, i), 1); mbar_init(bar(D_FREE, i), NFE); }
        for (int i = 0; i < 2; ++i) { mbar_init(bar(DZ_FULL, i), 1); mbar_init(bar(DZ_EMPTY, i), 4); }
        mbar_init(bar(W_FULL, 0), 1); mbar_init(bar(W_EMPTY, 0), 4); mbar_init(bar(A_READY, 0), 4); mbar_init(bar(TAPS_READY, 0), 4);
        fence_mbar_init();
    }
    if (warp == W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tslot), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tslot) : "memory");

    if (warp < NFE) {
        // ======== front end: lane = (row 16 warp + lane / 2, channels 8 (lane & 1) .. + 7) of each stream ================
        const int r = warp * WROWS + lane / 2, half = lane & 1, rr = CHUNK - 1 - r;
        const uint32_t lane_box = (uint32_t)(r * 32 + half * 16);
        uint32_t gc = 0, zc = 0;             // steps with g2 / with z so far: their tiles and stages
        bool ok = true;
        for (int t = 0; t < nmine && ok; ++t) {
            Stream st[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) st[s] = stream_of(a, item_set(t), s);
            const int c0 = item_group(t) * CH + 8 * half;
            for (int k = 0; k <= n + 1; ++k) {
                const bool has_g = k >= 1, has_z = k <= n;
                const uint32_t xs = zc % NXS, ds = gc % NDS, zs = zc % NZ, gs = gc % NG;
                uint4 x[NS], b[NS], dy[NS], c[NS], y2[NS];
                if (has_z) {
                    if (!mbar_wait(bar(X_FULL, xs), (zc / NXS) & 1u, 2)) { ok = false; break; }
                    const uint32_t base = sm_u + OFF_X + xs * X_STAGE + lane_box;
#pragma unroll
                    for (int s = 0; s < NS; ++s) { x[s] = ld_sh16(base + s * BOX); b[s] = ld_sh16(base + (NS + s) * BOX); }
                }
                if (has_g) {
                    if (!mbar_wait(bar(D_FULL, ds), (gc / NDS) & 1u, 3)) { ok = false; break; }
                    const uint32_t base = sm_u + OFF_D + ds * D_STAGE + lane_box;
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        dy[s] = ld_sh16(base + s * BOX);
                        c[s] = ld_sh16(base + (NS + s) * BOX);
                        y2[s] = ld_sh16(base + (2 * NS + s) * BOX);
                    }
                }
                if (has_z) {
                    if (zc >= NZ && !mbar_wait(bar(Z_FREE, zs), ((zc - NZ) / NZ) & 1u, 4)) { ok = false; break; }
#pragma unroll
                    for (int s = 0; s < NS; ++s) split_tile(sm_u + OFF_Z + zs * TILE, r, 2 * s + half, x[s], b[s]);
                }
                if (has_g) {
                    if (gc >= NG && !mbar_wait(bar(G_FREE, gs), ((gc - NG) / NG) & 1u, 5)) { ok = false; break; }
#pragma unroll
                    for (int s = 0; s < NS; ++s) split_tile(sm_u + OFF_G + gs * TILE, rr, 2 * s + half, dy[s], c[s]);
                }
                fence_proxy_async_smem();        // tiles -> the tensor core's async proxy
                __syncwarp();
                if (lane == 0) {
                    // (X_FREE first: whoever sees the tile then knows that this warp is done with the stage)
                    if (has_z) { mbar_arrive(bar(X_FREE, xs)); mbar_arrive(bar(Z_FULL, zs)); }
                    if (has_g) mbar_arrive(bar(G_FULL, gs));
                }
                if (has_g) {
                    if (has_z) {
#pragma unroll
                        for (int s = 0; s < NS; ++s) {
                            const int row = st[s].ts + (k - 1) * CHUNK + r;
                            const uint4 o = make_uint4(mul_pair(dy[s].x, y2[s].x), mul_pair(dy[s].y, y2[s].y),
                                                       mul_pair(dy[s].z, y2[s].z), mul_pair(dy[s].w, y2[s].w));
                            if (st[s].active && row < st[s].te)
                                *reinterpret_cast<uint4*>(a.dC + ((int64_t)st[s].b * a.L + row) * a.D + c0) = o;
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(D_FREE, ds));
                }
                gc += has_g; zc += has_z;
            }
        }
    } else if (warp < W_EP + 4) {
        // ======== epilogue: thread = TMEM lane = row of the chunk with time reversed ====================================
        const int e = warp - W_EP, i = e * 32 + lane, tt = CHUNK - 1 - i;
        const uint32_t lane_base = tmem + ((uint32_t)(e * 32) << 16);
        // Toeplitz operand of an item: taps through shared memory (zero padded, tp[m] = w[m - 128]), then row i of [T^|T]
        auto expand = [&](int t) {
            uint16_t* tp = reinterpret_cast<uint16_t*>(smp(OFF_TAPS));
            const int64_t hrow = (int64_t)((unsigned)(item_group(t) * CH) / (unsigned)a.dg) * K;
            // (the taps of the item before are no longer read: all four warps had expanded them before its MMAs began)
#pragma unroll
            for (int m = i; m < 384; m += 128) {
                const int l = m - 128;
                tp[m] = (l >= 0 && l < K) ? reinterpret_cast<const uint16_t*>(a.h)[hrow + (K - 1 - l)] : (uint16_t)0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(TAPS_READY, 0));
            if (!mbar_wait(bar(TAPS_READY, 0), (uint32_t)(t & 1), 17)) return false;
            for (int c0 = 0; c0 < 128; c0 += 16) {
                uint32_t v[16];
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const int j = 2 * (c0 + m);
                    const uint32_t e0 = tp[128 + 128 + i - j], e1 = tp[128 + 127 + i - j];
                    v[m] = e1 << 16 | e0;
                }
                tmem_st16(lane_base + A_COL + c0, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(A_READY, 0));
            return true;
        };
        uint32_t dc = 0, xc = 0;              // dz accumulators and (x, B) stages gone through
        bool ok = expand(0);
        for (int t = 0; t < nmine && ok; ++t) {
            const int g = item_group(t);
            int64_t yoff[NS];
            int nleft[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const Stream st = stream_of(a, item_set(t), s);
                yoff[s] = ((int64_t)st.b * a.L + st.ts + tt) * a.D + (int64_t)g * CH;
                nleft[s] = st.active ? st.te - st.ts - tt : 0;
            }
            if (lane == 0) mbar_arrive(bar(X_FREE, xc % NXS));      // the halo's stage has no epilogue
            ++xc;
            for (int k = 1; k <= n; ++k, ++dc, ++xc) {
                const uint32_t xs = xc % NXS, buf = dc & 1u;
                if (!mbar_wait(bar(X_FULL, xs), (xc / NXS) & 1u, 6)) { ok = false; break; }
                if (!mbar_wait(bar(DZ_FULL, buf), (dc >> 1) & 1u, 7)) { ok = false; break; }
                tc_fence_after();
                __syncwarp();
                const uint32_t xrow = sm_u + OFF_X + xs * X_STAGE + (uint32_t)(tt * 32);
                const int64_t step = (int64_t)(k - 1) * CHUNK * a.D;
#pragma unroll 1
                for (int s = 0; s < NS; ++s) {
                    uint32_t ah[16], al[16];
                    tmem_ld16(lane_base + DZ_COL + buf * 64 + s * 16, ah);
                    tmem_ld16(lane_base + DZ_COL + buf * 64 + 32 + s * 16, al);
                    tmem_ld_wait(ah, al);
                    if (s + 1 == NS) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(DZ_EMPTY, buf));
                    }
                    const int64_t yo = (s ? yoff[1] : yoff[0]) + step;
                    const int nl = s ? nleft[1] : nleft[0];
                    // (sums times zero are zero, or NaN if one of them is not finite)
                    f32x2 dz[CH / 2], finite = 0;
#pragma unroll
                    for (int j = 0; j < CH / 2; ++j) {
                        dz[j] = add2(pk2(__uint_as_float(ah[2 * j]), __uint_as_float(ah[2 * j + 1])),
                                     pk2(__uint_as_float(al[2 * j]), __uint_as_float(al[2 * j + 1])));
                        finite = fma2(dz[j], 0, finite);
                    }
                    float f0, f1;
                    up2(finite, f0, f1);
                    if (__any_sync(0xffffffffu, f0 + f1 != 0.f)) {
                        const Stream st = stream_of(a, item_set(t), s);
                        uint32_t sums[CH];
                        if (st.active) {
                            dz_under_taps(a, st.b, (int64_t)g * CH, st.ts + (int64_t)(k - 1) * CHUNK + tt, sums);
#pragma unroll
                            for (int j = 0; j < CH / 2; ++j) dz[j] = pk2(__uint_as_float(sums[2 * j]), __uint_as_float(sums[2 * j + 1]));
                        }
                    }
                    uint32_t ox[8], ob[8];
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const uint4 x4 = ld_sh16(xrow + s * BOX + hf * 16), b4 = ld_sh16(xrow + (NS + s) * BOX + hf * 16);
                        const uint32_t xw[4] = {x4.x, x4.y, x4.z, x4.w}, bw[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float d0, d1;
                            up2(dz[4 * hf + j], d0, d1);
                            ox[4 * hf + j] = pack_bf16(d0 * bf_lo(bw[j]), d1 * bf_hi(bw[j]));
                            ob[4 * hf + j] = pack_bf16(d0 * bf_lo(xw[j]), d1 * bf_hi(xw[j]));
                        }
                    }
                    if ((k - 1) * CHUNK < nl) {
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a.dx + yo), "r"(ox[0]),
                                     "r"(ox[1]), "r"(ox[2]), "r"(ox[3]), "r"(ox[4]), "r"(ox[5]), "r"(ox[6]), "r"(ox[7]) : "memory");
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a.dB + yo), "r"(ob[0]),
                                     "r"(ob[1]), "r"(ob[2]), "r"(ob[3]), "r"(ob[4]), "r"(ob[5]), "r"(ob[6]), "r"(ob[7]) : "memory");
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(X_FREE, xs));
            }
            if (ok && t + 1 < nmine && !expand(t + 1)) ok = false;
        }
    } else if (warp == W_MMA) {
        if (lane == 0) {
            // ======== MMA issue ====================================================================================
            const uint32_t id_dz = instr_desc(128, 64, 1), id_w1 = instr_desc(128, 128, 0), id_w2 = instr_desc(128, 256, 0);
            const uint64_t g_n = smem_desc(sm_u + OFF_G, TILE, 1024, 2);      // g2 as N-major B operand, head | remainder
            const uint64_t g_k = smem_desc(sm_u + OFF_G, 16, 1024, 2);        // g2 as K-major A operand
            const uint64_t z_k = smem_desc(sm_u + OFF_Z, 16, 1024, 2);        // z as K-major B operand
            constexpr uint64_t SLOT = TILE / 16;                              // in the descriptors' 16-byte units
            // T^ (g2 of the next chunk) or T (this chunk's, overwrites the accumulator)
            auto dz_half = [&](uint32_t gs, uint32_t buf, bool next) {
#pragma unroll
                for (int jj = 0; jj < 8; ++jj)
                    mma_ts(tmem + DZ_COL + buf * 64, tmem + A_COL + (next ? 0 : 64) + 8 * jj, g_n + gs * SLOT + (uint64_t)(jj * 128), id_dz,
                           (next || jj) ? 1u : 0u);
            };
            // all products of the 16-column K steps that hold the same channels: heads are steps 0, 1, remainders 2, 3; the
            // products of heads last (the tensor core truncates an accumulator at every step, the small ones cost little)
            auto w_part = [&](uint32_t gs, uint32_t zs, uint32_t col, uint32_t idesc, bool first) {
#pragma unroll
                for (int m = 7; m >= 0; --m) {
                    const int ka = (m & 1) + (m & 2), kb = (m & 1) + 2 * (m >> 2);
                    mma_ss(tmem + W_COL + col, g_k + gs * SLOT + (uint64_t)(2 * ka), z_k + zs * SLOT + (uint64_t)(2 * kb), idesc, (first && m == 7) ? 0u : 1u);
                }
            };
            uint32_t gc = 0, zc = 0, dc = 0, wc = 0;       // dz accumulators and fillings of W begun
            bool ok = true;
            for (int t = 0; t < nmine && ok; ++t) {
                if (!mbar_wait(bar(A_READY, 0), (uint32_t)(t & 1), 10)) break;
                if (!mbar_wait(bar(Z_FULL, zc % NZ), (zc / NZ) & 1u, 11)) break;
                ++zc;
                for (int k = 1; k <= n; ++k, ++gc, ++zc, ++dc) {
                    const uint32_t gs = gc % NG, zs = zc % NZ, zp = (zc - 1) % NZ;
                    if (!mbar_wait(bar(G_FULL, gs), (gc / NG) & 1u, 12)) { ok = false; break; }
                    tc_fence_after();
                    // W first if the last chunk's sums have left it: it is read while the dz halves run
                    const bool early = mbar_test_wait(bar(Z_FULL, zs), (zc / NZ) & 1u) && (wc == 0 || (k - 1) % WCHUNKS || mbar_test_wait(bar(W_EMPTY, 0), (wc - 1) & 1u));
#pragma unroll 1
                    for (int part = 0; part < 2; ++part) {
                        if ((part == 0) == early) {
                            if (!mbar_wait(bar(Z_FULL, zs), (zc / NZ) & 1u, 13)) { ok = false; break; }
                            const bool first = (k - 1) % WCHUNKS == 0;
                            if (wc >= 1 && first && !mbar_wait(bar(W_EMPTY, 0), (wc - 1) & 1u, 16)) { ok = false; break; }
                            tc_fence_after();
                            if (zs == zp + 1) {            // the two z tiles are neighbours in the ring: 256 rows at once
                                w_part(gs, zp, 0, id_w2, first);
                            } else {
                                w_part(gs, zp, 0, id_w1, first);
                                w_part(gs, zs, 128, id_w1, first);
                            }
                            const bool last = k % WCHUNKS == 0 || k == n;
                            if (last) mma_commit(bar(W_FULL, 0));
                            mma_commit(bar(Z_FREE, zp));
                            if (k == n) mma_commit(bar(Z_FREE, zs));
                            wc += last;
                        } else {
                            if (k > 1) {
                                dz_half(gs, (dc - 1) & 1u, true);
                                mma_commit(bar(DZ_FULL, (dc - 1) & 1u));
                            }
                            // the accumulator was last read by the epilogue of the chunk before the previous one
                            if (dc >= 2 && !mbar_wait(bar(DZ_EMPTY, dc & 1u), ((dc - 2) >> 1) & 1u, 14)) { ok = false; break; }
                            tc_fence_after();
                            dz_half(gs, dc & 1u, false);
                        }
                    }
                    if (!ok) break;
                    mma_commit(bar(G_FREE, gs));
                }
                if (!ok) break;
                const uint32_t gs = gc % NG;
                if (!mbar_wait(bar(G_FULL, gs), (gc / NG) & 1u, 15)) break;
                tc_fence_after();
                dz_half(gs, (dc - 1) & 1u, true);
                mma_commit(bar(DZ_FULL, (dc - 1) & 1u));
                mma_commit(bar(G_FREE, gs));
                ++gc;
            }
        }
    } else if (warp == W_TMA) {
        if (lane == 0) {
            // ======== TMA issue ======================================================================================
            tma_prefetch_desc(&maps.dy); tma_prefetch_desc(&maps.x); tma_prefetch_desc(&maps.Bg); tma_prefetch_desc(&maps.C);
            tma_prefetch_desc(&maps.y2);
            uint32_t gc = 0, zc = 0;
            bool ok = true;
            for (int t = 0; t < nmine && ok; ++t) {
                const int col = item_group(t) * CH;
                Stream st[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) st[s] = stream_of(a, item_set(t), s);
                for (int k = 0; k <= n + 1; ++k) {
                    if (k <= n) {
                        const uint32_t xs = zc % NXS, full = bar(X_FULL, xs), dst = sm_u + OFF_X + xs * X_STAGE;
                        if (zc >= NXS && !mbar_wait(bar(X_FREE, xs), ((zc - NXS) / NXS) & 1u, 20)) { ok = false; break; }
                        mbar_expect_tx(full, X_STAGE);
#pragma unroll
                        for (int s = 0; s < NS; ++s) {
                            const int row = st[s].ts + (k - 1) * CHUNK;
                            tma_load_3d(dst + s * BOX, &maps.x, full, col, row, st[s].b);
                            tma_load_3d(dst + (NS + s) * BOX, &maps.Bg, full, col, row, st[s].b);
                        }
                        ++zc;
                    }
                    if (k >= 1) {
                        const uint32_t ds = gc % NDS, full = bar(D_FULL, ds), dst = sm_u + OFF_D + ds * D_STAGE;
                        if (gc >= NDS && !mbar_wait(bar(D_FREE, ds), ((gc - NDS) / NDS) & 1u, 21)) { ok = false; break; }
                        mbar_expect_tx(full, k <= n ? D_STAGE : 2 * NS * BOX);
#pragma unroll
                        for (int s = 0; s < NS; ++s) {
                            const int row = st[s].ts + (k - 1) * CHUNK;
                            tma_load_3d(dst + s * BOX, &maps.dy, full, col, row, st[s].b);
                            tma_load_3d(dst + (NS + s) * BOX, &maps.C, full, col, row, st[s].b);
                            if (k <= n) tma_load_3d(dst + (2 * NS + s) * BOX, &maps.y2, full, col, row, st[s].b);
                        }
                        ++gc;
                    }
                }
            }
        }
    } else {
        // ======== dh: W out of TMEM after every other chunk, its anti-diagonals summed in fp32 registers over the item ============
        const int e = warp % 4;                              // the lane quarter that this warp may read
        const uint32_t lane_base = tmem + ((uint32_t)(e * 32) << 16);
        // Anti-diagonals of W: row i (g2 at time 127 - i of the chunk) and column c (z at time c - 128 of it) meet at lag
        // 255 - i - c, so a sum that moves one lane up per column to the left stays on its lag.  Columns from 255 - 32 e on
        // leftwards hold the lags of this warp's rows, K + 31 of them those below K; four independent runs of a quarter of
        // them hide the shuffle's latency.  Run q's lag rl q - 32 + p is complete in its word p: what has left lane 31 before
        // its column p, or, from rl on, what lane rl + 31 - p holds at the end.  All go to shared memory (as vectors: shared
        // memory and shuffles share a pipe that the tiles keep busy), and the sum over the runs is added to the lane's lags.
        const int rl = (K + 31 + 8 * RUNS - 1) / (8 * RUNS) * 8;
        const uint32_t sums = sm_u + OFF_RUNS + e * (RUNS * RUN_LAGS * 4);
        auto read_w = [&](float (&dw)[CHUNK / 32]) {
            float run[RUNS] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int c0 = 0; c0 < rl; c0 += 8) {
                uint32_t w8[RUNS][8];
#pragma unroll
                for (int q = 0; q < RUNS; ++q) tmem_ld8(lane_base + W_COL + (uint32_t)(255 - 32 * e - rl * q - c0 - 7), w8[q]);
                tmem_ld8_wait(w8[0], w8[1]);
                tmem_ld8_wait(w8[2], w8[3]);
                // the shuffle goes round: lane 0 gets what left lane 31, word c0 + j of the run
                float left[RUNS][8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int q = 0; q < RUNS; ++q) {
                        left[q][j] = __shfl_sync(0xffffffffu, run[q], lane + 31);
                        run[q] = (lane ? left[q][j] : 0.f) + __uint_as_float(w8[q][7 - j]);
                    }
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < RUNS; ++q)
#pragma unroll
                        for (int j = 0; j < 8; j += 4)
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(sums + (uint32_t)((q * RUN_LAGS + c0 + j) * 4)), "f"(left[q][j]),
                                         "f"(left[q][j + 1]), "f"(left[q][j + 2]), "f"(left[q][j + 3]) : "memory");
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(W_EMPTY, 0));
#pragma unroll
            for (int q = 0; q < RUNS; ++q)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(sums + (uint32_t)((q * RUN_LAGS + rl + 31 - lane) * 4)), "f"(run[q]) : "memory");
            __syncwarp();
#pragma unroll
            for (int m = 0; m < CHUNK / 32; ++m) {
                float v = 0.f;
#pragma unroll
                for (int q = 0; q < RUNS; ++q) {
                    const int at = 32 * m + lane - rl * q + 32;
                    if (at >= 1 && at < rl + 32) {
                        float u;
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u) : "r"(sums + (uint32_t)((q * RUN_LAGS + at) * 4)) : "memory");
                        v += u;
                    }
                }
                dw[m] += v;
            }
            __syncwarp();
        };
        uint32_t wc = 0;                      // fillings of W gone through
        bool ok = true;
        for (int t = 0; t < nmine && ok; ++t) {
            const int g = item_group(t);
            float dw[CHUNK / 32] = {};
            for (int k = WCHUNKS; k < n + WCHUNKS; k += WCHUNKS, ++wc) {
                if (!mbar_wait(bar(W_FULL, 0), wc & 1u, 8)) { ok = false; break; }
                tc_fence_after();
                __syncwarp();
                read_w(dw);
            }
            if (!ok) break;
            float* const dh = a.dh + (int64_t)((unsigned)(g * CH) / (unsigned)a.dg) * K;
#pragma unroll
            for (int m = 0; m < CHUNK / 32; ++m) {
                const int lag = 32 * m + lane;
                float v = dw[m];
                if (__any_sync(0xffffffffu, lag < K && !isfinite(v))) {
                    v = 0.f;
#pragma unroll 1
                    for (int s = 0; s < NS; ++s) {
                        const Stream st = stream_of(a, item_set(t), s);
                        if (st.active) v += dw_under_taps(a, st.b, (int64_t)g * CH, st.ts, st.te, CHUNK - 32 * (e + 1), lag);
                    }
                }
                if (lag < K) atomicAdd(dh + (K - 1 - lag), v);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// Segment length: the busiest CTA's steps, an item costing its chunks and about two more (two half halo steps, the sums
// along W, the next operand); ties go to fewer segments.
static void plan_items(Args& a) {
    const int64_t total = ceil_div<int64_t>(a.L, CHUNK);
    int64_t nseg = 1, best = INT64_MAX;
    for (int64_t seg = total; seg >= 1; --seg) {
        const int64_t ns = ceil_div<int64_t>(total, seg);
        if (ceil_div<int64_t>(total, ns) != seg) continue;
        const int64_t items = a.G * ceil_div<int64_t>(a.B * ns, NS);
        const int64_t cost = ceil_div<int64_t>(items, kNumSMs) * (seg + 2) * 64 + ns;
        if (cost < best) { best = cost; nseg = ns; }
        if (seg <= 2 || items > (int64_t)kNumSMs * 64) break;
    }
    a.seg_len = ceil_div<int64_t>(total, nseg) * CHUNK;
    a.nseg = ceil_div<int64_t>(a.L, a.seg_len);
    a.nstream = a.B * a.nseg;
    a.nset = ceil_div<int64_t>(a.nstream, NS);
    a.nitems = a.G * a.nset;
}

// Calls the kernel takes (the caller has checked the 16-byte alignment of every operand row); every other one runs the fp32
// kernels of gcg_bwd.cu.  A tensor map steps by positive pitches only, so expanded operands are among the others.
bool takes(const vtx_gcg_bwd_params* p) {
    auto al32 = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 32 == 0; };
    auto pitch = [&](int64_t sb, int64_t sl) {
        constexpr int64_t most = (int64_t)1 << 38;
        return sl > 0 && sl < most && (p->B == 1 || (sb > 0 && sb < most)) && sl * p->L < most;
    };
    return p->io_dtype == VTX_BF16 && p->h_dtype == VTX_BF16 && p->K <= CHUNK && (p->D / p->G) % CH == 0 && p->L < ((int64_t)1 << 30) &&
           p->D < ((int64_t)1 << 31) && al32(p->dx) && al32(p->dB) && al32(p->dC) && pitch(p->dy_stride_b, p->dy_stride_l) &&
           pitch(p->x_stride_b, p->x_stride_l) && pitch(p->b_stride_b, p->b_stride_l) && pitch(p->c_stride_b, p->c_stride_l) &&
           pitch(p->y2_stride_b, p->y2_stride_l) &&
           p->D / CH * ceil_div<int64_t>(p->B * ceil_div<int64_t>(p->L, CHUNK), NS) < ((int64_t)1 << 30);
}

int launch(const vtx_gcg_bwd_params* p, cudaStream_t stream) {
    Args a{};
    a.h = static_cast<const __nv_bfloat16*>(p->h);
    a.dx = static_cast<__nv_bfloat16*>(p->dx); a.dB = static_cast<__nv_bfloat16*>(p->dB); a.dC = static_cast<__nv_bfloat16*>(p->dC);
    a.dh = p->dh32;
    a.dy = static_cast<const __nv_bfloat16*>(p->dy); a.x = static_cast<const __nv_bfloat16*>(p->x);
    a.Bg = static_cast<const __nv_bfloat16*>(p->Bg); a.C = static_cast<const __nv_bfloat16*>(p->C);
    a.dy_sb = p->dy_stride_b; a.dy_sl = p->dy_stride_l; a.x_sb = p->x_stride_b; a.x_sl = p->x_stride_l;
    a.b_sb = p->b_stride_b; a.b_sl = p->b_stride_l; a.c_sb = p->c_stride_b; a.c_sl = p->c_stride_l;
    a.B = p->B; a.L = p->L; a.D = p->D; a.G = p->D / CH; a.K = p->K; a.dg = p->D / p->G;
    plan_items(a);
    Maps maps;
    auto map = [&](CUtensorMap* m, const void* base, int64_t sb, int64_t sl) {
        return make_tmap_3d(m, base, VTX_BF16, p->D, p->L, p->B, sl, sb, CH, CHUNK, 0, "gcg_bwd");
    };
    if (int rc = map(&maps.dy, p->dy, p->dy_stride_b, p->dy_stride_l)) return rc;
    if (int rc = map(&maps.x, p->x, p->x_stride_b, p->x_stride_l)) return rc;
    if (int rc = map(&maps.Bg, p->Bg, p->b_stride_b, p->b_stride_l)) return rc;
    if (int rc = map(&maps.C, p->C, p->c_stride_b, p->c_stride_l)) return rc;
    if (int rc = map(&maps.y2, p->y2, p->y2_stride_b, p->y2_stride_l)) return rc;
    static bool attr_set[64] = {};
    static int resident[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const bool known = dev >= 0 && dev < 64;
    if (!known || !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gcg_bwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return fail(VTX_ERR_LAUNCH, "gcg_bwd: shared memory opt-in: %s", cudaGetErrorString(e));
        if (known) attr_set[dev] = true;
    }
    int nres = known ? resident[dev] : 0;
    if (nres == 0) {
        cudaDeviceGetAttribute(&nres, cudaDevAttrMultiProcessorCount, dev);      // one CTA per SM: shared memory and TMEM
        if (known) resident[dev] = nres;
    }
    // launches of about 1000 steps per CTA (the forward kernel's 500 chunks of four streams): the CTAs drift apart over
    // longer ones
    int64_t rounds = 1000 / (a.seg_len / CHUNK + 2);
    if (rounds < 1) rounds = 1;
    long long launches = 0;
    for (int64_t i0 = 0; i0 < a.nitems; i0 += rounds * nres, ++launches) {
        a.item0 = i0;
        a.item1 = i0 + rounds * nres < a.nitems ? i0 + rounds * nres : a.nitems;
        const int64_t m = a.item1 - a.item0;
        gcg_bwd_tc_kernel<<<(unsigned)(m < nres ? m : nres), THREADS, SMEM_BYTES, stream>>>(maps, a);
    }
    return check_launch("gcg_bwd", launches);
}

}  // namespace gbt
}  // namespace vtx
