// Modal (IIR) long convolution on channel-first tensors, evaluated as the
// recurrence itself:  sigma_s[t] = p_s sigma_s[t-1] + kv[t],
//                     y[t] = q[t] * (sum_s Re(R_s sigma_s[t]) + bias * kv[t]).
// One lane owns one (batch, channel, time segment) and keeps all S <= 16
// states in registers; a warp is 32 neighbouring channels of one segment.  When
// batch*channels alone cannot fill the GPU the sequence is cut into segments and
// the carry is resolved in three phases:
//   A  end state of every segment from a zero start   (reads k, v)
//   B  sequential scan over the segments of a row     (tiny)
//   C  recurrence from the true start state, outputs  (reads q, k, v, writes y)
// With one segment per row only phase C runs.  The state after the last token
// (what the reference extracts with 2*S extra FFTs) is a by-product of C.
//
// Time is contiguous, so a lane's samples lie in a row of their own: the warp moves tiles of 32 rows x 32 samples through
// shared memory (16-byte asynchronous copies, one tile ahead; rows padded by 16 bytes, which makes the lanes' 16-byte
// reads of their own rows conflict-free), and the outputs leave the same way.  Rows whose start or pitch is not a
// multiple of 16 bytes are fetched or stored element by element, 32 samples of a row at a time.  Bound by the issue of the
// fp32 pipe like the channel-last kernels (fused_li_cc.cu).  B=1, L=4001, D=4096, bf16: 94 us from and to aligned rows, 96
// to dense ones (117 when every store waited for its own shared-memory read), 221 from and to dense ones; a thread per row
// that read its own 16 bytes, 4 segments: 510 us (1130 us).
#include "common.cuh"
#include "modal.cuh"

namespace vtx {

using modal::comps;
using modal::Modes;
using modal::Sys;

constexpr int IS = modal::NS;
constexpr int ITHREADS = 128;
constexpr int ITT = 32;       // samples per tile

struct IirPlan {
    int64_t nseg, seg_len;
};

// Scratch a caller of vtx_iir_fwd has always been asked for, and the limit vtx_iir_fwd_noalloc has always refused by: the
// carries of power-of-two segments of at least 512 samples, up to 1024 threads per SM.
static int64_t iir_classic_cuts(int64_t B, int64_t L, int64_t D) {
    int64_t nseg = 1;
    while (B * D * nseg < (int64_t)kNumSMs * 1024 && L / (nseg * 2) >= 512) nseg *= 2;
    return nseg;
}
static int64_t iir_classic_segments(int64_t B, int64_t L, int64_t D) {
    const int64_t nseg = iir_classic_cuts(B, L, D);
    const int64_t seg = ((L + nseg - 1) / nseg + 15) / 16 * 16;
    return (L + seg - 1) / seg;
}
static int64_t iir_carry_bytes(int64_t B, int64_t D, int64_t nseg, int64_t S, bool cplx) {
    return nseg <= 1 ? 0 : B * D * nseg * S * (cplx ? 2 : 1) * (int64_t)sizeof(float);
}

// Segments (whole tiles, at least two): the launch lasts as long as the SM with the most blocks, a sample costs about 55
// issue cycles in phase C and 22 more in phase A, and one block of four warps leaves its scheduler waiting for itself
// about a third of the time.  At most four blocks per SM: more only add carries.  (L=4001, D=4096: 9 segments, two blocks
// per SM, 98 us; 14 segments, which are 4 blocks too many for one round: 116 us.)
static int64_t iir_most_segments(int64_t B, int64_t L, int64_t D) {
    const int64_t by_blocks = (int64_t)kNumSMs * 4 * (ITHREADS / 32) / (B * ceil_div<int64_t>(D, 32)), by_length = L / (2 * ITT);
    const int64_t n = by_blocks < by_length ? by_blocks : by_length;
    return n > 1 ? n : 1;
}
static IirPlan iir_plan(int64_t B, int64_t L, int64_t D) {
    const int64_t warps = B * ceil_div<int64_t>(D, 32), most = iir_most_segments(B, L, D);
    IirPlan best{1, ceil_div<int64_t>(L, ITT) * ITT};
    int64_t best_cost = INT64_MAX;
    for (int64_t n = 1; n <= most; ++n) {
        const int64_t seg = ceil_div<int64_t>(ceil_div<int64_t>(L, n), ITT) * ITT, nseg = ceil_div<int64_t>(L, seg);
        const int64_t per_sm = ceil_div<int64_t>(ceil_div<int64_t>(warps * nseg, ITHREADS / 32), kNumSMs);
        const int64_t cost = seg * (per_sm == 1 ? 3 : 2 * per_sm) * (nseg > 1 ? 77 : 55);
        if (cost < best_cost) { best_cost = cost; best = IirPlan{nseg, seg}; }
    }
    return best;
}

// scratch[(seg * SS + j) * rows + row]: component j of a state vector of row (batch, channel)

// OUT: phase C, else phase A.  RND: k*v, the convolution, the skip term and their sum rounded to the I/O dtype.
template <typename T, bool CPLX, bool OUT, bool RND>
__global__ void __launch_bounds__(ITHREADS) iir_walk_kernel(vtx_iir_params p, IirPlan pl, bool vec_in, bool vec_out) {
    constexpr int N = 16 / sizeof(T), VPR = ITT / N, PITCH = ITT * (int)sizeof(T) + 16, NT = OUT ? 3 : 2;
    constexpr int TILE = 32 * PITCH, STAGES = 2;
    extern __shared__ __align__(16) uint8_t sm_raw[];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint8_t* const sm = sm_raw + warp * (STAGES * NT * TILE);
    const int64_t per_seg = p.B * ceil_div<int64_t>(p.D, 32), wid = (int64_t)blockIdx.x * (ITHREADS / 32) + warp;
    const int64_t seg = wid / per_seg, b = (wid % per_seg) / ceil_div<int64_t>(p.D, 32), c0 = (wid % ceil_div<int64_t>(p.D, 32)) * 32;
    if (seg >= (OUT ? pl.nseg : pl.nseg - 1)) return;      // whole warps; the last segment's end state is not a carry
    const bool valid = c0 + lane < p.D;
    const int64_t d = valid ? c0 + lane : p.D - 1;           // lanes past the last channel walk it again and store nothing
    const int64_t t0 = seg * pl.seg_len, t1 = t0 + pl.seg_len < p.L ? t0 + pl.seg_len : p.L;
    const int64_t rows = p.B * p.D, row = b * p.D + d;
    const int SS = comps<CPLX>((int)p.modal.S);

    const int64_t hn = d / p.head_dim, hj = d % p.head_dim;
    const T* src[NT];           // this lane's rows of k, v (, q)
    src[0] = static_cast<const T*>(p.k) + b * p.k_stride_b + hn * p.k_stride_h + hj * p.k_stride_d;
    src[1] = static_cast<const T*>(p.v) + b * p.v_stride_b + hn * p.v_stride_h + hj * p.v_stride_d;
    if (OUT) src[NT - 1] = static_cast<const T*>(p.q) + b * p.q_stride_b + hn * p.q_stride_h + hj * p.q_stride_d;
    auto row_ptr = [&](const T* mine, int r) {
        return reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), r));
    };
    auto issue = [&](int64_t t, int stage) {
        uint8_t* const dst = sm + stage * (NT * TILE);
        if (vec_in) {
#pragma unroll
            for (int x = 0; x < NT; ++x)
#pragma unroll
                for (int i = 0; i < VPR; ++i) {
                    const int r = i * (32 / VPR) + lane / VPR, v = lane % VPR;
                    const T* rp = row_ptr(src[x], r);
                    const int64_t ts = t + v * N, left = (t1 - ts) * (int64_t)sizeof(T);
                    const int bytes = left >= 16 ? 16 : left > 0 ? (int)left : 0;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + x * TILE + r * PITCH + v * 16)),
                                 "l"(bytes ? rp + ts : rp), "r"(bytes) : "memory");
                }
        } else {
            const bool in = t + lane < t1;
#pragma unroll 1
            for (int x = 0; x < NT; ++x) {
                const T* const mine = x == 0 ? src[0] : x == 1 ? src[1] : src[NT - 1];
                T e[32];
#pragma unroll
                for (int r = 0; r < 32; ++r) {
                    const T* rp = row_ptr(mine, r) + t + lane;
                    e[r] = from_f32<T>(0.f);
                    if (in) e[r] = *rp;
                }
#pragma unroll
                for (int r = 0; r < 32; ++r) *reinterpret_cast<T*>(dst + x * TILE + r * PITCH + lane * sizeof(T)) = e[r];
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int64_t ntile = (t1 - t0 + ITT - 1) / ITT;
    issue(t0, 0);
    if (ntile > 1) issue(t0 + ITT, 1);
    Sys<CPLX> sys;
    {
        Modes<CPLX> md;
        md.load(p.modal, d / (p.D / p.modal.G));
        sys.init(md);
    }
    if (OUT && pl.nseg > 1) sys.load(static_cast<const float*>(p.scratch) + seg * SS * rows + row, rows, SS);
    const float bias = OUT && p.bias ? ld_param(p.bias, p.bias_dtype, d) : 0.f;
    T* const y = OUT ? static_cast<T*>(p.y) + b * p.y_stride_b : nullptr;
    const bool y_rows = p.y_stride_l == 1;

    for (int64_t i = 0; i < ntile; ++i) {
        const int64_t t = t0 + i * ITT;
        if (i + 1 < ntile) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        uint8_t* const tile = sm + (i & 1) * (NT * TILE) + lane * PITCH;
#pragma unroll 1
        for (int v = 0; v < VPR; ++v) {
            alignas(16) T kk[N], vv[N], qq[N];
            *reinterpret_cast<uint4*>(kk) = *reinterpret_cast<const uint4*>(tile + v * 16);
            *reinterpret_cast<uint4*>(vv) = *reinterpret_cast<const uint4*>(tile + TILE + v * 16);
            if (OUT) *reinterpret_cast<uint4*>(qq) = *reinterpret_cast<const uint4*>(tile + (NT - 1) * TILE + v * 16);
            const int64_t ts = t + v * N;
            auto sample = [&](int e) {
                float x = to_f32<T>(kk[e]) * to_f32<T>(vv[e]);
                if (RND) x = round_io<T>(x);
                if (OUT) {
                    const float conv = round_io<T>(sys.step(x));
                    const float z = RND ? round_io<T>(conv + round_io<T>(bias * x)) : fmaf(bias, x, conv);
                    qq[e] = from_f32<T>(z * to_f32<T>(qq[e]));
                } else {
                    sys.advance(x);
                }
            };
            // a whole vector without a branch between its samples (they overlap), the end of a segment sample by sample
            if (ts + N <= t1) {
#pragma unroll
                for (int e = 0; e < N; ++e) sample(e);
            } else {
#pragma unroll
                for (int e = 0; e < N; ++e)
                    if (ts + e < t1) sample(e);
            }
            if (OUT && !y_rows && valid) {
#pragma unroll
                for (int e = 0; e < N; ++e)
                    if (ts + e < t1) y[d * p.y_stride_d + (ts + e) * p.y_stride_l] = qq[e];
            }
            if (OUT && y_rows) *reinterpret_cast<uint4*>(tile + (NT - 1) * TILE + v * 16) = *reinterpret_cast<const uint4*>(qq);
        }
        __syncwarp();
        if (OUT && y_rows) {
            const uint8_t* const out = sm + (i & 1) * (NT * TILE) + (NT - 1) * TILE;
            if (vec_out) {
#pragma unroll
                for (int m = 0; m < VPR; ++m) {
                    const int r = m * (32 / VPR) + lane / VPR, v = lane % VPR;
                    const int64_t ts = t + v * N;
                    T* const dst = y + (c0 + r) * p.y_stride_d + ts;
                    const uint8_t* const from = out + r * PITCH + v * 16;
                    if (c0 + r < p.D) {
                        if (ts + N <= t1) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(from);
                        else
                            for (int e = 0; ts + e < t1; ++e) dst[e] = reinterpret_cast<const T*>(from)[e];
                    }
                }
            } else if (t + lane < t1) {
                T* dst = y + c0 * p.y_stride_d + t + lane;
                const uint8_t* from = out + lane * sizeof(T);
                const int nrow = c0 + 32 <= p.D ? 32 : (int)(p.D - c0);
#pragma unroll 1
                for (int r0 = 0; r0 < nrow; r0 += 16, from += 16 * PITCH) {
                    T e[16];
#pragma unroll
                    for (int r = 0; r < 16; ++r) e[r] = *reinterpret_cast<const T*>(from + r * PITCH);
#pragma unroll
                    for (int r = 0; r < 16; ++r, dst += p.y_stride_d)
                        if (r0 + r < nrow) *dst = e[r];
                }
            }
            __syncwarp();
        }
        if (i + 2 < ntile) issue(t + 2 * ITT, (int)(i & 1));
    }
    if (!valid) return;
    if (!OUT) sys.store(static_cast<float*>(p.scratch) + seg * SS * rows + row, rows, SS);
    else if (p.state && seg == pl.nseg - 1) sys.store(p.state + row * SS, 1, SS);
}

// After this kernel scratch[seg] holds the state at the START of segment seg.
template <bool CPLX>
__global__ void iir_carry_kernel(vtx_iir_params p, IirPlan pl) {
    const int S = (int)p.modal.S, SS = comps<CPLX>(S);
    const int64_t rows = p.B * p.D, i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * S) return;
    const int64_t row = i % rows, d = row % p.D, g = d / (p.D / p.modal.G);
    const int s = (int)(i / rows);
    // p^seg_len in polar form
    float lam = static_cast<const float*>(p.modal.log_poles)[g * S + s];
    float mag = expf(lam * (float)pl.seg_len), pr = mag, pi = 0.f;
    if (CPLX) {
        double a = (double)static_cast<const float*>(p.modal.theta)[g * S + s] * (double)pl.seg_len;
        a -= 6.283185307179586 * floor(a / 6.283185307179586);
        float sn, cs;
        sincosf((float)a, &sn, &cs);
        pr = mag * cs; pi = mag * sn;
    }
    constexpr int C = CPLX ? 2 : 1, NB = 8;      // segments read together: their loads overlap
    float* base = static_cast<float*>(p.scratch) + (int64_t)(C * s) * rows + row;
    const int64_t step = (int64_t)SS * rows;
    float cr = 0.f, ci = 0.f;
    for (int64_t seg = 0; seg < pl.nseg; seg += NB) {
        float er[NB], ei[NB];
#pragma unroll
        for (int m = 0; m < NB; ++m) {          // end states from a zero start (the last segment's was not computed)
            const bool in = seg + m < pl.nseg - 1;
            er[m] = in ? base[(seg + m) * step] : 0.f;
            ei[m] = CPLX && in ? base[(seg + m) * step + rows] : 0.f;
        }
#pragma unroll
        for (int m = 0; m < NB; ++m) {
            if (seg + m >= pl.nseg) break;
            base[(seg + m) * step] = cr;
            if (CPLX) base[(seg + m) * step + rows] = ci;
            const float nr = pr * cr - pi * ci + er[m], ni = pr * ci + pi * cr + ei[m];
            cr = nr; ci = ni;
        }
    }
}

template <typename T, bool CPLX, bool OUT, bool RND>
static int iir_walk(const vtx_iir_params& p, const IirPlan& pl, bool vec_in, bool vec_out, cudaStream_t s) {
    constexpr int smem = (ITHREADS / 32) * 2 * (OUT ? 3 : 2) * 32 * (ITT * (int)sizeof(T) + 16);
    auto kern = iir_walk_kernel<T, CPLX, OUT, RND>;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > 48 * 1024 && (dev < 0 || dev >= 64 || !attr_set[dev])) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail(VTX_ERR_LAUNCH, "iir: shared memory opt-in: %s", cudaGetErrorString(e));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const int64_t warps = p.B * ceil_div<int64_t>(p.D, 32) * (OUT ? pl.nseg : pl.nseg - 1);
    kern<<<(unsigned)ceil_div<int64_t>(warps, ITHREADS / 32), ITHREADS, smem, s>>>(p, pl, vec_in, vec_out);
    return VTX_OK;
}

// The reference's legacy recurrent prefill (vortex/model/engine.py:473-504), step for step: complex poles and
// residues given as (re, im) pairs, the state kept in the I/O dtype (the reference builds it from x1*v, so with bf16
// activations every update is rounded to bf16), and the real part updated in place BEFORE the imaginary part reads
// it:   re' = pr re - pi im + x ;  im' = pr im + pi re'   (not a complex product: that is what the reference
// computes, and its cached state continues from it).  Every product, difference and sum is rounded on its own, as
// the reference's separate tensor operations are.  out[t] = sum_s Re(R_s) re_s[t] in the I/O dtype, then the same
// skip term and gate as the FFT branch.  One thread walks one (batch, channel) row: a compatibility path.
// modal.log_poles holds Re(p), modal.theta Im(p), modal.res_re Re(R), all fp32 [G, S].
template <typename T>
__global__ void __launch_bounds__(ITHREADS) iir_recurrence_kernel(vtx_iir_params p) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B * p.D) return;
    const int64_t b = i / p.D, d = i % p.D, g = d / (p.D / p.modal.G);
    const int S = (int)p.modal.S;
    float pr[IS], pi[IS], rr[IS], re[IS], im[IS];
#pragma unroll
    for (int s = 0; s < IS; ++s) {
        pr[s] = pi[s] = rr[s] = re[s] = im[s] = 0.f;
        if (s < S) {
            pr[s] = static_cast<const float*>(p.modal.log_poles)[g * S + s];
            pi[s] = static_cast<const float*>(p.modal.theta)[g * S + s];
            rr[s] = static_cast<const float*>(p.modal.res_re)[g * S + s];
        }
    }
    const int64_t hn = d / p.head_dim, hj = d % p.head_dim;
    const T* q = static_cast<const T*>(p.q) + b * p.q_stride_b + hn * p.q_stride_h + hj * p.q_stride_d;
    const T* k = static_cast<const T*>(p.k) + b * p.k_stride_b + hn * p.k_stride_h + hj * p.k_stride_d;
    const T* v = static_cast<const T*>(p.v) + b * p.v_stride_b + hn * p.v_stride_h + hj * p.v_stride_d;
    T* y = static_cast<T*>(p.y) + b * p.y_stride_b + d * p.y_stride_d;
    const float bias = p.bias ? ld_param(p.bias, p.bias_dtype, d) : 0.f;
    for (int64_t t = 0; t < p.L; ++t) {
        const float x = round_io<T>(to_f32<T>(k[t]) * to_f32<T>(v[t]));
        float acc = 0.f;
#pragma unroll
        for (int s = 0; s < IS; ++s) {
            const float nr = round_io<T>(__fadd_rn(__fsub_rn(__fmul_rn(pr[s], re[s]), __fmul_rn(pi[s], im[s])), x));
            const float ni = round_io<T>(__fadd_rn(__fmul_rn(pr[s], im[s]), __fmul_rn(pi[s], nr)));
            re[s] = nr; im[s] = ni;
            acc = __fadd_rn(acc, __fmul_rn(rr[s], nr));
        }
        const float conv = round_io<T>(acc);
        const float z = round_io<T>(conv + round_io<T>(bias * x));
        y[t * p.y_stride_l] = from_f32<T>(z * to_f32<T>(q[t]));
    }
    if (p.state) {
        float* so = p.state + (b * p.D + d) * S * 2;
        for (int s = 0; s < S; ++s) { so[2 * s] = re[s]; so[2 * s + 1] = im[s]; }
    }
}

__global__ void modal_filter_kernel(vtx_modal_params m, float* h, int64_t L) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.G * L) return;
    int64_t g = i / L, t = i % L;
    const float* lp = static_cast<const float*>(m.log_poles) + g * m.S;
    const float* rr = static_cast<const float*>(m.res_re) + g * m.S;
    float acc = 0.f;
    for (int s = 0; s < m.S; ++s) {
        float mag = expf(lp[s] * (float)t);
        if (m.theta) {
            double a = (double)static_cast<const float*>(m.theta)[g * m.S + s] * (double)t;
            a -= 6.283185307179586 * floor(a / 6.283185307179586);
            float sn, cs;
            sincosf((float)a, &sn, &cs);
            float ri = m.res_im ? static_cast<const float*>(m.res_im)[g * m.S + s] : 0.f;
            acc += mag * (rr[s] * cs - ri * sn);
        } else {
            acc += rr[s] * mag;
        }
    }
    h[i] = acc;
}

static int check_modal(const vtx_modal_params& m, const char* who) {
    VTX_REQUIRE(m.log_poles && m.res_re, VTX_ERR_BAD_ARG, "%s: null poles/residues", who);
    VTX_REQUIRE(m.G > 0 && m.S > 0, VTX_ERR_BAD_ARG, "%s: G and S must be positive", who);
    VTX_REQUIRE(!m.res_im || m.theta, VTX_ERR_BAD_ARG, "%s: complex residues need complex poles", who);
    return VTX_OK;
}

}  // namespace vtx

extern "C" int vtx_modal_filter(const vtx_modal_params* m, float* h, int64_t L, void* stream) {
    using namespace vtx;
    VTX_REQUIRE(m && h && L > 0, VTX_ERR_BAD_ARG, "modal_filter: bad argument");
    if (int rc = check_modal(*m, "modal_filter")) return rc;
    int64_t n = m->G * L;
    modal_filter_kernel<<<(unsigned)ceil_div<int64_t>(n, 256), 256, 0, (cudaStream_t)stream>>>(*m, h, L);
    return check_launch("modal_filter");
}

extern "C" int64_t vtx_iir_scratch_bytes(int64_t B, int64_t L, int64_t D, int64_t S, int64_t complex_poles) {
    using namespace vtx;
    if (B <= 0 || L <= 0 || D <= 0 || S <= 0) return 0;
    // The most segments a plan may have, not those it does have after rounding (D=4096: 14 at L=1156, 9 at L=4096): the
    // bytes never fall as L grows, so that a buffer sized for the longest sequence serves every shorter one.
    const int64_t now = iir_most_segments(B, L, D), classic = iir_classic_cuts(B, L, D);
    return iir_carry_bytes(B, D, now > classic ? now : classic, S, complex_poles != 0);
}

extern "C" int vtx_iir_fwd(const vtx_iir_params* p, void* stream) {
    using namespace vtx;
    VTX_REQUIRE(p && p->q && p->k && p->v && p->y, VTX_ERR_BAD_ARG, "iir: null pointer");
    VTX_REQUIRE(p->B > 0 && p->L > 0 && p->D > 0, VTX_ERR_BAD_ARG, "iir: sizes must be positive");
    VTX_REQUIRE(p->head_dim > 0 && p->D % p->head_dim == 0, VTX_ERR_BAD_ARG, "iir: head_dim must divide D");
    if (int rc = check_modal(p->modal, "iir")) return rc;
    VTX_REQUIRE(p->D % p->modal.G == 0, VTX_ERR_BAD_ARG, "iir: D not a multiple of the number of modal systems");
    VTX_REQUIRE(p->modal.S <= IS, VTX_ERR_UNSUPPORTED, "iir: state size %lld > %d", (long long)p->modal.S, IS);
    const bool cplx = p->modal.theta != nullptr;
    IirPlan pl = iir_plan(p->B, p->L, p->D);
    VTX_REQUIRE(iir_classic_segments(p->B, p->L, p->D) == 1 || p->scratch, VTX_ERR_BAD_ARG, "iir: scratch needed (%lld bytes)",
                (long long)vtx_iir_scratch_bytes(p->B, p->L, p->D, p->modal.S, cplx));
    if (!p->scratch) pl = IirPlan{1, ceil_div<int64_t>(p->L, ITT) * ITT};      // sizes that need none
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t es = dtype_size(p->io_dtype);
    auto al = [&](const void* q, int64_t s0, int64_t s1, int64_t s2) {
        return (reinterpret_cast<uintptr_t>(q) | (uintptr_t)(s0 * es) | (uintptr_t)(s1 * es) | (uintptr_t)(s2 * es)) % 16 == 0;
    };
    const bool vec_in = al(p->q, p->q_stride_b, p->q_stride_h, p->q_stride_d) && al(p->k, p->k_stride_b, p->k_stride_h, p->k_stride_d) &&
                        al(p->v, p->v_stride_b, p->v_stride_h, p->v_stride_d);
    const bool vec_out = al(p->y, p->y_stride_b, p->y_stride_d, 0);
    VTX_REQUIRE(ceil_div<int64_t>(p->B * ceil_div<int64_t>(p->D, 32) * pl.nseg, ITHREADS / 32) < ((int64_t)1 << 31), VTX_ERR_UNSUPPORTED,
                "iir: problem too large");
    int rc = VTX_OK;
    VTX_DISPATCH_IO(p->io_dtype, T, {
        auto walk = [&](bool c, bool out, bool rnd) {
            auto go = [&](auto f) { return f(*p, pl, vec_in, vec_out, s); };
            if (c) return out ? (rnd ? go(iir_walk<T, true, true, true>) : go(iir_walk<T, true, true, false>))
                              : (rnd ? go(iir_walk<T, true, false, true>) : go(iir_walk<T, true, false, false>));
            return out ? (rnd ? go(iir_walk<T, false, true, true>) : go(iir_walk<T, false, true, false>))
                       : (rnd ? go(iir_walk<T, false, false, true>) : go(iir_walk<T, false, false, false>));
        };
        if (pl.nseg > 1) {
            rc = walk(cplx, false, p->round_kv != 0);
            if (rc) return rc;
            const int64_t nc = p->B * p->D * p->modal.S;
            if (cplx) iir_carry_kernel<true><<<(unsigned)ceil_div<int64_t>(nc, 128), 128, 0, s>>>(*p, pl);
            else iir_carry_kernel<false><<<(unsigned)ceil_div<int64_t>(nc, 128), 128, 0, s>>>(*p, pl);
        }
        rc = walk(cplx, true, p->round_kv != 0);
        if (rc) return rc;
    });
    return check_launch("iir", pl.nseg > 1 ? 3 : 1);
}

extern "C" int vtx_iir_recurrence_fwd(const vtx_iir_params* p, void* stream) {
    using namespace vtx;
    VTX_REQUIRE(p && p->q && p->k && p->v && p->y, VTX_ERR_BAD_ARG, "iir(recurrence): null pointer");
    VTX_REQUIRE(p->B > 0 && p->L > 0 && p->D > 0, VTX_ERR_BAD_ARG, "iir(recurrence): sizes must be positive");
    VTX_REQUIRE(p->head_dim > 0 && p->D % p->head_dim == 0, VTX_ERR_BAD_ARG, "iir(recurrence): head_dim must divide D");
    VTX_REQUIRE(p->modal.log_poles && p->modal.theta && p->modal.res_re, VTX_ERR_BAD_ARG,
                "iir(recurrence): Re(p), Im(p) and Re(R) are needed");
    VTX_REQUIRE(p->modal.G > 0 && p->modal.S > 0 && p->D % p->modal.G == 0, VTX_ERR_BAD_ARG,
                "iir(recurrence): D not a multiple of the number of modal systems");
    VTX_REQUIRE(p->modal.S <= IS, VTX_ERR_UNSUPPORTED, "iir(recurrence): state size %lld > %d", (long long)p->modal.S, IS);
    const unsigned blocks = (unsigned)ceil_div<int64_t>(p->B * p->D, ITHREADS);
    VTX_DISPATCH_IO(p->io_dtype, T, { iir_recurrence_kernel<T><<<blocks, ITHREADS, 0, (cudaStream_t)stream>>>(*p); });
    return check_launch("iir(recurrence)");
}

// ---------------------------------------------------------------------------------------------------
// vtx_iir_fwd_noalloc: the same modal long convolution for callers that cannot allocate device memory.
//
// Some hosts of this library may not call cudaMalloc (or torch's allocator) at the point where they need the
// operator: an inference server that handed all free HBM to its KV-cache pool at start-up, a plain C caller
// that has no allocator of its own on the device, or code in the middle of a latency-critical loop where an
// allocation could stall or fail.  vtx_iir_fwd asks such a caller for a scratch buffer (the carries between
// time segments).  This variant brings its own: a fixed array in device global memory that is part of the
// library image, so every GPU that loads the library sets VTX_IIR_STATIC_SCRATCH_BYTES aside until the
// process exits.  Inputs and outputs are still the caller's.
//
// * Sizes whose carries do not fit are refused with VTX_ERR_UNSUPPORTED (vtx_iir_scratch_bytes is an upper bound of
//   them); nothing is launched.  (What the launch's own plan needs always fits: at
//   most 148 * 16 * 32 carries of at most 16 complex states, 9.3 of the 16 MiB.)
// * The first call on a device looks the array's device address up (cudaGetSymbolAddress with that device
//   current -- the array's name is only a host-side handle, never a pointer a kernel could use) and keeps it
//   per device.  Make that first call outside any stream capture -- and during start-up, before the host
//   commits the rest of the device memory: with CUDA's default lazy module loading the array is reserved on a
//   device when this file's module is first used there (this call, vtx_iir_fwd or vtx_modal_filter), not when
//   the library is loaded.
// * Calls of L < 1024, or of 148 * 1024 rows and more, do not touch the array (one segment per row).  All others
//   share it, and it keeps whatever the last of them left in it.  Nothing in it has to be zero at the start: every
//   word a call reads was written earlier by the same call.  Two of these that overlap on the GPU (different
//   streams, or different host threads) race on the array: serialise them.
// * No cudaMalloc / cudaFree / allocating library routine is called on this path.
constexpr size_t kIirStaticScratchBytes = VTX_IIR_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_iir_static_scratch[kIirStaticScratchBytes];

extern "C" int vtx_iir_fwd_noalloc(const vtx_iir_params* p, void* stream) {
    using namespace vtx;
    VTX_REQUIRE(p, VTX_ERR_BAD_ARG, "iir(noalloc): null parameter block");
    VTX_REQUIRE(p->B > 0 && p->L > 0 && p->D > 0 && p->modal.S > 0, VTX_ERR_BAD_ARG, "iir(noalloc): sizes must be positive");
    const bool cplx = p->modal.theta != nullptr;
    const int64_t need = iir_carry_bytes(p->B, p->D, iir_classic_segments(p->B, p->L, p->D), p->modal.S, cplx);
    VTX_REQUIRE(need <= (int64_t)kIirStaticScratchBytes, VTX_ERR_UNSUPPORTED,
                "iir(noalloc): this size needs %lld bytes of carries, the built-in scratch holds %lld; "
                "use vtx_iir_fwd with a caller-provided buffer",
                (long long)need, (long long)kIirStaticScratchBytes);
    constexpr int kMaxDevices = 64;
    static void* dev_ptr[kMaxDevices] = {nullptr};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(VTX_ERR_LAUNCH, "iir(noalloc): cudaGetDevice: %s", e == cudaSuccess ? "device index out of range" : cudaGetErrorString(e));
    if (!dev_ptr[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_iir_static_scratch);
        if (e != cudaSuccess || !ptr) return fail(VTX_ERR_LAUNCH, "iir(noalloc): cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        dev_ptr[dev] = ptr;
    }
    vtx_iir_params q = *p;
    // one segment per row where vtx_iir_fwd accepts no scratch: such calls may overlap
    q.scratch = iir_classic_segments(p->B, p->L, p->D) == 1 ? nullptr : dev_ptr[dev];
    return vtx_iir_fwd(&q, stream);
}
