// A modal system of one channel in a thread's registers: parameters and state of up to 16 modes, the recurrence
// sigma_s <- p_s sigma_s + x and its output sum_s Re(R_s sigma_s).  Shared by the channel-last and channel-first kernels.
#pragma once

#include "common.cuh"
#include "umma.cuh"

namespace vtx {
namespace modal {

using umma::f32x2;
using umma::fma2;
using umma::pk2;
using umma::up2;

constexpr int NS = 16;         // states per thread (shorter systems are padded with p = R = 0)
// floats of a state vector
template <bool CPLX> constexpr int comps(int S) { return CPLX ? 2 * S : S; }

template <bool CPLX>
struct Modes {
    float pr[NS], pi[CPLX ? NS : 1], rr[NS], ri[CPLX ? NS : 1];
    __device__ __forceinline__ void load(const vtx_modal_params& m, int64_t g) {
        const int S = (int)m.S;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            pr[s] = rr[s] = 0.f;
            if constexpr (CPLX) pi[s] = ri[s] = 0.f;
            if (s < S) {
                const float mag = expf(static_cast<const float*>(m.log_poles)[g * S + s]);
                rr[s] = static_cast<const float*>(m.res_re)[g * S + s];
                if constexpr (CPLX) {
                    float sn, cs;
                    sincosf(static_cast<const float*>(m.theta)[g * S + s], &sn, &cs);
                    pr[s] = mag * cs; pi[s] = mag * sn;
                    ri[s] = m.res_im ? static_cast<const float*>(m.res_im)[g * S + s] : 0.f;
                } else {
                    pr[s] = mag;
                }
            }
        }
    }
};

// Real systems keep poles, residues and states as f32x2 pairs: one packed FMA advances two states.
template <bool CPLX> struct Sys;

template <>
struct Sys<false> {
    f32x2 p2[NS / 2], r2[NS / 2], s2[NS / 2];
    __device__ __forceinline__ void init(const Modes<false>& m) {
#pragma unroll
        for (int j = 0; j < NS / 2; ++j) {
            p2[j] = pk2(m.pr[2 * j], m.pr[2 * j + 1]);
            r2[j] = pk2(m.rr[2 * j], m.rr[2 * j + 1]);
            s2[j] = pk2(0.f, 0.f);
        }
    }
    // components j < n of a state vector stored with the given stride
    __device__ __forceinline__ void load(const float* in, int64_t stride, int n) {
#pragma unroll
        for (int j = 0; j < NS / 2; ++j) {
            const float lo = 2 * j < n ? in[(2 * j) * stride] : 0.f;
            const float hi = 2 * j + 1 < n ? in[(2 * j + 1) * stride] : 0.f;
            s2[j] = pk2(lo, hi);
        }
    }
    __device__ __forceinline__ void store(float* out, int64_t stride, int n) const {
#pragma unroll
        for (int j = 0; j < NS / 2; ++j) {
            float lo, hi;
            up2(s2[j], lo, hi);
            if (2 * j < n) out[(2 * j) * stride] = lo;
            if (2 * j + 1 < n) out[(2 * j + 1) * stride] = hi;
        }
    }
    __device__ __forceinline__ void advance(float x) {
        const f32x2 x2 = pk2(x, x);
#pragma unroll
        for (int j = 0; j < NS / 2; ++j) s2[j] = fma2(p2[j], s2[j], x2);
    }
    __device__ __forceinline__ float step(float x) {
        const f32x2 x2 = pk2(x, x);
        f32x2 a0 = pk2(0.f, 0.f), a1 = a0;
#pragma unroll
        for (int j = 0; j < NS / 2; j += 2) {
            s2[j] = fma2(p2[j], s2[j], x2);
            s2[j + 1] = fma2(p2[j + 1], s2[j + 1], x2);
            a0 = fma2(r2[j], s2[j], a0);
            a1 = fma2(r2[j + 1], s2[j + 1], a1);
        }
        float u0, u1;
        up2(umma::add2(a0, a1), u0, u1);
        return u0 + u1;
    }
};

template <>
struct Sys<true> {
    float pr[NS], pi[NS], rr[NS], ri[NS], re[NS], im[NS];
    __device__ __forceinline__ void init(const Modes<true>& m) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            pr[s] = m.pr[s]; pi[s] = m.pi[s]; rr[s] = m.rr[s]; ri[s] = m.ri[s];
            re[s] = im[s] = 0.f;
        }
    }
    // components (re, im interleaved) j < n of a state vector stored with the given stride
    __device__ __forceinline__ void load(const float* in, int64_t stride, int n) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            re[s] = 2 * s < n ? in[(2 * s) * stride] : 0.f;
            im[s] = 2 * s + 1 < n ? in[(2 * s + 1) * stride] : 0.f;
        }
    }
    __device__ __forceinline__ void store(float* out, int64_t stride, int n) const {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            if (2 * s < n) out[(2 * s) * stride] = re[s];
            if (2 * s + 1 < n) out[(2 * s + 1) * stride] = im[s];
        }
    }
    __device__ __forceinline__ void advance(float x) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const float nr = fmaf(pr[s], re[s], fmaf(-pi[s], im[s], x));
            const float ni = fmaf(pr[s], im[s], pi[s] * re[s]);
            re[s] = nr; im[s] = ni;
        }
    }
    __device__ __forceinline__ float step(float x) {
        float acc = 0.f;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const float nr = fmaf(pr[s], re[s], fmaf(-pi[s], im[s], x));
            const float ni = fmaf(pr[s], im[s], pi[s] * re[s]);
            re[s] = nr; im[s] = ni;
            acc = fmaf(rr[s], nr, fmaf(-ri[s], ni, acc));
        }
        return acc;
    }
};

}  // namespace modal
}  // namespace vtx
