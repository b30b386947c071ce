// Delay-and-sum kernel template (Tabbed tables or Synthetic geometry).
//
// One thread per pixel; a CTA covers kBlock consecutive table columns (the
// host may store the tables in a locality-friendly pixel order and pass
// pixel_index to scatter the results back).  Loop order: receive outer,
// transmit inner.  The transmit-side delays and weights of a pixel are loaded
// (Tabbed) or computed (Synthetic) once, into registers when ntx <= kTxReg;
// beyond, the delays go to this thread's column of shared memory and the
// Tabbed weights are read from the table per receive (L1-resident rows);
// receive-side values are loaded or computed once per receive.  Each tap gathers one coefficient
// record of its channel (cubic) or one/two samples (nearest/linear) through
// the read-only path and accumulates in registers: no atomics, one store per
// output element.
//
// Tap decisions follow the reference's float32 C path exactly:
//   apod = apodtx*apodrx (one rounding), contributes iff |apod| >= thresh
//   x = tautx + taurx (one rounding); cubic/linear need t0 <= x <= xmax with
//   xmax = t0 + dt*(nt-1) rounded as two operations (pycbf.c:77,84);
//   knot j = (int)((x - t0)/dt) and nearest it = (int)((x - t0)/dt + 0.5)
//   use the correctly rounded quotient: the fast reciprocal product is used
//   unless its fraction lies within eps of the decision boundary, where the
//   IEEE division is taken instead.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace pgb {

constexpr int kTxReg = 12;
// Over receives, TX_AND_RX images are summed in blocks of kRxBlockSum consecutive
// receive indices: the sum over blocks, in order, of each block's sequential
// sum.  Every kernel (generic, staged, batched) sums this way, so they agree
// bit for bit, and the staged kernel can hand a tile's blocks to different CTAs.
constexpr int kRxBlockSum = 64;
constexpr float kDxMin = 1e-12f;

// (int)fl for an integral float 0 <= fl < 2^23 without a conversion instruction
__device__ __forceinline__ int small_int(float fl) {
    return __float_as_int(__fadd_rn(fl, 8388608.0f)) - 0x4B000000;
}

// The interpolation fractions as the reference rounds them (pycbf.c:93-98):
// xhi = t0 + dt*(j+1), xlo = t0 + dt*j, a = (xhi - x)/dt, b = (x - xlo)/dt.
// x carries ~q*2^-24 of rounding relative to dt, so deriving b from the
// quotient instead would differ from the reference by that much.
__device__ __forceinline__ void knot_fractions(float x, float fj, const DasArgs &a, float &am,
                                               float &b) {
    const float xlo = __fadd_rn(a.t0, __fmul_rn(a.dt, fj));
    const float xhi = __fadd_rn(a.t0, __fmul_rn(a.dt, __fadd_rn(fj, 1.0f)));
    am = __fmul_rn(__fsub_rn(xhi, x), a.inv_dt);
    b = __fmul_rn(__fsub_rn(x, xlo), a.inv_dt);
}

// ---------------------------------------------------------------------------
// Interpolation kinds.  Each tap goes through
//   index(x)        fast: in-range flag, sample index, and whether the
//                   reciprocal quotient sits within eps of a decision boundary
//   index_exact(x)  the same with the IEEE quotient (taken only when flagged)
//   load(idx)       the channel payload (one 16/8-byte record or 1-2 samples)
//   value(payload)  the interpolated sample
// so that a thread can put the gathers of several taps in flight at once.
// ---------------------------------------------------------------------------
template <int KIND, typename T> struct Kind;

template <typename T> struct Kind<PYCBF_GB_INTERP_CUBIC, T> {
    using P = float4;
    static __device__ __forceinline__ bool index(float x, const DasArgs &a, int &idx, bool &fix) {
        const bool inr = (x >= a.t0) && (x <= a.xmax);
        const float q = __fmul_rn(__fsub_rn(x, a.t0), a.inv_dt);
        const float fl = floorf(q);
        const float f = q - fl;
        fix = (f < a.eps) || (f > 1.f - a.eps);
        idx = min(small_int(fl), a.nt - 1);
        return inr;
    }
    static __device__ __forceinline__ bool index_exact(float x, const DasArgs &a, int &idx) {
        idx = min((int)floorf(__fdiv_rn(__fsub_rn(x, a.t0), a.dt)), a.nt - 1);
        return (x >= a.t0) && (x <= a.xmax);
    }
    static __device__ __forceinline__ P load(const void *data, long long ch, int idx,
                                            const DasArgs &a) {
        using rec = typename CoefRec<T>::raw;
        return CoefRec<T>::load(static_cast<const rec *>(data) + ch + idx);
    }
    // fj: the knot index as a float (exact: j < 2^23).
    // float32 records: b = (x - xlo) / dt with xlo = fl(t0 + fl(dt j)) as the
    // reference rounds it (x - xlo is exact), then the interval's polynomial.
    // 16-bit records (y, z): knot positions (xhi, xlo), fractions (a, b) and
    // cubic weights in packed float32 pairs, each lane rounded as
    // knot_fractions rounds it; b comes from (xlo - x) * -1/dt, the same bits
    // as (x - xlo) * 1/dt.
    static __device__ __forceinline__ float value(const P &c, float x, float fj, const DasArgs &a) {
        if constexpr (CoefRec<T>::kPoly) {
            const float xlo = __fadd_rn(a.t0, __fmul_rn(a.dt, fj));
            const float b = __fmul_rn(__fsub_rn(x, xlo), a.inv_dt);
            return fmaf(fmaf(fmaf(c.w, b, c.z), b, c.y), b, c.x);
        } else {
            const float2 K = add2_rn(make_float2(a.t0, a.t0),
                                     make_float2(__fmul_rn(a.dt, __fadd_rn(fj, 1.0f)), __fmul_rn(a.dt, fj)));
            const float2 AB = mul2_rn(add2_rn(K, make_float2(-x, -x)), make_float2(a.inv_dt, -a.inv_dt));
            const float2 W = fma2_rn(mul2_rn(AB, AB), AB, make_float2(-AB.x, -AB.y));
            return fmaf(AB.x, c.x, fmaf(AB.y, c.y, fmaf(W.x, c.z, W.y * c.w)));
        }
    }
    // dS/dx at x (the delay derivative of the adjoint): d(b)/dx = 1/dt, d(a)/dx = -1/dt
    static __device__ __forceinline__ float slope(const P &c, float x, float fj, const DasArgs &a) {
        if constexpr (CoefRec<T>::kPoly) {
            const float xlo = __fadd_rn(a.t0, __fmul_rn(a.dt, fj));
            const float b = __fmul_rn(__fsub_rn(x, xlo), a.inv_dt);
            return fmaf(fmaf(3.f * c.w, b, 2.f * c.z), b, c.y) * a.inv_dt;
        } else {
            float am, b;
            knot_fractions(x, fj, a, am, b);
            const float da = fmaf(3.f * am, am, -1.f);
            const float db = fmaf(3.f * b, b, -1.f);
            return (c.y - c.x + fmaf(db, c.w, -da * c.z)) * a.inv_dt;
        }
    }
};

template <typename T> struct Kind<PYCBF_GB_INTERP_LINEAR, T> {
    using P = float2;
    static __device__ __forceinline__ bool index(float x, const DasArgs &a, int &idx, bool &fix) {
        return Kind<PYCBF_GB_INTERP_CUBIC, T>::index(x, a, idx, fix);
    }
    static __device__ __forceinline__ bool index_exact(float x, const DasArgs &a, int &idx) {
        return Kind<PYCBF_GB_INTERP_CUBIC, T>::index_exact(x, a, idx);
    }
    static __device__ __forceinline__ P load(const void *data, long long ch, int idx,
                                            const DasArgs &a) {
        const T *y = static_cast<const T *>(data) + ch;
        return make_float2(load_sample(y + idx), idx + 1 < a.nt ? load_sample(y + idx + 1) : 0.f);
    }
    static __device__ __forceinline__ float value(const P &c, float x, float fj, const DasArgs &a) {
        float am, b;
        knot_fractions(x, fj, a, am, b);
        return fmaf(am, c.x, b * c.y);
    }
};

template <typename T> struct Kind<PYCBF_GB_INTERP_NEAREST, T> {
    using P = float;
    static __device__ __forceinline__ bool index(float x, const DasArgs &a, int &idx, bool &fix) {
        const float q = __fmul_rn(__fsub_rn(x, a.t0), a.inv_dt);
        const float f = q - floorf(q);
        fix = fabsf(f - 0.5f) < a.eps;
        const int it = __float2int_rz(q + 0.5f);
        idx = it;
        return (x == x) && (it >= 0) && (it < a.nt);
    }
    static __device__ __forceinline__ bool index_exact(float x, const DasArgs &a, int &idx) {
        const int it = __float2int_rz(__fdiv_rn(__fsub_rn(x, a.t0), a.dt) + 0.5f);
        idx = it;
        return (x == x) && (it >= 0) && (it < a.nt);
    }
    static __device__ __forceinline__ P load(const void *data, long long ch, int idx,
                                            const DasArgs &a) {
        return load_sample(static_cast<const T *>(data) + ch + idx);
    }
    static __device__ __forceinline__ float value(const P &c, float, float, const DasArgs &) {
        return c;
    }
};

// The reference CUDA linear_interp as written (__engines__.cu:36-53): the two
// weights multiply the same sample, so it returns (nearly) the floor sample.
template <typename T> struct Kind<PYCBF_GB_INTERP_LINEAR_FLOOR, T> {
    using P = float;
    static __device__ __forceinline__ bool index(float x, const DasArgs &a, int &idx, bool &fix) {
        const float q = __fmul_rn(__fsub_rn(x, a.t0), a.inv_dt);
        const float f = q - floorf(q);
        fix = (f < a.eps) || (f > 1.f - a.eps);
        return floor_in_range(x, __float2int_rz(q), a, idx);
    }
    static __device__ __forceinline__ bool index_exact(float x, const DasArgs &a, int &idx) {
        return floor_in_range(x, __float2int_rz(__fdiv_rn(__fsub_rn(x, a.t0), a.dt)), a, idx);
    }
    static __device__ __forceinline__ bool floor_in_range(float x, int ixo, const DasArgs &a,
                                                          int &idx) {
        if (x == a.xend) {
            idx = a.nt - 1;
            return true;
        }
        idx = ixo;
        return (x == x) && (ixo >= 0) && (ixo < a.nt);
    }
    static __device__ __forceinline__ P load(const void *data, long long ch, int idx,
                                            const DasArgs &a) {
        return load_sample(static_cast<const T *>(data) + ch + idx);
    }
    static __device__ __forceinline__ float value(const P &v, float x, float fixo, const DasArgs &a) {
        if (x == a.xend) return v;
        const float frac =
            __fdiv_rn(__fsub_rn(__fsub_rn(x, __fmul_rn(fixo, a.dt)), a.t0), a.dt);
        return __fadd_rn(__fmul_rn(v, __fsub_rn(1.0f, frac)), __fmul_rn(v, frac));
    }
};

// ---------------------------------------------------------------------------
// korder / akima / makima: one float32 record of cubic coefficients per
// interval (poly.cu), whatever the storage type.  Knot ixo = (int)((x-t0)/dt)
// with the correctly rounded quotient; korder fills outside [t0, xfma] or
// past the last knot, akima/makima outside [t0, xfma] and take the last knot
// at x == xfma (__engines__.cu:181-187, 266-269, 318-322).
// ---------------------------------------------------------------------------
template <int KIND, typename T> struct KindPoly {
    using P = float4;
    static __device__ __forceinline__ bool index(float x, const DasArgs &a, int &idx, bool &fix) {
        const float q = __fmul_rn(__fsub_rn(x, a.t0), a.inv_dt);
        const float fl = floorf(q);
        const float f = q - fl;
        fix = (f < a.eps) || (f > 1.f - a.eps);
        return finish(x, fl, a, idx);
    }
    static __device__ __forceinline__ bool index_exact(float x, const DasArgs &a, int &idx) {
        return finish(x, floorf(__fdiv_rn(__fsub_rn(x, a.t0), a.dt)), a, idx);
    }
    static __device__ __forceinline__ bool finish(float x, float fl, const DasArgs &a, int &idx) {
        const float last = (float)(a.nt - 1);
        bool inr = (x >= a.t0) && (x <= a.xfma);
        if (KIND == KIND_POLY_NORM) inr = inr && (fl <= last);
        float j = fminf(fl, last);
        if (KIND == KIND_POLY_DELTA && x == a.xfma) j = last;
        idx = inr ? (int)j : 0;
        return inr;
    }
    static __device__ __forceinline__ P load(const void *data, long long ch, int idx,
                                            const DasArgs &) {
        return __ldg(static_cast<const float4 *>(data) + ch + idx);
    }
    static __device__ __forceinline__ float value(const P &c, float x, float fj, const DasArgs &a) {
        float u;
        if (KIND == KIND_POLY_NORM)
            u = __fdiv_rn(fmaf(-a.dt, fj, __fsub_rn(x, a.t0)), a.dt);
        else
            u = __fsub_rn(x, fmaf(a.dt, fj, a.t0));
        const float s1 = __fadd_rn(c.x, __fmul_rn(c.y, u));
        const float s2 = __fadd_rn(s1, __fmul_rn(__fmul_rn(c.z, u), u));
        return __fadd_rn(s2, __fmul_rn(__fmul_rn(__fmul_rn(c.w, u), u), u));
    }
};
template <typename T> struct Kind<KIND_POLY_NORM, T> : KindPoly<KIND_POLY_NORM, T> {};
template <typename T> struct Kind<KIND_POLY_DELTA, T> : KindPoly<KIND_POLY_DELTA, T> {};

// ---------------------------------------------------------------------------
// synthetic-point delays (__engines__.cu:382-470, acos tests as cos compares).
// A masked delay is returned as +inf so the range test rejects the tap.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void synth_dist(const float *o, const float *n, const float *p, int nd,
                                           float &mag, float &proj) {
    float m2 = 0.f, pr = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // nd <= 3: constant indices keep p in registers
        if (k < nd) {
            const float d = __fsub_rn(p[k], __ldg(o + k));
            m2 = __fadd_rn(m2, __fmul_rn(d, d));
            pr = __fadd_rn(pr, __fmul_rn(d, __ldg(n + k)));
        }
    }
    mag = __fsqrt_rn(m2);
    proj = pr;
}

__device__ __forceinline__ float synth_tx_delay(const DasArgs &a, int t, const float *p) {
    const int nd = a.ndim;
    float mag, proj;
    synth_dist(a.geo.ovectx + t * nd, a.geo.nvectx + t * nd, p, nd, mag, proj);
    const float c0 = a.geo.c0;
    const float ala = __ldg(a.geo.alatx + t);
    const float t0 = __ldg(a.geo.t0tx + t);
    if (ala != 0.f) {
        const float sgn = (proj > 0.f) ? 1.f : -1.f;
        const float cosala = __ldg(a.geo.cosalatx + t);
        if (__ldg(a.geo.doftx + t) != 0.f) {
            if ((fabsf(proj) > kDxMin) && (mag > kDxMin) && (fabsf(__fdiv_rn(proj, mag)) >= cosala))
                return __fadd_rn(sgn * __fdiv_rn(mag, c0), t0);
            const float lat = __fsqrt_rn(fabsf(__fsub_rn(__fmul_rn(mag, mag), __fmul_rn(proj, proj))));
            if (lat < __ldg(a.geo.halfdofsintx + t))
                return __fadd_rn(__fdiv_rn(__fmul_rn(proj, __ldg(a.geo.secalatx + t)), c0), t0);
            return __int_as_float(0x7f800000);
        }
        const float tau = (fabsf(proj) > kDxMin) ? __fadd_rn(sgn * __fdiv_rn(mag, c0), t0) : t0;
        const bool off = (mag > kDxMin) && (fabsf(__fdiv_rn(proj, mag)) < cosala);
        return off ? __int_as_float(0x7f800000) : tau;
    }
    return __fdiv_rn(proj, c0);
}

// The same geometry as path lengths for the slowness form: a transmit delay
// is D*s + t0add, a receive delay D*s; false where the element masks the point.
__device__ __forceinline__ bool synth_tx_path(const DasArgs &a, int t, const float *p, float &D,
                                              float &t0add) {
    const int nd = a.ndim;
    float mag, proj;
    synth_dist(a.geo.ovectx + t * nd, a.geo.nvectx + t * nd, p, nd, mag, proj);
    const float ala = __ldg(a.geo.alatx + t);
    t0add = 0.f;
    D = proj;
    if (ala == 0.f) return true;
    t0add = __ldg(a.geo.t0tx + t);
    const float sgn = (proj > 0.f) ? 1.f : -1.f;
    const float cosala = __ldg(a.geo.cosalatx + t);
    if (__ldg(a.geo.doftx + t) != 0.f) {
        if ((fabsf(proj) > kDxMin) && (mag > kDxMin) && (fabsf(__fdiv_rn(proj, mag)) >= cosala)) {
            D = sgn * mag;
            return true;
        }
        const float lat = __fsqrt_rn(fabsf(__fsub_rn(__fmul_rn(mag, mag), __fmul_rn(proj, proj))));
        D = __fmul_rn(proj, __ldg(a.geo.secalatx + t));
        return lat < __ldg(a.geo.halfdofsintx + t);
    }
    D = (fabsf(proj) > kDxMin) ? sgn * mag : 0.f;
    return !((mag > kDxMin) && (fabsf(__fdiv_rn(proj, mag)) < cosala));
}

__device__ __forceinline__ bool synth_rx_path(const DasArgs &a, int r, const float *p, float &D) {
    const int nd = a.ndim;
    float mag, proj;
    synth_dist(a.geo.ovecrx + r * nd, a.geo.nvecrx + r * nd, p, nd, mag, proj);
    D = mag;
    return !((mag > kDxMin) && (__fdiv_rn(proj, mag) < __ldg(a.geo.cosalarx + r)));
}

__device__ __forceinline__ float slow_delay(bool ok, float D, float s, float t0add) {
    return ok ? __fadd_rn(__fmul_rn(D, s), t0add) : __int_as_float(0x7f800000);
}

__device__ __forceinline__ float synth_rx_delay(const DasArgs &a, int r, const float *p) {
    const int nd = a.ndim;
    float mag, proj;
    synth_dist(a.geo.ovecrx + r * nd, a.geo.nvecrx + r * nd, p, nd, mag, proj);
    const bool off = (mag > kDxMin) && (__fdiv_rn(proj, mag) < __ldg(a.geo.cosalarx + r));
    return off ? __int_as_float(0x7f800000) : __fdiv_rn(mag, a.geo.c0);
}

// synth_rx_delay for a whole warp: most receives mask every pixel of a tile, and
// there the projection alone shows it (proj < cos(ala) |d| from the squares, with
// a margin far above their rounding), so no root or quotient is taken.
__device__ __forceinline__ float synth_rx_delay_warp(const DasArgs &a, int r, const float *p) {
    const int nd = a.ndim;
    const float *o = a.geo.ovecrx + r * nd, *n = a.geo.nvecrx + r * nd;
    const float cosala = __ldg(a.geo.cosalarx + r);
    float m2 = 0.f, pr = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (k < nd) {
            const float d = __fsub_rn(p[k], __ldg(o + k));
            m2 = __fadd_rn(m2, __fmul_rn(d, d));
            pr = __fadd_rn(pr, __fmul_rn(d, __ldg(n + k)));
        }
    }
    const bool far = (m2 > 1e-20f) && (cosala > 1e-3f) &&
                     (pr <= 0.f || pr * pr < cosala * cosala * m2 * 0.9999f);
    if (__all_sync(0xffffffffu, far)) return __int_as_float(0x7f800000);
    const float mag = __fsqrt_rn(m2);
    const bool off = (mag > kDxMin) && (__fdiv_rn(pr, mag) < cosala);
    return off ? __int_as_float(0x7f800000) : __fdiv_rn(mag, a.geo.c0);
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
constexpr int kGroup = 6;  // taps whose gathers a thread keeps in flight together
// the same for cubic sums over transmits: at six, 3.76 against 3.91 ms for 75
// float32 transmits, but 0.83 against 0.74 ms for 31 and 122 against 112 ms for
// 25 in float16 (registers); at eight slower throughout
constexpr int kCubicGroup = 4;

// Smallest and largest transmit weight of a pixel: where they are equal the weights are
// all alike.  A NaN weight (its taps never count) is like no other.
__device__ __forceinline__ void weight_range(float w, float &lo, float &hi) {
    const bool nan = w != w;
    lo = nan ? -__int_as_float(0x7f800000) : fminf(lo, w);
    hi = nan ? __int_as_float(0x7f800000) : fmaxf(hi, w);
}

// The transmit delays of a pixel beyond kTxReg: a column of shared memory per
// thread.  Cubic sums keep them as pairs, padded with infinite delays to whole
// groups of kCubicGroup where that still fits; the padding of the last few
// sizes below the limit does not, and their last transmits go one by one (an odd
// one in half a row).
constexpr size_t kColumnSmemMax = kSmemMax;
__host__ __device__ inline int cubic_column_padded(int ntx) {
    const int full = (ntx + kCubicGroup - 1) / kCubicGroup * kCubicGroup;
    return (size_t)full * kBlock * sizeof(float) <= kColumnSmemMax ? full : ntx;
}

// ---------------------------------------------------------------------------
// Cubic taps summed over the transmits of one receive, for every kernel
// (generic, batched, staged): the same operations, so the same bits.
//
// What bounds them is the issue rate: a tap is one gather and a handful of
// float operations, and the L1 or shared-memory pipe is busy about a third of
// the time.  So a tap is kept to 20 instructions, 14 of them its decisions:
//   x   = fl(tautx + taurx)                      packed, two transmits each
//   s   = (x - t0) * 1/dt - 1/2                  packed subtract, packed fma
//   j   = s rounded to an integer: s + 1.5 * 2^23 holds it in its low bits,
//         and those bits scaled by the record size are the gather address
//   xlo = fl(t0 + fl(dt j)), b = (x - xlo) / dt  packed, as the reference rounds
//   three multiply-adds, and one into the running sum where the tap counts.
// 192 elements x 75 transmits x 4096 samples, 512 x 1024 pixels: 2.11e9 warp
// instructions and 3.6 ms (20 a tap, half the issue slots; the rest waits on the
// gathers) in das_kernel, against 3.84e9 and 4.9 ms with the tests and knots kept as bit
// masks, 64-bit addresses and every constant fetched again; with the receives over
// warps (das_rx_kernel) 2.6 ms.
// Every decision is the reference's: t0 <= x <= xmax and |w| >= thresh on the
// rounded x and w, and the knot of the correctly rounded quotient.  h = s - j is
// within 1/2 - eps_fast of zero unless the quotient is so near an integer that
// the two roundings could differ; a group with such a tap (a few in a hundred of
// a warp's groups at nt = 2048) takes those taps' knots from the IEEE quotient.
//
// A tap that counts has 0 <= j: x >= t0 gives s >= -1/2, which rounds to 0 or
// more; and j <= nt - 1 where the fast quotient of xmax rounds to at most nt -
// 1, which the host checks (DasArgs::fast_axis).  On the other time axes (one
// float step of the delay longer than two samples) the knot is clamped to nt - 1, as the
// reference clamps it, and 2^29 samples a transmit and more take 64-bit offsets: FAST false.
// There each tap by itself, with the quotient and a call, made das_kernel 2.7 times as
// slow as it had been before the packed decisions: nearest, 128 receives, 256 x 512 pixels
// from 1 s at 40 ns, 11 transmits 342 -> 912 us, now 293; 31 transmits 915 -> 1796, now 586;
// linear on 129 records of 2^22 samples 225 -> 367, now 179.
// ---------------------------------------------------------------------------
constexpr unsigned kKnotBits = 0x4B400000u;  // 1.5 * 2^23 as an integer

// the running sum over transmits: float32 records one value; 16-bit records the
// y and the z terms of the two ends of the interval side by side
template <typename T> struct CubicAcc {
    using type = float2;
    static __device__ __forceinline__ type zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ float total(type v) { return v.x + v.y; }
};
template <> struct CubicAcc<float> {
    using type = float;
    static __device__ __forceinline__ type zero() { return 0.f; }
    static __device__ __forceinline__ float total(type v) { return v; }
};

__device__ __forceinline__ float pair_lane(const float2 *v, int k) {
    return (k & 1) ? v[k >> 1].y : v[k >> 1].x;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The constants of the taps in registers, the packed operands twice over: left
// to itself the compiler fetches them from the argument bank for every tap.
__device__ __forceinline__ float in_register(float v) {
    float r;
    asm volatile("mov.b32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float2 twice(float v) {
    return make_float2(in_register(v), in_register(v));
}
struct TapConst {
    float2 t02, inv2, dt2, nz2, mh2, mag2;
    float t0, xmax, hmax, thresh;
    __device__ __forceinline__ explicit TapConst(const DasArgs &a)
        : t02(twice(a.t0)), inv2(twice(a.inv_dt)), dt2(twice(a.dt)), nz2(twice(a.neg_zero)),
          mh2(twice(-0.5f)), mag2(twice(12582912.f)), t0(in_register(a.t0)),
          xmax(in_register(a.xmax)), hmax(in_register(0.5f - a.eps_fast)),
          thresh(in_register(a.thresh)) {}
};

struct NoTapConst {  // for the kernels without groups of taps
    __device__ __forceinline__ explicit NoTapConst(const DasArgs &) {}
};

// delay sums x, knots fj (as floats) and r (kKnotBits + j) of NP pairs of
// transmits; a NaN or infinite x never counts, whatever its knot.  FAST false: knots past
// the record (quotients of nt and more, whose floor the fast one may miss) become its last.
template <int NP, bool FAST = true>
__device__ __forceinline__ void knot_pairs(const DasArgs &a, const TapConst &c, const float2 *tt2,
                                           float trx, float2 *x2, float2 *fj2, unsigned *r) {
    const float2 trx2 = make_float2(trx, trx);
    float2 h2[NP];
    float hm = 0.f;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        x2[p] = add2_rn(tt2[p], trx2);
        const float2 s2 = fma2_rn(sub2_rn(x2[p], c.t02), c.inv2, c.mh2);
        const float2 r2 = add2_rn(s2, c.mag2);
        fj2[p] = sub2_rn(r2, c.mag2);
        h2[p] = sub2_rn(s2, fj2[p]);
        hm = max3(hm, fabsf(h2[p].x), fabsf(h2[p].y));  // a NaN is passed over
        r[2 * p] = __float_as_uint(r2.x);
        r[2 * p + 1] = __float_as_uint(r2.y);
    }
    if (hm > c.hmax) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (fabsf(h ? h2[p].y : h2[p].x) > c.hmax) {
                    const float x = h ? x2[p].y : x2[p].x;
                    const float fl = fminf(floorf(__fdiv_rn(__fsub_rn(x, a.t0), a.dt)),
                                           (float)(a.nt - 1));
                    if (h) fj2[p].y = fl;
                    else fj2[p].x = fl;
                    r[2 * p + h] = kKnotBits + (unsigned)(int)fl;
                }
            }
        }
    }
    if (!FAST) {
        const unsigned last = (unsigned)(a.nt - 1);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            fj2[p].x = fminf(fj2[p].x, (float)last);
            fj2[p].y = fminf(fj2[p].y, (float)last);
            r[2 * p] = min(r[2 * p], kKnotBits + last);
            r[2 * p + 1] = min(r[2 * p + 1], kKnotBits + last);
        }
    }
}

// records between transmits, and the k-th transmit's record r (knot_pairs)
template <bool FAST> using ChannelStride = typename std::conditional<FAST, unsigned, long long>::type;
template <typename R>
__device__ __forceinline__ const R *tap_record(const R *rec, unsigned r, int k, unsigned chs) {
    return rec + (r + ((unsigned)k * chs - kKnotBits));
}
template <typename R>
__device__ __forceinline__ const R *tap_record(const R *rec, unsigned r, int k, long long chs) {
    return rec + k * chs + (r - kKnotBits);
}

// b = (x - xlo) / dt with xlo = fl(t0 + fl(dt j)) for two transmits: the product
// is an fma with -0 read from the arguments, so that it stays rounded on its own
__device__ __forceinline__ float2 knot_frac2(const TapConst &c, float2 x2, float2 fj2) {
    const float2 xlo2 = add2_rn(fma2_rn(c.dt2, fj2, c.nz2), c.t02);
    return mul2_rn(sub2_rn(x2, xlo2), c.inv2);
}

// v(b) of a float32 record (the interval's polynomial)
__device__ __forceinline__ float poly_value(const float4 &c, float b) {
    return fmaf(fmaf(fmaf(c.w, b, c.z), b, c.y), b, c.x);
}

// Interpolation weights of a 16-bit record (y_j, y_j+1, z_j, z_j+1): with a =
// (xhi - x)/dt, b = (x - xlo)/dt, wy = w (a, b) and wz = w (a^3 - a, b^3 - b).
template <bool WEIGHTED>
__device__ __forceinline__ void half_weights(const TapConst &c, float x, float fj, float w,
                                             float2 &wy, float2 &wz) {
    const float2 K = add2_rn(fma2_rn(c.dt2, make_float2(__fadd_rn(fj, 1.f), fj), c.nz2), c.t02);
    wy = mul2_rn(sub2_rn(K, make_float2(x, x)), make_float2(c.inv2.x, -c.inv2.x));
    const float2 t = fma2_rn(wy, wy, make_float2(-1.f, -1.f));
    if (WEIGHTED) wy = mul2_rn(wy, make_float2(w, w));
    wz = mul2_rn(t, wy);
}

__device__ __forceinline__ float2 half_add(const float4 &c, float2 wy, float2 wz, float2 acc) {
    return fma2_rn(wz, make_float2(c.z, c.w), fma2_rn(wy, make_float2(c.x, c.y), acc));
}

// One tap with the IEEE quotient and its knot clamped to the channel, added
// where it counts (transmits past the last whole group of an unpadded column, other time
// axes in a batch).
template <typename T, bool WEIGHTED>
__device__ __noinline__ typename CubicAcc<T>::type cubic_tap_clamped(
    const DasArgs &a, float x, float w, const typename CoefRec<T>::raw *rec,
    typename CubicAcc<T>::type acc) {
    if (!((x >= a.t0) && (x <= a.xmax)) || (WEIGHTED && !(fabsf(w) >= a.thresh))) return acc;
    const float fj = fminf(floorf(__fdiv_rn(__fsub_rn(x, a.t0), a.dt)), (float)(a.nt - 1));
    const float4 c = CoefRec<T>::load(rec + (int)fj);
    const TapConst tc(a);
    if constexpr (CoefRec<T>::kPoly) {
        const float v = poly_value(c, knot_frac2(tc, make_float2(x, x), make_float2(fj, fj)).x);
        return WEIGHTED ? fmaf(w, v, acc) : acc + v;
    } else {
        float2 wy, wz;
        half_weights<WEIGHTED>(tc, x, fj, w, wy, wz);
        return half_add(c, wy, wz, acc);
    }
}

// N taps gathered from global memory: transmits g .. g+N-1 of one receive, rec
// the channel of transmit g, chs records between transmits.  Padding transmits carry
// infinite delays, which never count.  The gather is predicated on the tap, so
// nothing is read for one that does not count; its address is 64-bit rec plus,
// with FAST (DasArgs::fast_axis: N chs < 2^32), 32-bit (j + k chs) records.
template <int GEOM, typename T, int N, bool FAST = true>
__device__ __forceinline__ typename CubicAcc<T>::type cubic_taps(
    const DasArgs &a, const TapConst &c, const float2 *tt2, const float2 *at2, float trx, float arx,
    const typename CoefRec<T>::raw *rec, ChannelStride<FAST> chs, typename CubicAcc<T>::type acc) {
    using raw = typename CoefRec<T>::raw;
    constexpr int NP = (N + 1) / 2;
    constexpr bool W = GEOM == GEOM_TABBED;
    float2 x2[NP], fj2[NP], w2[NP];
    unsigned r[2 * NP];
    knot_pairs<NP, FAST>(a, c, tt2, trx, x2, fj2, r);
    bool ok[N];
    raw pv[N];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        if (W) w2[p] = mul2_rn(at2[p], make_float2(arx, arx));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * p + h;
            if (k >= N) continue;
            const float x = h ? x2[p].y : x2[p].x;
            ok[k] = (x >= c.t0) && (x <= c.xmax);
            if (W) ok[k] = ok[k] && (fabsf(h ? w2[p].y : w2[p].x) >= c.thresh);
            if (ok[k]) pv[k] = __ldg(tap_record(rec, r[k], k, chs));
        }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        float2 b2;
        if constexpr (CoefRec<T>::kPoly) b2 = knot_frac2(c, x2[p], fj2[p]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * p + h;
            if (k >= N) continue;
            if constexpr (CoefRec<T>::kPoly) {
                const float v = poly_value(pv[k], h ? b2.y : b2.x);
                if (ok[k]) acc = W ? fmaf(h ? w2[p].y : w2[p].x, v, acc) : acc + v;
            } else {
                float2 wy, wz;
                half_weights<W>(c, h ? x2[p].y : x2[p].x, h ? fj2[p].y : fj2[p].x,
                                W ? (h ? w2[p].y : w2[p].x) : 1.f, wy, wz);
                const float2 s = half_add(CoefRec<T>::unpack(pv[k]), wy, wz, acc);
                if (ok[k]) acc = s;
            }
        }
    }
    return acc;
}

// ---------------------------------------------------------------------------
// Nearest and linear taps summed over the transmits of one receive, as cubic_taps:
// the decisions of Kind<KIND>::index two transmits at a time, a redo of the taps whose
// quotient is next to a rounding boundary, 32-bit offsets, the same values and order.
// Calls in float32, before and after: 7 transmits x 97 receives x 1999 int16 samples,
// 251 x 509 pixels, linear 251 -> 164 us, nearest 206 -> 155; 75 Synthetic transmits, 192
// receives, 128 x 1024 pixels, linear 2.83 -> 1.55 ms, nearest 2.23 -> 1.28.
// ---------------------------------------------------------------------------
// one tap, decided with the IEEE quotient (unpadded columns)
template <int KIND, typename T, bool WEIGHTED>
__device__ __noinline__ float sample_tap_exact(const DasArgs &a, float x, float w, const T *ch,
                                               float acc) {
    using K = Kind<KIND, T>;
    int idx;
    if (!K::index_exact(x, a, idx) || (WEIGHTED && !(fabsf(w) >= a.thresh))) return acc;
    const float v = K::value(K::load(ch, 0, idx, a), x, (float)idx, a);
    return WEIGHTED ? fmaf(w, v, acc) : acc + v;
}

template <int GEOM, int KIND, typename T, int N, bool FAST>
__device__ __forceinline__ float sample_taps(const DasArgs &a, const TapConst &c, const float2 *tt2,
                                             const float2 *at2, float trx, float arx, const T *rec,
                                             ChannelStride<FAST> chs, float acc) {
    constexpr int NP = (N + 1) / 2;
    constexpr bool W = GEOM == GEOM_TABBED;
    float2 x2[NP], fj2[NP], w2[NP];
    unsigned r[2 * NP];
    if constexpr (KIND == PYCBF_GB_INTERP_LINEAR) {
        knot_pairs<NP, FAST>(a, c, tt2, trx, x2, fj2, r);
    } else {
        // it = (int)(q + 1/2): the nearest integer, but 0 for all of -3/2 < q < 1/2
        const float2 trx2 = make_float2(trx, trx);
        const float hmax = 0.5f - 2.f * a.eps_fast;  // q + 1/2 is rounded too
        float2 h2[NP];
        float hm = 0.f;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            x2[p] = add2_rn(tt2[p], trx2);
            const float2 q2 = fma2_rn(sub2_rn(x2[p], c.t02), c.inv2, c.nz2);
            const float2 r2 = add2_rn(q2, c.mag2);
            fj2[p] = sub2_rn(r2, c.mag2);
            h2[p] = sub2_rn(q2, fj2[p]);
            hm = max3(hm, fabsf(h2[p].x), fabsf(h2[p].y));
            r[2 * p] = max(__float_as_uint(r2.x), kKnotBits);
            r[2 * p + 1] = max(__float_as_uint(r2.y), kKnotBits);
        }
        if (hm > hmax) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                if (fabsf(pair_lane(h2, k)) > hmax) {
                    int idx;
                    const bool in = Kind<KIND, T>::index_exact(pair_lane(x2, k), a, idx);
                    r[k] = kKnotBits + (in ? (unsigned)idx : 0u);
                    if (k & 1) fj2[k >> 1].y = in ? (float)idx : -2.f;
                    else fj2[k >> 1].x = in ? (float)idx : -2.f;
                }
            }
        }
    }
    bool ok[N];
    // samples as they are stored: a conversion next to the load would wait for it, and with
    // two samples a tap the loads of a group would go one after another (float16, linear,
    // 11 transmits, 128 receives, 256 x 512 pixels: 241 us, now 187)
    T lo[N], hi[N];
    const float top = (float)(a.nt - 1);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        if (W) w2[p] = mul2_rn(at2[p], make_float2(arx, arx));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * p + h;
            if (k >= N) continue;
            const float x = h ? x2[p].y : x2[p].x, fj = h ? fj2[p].y : fj2[p].x;
            ok[k] = KIND == PYCBF_GB_INTERP_LINEAR ? (x >= c.t0) && (x <= c.xmax)
                                                   : (fj >= -1.f) && (fj <= top);
            if (W) ok[k] = ok[k] && (fabsf(h ? w2[p].y : w2[p].x) >= c.thresh);
            if (ok[k]) {
                const T *s = tap_record(rec, r[k], k, chs);
                lo[k] = __ldg(s);
                if (KIND == PYCBF_GB_INTERP_LINEAR) hi[k] = fj < top ? __ldg(s + 1) : T{};
            }
        }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        float v;
        if constexpr (KIND == PYCBF_GB_INTERP_LINEAR) {
            const float fj = pair_lane(fj2, k), x = pair_lane(x2, k);
            const float2 K = add2_rn(
                fma2_rn(c.dt2, make_float2(__fadd_rn(fj, 1.f), fj), c.nz2), c.t02);
            const float2 ab = mul2_rn(sub2_rn(K, make_float2(x, x)), make_float2(c.inv2.x, -c.inv2.x));
            v = fmaf(ab.x, load_sample_reg(lo[k]), ab.y * load_sample_reg(hi[k]));
        } else {
            v = load_sample_reg(lo[k]);
        }
        if (ok[k]) acc = W ? fmaf(pair_lane(w2, k), v, acc) : acc + v;
    }
    return acc;
}

// What a receive's sum over transmits gathers and accumulates, by kind: records of a
// cubic, or samples
template <int GEOM, int KIND, typename T> struct TapSum {
    using Rec = T;
    using Acc = float;
    static __device__ __forceinline__ Acc zero() { return 0.f; }
    static __device__ __forceinline__ float total(Acc v) { return v; }
    template <int N, bool FAST>
    static __device__ __forceinline__ Acc taps(const DasArgs &a, const TapConst &c, const float2 *tt2,
                                               const float2 *at2, float trx, float arx,
                                               const Rec *rec, long long chs, Acc acc) {
        return sample_taps<GEOM, KIND, T, N, FAST>(a, c, tt2, at2, trx, arx, rec,
                                                   (ChannelStride<FAST>)chs, acc);
    }
    static __device__ __forceinline__ Acc tap(const DasArgs &a, float x, float w, const Rec *rec,
                                              Acc acc) {
        return sample_tap_exact<KIND, T, GEOM == GEOM_TABBED>(a, x, w, rec, acc);
    }
};
template <int GEOM, typename T> struct TapSum<GEOM, PYCBF_GB_INTERP_CUBIC, T> {
    using Rec = typename CoefRec<T>::raw;
    using Acc = typename CubicAcc<T>::type;
    static __device__ __forceinline__ Acc zero() { return CubicAcc<T>::zero(); }
    static __device__ __forceinline__ float total(Acc v) { return CubicAcc<T>::total(v); }
    template <int N, bool FAST>
    static __device__ __forceinline__ Acc taps(const DasArgs &a, const TapConst &c, const float2 *tt2,
                                               const float2 *at2, float trx, float arx,
                                               const Rec *rec, long long chs, Acc acc) {
        return cubic_taps<GEOM, T, N, FAST>(a, c, tt2, at2, trx, arx, rec, (ChannelStride<FAST>)chs,
                                            acc);
    }
    static __device__ __forceinline__ Acc tap(const DasArgs &a, float x, float w, const Rec *rec,
                                              Acc acc) {
        return cubic_tap_clamped<T, GEOM == GEOM_TABBED>(a, x, w, rec, acc);
    }
};

// Where the transmit side of a pixel lives: decided per launch from ntx
// (kTxAuto, one kernel for both), or fixed at compile time so that a kernel
// carries the registers of one form only (kTxRegs: ntx <= kTxReg in
// registers; kTxSmem: the thread's column of shared memory).
constexpr int kTxAuto = 0, kTxRegs = 1, kTxSmem = 2;

// One pixel (table column i of frame f) of the generic delay-and-sum: the
// body of das_kernel, also run by the batched kernel for each of its jobs.
// sm: the CTA's dynamic shared memory (das_smem_bytes), a column per thread.
// FAST: the groups of taps are those of axes with fast_axis, and on others the taps go one
// by one (the batched kernel: with both forms of the groups it spills, 60 bytes against
// none); otherwise the groups are those of every axis.
// cubic, linear and nearest sums over the transmits of a receive take cubic_taps and
// sample_taps; the rest (census, per-tap outputs, other kinds) the general group
template <int KIND, int SUM, bool CENSUS> __host__ __device__ constexpr bool fast_sum() {
    return (KIND == PYCBF_GB_INTERP_CUBIC || KIND == PYCBF_GB_INTERP_LINEAR ||
            KIND == PYCBF_GB_INTERP_NEAREST) &&
           !CENSUS && SUM != PYCBF_GB_SUM_NONE && SUM != PYCBF_GB_SUM_RX_ONLY;
}

template <int GEOM, int KIND, int SUM, typename T, bool CENSUS, int TXM = kTxAuto, bool FAST = false>
__device__ __forceinline__ void das_pixel(const DasArgs &a, long long i, int f, float *sm) {
    using K = Kind<KIND, T>;
    constexpr bool kFast = fast_sum<KIND, SUM, CENSUS>();
    constexpr unsigned kFull = 0xffffffffu;
    const int tid = threadIdx.x;
    const long long np = a.np;
    // The receive loop votes per warp where it pays: sums by groups of taps, outputs per
    // transmit (but akima's).  There threads past the end walk the last pixel along and write
    // nothing.  Elsewhere they leave: a vote and its clamped threads cost outputs per tap 4
    // to 11 % (11 transmits, 64 receives, 64 x 128 pixels: nearest 103 us with, 91 without,
    // Synthetic 105 and 95), akima's per transmit 4 % (256 x 512 pixels, 25 transmits 694
    // and 664; nearest from float16 455 and 470).
    constexpr bool kVote = kFast || (GEOM == GEOM_SYNTH && SUM != PYCBF_GB_SUM_NONE) ||
                           (SUM == PYCBF_GB_SUM_RX_ONLY && KIND <= PYCBF_GB_INTERP_CUBIC);
    const bool valid = !kVote || i < np;
    if (i >= np) {
        if (!kVote) return;
        i = np - 1;
    }
    const int ntx = a.ntx, nrx = a.nrx;
    const long long op = a.pixel_index ? (long long)__ldg(a.pixel_index + i) : i;
    const bool in_regs = TXM == kTxAuto ? ntx <= kTxReg : TXM == kTxRegs;
    const long long frame_ch = (long long)f * ntx * nrx;
    const long long chs = (long long)nrx * a.nt;  // channel stride between transmits

    float pnt[3] = {0.f, 0.f, 0.f};
    if (GEOM != GEOM_TABBED)
        for (int k = 0; k < 3; ++k) if (k < a.ndim) pnt[k] = __ldg(a.geo.pnts + i * a.ndim + k);
    const float slow = (GEOM == GEOM_SYNTH_SLOW) ? __ldg(a.slow + i) : 0.f;

    // transmit side: registers (ntx <= kTxReg) or this thread's column of shared memory.
    // Synthetic masks travel as +inf delays, which the range test rejects.
    float rtau[kTxReg], rapod[kTxReg], racc[kTxReg];
    float2 tt2[kTxReg / 2], at2[kTxReg / 2];  // kFast: the same in pairs
    float *stau = sm + tid;
    float2 *spair = reinterpret_cast<float2 *>(sm) + tid;  // kFast: the column in pairs
    const int ncol = kFast && !in_regs ? cubic_column_padded(ntx) : ntx;
    const int ngroups = FAST && !a.fast_axis ? 0 : ncol / kCubicGroup * kCubicGroup;  // taps by whole groups
    const typename std::conditional<kFast, TapConst, NoTapConst>::type tc(a);
    // Tabbed transmit weights beyond kTxReg are read from the table per
    // receive (L1-resident: a tile's rows), which halves the shared memory of
    // the column form and so raises the CTAs per SM (two -> five at 75 transmits)
    float *sacc = stau + (size_t)ntx * kBlock;
    float amax = 0.f;  // max |apodtx| of this pixel, for the exact receive-level reject
    float amin = __int_as_float(0x7f800000), atop = -amin;  // weight_range
    auto tx_side = [&](int t, float &tau, float &apod) {
        if (GEOM == GEOM_TABBED) {
            tau = __ldg(a.tautx + (long long)t * np + i);
            apod = __ldg(a.apodtx + (long long)t * np + i);
            amax = fmaxf(amax, fabsf(apod));
            weight_range(apod, amin, atop);
        } else if (GEOM == GEOM_SYNTH) {
            tau = synth_tx_delay(a, t, pnt);
            apod = 1.f;
        } else {
            float D, t0add;
            const bool ok = synth_tx_path(a, t, pnt, D, t0add);
            tau = slow_delay(ok, D, slow, t0add);
            apod = 1.f;
        }
    };
    const float inf = __int_as_float(0x7f800000);
    if constexpr (kFast) {
        if (in_regs) {
#pragma unroll
            for (int k = 0; k < kTxReg; ++k) {
                float tau = inf, apod = 0.f;
                if (k < ntx) tx_side(k, tau, apod);
                if (k & 1) {
                    tt2[k >> 1].y = tau;
                    at2[k >> 1].y = apod;
                } else {
                    tt2[k >> 1].x = tau;
                    at2[k >> 1].x = apod;
                }
            }
        } else {
            int k = 0;
            constexpr int kAhead = GEOM == GEOM_TABBED ? 4 : 1;  // pairs of table rows in flight
#pragma unroll kAhead
            for (; k + 1 < ntx; k += 2) {
                float2 t;
                float apod;
                tx_side(k, t.x, apod);
                tx_side(k + 1, t.y, apod);
                spair[(size_t)(k >> 1) * kBlock] = t;
            }
            for (; k < ncol; k += 2) {
                float2 t = make_float2(inf, inf);
                float apod;
                if (k < ntx) tx_side(k, t.x, apod);
                if (k + 1 < ntx) tx_side(k + 1, t.y, apod);
                if (k + 1 < ncol) spair[(size_t)(k >> 1) * kBlock] = t;
                else stau[(size_t)k * kBlock] = t.x;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < kTxReg; ++k) {
            rtau[k] = 0.f;
            rapod[k] = 0.f;
            racc[k] = 0.f;
        }
        if (in_regs) {
#pragma unroll
            for (int k = 0; k < kTxReg; ++k)
                if (k < ntx) tx_side(k, rtau[k], rapod[k]);
        } else {
            for (int k = 0; k < ntx; ++k) {
                float tau, apod;
                tx_side(k, tau, apod);
                stau[(size_t)k * kBlock] = tau;
                if (SUM == PYCBF_GB_SUM_RX_ONLY) sacc[(size_t)k * kBlock] = 0.f;
            }
        }
    }
    // Tabbed weights beyond kTxReg: one value for every transmit of every pixel of the warp
    // (apodtx all ones), or read from the table per tap
    bool one_weight = false;
    if (kFast && GEOM == GEOM_TABBED) one_weight = __all_sync(kFull, amin == atop);

    float acc = 0.f, s1 = 0.f;
    float bacc = 0.f;  // TX_AND_RX: sequential sum of the current block of kRxBlockSum receives
    int cnt = 0;
    long long isum = 0;

    // receive-side values, fetched one receive ahead
    auto rx_side = [&](int r, float &trx, float &arx) {
        if (GEOM == GEOM_TABBED) {
            trx = __ldg(a.taurx + (long long)r * np + i);
            arx = __ldg(a.apodrx + (long long)r * np + i);
        } else if (GEOM == GEOM_SYNTH) {
            trx = kVote ? synth_rx_delay_warp(a, r, pnt) : synth_rx_delay(a, r, pnt);
            arx = 1.f;
        } else {
            float D;
            const bool ok = synth_rx_path(a, r, pnt, D);
            trx = slow_delay(ok, D, slow, 0.f);
            arx = 1.f;
        }
    };
    float trx_next = 0.f, arx_next = 0.f;
    if (GEOM == GEOM_TABBED && nrx > 0) rx_side(0, trx_next, arx_next);
    for (int r = 0; r < nrx; ++r) {
        if (SUM == PYCBF_GB_SUM_TX_AND_RX && r > 0 && r % kRxBlockSum == 0) {
            acc += bacc;  // the image is the sum of the blocks' sums, in block order
            bacc = 0.f;
        }
        float trx, arx;
        if (GEOM == GEOM_TABBED) {
            trx = trx_next;
            arx = arx_next;
            if (r + 1 < nrx) rx_side(r + 1, trx_next, arx_next);
        } else {
            rx_side(r, trx, arx);
        }
        // Exact reject of the whole receive: rounding is monotonic, so
        // fl(amax*|arx|) < thresh implies fl(|apodtx*apodrx|) < thresh for every
        // transmit.  A masked synthetic receive has an infinite delay.
        bool live;
        if (GEOM == GEOM_TABBED) live = __fmul_rn(amax, fabsf(arx)) >= a.thresh;
        else live = trx != inf;
        // a warp that votes leaves a receive together; the taps of a pixel that it cannot
        // reach fail their own tests (weight below thresh, infinite delay)
        if (SUM != PYCBF_GB_SUM_NONE && !(kVote ? __any_sync(kFull, live) : live)) {
            if (!CENSUS && SUM == PYCBF_GB_SUM_TX_ONLY && valid)
                a.out[((long long)f * nrx + r) * np + op] = 0.f;
            continue;
        }
        const long long ch0 = (frame_ch + r) * a.nt;  // channel (tx 0, rx r)
        float accr = 0.f;

        // one group of up to kGroup transmits taken from registers or shared memory
        auto group = [&](int k0, int nk, const float *tt, const float *at) {
            float xs[kGroup], ap[kGroup];
            int ix[kGroup];
            unsigned hit = 0u, fix = 0u;
#pragma unroll
            for (int k = 0; k < kGroup; ++k) {
                xs[k] = 0.f;
                ap[k] = 0.f;
                ix[k] = 0;
                if (k < nk) {
                    const float x = __fadd_rn(tt[k], trx);
                    float apod = 1.f;
                    bool h = true;
                    if (GEOM == GEOM_TABBED) {
                        apod = __fmul_rn(at[k], arx);
                        h = fabsf(apod) >= a.thresh;
                    }
                    bool fx;
                    int idx;
                    const bool inr = K::index(x, a, idx, fx);
                    xs[k] = x;
                    ap[k] = apod;
                    ix[k] = idx;
                    hit |= (unsigned)(h && inr) << k;
                    fix |= (unsigned)(h && fx) << k;
                }
            }
            if (fix) {  // rare: a quotient next to a rounding boundary, redo it exactly
#pragma unroll
                for (int k = 0; k < kGroup; ++k) {
                    if ((fix >> k) & 1u) {
                        int idx;
                        const bool inr = K::index_exact(xs[k], a, idx);
                        ix[k] = idx;
                        hit = inr ? (hit | (1u << k)) : (hit & ~(1u << k));
                    }
                }
            }
            typename K::P pv[kGroup];
#pragma unroll
            for (int k = 0; k < kGroup; ++k)
                if ((hit >> k) & 1u) pv[k] = K::load(a.data, ch0 + (long long)(k0 + k) * chs, ix[k], a);
#pragma unroll
            for (int k = 0; k < kGroup; ++k) {
                if (k < nk) {
                    // per-receive sums accumulate with one fma per tap (the staged
                    // kernel does the same, so both give identical bits)
                    constexpr bool kPerTap = SUM == PYCBF_GB_SUM_NONE || SUM == PYCBF_GB_SUM_RX_ONLY;
                    float c = 0.f;
                    if ((hit >> k) & 1u) {
                        if (!CENSUS) {
                            const float v = K::value(pv[k], xs[k], (float)ix[k], a);
                            if (kPerTap) c = (GEOM == GEOM_TABBED) ? ap[k] * v : v;
                            else accr = fmaf(ap[k], v, accr);
                        } else {
                            cnt += 1;
                            isum += ix[k];
                        }
                    }
                    const int t = k0 + k;
                    if (!CENSUS && SUM == PYCBF_GB_SUM_NONE && valid)
                        a.out[(((long long)f * ntx + t) * nrx + r) * np + op] = c;
                    if (SUM == PYCBF_GB_SUM_RX_ONLY) {
                        if (in_regs) {
#pragma unroll
                            for (int kk = 0; kk < kTxReg; ++kk)
                                if (kk == t) racc[kk] += c;
                        } else {
                            sacc[(size_t)t * kBlock] += c;
                        }
                    }
                }
            }
        };

        if constexpr (kFast) {
            using S = TapSum<GEOM, KIND, T>;
            using Rec = typename S::Rec;
            const Rec *rec = static_cast<const Rec *>(a.data) + ch0;
            auto sum = S::zero();
            if (in_regs) {
#pragma unroll
                for (int g = 0; g < kTxReg; g += kCubicGroup) {
                    if (g < ntx) {
                        const Rec *rg = rec + (long long)g * chs;
                        sum = S::template taps<kCubicGroup, FAST>(a, tc, tt2 + g / 2, at2 + g / 2,
                                                                  trx, arx, rg, chs, sum);
                    }
                }
            } else {
                int g = 0;
                for (; g < ngroups; g += kCubicGroup) {
                    float2 t2[kCubicGroup / 2], w2[kCubicGroup / 2];
#pragma unroll
                    for (int p = 0; p < kCubicGroup / 2; ++p) {
                        t2[p] = spair[(size_t)(g / 2 + p) * kBlock];
                        w2[p] = make_float2(amin, amin);
                    }
                    if (GEOM == GEOM_TABBED && !one_weight) {
                        float *w = reinterpret_cast<float *>(w2);
#pragma unroll
                        for (int k = 0; k < kCubicGroup; ++k)
                            w[k] = __ldg(a.apodtx + (long long)min(g + k, ntx - 1) * np + i);
                    }
                    sum = S::template taps<kCubicGroup, FAST>(a, tc, t2, w2, trx, arx, rec, chs, sum);
                    rec += kCubicGroup * chs;
                }
                for (; g < ntx; ++g) {  // the others: an unpadded column's last transmits
                    float2 t = make_float2(0.f, 0.f);
                    if (g + 1 == ncol && !(g & 1)) t.x = stau[(size_t)g * kBlock];
                    else t = spair[(size_t)(g >> 1) * kBlock];
                    float w = 1.f;
                    if (GEOM == GEOM_TABBED)
                        w = __fmul_rn(__ldg(a.apodtx + (long long)g * np + i), arx);
                    sum = S::tap(a, __fadd_rn((g & 1) ? t.y : t.x, trx), w, rec, sum);
                    rec += chs;
                }
            }
            accr = S::total(sum);
        } else if (in_regs) {
#pragma unroll
            for (int g = 0; g < kTxReg; g += kGroup)
                if (g < ntx) group(g, min(kGroup, ntx - g), rtau + g, rapod + g);
        } else {
            for (int g = 0; g < ntx; g += kGroup) {
                const int nk = min(kGroup, ntx - g);
                float tt[kGroup], at[kGroup];
#pragma unroll
                for (int k = 0; k < kGroup; ++k) {
                    tt[k] = (k < nk) ? stau[(size_t)(g + k) * kBlock] : 0.f;
                    at[k] = (GEOM == GEOM_TABBED && k < nk)
                                ? __ldg(a.apodtx + (long long)(g + k) * np + i)
                                : 1.f;
                }
                group(g, nk, tt, at);
            }
        }

        if (SUM == PYCBF_GB_SUM_TX_AND_RX) bacc += accr;
        if (!CENSUS && SUM == PYCBF_GB_SUM_TX_ONLY && valid)
            a.out[((long long)f * nrx + r) * np + op] = accr;
        if ((SUM == PYCBF_GB_SUM_DMAS_SSR || SUM == PYCBF_GB_SUM_DMAS_POWER) && live) {
            // pairwise sum over receives i<j of s_i s_j as sum_j s_j * (sum_{i<j} s_i):
            // no cancellation, two FMAs per receive
            const float s = (SUM == PYCBF_GB_SUM_DMAS_SSR) ? copysignf(sqrtf(fabsf(accr)), accr) : accr;
            acc = fmaf(s, s1, acc);
            s1 += s;
        }
    }

    if (!valid) return;
    if (SUM == PYCBF_GB_SUM_TX_AND_RX) acc += bacc;
    // census launches carry no image buffer (out is NULL): they store counts only
    if (!CENSUS && (SUM == PYCBF_GB_SUM_TX_AND_RX || SUM == PYCBF_GB_SUM_DMAS_SSR ||
                    SUM == PYCBF_GB_SUM_DMAS_POWER))
        a.out[(long long)f * np + op] = acc;
    if (!CENSUS && SUM == PYCBF_GB_SUM_RX_ONLY) {
        if (in_regs) {
#pragma unroll
            for (int k = 0; k < kTxReg; ++k)
                if (k < ntx) a.out[((long long)f * ntx + k) * np + op] = racc[k];
        } else {
            for (int k = 0; k < ntx; ++k) a.out[((long long)f * ntx + k) * np + op] = sacc[(size_t)k * kBlock];
        }
    }
    if (CENSUS) {
        a.census_count[i] = cnt;
        a.census_isum[i] = isum;
    }
}

// Five CTAs per SM for the shared-memory form (its registers fit 96 per
// thread; 3-D 25-transmit launches measured 5 % faster than at four).
template <int GEOM, int KIND, int SUM, typename T, bool CENSUS, int TXM>
__global__ void __launch_bounds__(kBlock, TXM == kTxSmem ? 5 : 4) das_kernel(const __grid_constant__ DasArgs a) {
    extern __shared__ float sm[];
    das_pixel<GEOM, KIND, SUM, T, CENSUS, TXM>(a, (long long)blockIdx.x * kBlock + threadIdx.x,
                                          (int)blockIdx.y, sm);
}

// the column form: per transmit the delay (and the RX_ONLY accumulator)
inline size_t das_smem_bytes(int geom, int sum, int ntx) {
    (void)geom;
    if (ntx <= kTxReg) return 0;
    const size_t per = 1 + (sum == PYCBF_GB_SUM_RX_ONLY ? 1 : 0);
    const size_t cols = per > 1 ? per * (size_t)ntx : (size_t)std::max(ntx, cubic_column_padded(ntx));
    return cols * kBlock * sizeof(float);
}

template <int GEOM, int KIND, int SUM, typename T, bool CENSUS, int TXM>
cudaError_t launch_das_txm(const DasArgs &a, cudaStream_t s) {
    const size_t smem = das_smem_bytes(GEOM, SUM, a.ntx);
    auto kern = das_kernel<GEOM, KIND, SUM, T, CENSUS, TXM>;
    if (smem > 48 * 1024) {
        cudaError_t err = allow_smem(kern, kColumnSmemMax);
        if (err != cudaSuccess) return err;
    }
    const long long bx = (a.np + kBlock - 1) / kBlock;
    dim3 grid((unsigned)bx, CENSUS ? 1u : (unsigned)a.nframes);
    kern<<<grid, kBlock, smem, s>>>(a);
    return cudaGetLastError();
}

// cubic images and sums by taps: a kernel per transmit-side form (fewer registers
// each); census launches and the rest: one kernel for both
template <int GEOM, int KIND, int SUM, typename T, bool CENSUS>
cudaError_t launch_das_one(const DasArgs &a, cudaStream_t s) {
    if constexpr ((KIND == PYCBF_GB_INTERP_CUBIC || fast_sum<KIND, SUM, CENSUS>()) && !CENSUS) {
        if (a.ntx <= kTxReg) return launch_das_txm<GEOM, KIND, SUM, T, CENSUS, kTxRegs>(a, s);
        return launch_das_txm<GEOM, KIND, SUM, T, CENSUS, kTxSmem>(a, s);
    } else {
        return launch_das_txm<GEOM, KIND, SUM, T, CENSUS, kTxAuto>(a, s);
    }
}

template <int GEOM, int KIND, typename T>
cudaError_t launch_das_sum(const DasArgs &a, int sum, cudaStream_t s) {
    switch (sum) {
        case PYCBF_GB_SUM_NONE: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_NONE, T, false>(a, s);
        case PYCBF_GB_SUM_TX_ONLY: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_TX_ONLY, T, false>(a, s);
        case PYCBF_GB_SUM_RX_ONLY: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_RX_ONLY, T, false>(a, s);
        case PYCBF_GB_SUM_TX_AND_RX: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_TX_AND_RX, T, false>(a, s);
        case PYCBF_GB_SUM_DMAS_SSR: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_DMAS_SSR, T, false>(a, s);
        case PYCBF_GB_SUM_DMAS_POWER: return launch_das_one<GEOM, KIND, PYCBF_GB_SUM_DMAS_POWER, T, false>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <int GEOM, typename T>
cudaError_t launch_das_geom_type(const DasArgs &a, int interp, int sum, bool census, cudaStream_t s) {
    if (census) {
        if constexpr (std::is_same<T, float>::value) {
            if (interp == KIND_POLY_NORM)
                return launch_das_one<GEOM, KIND_POLY_NORM, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
            if (interp == KIND_POLY_DELTA)
                return launch_das_one<GEOM, KIND_POLY_DELTA, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
        }
        switch (interp) {
            case PYCBF_GB_INTERP_CUBIC: return launch_das_one<GEOM, PYCBF_GB_INTERP_CUBIC, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
            case PYCBF_GB_INTERP_LINEAR: return launch_das_one<GEOM, PYCBF_GB_INTERP_LINEAR, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
            case PYCBF_GB_INTERP_NEAREST: return launch_das_one<GEOM, PYCBF_GB_INTERP_NEAREST, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
            case PYCBF_GB_INTERP_LINEAR_FLOOR: return launch_das_one<GEOM, PYCBF_GB_INTERP_LINEAR_FLOOR, PYCBF_GB_SUM_TX_AND_RX, T, true>(a, s);
            default: return cudaErrorInvalidValue;
        }
    }
    if constexpr (std::is_same<T, float>::value) {  // polynomial records are float32 always
        if (interp == KIND_POLY_NORM) return launch_das_sum<GEOM, KIND_POLY_NORM, T>(a, sum, s);
        if (interp == KIND_POLY_DELTA) return launch_das_sum<GEOM, KIND_POLY_DELTA, T>(a, sum, s);
    }
    switch (interp) {
        case PYCBF_GB_INTERP_CUBIC: return launch_das_sum<GEOM, PYCBF_GB_INTERP_CUBIC, T>(a, sum, s);
        case PYCBF_GB_INTERP_LINEAR: return launch_das_sum<GEOM, PYCBF_GB_INTERP_LINEAR, T>(a, sum, s);
        case PYCBF_GB_INTERP_NEAREST: return launch_das_sum<GEOM, PYCBF_GB_INTERP_NEAREST, T>(a, sum, s);
        case PYCBF_GB_INTERP_LINEAR_FLOOR: return launch_das_sum<GEOM, PYCBF_GB_INTERP_LINEAR_FLOOR, T>(a, sum, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pgb
