// Per-pixel augmented-Lagrangian / projected L-BFGS solve, one pixel per lane.
//
// The method, its arithmetic and its operation order are those of solver.cuh
// (FP64: rounded multiplies and adds; FP32: its fused and approximate forms; a
// pixel's sums over the three channels and the alphas are added in the tree in
// which a quad's lanes add theirs), so outputs, statuses and counters equal
// its kernels' bit for bit in both precisions. (Two edges are not the same
// operations: a zero numerator's quotient loses its sign, and FP64 steps of
// 2^-537.5 to 2^-537 count as no motion. Neither reaches an output that any
// test has seen.) Figures below are FP64's.
//
// Why one pixel per lane: on a quad, all four lanes repeat the composite alpha
// chain and the 3x3 colour prior, lane 3 idles through the colour arithmetic,
// every sum costs shuffles, and a trip issues about four times the
// instructions a pixel needs. Here a pixel's three channels are three
// independent chains of one lane. The price is state: x, g and d (12 L
// doubles) live in shared memory (conflict-free 16-byte accesses), the L-BFGS
// ring, the best point and the outer step's start in global memory, one
// 32-byte sector per layer and lane, so a lane's loads use whole sectors
// whatever ring slot its neighbours are at.
//
// Phases: a block's lanes are at different actions (a line-search trial, a
// gradient, a new direction, the end of an outer step). The block runs the
// actions as phases, all warps at once: every trip evaluates the lanes with a
// trial, and the other actions run when a share of the block's lanes waits
// for them (or none has a trial). With each warp on its own schedule, the
// instruction cache thrashed between the phases' code (85-100 KB; 4 to 7 cycles
// of fetch stall per issue): putting the block in phase took the two passes of
// the 1024x1024 five-layer image from 75 + 45 to 53 + 33 ms. (The quads take
// 130 + 88 ms; the steps since the phases, 35 + 21. The fetch stall is now 0.46
// and 0.34 cycles per issue.) Even a block whose warps meet once a trip only is
// slower (measured at 42 + 26 ms: 47 + 28).
//
// What bounds it (a 512x512 image of five layers, first pass and refinement):
// latency at three warps per scheduler (the shared memory and registers that a
// pixel's state and the direction's loops take) and lanes that wait for a
// phase: 49 and 51 % of issue slots, 45 % of the FP64 pipe, 14 to 15 of 32
// lanes active. At 1024x1024 trials take 38 and 52 % of the time, directions 34
// and 14 %, gradients 13 %, outer steps 4 and 6 %, the meetings 10 and 15 %.
//
// An accepted trial needs its gradient once; the lane's values repeat their
// evaluation during the next trial phase, beside the lanes that evaluate
// anyway, and keep what the reverse sweep reads.
#pragma once
#include "blend.cuh"
#include "common.cuh"
#include "quotient.hpp"
#include "solver.cuh"

namespace unb {

// Blend values of three channels of one layer (blend_value of each).
__device__ __forceinline__ void blend_value3(int mode, const double* s, const double* d, double* f) {
    const double eps = 1e-5;
    switch (mode) {
    case 0:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c];
        return;
    case 1:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] * d[c];
        return;
    case 2:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = 1.0 - (1.0 - s[c]) * (1.0 - d[c]);
        return;
    case 3:
    case 8:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double t = mode == 3 ? d[c] : s[c];
            const double lowv = 2.0 * s[c] * d[c], highv = 1.0 - 2.0 * (1.0 - s[c]) * (1.0 - d[c]);
            f[c] = t <= 0.5 ? lowv : highv;
        }
        return;
    case 4:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] < d[c] ? s[c] : d[c];
        return;
    case 5:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] < d[c] ? d[c] : s[c];
        return;
    case 6:     // d / (1 - s), and Burn, 1 - (1 - d) / s, by the same code
    case 7:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double p = mode == 6 ? d[c] : 1.0 - d[c], q = mode == 6 ? 1.0 - s[c] : s[c];
            const double v = quotient(p, q, reciprocal(q));
            const double r = p < eps ? 0.0 : (q < eps ? 1.0 : (v < 1.0 ? v : 1.0));
            f[c] = mode == 6 ? r : 1.0 - r;
        }
        return;
    case 9:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double lowv = d[c] - (1.0 - 2.0 * s[c]) * d[c] * (1.0 - d[c]);
            const double highv = d[c] + (2.0 * s[c] - 1.0) * (softlight_g(d[c]) - d[c]);
            f[c] = s[c] <= 0.5 ? lowv : highv;
        }
        return;
    case 10:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] < d[c] ? d[c] - s[c] : s[c] - d[c];
        return;
    case 11:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] + d[c] - 2.0 * s[c] * d[c];
        return;
    case 12:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s[c] + d[c];
        return;
    default:
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = 0.0;
        return;
    }
}

// Blend values and partials of three channels (blend_all of each).
__device__ __forceinline__ void blend_all3(int mode, const double* s, const double* d, double* f, double* fs,
                                           double* fd) {
    const double eps = 1e-5;
    if (mode == 6 || mode == 7) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double p = mode == 6 ? d[c] : 1.0 - d[c], q = mode == 6 ? 1.0 - s[c] : s[c];
            const double y = reciprocal(q), qq = q * q;
            const double v = quotient(p, q, y), g = quotient(p, qq, reciprocal(qq));
            const bool dark = p < eps, flat = dark || q < eps || 1.0 < v;
            const double r = dark ? 0.0 : (flat ? 1.0 : v);
            f[c] = mode == 6 ? r : 1.0 - r;
            fs[c] = flat ? 0.0 : g;
            fd[c] = flat ? 0.0 : y;
        }
    } else {
        // The remaining modes have no division but SoftLight's, which keeps
        // the one-channel form.
        switch (mode) {
        case 0:
#pragma unroll
            for (int c = 0; c < 3; ++c) { f[c] = s[c]; fs[c] = 1.0; fd[c] = 0.0; }
            return;
        case 1:
#pragma unroll
            for (int c = 0; c < 3; ++c) { f[c] = s[c] * d[c]; fs[c] = d[c]; fd[c] = s[c]; }
            return;
        case 2:
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double p = 1.0 - s[c], q = 1.0 - d[c];
                f[c] = 1.0 - p * q; fs[c] = q; fd[c] = p;
            }
            return;
        case 3:
        case 8:
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double t = mode == 3 ? d[c] : s[c];
                const bool low = t <= 0.5;
                const double a = low ? s[c] : 1.0 - s[c], b = low ? d[c] : 1.0 - d[c];
                const double p = 2.0 * a * b;
                f[c] = low ? p : 1.0 - p; fs[c] = 2.0 * b; fd[c] = 2.0 * a;
            }
            return;
        case 4:
        case 5:
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const bool less = s[c] < d[c], src = mode == 4 ? less : !less;
                f[c] = src ? s[c] : d[c]; fs[c] = src ? 1.0 : 0.0; fd[c] = src ? 0.0 : 1.0;
            }
            return;
        case 10:
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const bool less = s[c] < d[c];
                f[c] = less ? d[c] - s[c] : s[c] - d[c]; fs[c] = less ? -1.0 : 1.0; fd[c] = less ? 1.0 : -1.0;
            }
            return;
        case 11:
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f[c] = s[c] + d[c] - 2.0 * s[c] * d[c]; fs[c] = 1.0 - 2.0 * d[c]; fd[c] = 1.0 - 2.0 * s[c];
            }
            return;
        case 12:
#pragma unroll
            for (int c = 0; c < 3; ++c) { f[c] = s[c] + d[c]; fs[c] = 1.0; fd[c] = 1.0; }
            return;
        case 9:
#pragma unroll
            for (int c = 0; c < 3; ++c) blend_all<double>(9, s[c], d[c], f[c], fs[c], fd[c]);
            return;
        default:
#pragma unroll
            for (int c = 0; c < 3; ++c) { f[c] = 0.0; fs[c] = 0.0; fd[c] = 0.0; }
            return;
        }
    }
}

// FP32: the solver's table-driven blends, channel by channel.
__device__ __forceinline__ void blend_values(const Models<float>& m, int l, const float* s, const float* d, float* f) {
    float fs, fd;
#pragma unroll
    for (int c = 0; c < 3; ++c) blend_table<float>(m, l, s[c], d[c], f[c], fs, fd, false);
}
__device__ __forceinline__ void blend_all(const Models<float>& m, int l, const float* s, const float* d, float* f,
                                          float* fs, float* fd) {
#pragma unroll
    for (int c = 0; c < 3; ++c) blend_table<float>(m, l, s[c], d[c], f[c], fs[c], fd[c], true);
}
__device__ __forceinline__ void blend_values(const Models<double>& m, int l, const double* s, const double* d, double* f) {
    blend_value3(m.mode[l], s, d, f);
}
__device__ __forceinline__ void blend_all(const Models<double>& m, int l, const double* s, const double* d, double* f,
                                          double* fs, double* fd) {
    blend_all3(m.mode[l], s, d, f, fs, fd);
}

// ----------------------------------------------------------------- storage --
// A lane's four values of one layer (three colours, alpha) as one 32-byte
// sector of global memory.
__device__ __forceinline__ void load_rec(const double* p, double* v) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void store_rec(double* p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

__device__ __forceinline__ void load_rec(const float* p, float* v) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void store_rec(float* p, float a, float b, float c, float d) {
    asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// Bits of the magnitude (double: of its high word), ordered as magnitudes are.
__device__ __forceinline__ uint32_t magnitude_bits(double v) { return uint32_t(__double2hiint(v)) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t magnitude_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

extern __shared__ __align__(16) unsigned char lane_smem[];

// Eighths of a block's live lanes that start a phase: the end of an outer
// step, a direction, a gradient. Measured on the 1024x1024 five-layer image,
// first pass + refinement in ms: 2, 2, 2: 42.1 + 26.5; 4, 2, 2: 41.5 + 27.1; 1.5, 2, 2:
// 42.8 + 27.0; 1.5, 1.5, 1.5: 44.8 + 27.6; 1.5, 3, 3: 42.2 + 27.7; 1, 1, 1: 49.2 + 30.1.
constexpr int kOuterQuorum = 2, kDirectionQuorum = 2, kGradientQuorum = 2;
enum : int { kLaneIdle = 0, kLaneTrial, kLaneOuter, kLaneGrad, kLaneDir, kLaneSteep, kLaneEnd, kLaneFetch };

template <class T, int L, bool REFINE, bool BATCH> struct LaneSolver {
    static constexpr bool kFast = sizeof(T) == 4;   // the FP32 solver's arithmetic: fused, approximate division
    static constexpr int NV = REFINE ? 3 : 4;    // components of a layer that the method moves
    // The evaluation's layers are unrolled for up to three; at five the code
    // outgrows the instruction cache (42 -> 48 ms).
    static constexpr int kUnroll = L <= 3 ? L : 1;
    const Models<T>* models_;
    const SolverControls& ctl;
    const SolveArgs& a;
    const int lane = threadIdx.x & 31;
    T* rec_base;       // this lane's records, kLaneBlock apart: a block's are contiguous
    uint32_t n_value = 0, n_grad = 0;

    // The pixel's state that its trials read. The rest, read once an outer
    // step, is in two records: the constraint residual at x, and `Outer`.
    int state = kLaneFetch;
    T rho, f, step;
    T best_step;   // kBestAtTrial: its step along d
    int it, bt, valid, next;
    bool second;        // the line search's steepest-descent attempt
    bool from_trial;    // kLaneGrad: the point is an accepted trial (else the outer step's start)
    bool small_change, best_moved;
    // Where the best point is: nowhere yet, in its records, x itself, or the
    // trial point of step best_step. It is written to its records when x or d
    // is about to change and it would be lost: most accepted points are better
    // than the one before, so most best points never are (a copy at each new
    // best point was a fifth of a trial's instructions).
    enum : int { kNoBest = 0, kBestStored, kBestAtX, kBestAtTrial };
    int best_at;
    bool pending = false;   // the gradient phase of this trip is this lane's too

    __device__ LaneSolver(const Models<T>* m, const SolverControls& c, const SolveArgs& args)
        : models_(m), ctl(c), a(args) {
        rec_base = static_cast<T*>(a.history) + (size_t(blockIdx.x) * lane_records(L, kFast) * kLaneBlock + threadIdx.x) * 4;
        if constexpr (BATCH) models_ = static_cast<const Models<T>*>(a.models);
    }

    // ------------------------------------------------------------ storage --
    // A layer's four values of a lane: two 16-byte units (FP64) or one (FP32).
    static constexpr int kUnits = kFast ? 1 : 2;
    __device__ __forceinline__ static double2* slot(int unit) {
        return reinterpret_cast<double2*>(lane_smem) + unit * kLaneBlock + threadIdx.x;
    }
    __device__ __forceinline__ static void get(int vec, int l, T* v) {
        const double2* p = slot((vec * L + l) * kUnits);
        if constexpr (kFast) {
            const float4 u = *reinterpret_cast<const float4*>(p);
            v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
        } else {
            const double2 u = p[0], w = p[kLaneBlock];
            v[0] = u.x; v[1] = u.y; v[2] = w.x; v[3] = w.y;
        }
    }
    __device__ __forceinline__ static void put(int vec, int l, T v0, T v1, T v2, T v3) {
        double2* p = slot((vec * L + l) * kUnits);
        if constexpr (kFast) {
            *reinterpret_cast<float4*>(p) = make_float4(v0, v1, v2, v3);
        } else {
            p[0] = make_double2(v0, v1);
            p[kLaneBlock] = make_double2(v2, v3);
        }
    }
    enum : int { kX = 0, kG = 1, kD = 2 };
    // What a trial reads or leaves once: in shared memory, for the registers
    // that the loops need (at 168 a thread every spilled value is read back
    // through a first-level cache of 28 KB: the four-layer kernels with 128
    // registers and a fourth block spilled 600 bytes and took 38 ms where
    // they take 24).
    __device__ __forceinline__ static T& extra(int k) {
        return reinterpret_cast<T*>(lane_smem + lane_smem_units(L, kFast) * kLaneBlock * 16)[k * kLaneBlock + threadIdx.x];
    }
    __device__ __forceinline__ static T& target(int c) { return extra(c); }
    __device__ __forceinline__ static T& lam(int c) { return extra(3 + c); }
    __device__ __forceinline__ static T& best_norm() { return extra(7); }
    __device__ __forceinline__ static T& best_energy() { return extra(8); }
    // From the trial phase to the gradient phase of one trip.
    __device__ __forceinline__ static T& ss_kept() { return extra(9); }
    __device__ __forceinline__ static T& res_kept(int c) { return extra(10 + c); }
    // Record k of a lane whose records start at `base`.
    __device__ __forceinline__ static T* rec(T* base, int k) { return base + k * (kLaneBlock * 4); }
    __device__ __forceinline__ static T* ring(T* base, int s, int w, int l) { return rec(base, (s * 2 + w) * L + l); }
    __device__ __forceinline__ T* ring(int s, int w, int l) const { return ring(rec_base, s, w, l); }
    __device__ __forceinline__ T* best_rec(int l) const { return rec(rec_base, 2 * kLaneRing * L + l); }
    __device__ __forceinline__ T* ox_rec(int l) const { return rec(rec_base, (2 * kLaneRing + 1) * L + l); }
    __device__ __forceinline__ T* residual_rec() const { return rec(rec_base, (2 * kLaneRing + 2) * L); }
    __device__ __forceinline__ T* outer_rec() const { return rec(rec_base, (2 * kLaneRing + 2) * L + 1); }

    // What the method keeps of a pixel between its outer steps.
    struct Outer {
        T oldnorm;     // squared residual at the outer step's start
        int outer, frozen, pixel, gidx, start, job;
    };
    __device__ __forceinline__ Outer load_outer() const {
        T v[4];
        load_rec(outer_rec(), v);
        if constexpr (kFast) {
            T w[4];
            load_rec(outer_rec() + kLaneBlock * 4, w);
            return Outer{v[0], __float_as_int(v[1]), __float_as_int(v[2]), __float_as_int(v[3]), __float_as_int(w[0]),
                         __float_as_int(w[1]), __float_as_int(w[2])};
        } else {
            return Outer{v[0], __double2hiint(v[1]), __double2loint(v[1]), __double2hiint(v[2]), __double2loint(v[2]),
                         __double2hiint(v[3]), __double2loint(v[3])};
        }
    }
    __device__ __forceinline__ void store_outer(const Outer& o) const {
        if constexpr (kFast) {
            store_rec(outer_rec(), o.oldnorm, __int_as_float(o.outer), __int_as_float(o.frozen), __int_as_float(o.pixel));
            store_rec(outer_rec() + kLaneBlock * 4, __int_as_float(o.gidx), __int_as_float(o.start), __int_as_float(o.job), 0.0f);
        } else {
            store_rec(outer_rec(), o.oldnorm, __hiloint2double(o.outer, o.frozen), __hiloint2double(o.pixel, o.gidx),
                      __hiloint2double(o.start, o.job));
        }
    }
    // Work counters (only when requested).
    __device__ __forceinline__ void count(int k) const { if (a.counters) ++a.counters[5 * size_t(load_outer().gidx) + k]; }
    __device__ __forceinline__ static bool fixed_bounds(bool opaque, bool smooth, int l, int c) {
        return l == 0 && (c == 3 ? opaque : (REFINE && smooth));
    }
    __device__ __forceinline__ static bool fixed_at(bool opaque, bool smooth, int l, int c, T x, T g) {
        return fixed_bounds(opaque, smooth, l, c) || (x <= T(0.0) && g > T(0.0)) || (x >= T(1.0) && g < T(0.0));
    }
    // v in [0, 1] (NaN stays NaN), by its bits: the FP64 pipe has the
    // arithmetic, and its compares are as slow as it is.
    __device__ __forceinline__ static double clamp01(double v) {
        const int hi = __double2hiint(v);
        const bool keep = uint32_t(hi) < 0x3ff00000u || (uint32_t(hi) & 0x7fffffffu) > 0x7ff00000u;
        return __hiloint2double(keep ? hi : (hi < 0 ? 0 : 0x3ff00000), keep ? __double2loint(v) : 0);
    }
    __device__ __forceinline__ static float clamp01(float v) { return v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v); }

    // The per-channel partial sums, added as the lanes of a group add theirs.
    __device__ __forceinline__ static T sum(const T* v) {
        if constexpr (REFINE) return (v[0] + v[1]) + v[2];
        else return (v[0] + v[1]) + (v[2] + v[3]);
    }

    // ------------------------------------------------------------ forward --
    // One layer of the composite: A, pc in/out.
    __device__ __forceinline__ void compose(const Models<T>& m, int l, const T* t, T av, T& A,
                                            T* pc) const {
        if (l == 0) {
            A = av;
#pragma unroll
            for (int c = 0; c < 3; ++c) pc[c] = t[c];
            return;
        }
        const T dd = A, X = m.fX[l], Y = m.fY[l], Z = m.fZ[l];
        const T n_dd = T(1.0) - dd, n_av = T(1.0) - av;
        const T ya = Y * av * n_dd, zd = Z * dd * n_av;
        const T Al = madd<T>(Z * dd, n_av, madd<T>(X * av, dd, ya));
        T fv[3], y = T(0);
        if constexpr (!kFast) y = reciprocal(Al);
        blend_values(m, l, t, pc, fv);
        const bool big = Al > T(1e-12);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T pre = madd<T>(zd, pc[c], madd<T>(fv[c] * av, dd, ya * t[c]));
            T q;
            if constexpr (kFast) q = qdiv(pre, Al); else q = quotient(pre, Al, y);
            pc[c] = big ? q : pre;
        }
        A = Al;
    }

    // Point of layer l at step s along d, within bounds (the fixed values have
    // d = 0 and x in [0, 1]; at the start of an outer step d is zero).
    __device__ __forceinline__ static void point(const T* x, const T* d, T s, T* t) {
#pragma unroll
        for (int c = 0; c < 4; ++c) t[c] = REFINE && c == 3 ? x[c] : clamp01(madd<T>(s, d[c], x[c]));
    }

    // Layer l of the best point, at x or at the trial point of step best_step, to
    // its record (x as it is: a step of zero along an infinite d would not be x).
    __device__ __forceinline__ void store_best(int l, const T* x, const T* d) const {
        const bool at_x = best_at == kBestAtX;
        T t[4];
        point(x, d, best_step, t);
        store_rec(best_rec(l), at_x ? x[0] : t[0], at_x ? x[1] : t[1], at_x ? x[2] : t[2], at_x ? x[3] : t[3]);
    }

    // Writes the best point to its records before x or d changes.
    __device__ __forceinline__ void save_best() {
#pragma unroll 1
        for (int l = 0; l < L; ++l) {
            T x[4], d[4];
            get(kX, l, x); get(kD, l, d);
            store_best(l, x, d);
        }
        best_at = kBestStored;
    }

    // Evaluates the objective at the trial point (kLaneTrial) or at x
    // (kLaneOuter) and decides the trial. A lane whose point is accepted and
    // whose gradient comes next (kLaneGrad) repeats its evaluation beside the
    // others', at no cost of its own, and keeps what the reverse sweep needs:
    // x becomes the accepted point, its step goes to the ring's free slot, and
    // d's slots take the composite's colours and alpha.
    __device__ __forceinline__ void forward() {
        const Models<T>& m = *models_;
        const bool keep = state == kLaneGrad, at_x = state == kLaneOuter || (keep && !from_trial);
        // (keep) the accepted point is the best point; the best point is lost with x and d.
        const bool best_here = best_at == kBestAtTrial && best_step == step;
        const bool best_lost = !at_x && (best_at == kBestAtX || (best_at == kBestAtTrial && !best_here));
        bool moved = false;     // (keep) some component moved by at least the inner tolerance
        [[maybe_unused]] const T tol_lo = ctl.inner_tolerance * (1.0 - 0x1p-48), tol_hi = ctl.inner_tolerance * (1.0 + 0x1p-48);
        T sl[NV], ss[NV], A = T(0.0), pc[3], energy = T(0.0), asum = T(0.0);
        uint32_t largest = 0;   // high word of the largest motion of a component
#pragma unroll
        for (int c = 0; c < NV; ++c) { sl[c] = T(0.0); ss[c] = T(0.0); }
#pragma unroll kUnroll
        for (int l = 0; l < L; ++l) {
            T x[4], d[4], g[4], t[4], s[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
            get(kX, l, x); get(kD, l, d); get(kG, l, g);
            point(x, d, step, t);
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                s[c] = t[c] - x[c];
                sl[c] = madd<T>(g[c], s[c], sl[c]);
                largest = max(largest, magnitude_bits(s[c]));
            }
            const T av = t[3];
            const T d0 = t[0] - m.mean[l][0], d1 = t[1] - m.mean[l][1], d2 = t[2] - m.mean[l][2];
            const T* P = m.prec[l];
            const T v0 = madd<T>(P[2], d2, madd<T>(P[0], d0, P[1] * d1));
            const T v1 = madd<T>(P[5], d2, madd<T>(P[3], d0, P[4] * d1));
            const T v2 = madd<T>(P[8], d2, madd<T>(P[6], d0, P[7] * d1));
            const T D = madd<T>(d2, v2, madd<T>(d0, v0, d1 * v1));
            energy = madd<T>(av, D, energy);
            asum += av;
            compose(m, l, t, av, A, pc);
            if (keep) {
#pragma unroll
                for (int c = 0; c < NV; ++c) {
                    ss[c] = madd<T>(s[c], s[c], ss[c]);
                    // |s| / (1 + |x|) against the tolerance without the
                    // division, except where rounding could decide.
                    const T w = T(1.0) + fabs(x[c]), as = fabs(s[c]);
                    if constexpr (kFast) moved = moved || !(qdiv(as, w) < T(ctl.inner_tolerance));
                    else if (!(as < tol_lo * w)) moved = moved || as > tol_hi * w || step_reaches(as, w, ctl.inner_tolerance);
                }
                if (best_lost) {
                    store_best(l, x, d);
                }
                store_rec(ring(next, 0, l), s[0], s[1], s[2], s[3]);
                put(kX, l, t[0], t[1], t[2], t[3]);
                put(kD, l, pc[0], pc[1], pc[2], A);
            }
        }
        T res[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) res[c] = c < 3 ? pc[c < 3 ? c : 0] - target(c < 3 ? c : 0) : A - T(1.0);
        if (keep) {
            small_change = small_change || !moved;
            if (best_here) best_at = kBestAtX;
            if (best_lost) best_at = kBestStored;
            ss_kept() = sum(ss);
#pragma unroll
            for (int c = 0; c < NV; ++c) res_kept(c) = res[c];
            store_rec(residual_rec(), res[0], res[1], res[2], res[NV - 1]);
            return;
        }
        if (!REFINE) energy += T(0.01) * asum;
        T terms[NV], nn[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            terms[c] = madd<T>(T(0.5) * rho * res[c], res[c], -(lam(c) * res[c]));
            nn[c] = res[c] * res[c];
        }
        const T norm = sum(nn), value = energy + sum(terms), slope = sum(sl);

        // A trial that does not move (whose sum of squared motions is zero)
        // ends the attempt, unevaluated. FP32: squares that round to zero, up to
        // 2^-75; FP64 by the high word, below 2^-537 (squares round to zero
        // below 2^-537.5).
        if (!at_x && largest < (kFast ? 0x1a000001u : 0x1e600000u)) { attempt_failed(); return; }
        const T tol2 = ctl.outer_tolerance * ctl.outer_tolerance;
        const bool feasible = norm < tol2;
        if (isfinite(energy) && isfinite(norm) &&
            (best_at == kNoBest || (feasible && (best_norm() >= tol2 || energy < best_energy())) ||
             (!feasible && best_norm() >= tol2 && norm < best_norm()))) {
            best_norm() = norm; best_energy() = energy; best_moved = true;
            best_at = at_x ? kBestAtX : kBestAtTrial;
            best_step = step;
        }
        // Evaluations are counted as the method makes them: a first trial
        // with its gradient, and a later trial that is accepted once more,
        // with its gradient.
        const bool counted_grad = at_x || (bt == 0 && ctl.gradient_on_first_trial);
        count(0); ++n_value;
        if (counted_grad) { count(1); ++n_grad; }
        if (at_x) {
            f = value;
            outer_rec()[0] = norm;
            valid = 0; next = 0; it = 0;
            from_trial = false;
            state = kLaneGrad;
        } else {
            count(3);
            if (slope < T(0.0) && isfinite(value) && value <= f + T(1e-4) * slope) {
                if (!counted_grad) { count(0); count(1); ++n_value; ++n_grad; }
                const T delta = fabs(f - value), size = T(0.5) * (fabs(f) + fabs(value));
                small_change = delta < T(ctl.inner_tolerance) * size;
                f = value;
                from_trial = true;
                state = kLaneGrad;
            } else {
                step *= T(0.5);
                if (++bt >= 32) attempt_failed();
            }
        }
    }

    __device__ __noinline__ static bool step_reaches(T as, T w, T tol) { return !(as / w < tol); }

    // The line search ran out of trials: once more from steepest descent,
    // then the end of the inner solve.
    __device__ __forceinline__ void attempt_failed() {
        valid = 0; next = 0;
        state = second ? kLaneEnd : kLaneSteep;
    }

    // ----------------------------------------------------------- backward --
    // Gradient at the evaluated point (kLaneGrad, after forward()), and the
    // accepted step's curvature pair and termination test.
    __device__ __forceinline__ void backward() {
        const Models<T>& m = *models_;
        const bool at_x = !from_trial;
        // Reverse sweep; layer l's slot of d turns from its composite into its gradient.
        T adj[3], adj3 = REFINE ? T(0.0) : rho * res_kept(NV - 1) - lam(NV - 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) adj[c] = rho * res_kept(c) - lam(c);
#pragma unroll 1
        for (int l = L - 1; l >= 0; --l) {
            T t[4], ng[4];
            get(kX, l, t);
            const T av = t[3];
            {
                const T d0 = t[0] - m.mean[l][0], d1 = t[1] - m.mean[l][1], d2 = t[2] - m.mean[l][2];
                const T* P = m.prec[l];
                const T v0 = madd<T>(P[2], d2, madd<T>(P[0], d0, P[1] * d1));
                const T v1 = madd<T>(P[5], d2, madd<T>(P[3], d0, P[4] * d1));
                const T v2 = madd<T>(P[8], d2, madd<T>(P[6], d0, P[7] * d1));
                const T D = madd<T>(d2, v2, madd<T>(d0, v0, d1 * v1));
                const T t0 = madd<T>(P[6], d2, madd<T>(P[0], d0, P[3] * d1));
                const T t1 = madd<T>(P[7], d2, madd<T>(P[1], d0, P[4] * d1));
                const T t2 = madd<T>(P[8], d2, madd<T>(P[2], d0, P[5] * d1));
                ng[0] = av * (v0 + t0); ng[1] = av * (v1 + t1); ng[2] = av * (v2 + t2);
                ng[3] = REFINE ? D : D + T(0.01);
            }
            if (l > 0) {
                T o[4], q[4];
                get(kD, l, o); get(kD, l - 1, q);
                const T Al = o[3], dd = q[3], X = m.fX[l], Y = m.fY[l], Z = m.fZ[l];
                const T n_dd = T(1.0) - dd, n_av = T(1.0) - av;
                const T da = madd<T>(X, dd, Y * n_dd) - Z * dd;
                const T db = madd<T>(Z, n_av, X * av - Y * av);
                const T ya = Y * av * n_dd, yd = Y * n_dd, zd = Z * dd, zdn = zd * n_av, zn = Z * n_av, ad = av * dd;
                const bool big = Al > T(1e-12);
                T fv[3], fs[3], fd[3], ga[3], gp[3];
                blend_all(m, l, t, q, fv, fs, fd);
                T y;   // (FP32: times the approximate reciprocal)
                if constexpr (kFast) y = big ? qdiv(T(1), Al) : T(1); else y = reciprocal(Al);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const T v = adj[c], s = t[c], cc = q[c];
                    const T ds = madd<T>(ad, fs[c], ya);
                    const T dc = madd<T>(ad, fd[c], zdn);
                    const T pa = madd<T>(fv[c], dd, yd * s) - zd * cc;
                    const T pd = madd<T>(zn, cc, fv[c] * av - Y * av * s);
                    if constexpr (kFast) {
                        ga[c] = v * (big ? madd<T>(-o[c], da, pa) * y : pa);
                        gp[c] = v * (big ? madd<T>(-o[c], db, pd) * y : pd);
                        ng[c] += v * (big ? ds * y : ds);
                        adj[c] = v * (big ? dc * y : dc);
                    } else {
                        const T na = pa - o[c] * da, np = pd - o[c] * db;
                        const T qa = quotient(na, Al, y), qp = quotient(np, Al, y), qs = quotient(ds, Al, y),
                                qc = quotient(dc, Al, y);
                        ga[c] = v * (big ? qa : pa);
                        gp[c] = v * (big ? qp : pd);
                        ng[c] += v * (big ? qs : ds);
                        adj[c] = v * (big ? qc : dc);
                    }
                }
                if constexpr (REFINE) {
                    T ta = adj3 * da, tp = adj3 * db;
                    ta += ga[0]; ta += ga[1]; ta += ga[2];
                    tp += gp[0]; tp += gp[1]; tp += gp[2];
                    ng[3] += ta;
                    adj3 = tp;
                } else {
                    const T g3 = adj3 * da, p3 = adj3 * db;
                    ng[3] += (ga[0] + ga[1]) + (ga[2] + g3);
                    adj3 = (gp[0] + gp[1]) + (gp[2] + p3);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) ng[c] += adj[c];
                ng[3] += adj3;
            }
            put(kD, l, ng[0], ng[1], ng[2], ng[3]);
        }
        if (at_x) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
                T ng[4];
                get(kD, l, ng);
                put(kG, l, ng[0], ng[1], ng[2], ng[3]);
            }
            state = kLaneDir;
            return;
        }
        T sy[NV], yy[NV], ya = T(0.0);
#pragma unroll
        for (int c = 0; c < NV; ++c) { sy[c] = T(0.0); yy[c] = T(0.0); }
        T step_taken[L][4];
#pragma unroll
        for (int l = 0; l < L; ++l) load_rec(ring(next, 0, l), step_taken[l]);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            T ng[4], g[4], yv[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
            const T* s = step_taken[l];
            get(kD, l, ng); get(kG, l, g);
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                yv[c] = ng[c] - g[c];
                sy[c] = madd<T>(s[c], yv[c], sy[c]);
                yy[c] = madd<T>(yv[c], yv[c], yy[c]);
            }
            if (REFINE) { const T dy = ng[3] - g[3]; ya = madd<T>(dy, dy, ya); }
            store_rec(ring(next, 1, l), yv[0], yv[1], yv[2], yv[3]);
            put(kG, l, ng[0], ng[1], ng[2], ng[3]);
        }
        T yyt = sum(yy);
        if (REFINE) yyt += ya;
        if (curvature(sum(sy), ss_kept(), yyt)) {
            next = next + 1 == kLaneRing ? 0 : next + 1;
            valid = valid + 1 < kHistory ? valid + 1 : kHistory;
        }
        if (small_change) state = kLaneEnd;
        else if (++it >= ctl.inner) state = kLaneEnd;
        else state = kLaneDir;
    }

    __device__ __forceinline__ static T inverse(T v) {
        if constexpr (kFast) return qdiv(T(1), v); else return __drcp_rn(v);
    }
    // sy > 1e-9 sqrt(ss yy), sy > 0 and 1 / sy finite: by squares, except
    // where rounding, under- or overflow could decide.
    __device__ __forceinline__ static bool curvature(T sy, T ss, T yy) {
        if constexpr (kFast) return sy > T(0) && sy * sy > T(1e-18) * (ss * yy) && isfinite(qdiv(T(1), sy));
        if (!(sy > T(0.0))) return false;
        const T t = T(1e-18) * (ss * yy), r = sy * sy;
        if (t > 1e-250 && t < 1e250 && r < 1e250 && fabs(r - t) > 1e-12 * t) return r > t;
        return curvature_exact(sy, ss, yy);
    }
    __device__ __noinline__ static bool curvature_exact(T sy, T ss, T yy) {
        return sy > T(1e-9) * sqrt(ss * yy) && sy > T(0.0) && isfinite(T(1.0) / sy);
    }

    // ---------------------------------------------------------- direction --
    // Top of an inner iteration (kLaneDir: projected gradient test, two-loop
    // direction) or the steepest-descent attempt (kLaneSteep).
    __device__ __forceinline__ void direction() {
        const bool steep = state == kLaneSteep;
        if (!steep) count(2);
        if (best_at == kBestAtTrial) save_best();
        const int what = form_direction(rec_base, valid, next, steep, a.opaque != 0, a.smooth != 0, isfinite(f));
        if (what == kStationary) { state = kLaneEnd; return; }
        if (what == kReset) { valid = 0; next = 0; }
        second = steep;
        bt = 0;
        step = T(1.0);
        state = kLaneTrial;
    }

    // Forms d from x, g and the ring (static: it touches none of the pixel's
    // other state).
    enum : int { kStationary = 0, kFormed = 1, kReset = 2 };
    __device__ __forceinline__ static int form_direction(T* base, int valid, int next, bool steep, bool opaque,
                                                      bool smooth, bool finite_f) {
        uint32_t freem = 0;
        {
            T pg[NV];
#pragma unroll
            for (int c = 0; c < NV; ++c) pg[c] = T(0.0);
#pragma unroll 1
            for (int l = 0; l < L; ++l) {
                T x[4], g[4], v[4];
                get(kX, l, x); get(kG, l, g);
                v[3] = T(0.0);
#pragma unroll
                for (int c = 0; c < NV; ++c) {
                    const bool fr = !fixed_at(opaque, smooth, l, c, x[c], g[c]);
                    freem |= fr ? 1u << (l * 4 + c) : 0u;
                    v[c] = fr ? g[c] : T(0.0);
                    pg[c] = madd<T>(v[c], v[c], pg[c]);
                }
                put(kD, l, v[0], v[1], v[2], v[3]);
            }
            if (!steep && (sum(pg) < T(1e-16) || !finite_f)) return kStationary;
        }
        T q[L][4];
#pragma unroll
        for (int l = 0; l < L; ++l) get(kD, l, q[l]);
        // The pairs' components outside the free set are read as zeros (a
        // select each; skipping their operations instead takes a branch each,
        // and the kernel 1.1 times as long). q is zero there throughout, so
        // its own products need no select.
        T scaling = T(1.0);
        bool have_scaling = false;
        double2* coeff = slot(2 * L * kUnits);   // (one pair a unit)
#pragma unroll 1
        for (int j = 0; j < valid; ++j) {
            int k = next - 1 - j;
            k = k < 0 ? k + kLaneRing : k;
            T dot[NV], sy[NV], ss[NV], yy[NV];
#pragma unroll
            for (int c = 0; c < NV; ++c) { dot[c] = T(0.0); sy[c] = T(0.0); ss[c] = T(0.0); yy[c] = T(0.0); }
            T ym[L][4];
#pragma unroll
            for (int l = 0; l < L; ++l) load_rec(ring(base, k, 1, l), ym[l]);
#pragma unroll
            for (int l = 0; l < L; ++l) {
                T sv[4];
                T* yv = ym[l];
                load_rec(ring(base, k, 0, l), sv);
#pragma unroll
                for (int c = 0; c < NV; ++c) {
                    const bool fr = freem >> (l * 4 + c) & 1u;
                    const T s1 = fr ? sv[c] : T(0.0), y1 = fr ? yv[c] : T(0.0);
                    yv[c] = y1;
                    dot[c] = madd<T>(s1, q[l][c], dot[c]);
                    sy[c] = madd<T>(s1, y1, sy[c]);
                    ss[c] = madd<T>(s1, s1, ss[c]);
                    yy[c] = madd<T>(y1, y1, yy[c]);
                }
            }
            const T syt = sum(sy), yyt = sum(yy);
            const T inv = curvature(syt, sum(ss), yyt) ? inverse(syt) : T(0.0);
            const T co = sum(dot) * inv;
#pragma unroll
            for (int l = 0; l < L; ++l)
#pragma unroll
                for (int c = 0; c < NV; ++c) q[l][c] = madd<T>(-co, ym[l][c], q[l][c]);
            if (!have_scaling && inv > T(0.0) && yyt > T(0.0)) { scaling = qdiv(syt, yyt); have_scaling = true; }
            coeff[j * kLaneBlock] = make_double2(co, inv);   // (exact in FP32 too)
        }
        scaling = fmax(T(1e-12), fmin(T(1e3), scaling));
#pragma unroll
        for (int l = 0; l < L; ++l)
#pragma unroll
            for (int c = 0; c < NV; ++c) q[l][c] *= scaling;
#pragma unroll 1
        for (int j = valid - 1; j >= 0; --j) {
            int k = next - 1 - j;
            k = k < 0 ? k + kLaneRing : k;
            T dot[NV], sv[L][4];
#pragma unroll
            for (int c = 0; c < NV; ++c) dot[c] = T(0.0);
#pragma unroll
            for (int l = 0; l < L; ++l) {
                T yv[4];
                load_rec(ring(base, k, 1, l), yv); load_rec(ring(base, k, 0, l), sv[l]);
#pragma unroll
                for (int c = 0; c < NV; ++c) dot[c] = madd<T>(yv[c], q[l][c], dot[c]);
            }
            const double2 ci = coeff[j * kLaneBlock];
            const T w = madd<T>(-sum(dot), T(ci.y), T(ci.x));
#pragma unroll
            for (int l = 0; l < L; ++l)
#pragma unroll
                for (int c = 0; c < NV; ++c)
                    q[l][c] = madd<T>(w, freem >> (l * 4 + c) & 1u ? sv[l][c] : T(0.0), q[l][c]);
        }
#pragma unroll
        for (int l = 0; l < L; ++l) put(kD, l, q[l][0], q[l][1], q[l][2], q[l][3]);
        T descent[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) descent[c] = T(0.0);
#pragma unroll 1
        for (int l = 0; l < L; ++l) {
            T x[4], g[4], d[4];
            get(kX, l, x); get(kG, l, g); get(kD, l, d);
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                T v = -d[c];
                if (fixed_bounds(opaque, smooth, l, c) || (x[c] <= T(0.0) && v < T(0.0)) || (x[c] >= T(1.0) && v > T(0.0))) v = T(0.0);
                d[c] = v;
                descent[c] = madd<T>(v, g[c], descent[c]);
            }
            put(kD, l, d[0], d[1], d[2], d[3]);
        }
        if (!steep && !(sum(descent) < T(0.0))) {
#pragma unroll 1
            for (int l = 0; l < L; ++l) {
                T x[4], g[4], d[4];
                get(kX, l, x); get(kG, l, g);
                d[3] = T(0.0);
#pragma unroll
                for (int c = 0; c < NV; ++c) d[c] = fixed_at(opaque, smooth, l, c, x[c], g[c]) ? T(0.0) : -g[c];
                put(kD, l, d[0], d[1], d[2], d[3]);
            }
            return kReset;
        }
        return kFormed;
    }

    // -------------------------------------------------------- outer steps --
    // End of an outer step (kLaneEnd): multipliers, penalty, and the next
    // outer step, the next start, or the pixel's result.
    enum : int { kNextOuter, kNextStart, kFinished };
    __device__ __forceinline__ int end_outer(Outer& o, bool& capped) {
        T r[4], ox[L][4], nn[NV], mo[NV];
        o = load_outer();
        load_rec(residual_rec(), r);
#pragma unroll
        for (int l = 0; l < L; ++l) load_rec(ox_rec(l), ox[l]);
        const T tol2 = ctl.outer_tolerance * ctl.outer_tolerance;
#pragma unroll
        for (int c = 0; c < NV; ++c) { nn[c] = r[c] * r[c]; mo[c] = T(0.0); }
        const T norm = sum(nn);
        const bool feasible = norm < tol2;
#pragma unroll
        for (int c = 0; c < NV; ++c) lam(c) = madd<T>(-rho, r[c], lam(c));
        if (norm > T(0.0625) * o.oldnorm) rho *= T(10.0);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            T x[4];
            get(kX, l, x);
#pragma unroll
            for (int c = 0; c < NV; ++c) { const T dl = x[c] - ox[l][c]; mo[c] = madd<T>(dl, dl, mo[c]); }
        }
        const T motion = sum(mo);
        o.frozen = (motion == T(0.0) && !best_moved) ? o.frozen + 1 : 0;
        int what = kFinished;
        if (!(ctl.frozen_stop > 0 && o.frozen >= ctl.frozen_stop) && !(motion < tol2 && feasible) &&
            o.outer + 1 < ctl.outer) {
            ++o.outer;
            what = kNextOuter;
        } else if (kFast && ctl.cap_is_miss && !(motion < tol2 && feasible)) {
            capped = true;   // the FP64 re-solve gives the pixel the method's own result
        } else if (o.start + 1 < ctl.starts) {
            ++o.start;
            what = kNextStart;
        }
        if (best_at == kBestAtTrial || (best_at == kBestAtX && what == kNextStart)) save_best();
        return what;
    }

    __device__ __forceinline__ void begin_outer(const Outer& o) {
        store_outer(o);
        count(4);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            T x[4];
            get(kX, l, x);
            store_rec(ox_rec(l), x[0], x[1], x[2], x[3]);
            put(kD, l, T(0.0), T(0.0), T(0.0), T(0.0));
        }
        best_moved = false;
        step = T(0.0);
        state = kLaneOuter;
    }

    __device__ __forceinline__ const double* image(const Outer& o) const {
        if constexpr (BATCH) return a.jobs[o.job].image; else return a.image;
    }
    __device__ __forceinline__ size_t pixels(const Outer& o) const {
        if constexpr (BATCH) return size_t(a.jobs[o.job].n); else return size_t(a.n);
    }
    __device__ __forceinline__ double pinned_alpha(const Outer& o, int l) const {
        return (a.opaque && l == 0) ? 1.0 : a.targets[size_t(l) * size_t(a.n) + o.pixel];
    }
    __device__ __forceinline__ double background(const Outer& o, int c) const {
        return a.targets[(size_t(L) + c) * size_t(a.n) + o.pixel];
    }

    // The start-0 seed of component c of layer l.
    __device__ __forceinline__ T seed(const Outer& o, int l, int c) const {
        const size_t i = size_t(o.pixel);
        if constexpr (REFINE) {
            if (c == 3) return T(pinned_alpha(o, l));
            return T((a.smooth && l == 0) ? background(o, c) : a.first[(size_t(l) * size_t(a.n) + i) * 4 + c]);
        } else {
            const float* wp;
            if constexpr (BATCH) wp = a.jobs[o.job].warm; else wp = a.warm;
            if (wp) return T(wp[i * size_t(4 * L) + (c == 3 ? l : L + 3 * l + c)]);
            if (c == 3) return (a.opaque && l == 0) ? T(1.0) : T(0.5);
            return fmin(T(1.0), fmax(T(0.0), models_->mean[l][c]));
        }
    }

    // Bounds of component c of layer l applied to v.
    __device__ __forceinline__ T clamp_bounds(const Outer& o, int l, int c, T v) const {
        if (REFINE && c == 3) return v;
        T lo = T(0.0), hi = T(1.0);
        if (l == 0 && c == 3 && a.opaque) lo = T(1.0);
        if (REFINE && l == 0 && c != 3 && a.smooth) lo = hi = T(background(o, c));
        return v < lo ? lo : (v > hi ? hi : v);
    }

    // Component c of layer l of x in shared memory.
    __device__ __forceinline__ static T* x_at(int l, int c) {
        if constexpr (kFast) return reinterpret_cast<T*>(slot(l)) + c;
        else return reinterpret_cast<T*>(slot(2 * l + (c >> 1))) + (c & 1);
    }

    // Starting point o.start: the seeds, all loads in flight at once; the
    // further starts one component at a time (rare).
    __device__ __forceinline__ void begin_start(Outer& o) {
        if (o.start == 0) {
            T v[L][4];
#pragma unroll
            for (int l = 0; l < L; ++l)
#pragma unroll
                for (int c = 0; c < 4; ++c) v[l][c] = seed(o, l, c);
#pragma unroll
            for (int l = 0; l < L; ++l) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (!(REFINE && l == 0 && c != 3 && a.smooth)) v[l][c] = clamp_bounds(o, l, c, v[l][c]);
                put(kX, l, v[l][0], v[l][1], v[l][2], v[l][3]);
            }
        } else {
            further_start(o);
        }
#pragma unroll
        for (int c = 0; c < NV; ++c) lam(c) = T(0.0);
        rho = T(100.0);
        o.outer = 0;
        o.frozen = 0;
    }

    __device__ __forceinline__ void further_start(const Outer& o) const {
        const Models<T>& m = *models_;
        const int s = o.start;
#pragma unroll 1
        for (int k = 0; k < 4 * L; ++k) {
            const int l = k >> 2, c = k & 3;
            T v;
            if (c == 3) v = REFINE ? T(pinned_alpha(o, l)) : (s == 1 ? (l == 0 ? T(1.0) : T(0.0)) : T(0.5));
            else if (s == 2) v = fmax(T(0.05), fmin(T(0.95), m.mean[l][c]));
            else v = (!REFINE && l == 0) ? fmin(T(1.0), fmax(T(0.0), T(image(o)[3 * size_t(o.pixel) + c]))) : m.mean[l][c];
            *x_at(l, c) = clamp_bounds(o, l, c, v);
        }
        if (s != 2) return;
        // Move Dodge/Burn sources into the unsaturated branch.
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
            T da = *x_at(0, 3), dest = *x_at(0, c);
#pragma unroll 1
            for (int l = 1; l < L; ++l) {
                const T al = *x_at(l, 3), X = m.fX[l], Y = m.fY[l], Z = m.fZ[l];
                const T Al = X * al * da + Y * al * (T(1.0) - da) + Z * da * (T(1.0) - al);
                T sv = *x_at(l, c);
                if (dest >= T(0.0) && dest <= T(1.0) && m.mode[l] == 6) sv = fmin(sv, fmax(T(0.0), T(1.0) - dest - T(0.05)));
                if (dest >= T(0.0) && dest <= T(1.0) && m.mode[l] == 7) sv = fmax(sv, fmin(T(1.0), T(1.0) - dest + T(0.05)));
                sv = clamp_bounds(o, l, c, sv);
                *x_at(l, c) = sv;
                const T pre = blend_value_call<T>(m.mode[l], sv, dest) * al * da +
                                   Y * al * (T(1.0) - da) * sv + Z * da * (T(1.0) - al) * dest;
                dest = Al > T(1e-12) ? pre / Al : pre;
                da = Al;
            }
        }
    }

    // ------------------------------------------------------------- pixels --
    // Writes the finished pixel: output (pinned values exactly), status, miss
    // list. The point written is the best point, whose constraint norm is
    // best_norm (the same operations on the same values as a check of the
    // written point); a pixel without one writes its seed, checked here.
    __device__ __forceinline__ void store(const Outer& o, bool skipped, bool capped) {
        const size_t n = pixels(o), i = size_t(o.pixel);
        double* outp;
        int32_t* stp;
        if constexpr (BATCH) { outp = a.jobs[o.job].out; stp = a.jobs[o.job].status; }
        else { outp = a.out; stp = a.status; }
        T w[L][4];
        double v[L][4];
        if (best_at == kBestStored) {
#pragma unroll
            for (int l = 0; l < L; ++l) load_rec(best_rec(l), w[l]);
        } else if (best_at == kBestAtX) {
#pragma unroll
            for (int l = 0; l < L; ++l) get(kX, l, w[l]);
        } else {
#pragma unroll
            for (int l = 0; l < L; ++l)
#pragma unroll
                for (int c = 0; c < 4; ++c) w[l][c] = seed(o, l, c);
        }
#pragma unroll
        for (int l = 0; l < L; ++l) {
#pragma unroll
            for (int c = 0; c < 4; ++c) v[l][c] = double(w[l][c]);
            if (REFINE) v[l][3] = pinned_alpha(o, l);
            else if (l == 0 && a.opaque) v[l][3] = 1.0;
            if (REFINE && l == 0 && a.smooth)
#pragma unroll
                for (int c = 0; c < 3; ++c) v[l][c] = background(o, c);
        }
#pragma unroll
        for (int l = 0; l < L; ++l)
#pragma unroll
            for (int c = 0; c < 4; ++c) outp[(size_t(l) * n + i) * 4 + c] = v[l][c];   // (8-byte aligned, as the caller's buffer)
        if (skipped) {
            if (stp) stp[i] = 8;
            if (a.input_failed) atomicAdd(a.input_failed, 1);
            return;
        }
        // FP64: the written best point's norm is best_norm, the same operations
        // on the same values. FP32, and a pixel without a best point: checked.
        const double norm = kFast || best_at == kNoBest ? written_norm(*models_, outp, image(o) + 3 * i, n, i) : double(best_norm());
        const bool miss = capped || !(norm < ctl.outer_tolerance * ctl.outer_tolerance);
        if (stp) stp[i] = miss ? 3 : 0;
        if (miss && a.miss_list) a.miss_list[atomicAdd(a.miss_count, 1)] = int32_t(o.gidx);
    }

    // Constraint norm of the written point, one channel at a time.
    __device__ __noinline__ static double written_norm(const Models<T>& m, const double* outp, const double* rgb,
                                                       size_t n, size_t i) {
        double total = 0.0, A = 0.0, first_two = 0.0;
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
            double cc = 0.0;
#pragma unroll 1
            for (int l = 0; l < L; ++l) {
                const double* o = outp + (size_t(l) * n + i) * 4;
                const double sv = o[c], al = o[3];
                if (l == 0) { A = al; cc = sv; continue; }
                const double dd = A, X = m.fX[l], Y = m.fY[l], Z = m.fZ[l];
                const double Al = X * al * dd + Y * al * (1.0 - dd) + Z * dd * (1.0 - al);
                const double pre = blend_value<double>(m.mode[l], sv, cc) * al * dd + Y * al * (1.0 - dd) * sv +
                                   Z * dd * (1.0 - al) * cc;
                cc = Al > 1e-12 ? pre / Al : pre;
                A = Al;
            }
            const double r = cc - rgb[c];
            if (c == 0) first_two = r * r;
            else if (c == 1) first_two += r * r;
            else total = r * r;
        }
        if (!REFINE) total += (A - 1.0) * (A - 1.0);
        return first_two + total;
    }

    // Loads the pixel of queue entry `job`; false when it is written without
    // a solve (refinement targets that cannot be normalized).
    __device__ __forceinline__ bool load(Outer& o, int job) {
        o.gidx = a.list ? a.list[job] : (a.order ? a.order[job] : a.first_pixel + job);
        o.pixel = o.gidx;
        o.job = 0;
        if constexpr (BATCH) {
            int lo = 0, hi = a.job_count - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.jobs[mid].offset <= int64_t(o.gidx)) lo = mid; else hi = mid - 1;
            }
            o.job = lo;
            models_ = static_cast<const Models<T>*>(a.models) + a.jobs[lo].model;
            o.pixel = o.gidx - int(a.jobs[lo].offset);
        }
        const size_t i = size_t(o.pixel);
        const double* p = image(o) + 3 * i;
#pragma unroll
        for (int c = 0; c < 3; ++c) target(c) = T(p[c]);
        best_at = kNoBest;
        best_norm() = INFINITY; best_energy() = INFINITY;
        if (a.counters)
#pragma unroll
            for (int k = 0; k < 5; ++k) a.counters[5 * size_t(o.gidx) + k] = 0;
        o.start = 0;
        o.oldnorm = T(0.0);
        return !(REFINE && a.input_status && a.input_status[i] != 0);
    }

    // --------------------------------------------------------------- loop --
    __device__ void run() {
        const unsigned full = 0xffffffffu;
        const int total = a.list ? min(*a.list_count, a.list_limit) : (a.pixel_count >= 0 ? a.pixel_count : a.n);
        // A small launch spreads its pixels over all blocks, and in a block over
        // its warps: the fewer pixels share a block's phases, the shorter the
        // last one's chain. Not so the groups of a batch, which run side by side
        // (also as re-solves, of a few thousand hard pixels each): spread over all
        // blocks, each would hold the others off the SMs until its last chain
        // ends. A group whose pixels fit its share of the blocks leaves the
        // rest of them to the others, unless it has less than two pixels a block
        // there. FP32 batches, ms, every block / share / quad re-solve: 162,387
        // pixels in four groups (16,086 misses) 17.4 / 13.6 / 16.0, 26,674
        // (3,700) 8.6 / 6.3 / 7.8, 3,241 (830) 4.5 / 4.9 / 6.9; FP64 batches, every
        // block / share: 26,674 8.1 / 4.9, 3,941 5.6 / 4.1, 2,029 3.6 / 4.1.
        static_assert(kLaneBlock == 128, "four warps a block");
        int blocks = gridDim.x;
        if constexpr (BATCH) {
            const int share = max(1, blocks / a.groups);
            if (total > 2 * share && total <= share * kLaneBlock) blocks = share;
            if (int(blockIdx.x) >= blocks) return;
        }
        if (int64_t((threadIdx.x & 31u) << 2 | threadIdx.x >> 5) * blocks >= total) state = kLaneIdle;
        // Lanes waiting for each phase, one byte a phase (trial, direction,
        // gradient, outer step), counted over the block with one barrier, in
        // two buffers in turn.
        __shared__ uint32_t counts[2][kLaneBlock / 32];
        int turn = 0, nf = 0, nd = 0, nb = 0, ne = 0, live = 0;
        auto recount = [&]() {
            const uint32_t mine = uint32_t(__popc(__ballot_sync(full, state == kLaneTrial || state == kLaneOuter))) |
                                  uint32_t(__popc(__ballot_sync(full, state == kLaneDir || state == kLaneSteep))) << 8 |
                                  uint32_t(__popc(__ballot_sync(full, state == kLaneGrad))) << 16 |
                                  uint32_t(__popc(__ballot_sync(full, state == kLaneEnd || state == kLaneFetch))) << 24;
            if (lane == 0) counts[turn][threadIdx.x >> 5] = mine;
            __syncthreads();
            uint32_t all = 0;
#pragma unroll
            for (int w = 0; w < kLaneBlock / 32; ++w) all += counts[turn][w];
            nf = all & 255; nd = all >> 8 & 255; nb = all >> 16 & 255; ne = all >> 24;
            live = nf + nd + nb + ne;
            turn ^= 1;
        };
        for (;;) {
            recount();
            if (live == 0) break;
            if (ne > 0 && (8 * ne >= kOuterQuorum * live || nf == 0)) {
                int what = kFinished;
                bool write = false, skipped = false, capped = false;
                Outer o{};
                if (state == kLaneEnd) {
                    what = end_outer(o, capped);
                    write = what == kFinished;
                }
                // Finished pixels are written, and the lanes without a pixel
                // take the next queue entries together. (The queue's head passes
                // the total, which may be close to 2^31, by up to one a lane.)
                for (;;) {
                    if (write) { store(o, skipped, capped); write = false; capped = false; state = kLaneFetch; }
                    const unsigned want = __ballot_sync(full, state == kLaneFetch);
                    if (want == 0) break;
                    const int leader = __ffs(want) - 1;
                    int base = 0;
                    if (lane == leader) base = int(atomicAdd(a.queue, unsigned(__popc(want))));
                    base = __shfl_sync(full, base, leader);
                    if (state == kLaneFetch) {
                        const int job = base + __popc(want & ((1u << lane) - 1u));
                        if (uint32_t(job) >= uint32_t(total)) state = kLaneIdle;
                        else {
                            state = kLaneEnd;
                            what = kNextStart;
                            if (!load(o, job)) write = skipped = true;
                        }
                    }
                }
                if (state == kLaneEnd) {
                    if (what == kNextStart) begin_start(o);
                    begin_outer(o);
                }
                __syncwarp();
                recount();
            }
            if (nd > 0 && (8 * nd >= kDirectionQuorum * live || nf == 0)) {
                if (state == kLaneDir || state == kLaneSteep) direction();
                recount();
            }
            const bool gradients = nb > 0 && (8 * nb >= kGradientQuorum * live || nf == 0);
            if (state == kLaneTrial || state == kLaneOuter || (gradients && state == kLaneGrad)) {
                const bool mine = state == kLaneGrad;
                forward();
                pending = mine;
            }
            __syncwarp();
            if (gradients) {
                if (pending) backward();
                pending = false;
                __syncwarp();
            }
        }
        if (a.tally) {
            const uint32_t v = __reduce_add_sync(full, n_value), g = __reduce_add_sync(full, n_grad);
            if (lane == 0) {
                atomicAdd(a.tally + 0, (unsigned long long)v);
                atomicAdd(a.tally + 1, (unsigned long long)g);
            }
        }
    }
};

template <class T, int L, bool REFINE, bool BATCH>
__global__ void __launch_bounds__(kLaneBlock, lane_blocks_per_sm(L, sizeof(T) == 4))
solve_lanes(const __grid_constant__ Models<T> m, const __grid_constant__ SolverControls ctl,
            const __grid_constant__ SolveArgs a) {
    LaneSolver<T, L, REFINE, BATCH> solver(&m, ctl, a);
    solver.run();
}

}  // namespace unb
