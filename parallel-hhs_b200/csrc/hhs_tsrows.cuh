// hhs_tsrows.cuh -- timesteps of a block of particles by one CTA, in either precision: the
// standalone timesteps call and the batched step's nodes (the device step's grid nodes have
// their own form, over pairs, in hhs_engine.cu).
#pragma once
#include "hhs_common.cuh"
#include "hhs_pairmath.cuh"

namespace hhs {

constexpr double kHuge = 1.e30;  // src/timestep.cuh:4

__device__ __forceinline__ int ts_list_at(const int32_t* list, int i) { return list ? list[i] : i; }

// A CTA takes T rows (particles) and passes over all n columns, 512 at a time, two a thread in
// registers, with the pair test of the device step's filtered timestep (hhs_engine.cu): a pair
// below a row's best rate so far is left out by 9 packed FP32 operations for two pairs, and the
// few that pass are listed and evaluated exactly, in either precision, some dozens at a time.
// Each row starts from its exact rates over the first 32 columns. The result is the maximum
// over all pairs, as if every one had been evaluated.
//
// The squares come from dot products, whose rounding grows with |x|^2 and |v|^2, so the test takes
// positions and velocities from a centre: the medians of some members, which neither a distant
// origin, a common velocity nor a few outlying members move away from the rest. (The subtraction
// is one FP64 rounding of the difference itself.) In FP32 from there on: rounded coordinates, their
// squares and the dot products err by less than 1.2e-6 of |x_i|^2 + |x_j|^2, which shrinking
// |x|^2 and growing |v|^2 by 4e-6 covers.
//
// The test here is for the row alone, with its rate T = 0.99 best: a pair may be left out if
//     A >= kappa B + C (p_i + p_j) and B >= D (p_i + p_j),  p = |m|^(2/3),
// A = |x_i - x_j|^2, B = |v_i - v_j|^2, C = (2 / (eta beta T)^2)^(2/3), D = (1 / (2 (1 - alpha)
// T C))^2: C (p_i + p_j) is at least the `a` and D (p_i + p_j) at least the `b` of the pair's
// mass sum there, since (m_i + m_j)^(2/3) <= p_i + p_j.
//
// Measured, one call: 2051 particles in FP64 1384 -> 23 us, 16384 mixed 1652 -> 261 us. What
// bounds it: the latency of a row's test (a chain of six packed operations, its shared-memory
// reads and a branch, hidden by eight warps per scheduler at most), and below about 4000
// particles that of a tile's loads and listed pairs.
constexpr int kTsThreads = 256;
constexpr int kTsCols = 2 * kTsThreads;  // columns of a tile
constexpr int kTsSeed = 32;              // columns that every row evaluates first
// No more columns than these are evaluated without a test, whose phases cost a small call more than
// its pairs: FP64 / mixed 7 particles 8.3 / 8.3 -> 5.2 / 4.2 us, 33 8.3 / 8.3 -> 6.2 / 4.4 (a thread a
// particle: 8.3 / 4.2, 24.6 / 6.2). At 64 the evaluation is still the shorter (6.2 / 5.0 against 9.3 / 8.3).
constexpr int kTsDirect = 64;
constexpr int kTsCap = 2048;             // pairs listed at a time
constexpr unsigned kTsBatch = 64;        // listed pairs that are worth evaluating together
constexpr int kTsMaxRows = 32;
constexpr int kTsDense = 7;
constexpr float kTsAlpha = 0.9f;
constexpr float kTsAll = 1.0e38f;

struct __align__(16) TsRowTest {  // -2 x, -2 v, -kappa, -C, -D, each in both lanes; pass: v <= c1 or w < c2
    float2 x, y, z, vx, vy, vz, nk, nC, nD;
    float c1, c2;
};

struct TsArgs {
    double eta, eta_s2;
    float inv_eta_s2, inv_eta;
};

struct TsState {
    double x, y, z, vx, vy, vz, m;
};

__device__ __forceinline__ TsState ts_load(const SoA& P, int g) {
    return TsState{P.x[g], P.y[g], P.z[g], P.vx[g], P.vy[g], P.vz[g], P.m[g]};
}

// the pair's rate as FP32 bits (mixed) or the complement of its timescale's bits (FP64): the
// largest key is the timestep; 0 for none
template <int PREC>
__device__ __forceinline__ unsigned long long ts_key(const TsState& a, const TsState& b,
                                                     const TsArgs& A) {
    if constexpr (PREC == HHS_PREC_FP64) {
        double t = kHuge;
        ts_pair_fp64(f64_sub(a.x, b.x), f64_sub(a.y, b.y), f64_sub(a.z, b.z), f64_sub(a.vx, b.vx),
                     f64_sub(a.vy, b.vy), f64_sub(a.vz, b.vz), a.m, b.m, A.eta, A.eta_s2, t);
        // (+ 0: a coincident pair of negative mass sum has a timescale of -0, the least there is)
        return t < kHuge ? ~(unsigned long long)__double_as_longlong(f64_add(t, 0.0)) : 0ull;
    } else {
        const DS ax = ds_split(a.x), ay = ds_split(a.y), az = ds_split(a.z);
        const DS bx = ds_split(b.x), by = ds_split(b.y), bz = ds_split(b.z);
        const float r = ts_pair_rate_mixed(
            ds_diff(ax.hi, ax.lo, bx.hi, bx.lo), ds_diff(ay.hi, ay.lo, by.hi, by.lo),
            ds_diff(az.hi, az.lo, bz.hi, bz.lo), (float)a.vx - (float)b.vx,
            (float)a.vy - (float)b.vy, (float)a.vz - (float)b.vz, (float)a.m + (float)b.m,
            A.inv_eta_s2, A.inv_eta);
        return r > 0.0f ? (unsigned long long)__float_as_uint(r) : 0ull;
    }
}
template <int PREC>
__device__ __forceinline__ double ts_of_key(unsigned long long key) {
    if (key == 0ull) return kHuge;
    if (PREC == HHS_PREC_FP64) return __longlong_as_double((long long)~key);
    const double t = 1.0 / (double)__uint_as_float((unsigned)key);
    return t < kHuge ? t : kHuge;
}

// 1.01 |m|^(2/3); the hardware's base-2 functions are within 2e-5 over the range of a float
__device__ __forceinline__ float ts_mass_term(double m) {
    return 1.01f * exp2f(0.66666667f * __log2f((float)fabs(m)));
}

template <int PREC>
__device__ __forceinline__ TsRowTest ts_row_test(const TsState& q, unsigned long long key,
                                                 const TsArgs& A) {
    TsRowTest r;
    const double rate = 1.0 / ts_of_key<PREC>(key), r2 = q.x * q.x + q.y * q.y + q.z * q.z,
                 v2 = q.vx * q.vx + q.vy * q.vy + q.vz * q.vz;
    const float T = 0.99f * (float)rate, eta = (float)A.eta;
    const float e = 1.0f / eta + 0.5f, beta = 1.0f - 0.75f * kTsAlpha / e;
    const float k = e / (kTsAlpha * T), f = eta * beta * T, c = cbrtf(2.01f / (f * f));
    const float kappa = 1.01f * k * k, C = 1.02f * c * c;
    const float h = 0.5f / ((1.0f - kTsAlpha) * T * C), D = 1.02f * h * h;
    const float p = ts_mass_term(q.m);
    const float W = (float)(r2 * (1.0 - 4e-6)), U = (float)(v2 * (1.0 + 4e-6));
    // without a usable rate (or for eta beyond the test's range) every pair passes
    const bool ok = A.eta <= 1.0 && rate > 1e-12 && rate < 1e12 && r2 < 1e24 && v2 < 1e24 &&
                    kappa < 1e24f && C * p < 1e24f && D * p < 1e24f;
    r.x = f2dup(ok ? -2.0f * (float)q.x : 0.0f);
    r.y = f2dup(ok ? -2.0f * (float)q.y : 0.0f);
    r.z = f2dup(ok ? -2.0f * (float)q.z : 0.0f);
    r.vx = f2dup(ok ? -2.0f * (float)q.vx : 0.0f);
    r.vy = f2dup(ok ? -2.0f * (float)q.vy : 0.0f);
    r.vz = f2dup(ok ? -2.0f * (float)q.vz : 0.0f);
    r.nk = f2dup(ok ? -kappa : 0.0f);
    r.nC = f2dup(ok ? -C : 0.0f);
    r.nD = f2dup(ok ? -D : 0.0f);
    const float a = C * p + 1e-30f;
    r.c1 = ok ? (a - W + kappa * U) + 2e-6f * (a + W + kappa * U) : 3e38f;
    r.c2 = ok ? D * p + 4e-5f * U + 1e-30f - U : 3e38f;
    return r;
}

// The centre: medians (upper ones) over 8 members spread over the n. ts_centre_sample is the calling
// lane's member (lane modulo 8) in component 0..5 = x, y, z, vx, vy, vz; ts_median the median of a
// warp's samples in all lanes, NaNs left out; 0 if they are half of them.
__device__ __forceinline__ double ts_centre_sample(const SoA& P, const int32_t* list, int n,
                                                   int component) {
    const double* a = component == 0 ? P.x : component == 1 ? P.y : component == 2 ? P.z
                      : component == 3 ? P.vx : component == 4 ? P.vy : P.vz;
    return a[ts_list_at(list, (int)((long long)(threadIdx.x & 7) * n >> 3))];
}
__device__ __forceinline__ double ts_median(double v) {
    const int q = threadIdx.x & 7;
    const float f = (float)v;  // ranked in FP32: a centre need not be exact
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float o = __shfl_sync(HHS_FULL_MASK, f, j);
        rank += o < f || (o == f && j < q) ? 1 : 0;
    }
    const unsigned mid = __ballot_sync(HHS_FULL_MASK, rank == 4 && f == f);
    const double c = __shfl_sync(HHS_FULL_MASK, v, mid ? __ffs(mid) - 1 : 0);
    return mid ? c : 0.0;
}
__device__ __forceinline__ TsState ts_from(const TsState& q, const double* centre) {
    return TsState{q.x - centre[0], q.y - centre[1], q.z - centre[2], q.vx - centre[3],
                   q.vy - centre[4], q.vz - centre[5], q.m};
}

// A row of the mixed rates: the negated particle, each value in both lanes when used.
struct TsSink {
    float nxh, nyh, nzh, nxl, nyl, nzl, nvx, nvy, nvz, m;
};
__device__ __forceinline__ TsSink ts_sink(const TsState& q) {
    const DS x = ds_split(q.x), y = ds_split(q.y), z = ds_split(q.z);
    return TsSink{-x.hi, -y.hi, -z.hi, -x.lo, -y.lo, -z.lo,
                  -(float)q.vx, -(float)q.vy, -(float)q.vz, (float)q.m};
}

struct TsRows {  // shared memory of ts_rows
    TsState row[kTsMaxRows];
    TsRowTest test[kTsMaxRows];
    unsigned long long best[kTsMaxRows];
    double centre[6];
    TsSink sink[kTsMaxRows];  // mixed
    int2 hit[kTsCap];  // (row, column)
    unsigned cnt;
};

// Every rate of the rows against the columns t0 .. t0 + kTsCols - 1 in mixed precision, two columns
// a thread, without a list.
__device__ __forceinline__ void ts_dense_tile(const SoA& P, const int32_t* list, int n, int i0,
                                              int nrow, int t0, const TsArgs& A, TsRows& sm) {
    const int j0 = t0 + 2 * (int)threadIdx.x;
    float2 xh, yh, zh, xl, yl, zl, vx, vy, vz, m;
    {
        // (past the end: the last particle again, left out below)
        const TsState a = ts_load(P, ts_list_at(list, min(j0, n - 1))),
                      b = ts_load(P, ts_list_at(list, min(j0 + 1, n - 1)));
        const DS ax = ds_split(a.x), ay = ds_split(a.y), az = ds_split(a.z);
        const DS bx = ds_split(b.x), by = ds_split(b.y), bz = ds_split(b.z);
        xh = make_float2(ax.hi, bx.hi); yh = make_float2(ay.hi, by.hi); zh = make_float2(az.hi, bz.hi);
        xl = make_float2(ax.lo, bx.lo); yl = make_float2(ay.lo, by.lo); zl = make_float2(az.lo, bz.lo);
        vx = make_float2((float)a.vx, (float)b.vx); vy = make_float2((float)a.vy, (float)b.vy);
        vz = make_float2((float)a.vz, (float)b.vz); m = make_float2((float)a.m, (float)b.m);
    }
    for (int r = 0; r < nrow; r++) {
        const TsSink q = sm.sink[r];
        const TsSink2 s{f2dup(q.nxh), f2dup(q.nyh), f2dup(q.nzh), f2dup(q.nxl), f2dup(q.nyl),
                        f2dup(q.nzl), f2dup(q.nvx), f2dup(q.nvy), f2dup(q.nvz), f2dup(q.m)};
        const float2 rate = ts_pair_rate_mixed2(xh, yh, zh, xl, yl, zl, vx, vy, vz, m, s,
                                                A.inv_eta_s2, A.inv_eta);
        const int i = i0 + r;
        const float best = fmaxf(fmaxf(j0 < n && j0 != i ? rate.x : 0.0f,
                                       j0 + 1 < n && j0 + 1 != i ? rate.y : 0.0f), 0.0f);
        const unsigned key = __reduce_max_sync(HHS_FULL_MASK, __float_as_uint(best));
        if ((threadIdx.x & 31) == 0 && key > *(volatile unsigned long long*)&sm.best[r])
            atomicMax(&sm.best[r], (unsigned long long)key);
    }
}

// The keys of rows i0 .. i0 + nrow - 1 (at most kTsMaxRows) of the n particles of `list` into
// sm.best. Called by all kTsThreads threads of the CTA; ends with a CTA barrier.
template <int PREC>
__device__ __forceinline__ void ts_rows(const SoA& P, const int32_t* list, int n, int i0, int nrow,
                                        const TsArgs& A, TsRows& sm) {
    const int tid = threadIdx.x;
    if (tid < nrow) {
        sm.row[tid] = ts_load(P, ts_list_at(list, i0 + tid));
        if (PREC == HHS_PREC_MIXED) sm.sink[tid] = ts_sink(sm.row[tid]);
    }
    if (tid < kTsMaxRows) sm.best[tid] = 0ull;
    if (tid == 0) sm.cnt = 0u;
    const int seed = n <= kTsDirect ? kTsDirect : kTsSeed;
    const double sample = n > kTsDirect && tid < 6 * 32 ? ts_centre_sample(P, list, n, tid >> 5) : 0.0;
    __syncthreads();
    for (int k = tid; k < nrow * seed; k += kTsThreads) {
        const int r = k / seed, j = k % seed;
        if (j < n && j != i0 + r) {
            const unsigned long long q = ts_key<PREC>(sm.row[r], ts_load(P, ts_list_at(list, j)), A);
            if (q > sm.best[r]) atomicMax(&sm.best[r], q);
        }
    }
    if (n <= kTsDirect) {
        __syncthreads();
        return;
    }
    __syncwarp();
    const double median = ts_median(sample);
    if (tid < 6 * 32 && (tid & 31) == 0) sm.centre[tid >> 5] = median;
    __syncthreads();
    if (tid < nrow) sm.test[tid] = ts_row_test<PREC>(ts_from(sm.row[tid], sm.centre), sm.best[tid], A);
    __syncthreads();
    unsigned held = 0u;
    int dense = 0;  // tiles to come that are not tested
    for (int t0 = 0; t0 < n; t0 += kTsCols) {
        if (PREC == HHS_PREC_MIXED && dense > 0) {
            dense--;
            ts_dense_tile(P, list, n, i0, nrow, t0, A, sm);
            continue;
        }
        const int j0 = t0 + 2 * tid;
        float2 X, Y, Z, VX, VY, VZ, W, U, p;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const TsState q = j0 + c < n
                                  ? ts_from(ts_load(P, ts_list_at(list, j0 + c)), sm.centre)
                                  : TsState{0, 0, 0, 0, 0, 0, 0};
            const float x = (float)q.x, y = (float)q.y, z = (float)q.z;
            const float vx = (float)q.vx, vy = (float)q.vy, vz = (float)q.vz;
            const float r2 = x * x + y * y + z * z, v2 = vx * vx + vy * vy + vz * vz;
            const float pc = ts_mass_term(q.m);
            const bool ok = r2 < 1e24f && v2 < 1e24f && pc < 1e20f;  // else it passes every test
            auto put = [&](float2& v, float f) {
                if (c) v.y = f;
                else v.x = f;
            };
            put(X, ok ? x : 0.0f);
            put(Y, ok ? y : 0.0f);
            put(Z, ok ? z : 0.0f);
            put(VX, ok ? vx : 0.0f);
            put(VY, ok ? vy : 0.0f);
            put(VZ, ok ? vz : 0.0f);
            put(p, ok ? pc : 0.0f);
            put(W, ok ? r2 * (1.0f - 4e-6f) : -kTsAll);
            put(U, ok ? v2 * (1.0f + 4e-6f) : 0.0f);
        }
        for (int r = 0; r < nrow; r++) {
            __syncwarp();  // lanes that listed pairs rejoin the others here
            const TsRowTest t = sm.test[r];
            float2 w = __ffma2_rn(t.vx, VX, U), v = __ffma2_rn(t.x, X, W);
            w = __ffma2_rn(t.vy, VY, w);
            v = __ffma2_rn(t.y, Y, v);
            w = __ffma2_rn(t.vz, VZ, w);
            v = __ffma2_rn(t.z, Z, v);
            v = __ffma2_rn(t.nk, w, v);
            v = __ffma2_rn(t.nC, p, v);
            w = __ffma2_rn(t.nD, p, w);
            if (fminf(v.x, v.y) <= t.c1 || fminf(w.x, w.y) < t.c2) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const float vc = c ? v.y : v.x, wc = c ? w.y : w.x;
                    if ((vc <= t.c1 || wc < t.c2) && j0 + c < n && j0 + c != i0 + r) {
                        const unsigned k = atomicAdd(&sm.cnt, 1u);
                        if (k < kTsCap) sm.hit[k] = make_int2(r, j0 + c);
                    }
                }
            }
        }
        __syncthreads();
        const unsigned cnt = sm.cnt;
        __syncthreads();  // every thread has the count
        if (cnt < kTsBatch && t0 + kTsCols < n) {
            held = cnt;
            continue;
        }
        // the listed pairs; if the list overflowed, those of earlier tiles and every pair of
        // this one, in mixed precision also of the next kTsDense tiles without a test. (A listed
        // pair takes as long as five in dense tiles: 16384 mixed, all pairs pass, 3104 us with lists, 755)
        const bool all = cnt > kTsCap;
        const int listed = (int)(all ? held : cnt),
                  total = listed + (all && PREC == HHS_PREC_FP64 ? nrow * kTsCols : 0);
        if (PREC == HHS_PREC_MIXED && all) {
            ts_dense_tile(P, list, n, i0, nrow, t0, A, sm);
            dense = kTsDense;
        }
        for (int k = tid; k < total; k += kTsThreads) {
            const int2 h = k < listed ? sm.hit[k]
                                      : make_int2((k - listed) / kTsCols, t0 + (k - listed) % kTsCols);
            if (h.y >= n || h.y == i0 + h.x) continue;
            const unsigned long long key =
                ts_key<PREC>(sm.row[h.x], ts_load(P, ts_list_at(list, h.y)), A);
            if (key > *(volatile unsigned long long*)&sm.best[h.x]) atomicMax(&sm.best[h.x], key);
        }
        __syncthreads();
        if (tid == 0) sm.cnt = 0u;
        if (tid < nrow) sm.test[tid] = ts_row_test<PREC>(ts_from(sm.row[tid], sm.centre), sm.best[tid], A);
        __syncthreads();
        held = 0u;
    }
    if (PREC == HHS_PREC_MIXED) __syncthreads();  // the last tile may have been a dense one
}

}  // namespace hhs
