// krylov_resident.cu -- Jacobi-PCG and BiCGStab as one cooperative kernel per chunk of
// iterations, for systems small enough that each SM keeps its rows' vectors in shared
// memory (the solver of krylov.cu otherwise, one launch per phase).
//
// One CTA per SM owns a contiguous range of nodes: x, r, z, p, q, D^-1 of its rows (and
// BiCGStab's further vectors) live in its shared memory for the whole launch.  The
// operand of the product is published in global memory (double-buffered) and gathered by
// the other CTAs after a grid barrier; the matrix streams from L2 / HBM.
//
// A reduction is a grid barrier with values: each CTA stores its partial sum, adds one to
// a counter (release), polls the counter (acquire) and one warp sums all partials in a
// fixed order, so every CTA forms the same scalars by itself: no last-block pass, no
// launch.  The partials alternate between two sets (a CTA is at most one exchange ahead of
// another).  Polls are bounded: a wait that runs out sets *err and every CTA leaves (the
// others' waits run out in turn).
//
// What bounds it: at a few thousand nodes the exchanges of an iteration (a barrier about
// 1.3 us and two reductions of about 2.2 us; an L2 round trip is 700 cycles and a dependent
// FP64 addition 75), above that the FP64 pipe (two DFMA per cycle and SM; 243 per node).
// Measured and slower: all CTAs polling one array of value-and-epoch slots, one inbox per
// CTA written by all the others, and a cluster level in front (1,150 cycles a cluster barrier).
// Microseconds per CG iteration, three launches an iteration -> this form: HEX8 24x12x12
// 25.0 -> 11.0, 40x20x20 30.9 -> 19.8, 64x32x32 84 -> 58, 80x40x40 132 -> 94; heat 200x200
// 25.4 -> 10.3 (and BiCGStab, 15.0 -> 5.2 ms a solve), 400x400 49 -> 15.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "mg_internal.h"

namespace mg {

namespace {

constexpr int kRThreads = 512;
constexpr int kRVec = 256;            // threads of the elementwise phases (FP64-pipe bound: more add no rate)
constexpr int kRMaxCtas = 160;        // five slots per polling lane
constexpr int kRSmemMax = 200 * 1024;

// A load of another CTA's data: from L2, and never moved across a barrier (the __ldcg
// intrinsic is an asm statement without a memory clobber, which the compiler may hoist).
__device__ __forceinline__ double load_gpu(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

struct Xch {
    double *parts;        // [2 sets][2 values][kRMaxCtas]
    unsigned *count;      // arrivals since the launch
    unsigned target;      // arrivals that complete the next exchange, less this one's
    int set;
    int *err;
};

// One warp per value: this CTA's total v (the same in every lane) -> the sum over the CTAs,
// the same bits in every CTA.  `warps` of every CTA take part in the exchange; SUM false: a
// barrier only.  False after the poll bound.
template <bool SUM>
__device__ __forceinline__ bool xch_warp(const Xch &X, int warps, double &v) {
    const int lane = threadIdx.x & 31, which = threadIdx.x >> 5, n = gridDim.x;
    double *part = X.parts + (X.set * 2 + which) * kRMaxCtas;
    bool ok = true;
    if (lane == 0) {
        if (SUM) asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(part + blockIdx.x), "d"(v) : "memory");
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(X.count) : "memory");
        const unsigned target = X.target + (unsigned)(n * warps);
        unsigned c;
        for (int tries = 0;; tries++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(X.count) : "memory");
            if ((int)(c - target) >= 0) break;
            if (tries >= (1 << 22)) {
                ok = false;
                *X.err = 1;
                break;
            }
        }
    }
    __syncwarp();  // orders the other lanes' reads after lane 0's acquire
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (SUM) {
        static_assert(kRMaxCtas == 160, "five partials per lane");
        double g[5];
#pragma unroll
        for (int j = 0; j < 5; j++) g[j] = lane + 32 * j < n ? load_gpu(part + lane + 32 * j) : 0.0;
        v = ((g[0] + g[1]) + (g[2] + g[3])) + g[4];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return ok;
}

// one warp: the CTA's total of the first `rows` x 32 partials in red, the same in every lane
__device__ __forceinline__ double cta_total(const double *red, int rows) {
    const int lane = threadIdx.x & 31;
    double a = red[lane], b = 0.0;
    for (int j = 1; j + 1 < rows; j += 2) {
        b += red[lane + 32 * j];
        a += red[lane + 32 * (j + 1)];
    }
    if (!(rows & 1)) b += red[lane + 32 * (rows - 1)];
    a += b;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// All-reduce of the NV block sums whose kRVec partials are in red: warp k does value k; the
// totals are in s_tot after the closing barrier.  Uniform result: false after a poll bound.
template <int NV>
__device__ __forceinline__ bool all_sum(Xch &X, const double (*red)[kRVec], int rows, double *s_tot, int *s_ok) {
    __syncthreads();
    if (threadIdx.x < 32 * NV) {
        const int k = threadIdx.x >> 5;
        double v = cta_total(red[k], rows);
        const bool ok = xch_warp<true>(X, NV, v);
        if ((threadIdx.x & 31) == 0) {
            s_tot[k] = v;
            s_ok[k] = ok;
        }
    }
    X.target += NV * gridDim.x;
    X.set ^= 1;
    __syncthreads();
    return s_ok[0] && (NV == 1 || s_ok[1]);
}

__device__ __forceinline__ bool bad(double x) { return !isfinite(x); }

struct ResidentArgs {
    const int32_t *rowptr, *cols;
    const double *vals, *dinv;
    int64_t n_nodes;
    int npc;                       // nodes per CTA
    double *x, *r, *z, *p;         // solver vectors between launches (BiCGStab: r, p, v, rh)
    double *rh, *v;
    double *pub0, *pub1;           // published operand, double-buffered
    KrylovState *st;
    double *parts;
    unsigned *count;
    int max_iters;
    int *err;
};

// Shape of the product per dofs per node: G lanes share a node, a lane holds B columns of
// all the node's rows at a time (NB such batches cover 81, 18 and 9 columns a row: the
// structured HEX8 and QUAD4 stencils; longer rows take further rounds).  RG, RB: the same
// for the register-resident form (every value of the CTA's rows in registers, at most one
// node per group).
template <int DPN> struct Shape;
template <> struct Shape<3> { static constexpr int G = 4, NB = 3, B = 7, RG = 8, RB = 11; };
template <> struct Shape<2> { static constexpr int G = 2, NB = 1, B = 9, RG = 2, RB = 9; };
template <> struct Shape<1> { static constexpr int G = 1, NB = 1, B = 9, RG = 1, RB = 9; };

// Sums the lanes' partial rows: each step of the butterfly also halves the rows a lane
// keeps (4 additions instead of 9 for three rows over eight lanes).  Returns the sum of
// row `row` (row >= DPN: none) in the lanes that write it.
template <int DPN, int G>
__device__ __forceinline__ double lane_rows(const double (&acc)[DPN], int sub, int &row) {
    if constexpr (G == 1) {
        static_assert(DPN == 1, "one row per lane");
        row = 0;
        return acc[0];
    } else if constexpr (G == 2) {
        static_assert(DPN == 2, "one row per lane");
        const bool odd = sub & 1;
        row = sub;
        return (odd ? acc[1] : acc[0]) + __shfl_xor_sync(0xffffffffu, odd ? acc[0] : acc[1], 1);
    } else {
        static_assert(DPN == 3 && (G == 4 || G == 8), "three rows over four or eight lanes");
        // upper half of the group: row 2; lower half: rows 0 and 1
        const bool hi = sub & (G / 2), mid = sub & (G / 4);
        const double g0 = __shfl_xor_sync(0xffffffffu, hi ? acc[0] : acc[2], G / 2);
        const double g1 = __shfl_xor_sync(0xffffffffu, hi ? acc[1] : 0.0, G / 2);
        const double m0 = (hi ? acc[2] : acc[0]) + g0;
        const double m1 = hi ? 0.0 : acc[1] + g1;
        double s = (mid ? m1 : m0) + __shfl_xor_sync(0xffffffffu, mid ? m0 : m1, G / 4);
        row = (hi ? 2 : 0) + (mid ? 1 : 0);
        if constexpr (G == 8) {
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (sub & 1) row = DPN;  // the even lane writes
        }
        return s;
    }
}

// y = A u over the CTA's rows, u gathered from the published operand, y in shared memory
template <int DPN>
__device__ __forceinline__ void stream_spmv(const ResidentArgs &A, int64_t node0, int nloc,
                                            const double *__restrict__ u, double *y) {
    using H = Shape<DPN>;
    constexpr int G = H::G, NPW = 32 / G;
    const int warp = threadIdx.x >> 5, gsub = (threadIdx.x & 31) / G, sub = threadIdx.x % G;
    for (int base = warp * NPW; base < nloc; base += (kRThreads / 32) * NPW) {  // warp-uniform
        const int loc = base + gsub;
        const bool valid = loc < nloc;
        const int64_t r0 = (node0 + (valid ? loc : 0)) * DPN;
        int32_t rp[DPN];
#pragma unroll
        for (int d = 0; d < DPN; d++) rp[d] = __ldg(A.rowptr + r0 + d);
        const int32_t len = valid ? __ldg(A.rowptr + r0 + 1) - rp[0] : 0;
        double acc[DPN];
#pragma unroll
        for (int d = 0; d < DPN; d++) acc[d] = 0.0;
        for (int32_t k0 = sub; k0 < len; k0 += H::NB * H::B * G) {
            int32_t c[H::NB * H::B];
#pragma unroll
            for (int j = 0; j < H::NB * H::B; j++) c[j] = k0 + j * G < len ? __ldg(A.cols + rp[0] + k0 + j * G) : -1;
#pragma unroll
            for (int b = 0; b < H::NB; b++) {
                double a[DPN][H::B], uc[H::B];
#pragma unroll
                for (int j = 0; j < H::B; j++)
#pragma unroll
                    for (int d = 0; d < DPN; d++)
                        a[d][j] = k0 + (b * H::B + j) * G < len ? __ldg(A.vals + rp[d] + k0 + (b * H::B + j) * G) : 0.0;
#pragma unroll
                for (int j = 0; j < H::B; j++) uc[j] = c[b * H::B + j] >= 0 ? load_gpu(u + c[b * H::B + j]) : 0.0;
#pragma unroll
                for (int j = 0; j < H::B; j++)
#pragma unroll
                    for (int d = 0; d < DPN; d++) acc[d] = fma(a[d][j], uc[j], acc[d]);
            }
        }
        int row;
        const double s = lane_rows<DPN, G>(acc, sub, row);
        if (valid && row < DPN) y[loc * DPN + row] = s;
    }
}

// the rows of one node per group of lanes, held in registers for the whole launch
template <int DPN>
struct RegisterRows {
    using H = Shape<DPN>;
    int32_t c[H::RB];
    double a[DPN][H::RB];
    int loc, sub;
    bool valid;
    __device__ __forceinline__ void load(const ResidentArgs &A, int64_t node0, int nloc) {
        loc = threadIdx.x / H::RG;
        sub = threadIdx.x % H::RG;
        valid = loc < nloc;
        const int64_t r0 = (node0 + (valid ? loc : 0)) * DPN;
        int32_t rp[DPN];
#pragma unroll
        for (int d = 0; d < DPN; d++) rp[d] = __ldg(A.rowptr + r0 + d);
        const int32_t len = valid ? __ldg(A.rowptr + r0 + 1) - rp[0] : 0;
#pragma unroll
        for (int j = 0; j < H::RB; j++) {
            const int32_t k = sub + j * H::RG;
            c[j] = k < len ? __ldg(A.cols + rp[0] + k) : (int32_t)r0;  // a zero value times the own dof
#pragma unroll
            for (int d = 0; d < DPN; d++) a[d][j] = k < len ? __ldg(A.vals + rp[d] + k) : 0.0;
        }
    }
    __device__ __forceinline__ void apply(int nloc, const double *__restrict__ u, double *y) const {
        // a warp without a node leaves the FP64 pipe to the others
        if ((int)(threadIdx.x & ~31u) / H::RG >= nloc) return;
        double uc[H::RB], acc[DPN], odd[DPN];  // two chains per row: a DFMA's latency is 75 cycles
#pragma unroll
        for (int j = 0; j < H::RB; j++) uc[j] = load_gpu(u + c[j]);
#pragma unroll
        for (int d = 0; d < DPN; d++) {
            acc[d] = a[d][0] * uc[0];
            odd[d] = a[d][1] * uc[1];
        }
#pragma unroll
        for (int j = 2; j < H::RB; j++)
#pragma unroll
            for (int d = 0; d < DPN; d++) {
                if (j & 1) odd[d] = fma(a[d][j], uc[j], odd[d]);
                else acc[d] = fma(a[d][j], uc[j], acc[d]);
            }
#pragma unroll
        for (int d = 0; d < DPN; d++) acc[d] += odd[d];
        int row;
        const double s = lane_rows<DPN, H::RG>(acc, sub, row);
        if (valid && row < DPN) y[loc * DPN + row] = s;
    }
};
template <>
struct RegisterRows<0> {  // the streaming form holds nothing
};

template <int DPN, bool REG, class R>
__device__ __forceinline__ void resident_spmv(const ResidentArgs &A, const R &rows, int64_t node0, int nloc,
                                              const double *__restrict__ u, double *y) {
    if constexpr (REG) rows.apply(nloc, u, y);
    else stream_spmv<DPN>(A, node0, nloc, u, y);
}

// grid barrier that publishes the operand written before it; uniform result
__device__ __forceinline__ bool publish_barrier(Xch &X, int *s_ok) {
    __syncthreads();
    if (threadIdx.x < 32) {
        double none = 0.0;
        const bool ok = xch_warp<false>(X, 1, none);
        if (threadIdx.x == 0) *s_ok = ok;
    }
    X.target += gridDim.x;
    __syncthreads();
    return *s_ok != 0;
}

template <int DPN, bool REG>
__global__ void __launch_bounds__(kRThreads, 1) cg_resident_kernel(const ResidentArgs A) {
    extern __shared__ double sv[];
    __shared__ double red[2][kRVec];
    __shared__ double s_tot[2], s_scal[2];
    __shared__ int s_ok[2], s_done;
    __shared__ KrylovState S;  // updated by thread 0, the same in every CTA
    const int tid = threadIdx.x;
    const int64_t node0 = (int64_t)blockIdx.x * A.npc;
    const int nloc = (int)min((int64_t)A.npc, A.n_nodes - node0), nd = nloc * DPN;
    const int64_t d0 = node0 * DPN;
    const int rrows = min(kRVec, (nd + 31) & ~31) / 32;  // warps of the elementwise phases with work
    const int cap = A.npc * DPN;
    double *x = sv, *r = x + cap, *z = r + cap, *p = z + cap, *q = p + cap, *di = q + cap;
    if (tid == 0) S = *A.st;
    __syncthreads();
    if (S.done) return;  // the same state in every CTA
    for (int i = tid; i < nd; i += kRThreads) {
        x[i] = A.x[d0 + i];
        r[i] = A.r[d0 + i];
        z[i] = A.z[d0 + i];
        p[i] = A.p[d0 + i];
        di[i] = A.dinv[d0 + i];
    }
    RegisterRows<REG ? DPN : 0> rows;
    if constexpr (REG) rows.load(A, node0, nloc);
    Xch X{A.parts, A.count, 0u, 0, A.err};
    __syncthreads();  // the vectors are loaded by other threads than use them
    double beta = S.beta, rz = S.rz;
    int iter = 0;
    bool ok = true;
    for (; iter < A.max_iters; iter++) {
        double *pub = iter & 1 ? A.pub1 : A.pub0;
        if (tid < kRVec)
            for (int i = tid; i < nd; i += kRVec) {
                const double pi = fma(beta, p[i], z[i]);
                p[i] = pi;
                __stcg(pub + d0 + i, pi);
            }
        if (!(ok = publish_barrier(X, s_ok))) break;
        resident_spmv<DPN, REG>(A, rows, node0, nloc, pub, q);
        __syncthreads();
        if (tid < kRVec) {
            double pq = 0.0;
            for (int i = tid; i < nd; i += kRVec) pq = fma(p[i], q[i], pq);
            red[0][tid] = pq;
        }
        if (!(ok = all_sum<1>(X, red, rrows, s_tot, s_ok))) break;
        if (tid == 0) {
            const double pq = s_tot[0];
            S.pq = pq;
            s_done = 0;
            if (bad(pq)) { S.status = MG_ENAN; s_done = 1; }
            else if (!(pq > 0.0)) { S.status = MG_EBREAKDOWN; s_done = 1; }
            else s_scal[0] = rz / pq;
        }
        __syncthreads();
        if (s_done) break;
        const double alpha = s_scal[0];
        if (tid < kRVec) {
            double a = 0.0, b = 0.0;
            for (int i = tid; i < nd; i += kRVec) {
                x[i] = fma(alpha, p[i], x[i]);
                const double ri = fma(-alpha, q[i], r[i]);
                r[i] = ri;
                const double zi = di[i] * ri;
                z[i] = zi;
                a = fma(ri, zi, a);
                b = fma(ri, ri, b);
            }
            red[0][tid] = a;
            red[1][tid] = b;
        }
        if (!(ok = all_sum<2>(X, red, rrows, s_tot, s_ok))) break;
        if (tid == 0) {
            const double nrz = s_tot[0], nrr = s_tot[1];
            S.iter += 1;
            S.rr = nrr;
            s_done = 0;
            if (bad(nrz) || bad(nrr)) {
                S.status = MG_ENAN;
                s_done = 1;
            } else {
                s_scal[0] = nrz / rz;
                s_scal[1] = nrz;
                if (nrr <= S.tol2) s_done = 1;
                else if (S.iter >= S.maxit) { S.status = MG_ENOCONV; s_done = 1; }
            }
        }
        __syncthreads();
        if (S.status == MG_ENAN) break;
        beta = s_scal[0];
        rz = s_scal[1];
        if (s_done) break;
    }
    for (int i = tid; i < nd; i += kRThreads) {
        A.x[d0 + i] = x[i];
        A.r[d0 + i] = r[i];
        A.z[d0 + i] = z[i];
        A.p[d0 + i] = p[i];
    }
    if (blockIdx.x == 0 && tid == 0 && ok) {
        S.done = (iter < A.max_iters) ? 1 : 0;
        S.beta = beta;
        S.rz = rz;
        *A.st = S;
    }
}

template <int DPN, bool REG>
__global__ void __launch_bounds__(kRThreads, 1) bicg_resident_kernel(const ResidentArgs A) {
    extern __shared__ double sv[];
    __shared__ double red[2][kRVec];
    __shared__ double s_tot[2], s_scal[2];
    __shared__ int s_ok[2], s_done;
    __shared__ KrylovState S;  // updated by thread 0, the same in every CTA
    const int tid = threadIdx.x;
    const int64_t node0 = (int64_t)blockIdx.x * A.npc;
    const int nloc = (int)min((int64_t)A.npc, A.n_nodes - node0), nd = nloc * DPN;
    const int64_t d0 = node0 * DPN;
    const int rrows = min(kRVec, (nd + 31) & ~31) / 32;  // warps of the elementwise phases with work
    const int cap = A.npc * DPN;
    double *x = sv, *r = x + cap, *p = r + cap, *v = p + cap, *s = v + cap, *t = s + cap, *y = t + cap,
           *z = y + cap, *rh = z + cap, *di = rh + cap;
    if (tid == 0) S = *A.st;
    __syncthreads();
    if (S.done) return;
    for (int i = tid; i < nd; i += kRThreads) {
        x[i] = A.x[d0 + i];
        r[i] = A.r[d0 + i];
        p[i] = A.p[d0 + i];
        v[i] = A.v[d0 + i];
        rh[i] = A.rh[d0 + i];
        di[i] = A.dinv[d0 + i];
    }
    RegisterRows<REG ? DPN : 0> rows;
    if constexpr (REG) rows.load(A, node0, nloc);
    Xch X{A.parts, A.count, 0u, 0, A.err};
    __syncthreads();  // the vectors are loaded by other threads than use them
    double alpha = S.alpha, beta = S.beta, omega = S.omega, rho = S.rho;
    int iter = 0;
    bool ok = true;
    for (; iter < A.max_iters; iter++) {
        // p = r + beta (p - omega v), y = D^-1 p
        if (tid < kRVec)
            for (int i = tid; i < nd; i += kRVec) {
                const double pi = fma(beta, fma(-omega, v[i], p[i]), r[i]);
                p[i] = pi;
                const double yi = di[i] * pi;
                y[i] = yi;
                __stcg(A.pub0 + d0 + i, yi);
            }
        if (!(ok = publish_barrier(X, s_ok))) break;
        resident_spmv<DPN, REG>(A, rows, node0, nloc, A.pub0, v);
        __syncthreads();
        if (tid < kRVec) {
            double a = 0.0;
            for (int i = tid; i < nd; i += kRVec) a = fma(rh[i], v[i], a);
            red[0][tid] = a;
        }
        if (!(ok = all_sum<1>(X, red, rrows, s_tot, s_ok))) break;
        if (tid == 0) {
            const double rv = s_tot[0];
            S.rv = rv;
            s_done = 0;
            if (bad(rv)) { S.status = MG_ENAN; s_done = 1; }
            else if (rv == 0.0) { S.status = MG_EBREAKDOWN; s_done = 1; }
            else s_scal[0] = rho / rv;
        }
        __syncthreads();
        if (s_done) break;
        alpha = s_scal[0];
        // s = r - alpha v, z = D^-1 s
        if (tid < kRVec)
            for (int i = tid; i < nd; i += kRVec) {
                const double si = fma(-alpha, v[i], r[i]);
                s[i] = si;
                const double zi = di[i] * si;
                z[i] = zi;
                __stcg(A.pub1 + d0 + i, zi);
            }
        if (!(ok = publish_barrier(X, s_ok))) break;
        resident_spmv<DPN, REG>(A, rows, node0, nloc, A.pub1, t);
        __syncthreads();
        if (tid < kRVec) {
            double a = 0.0, b = 0.0;
            for (int i = tid; i < nd; i += kRVec) {
                a = fma(t[i], s[i], a);
                b = fma(t[i], t[i], b);
            }
            red[0][tid] = a;
            red[1][tid] = b;
        }
        if (!(ok = all_sum<2>(X, red, rrows, s_tot, s_ok))) break;
        if (tid == 0) {
            S.ts = s_tot[0];
            S.tt = s_tot[1];
            s_done = 0;
            if (bad(S.ts) || bad(S.tt)) { S.status = MG_ENAN; s_done = 1; }
            else s_scal[0] = (S.tt > 0.0) ? S.ts / S.tt : 0.0;
        }
        __syncthreads();
        if (s_done) break;
        omega = s_scal[0];
        // x += alpha y + omega z, r = s - omega t
        if (tid < kRVec) {
            double a = 0.0, b = 0.0;
            for (int i = tid; i < nd; i += kRVec) {
                x[i] = fma(omega, z[i], fma(alpha, y[i], x[i]));
                const double ri = fma(-omega, t[i], s[i]);
                r[i] = ri;
                a = fma(rh[i], ri, a);
                b = fma(ri, ri, b);
            }
            red[0][tid] = a;
            red[1][tid] = b;
        }
        if (!(ok = all_sum<2>(X, red, rrows, s_tot, s_ok))) break;
        if (tid == 0) {
            const double nrho = s_tot[0], nrr = s_tot[1];
            S.iter += 1;
            S.rr = nrr;
            s_done = 1;
            if (bad(nrho) || bad(nrr)) S.status = MG_ENAN;
            else if (nrr <= S.tol2) {
            } else if (omega == 0.0 || nrho == 0.0) S.status = MG_EBREAKDOWN;
            else if (S.iter >= S.maxit) S.status = MG_ENOCONV;
            else {
                s_scal[0] = (nrho / rho) * (alpha / omega);
                s_scal[1] = nrho;
                s_done = 0;
            }
        }
        __syncthreads();
        if (s_done) break;
        beta = s_scal[0];
        rho = s_scal[1];
    }
    for (int i = tid; i < nd; i += kRThreads) {
        A.x[d0 + i] = x[i];
        A.r[d0 + i] = r[i];
        A.p[d0 + i] = p[i];
        A.v[d0 + i] = v[i];
    }
    if (blockIdx.x == 0 && tid == 0 && ok) {
        S.done = (iter < A.max_iters) ? 1 : 0;
        S.alpha = alpha;
        S.beta = beta;
        S.omega = omega;
        S.rho = rho;
        *A.st = S;
    }
}

using ResidentKernel = void (*)(const ResidentArgs);

template <int DPN>
ResidentKernel pick(bool cg, bool reg) {
    if (cg) return reg ? cg_resident_kernel<DPN, true> : cg_resident_kernel<DPN, false>;
    return reg ? bicg_resident_kernel<DPN, true> : bicg_resident_kernel<DPN, false>;
}

}  // namespace

size_t krylov_resident_bytes() { return sizeof(double) * (4 * kRMaxCtas + 1); }

// Runs up to max_iters iterations of the solve whose state krylov_solve has initialised;
// *launched = 0 when the system does not fit (the caller then uses the launch-per-phase form).
int krylov_resident_launch(mg_problem *p, const CsrMatrix &A, double *d_x, bool cg,
                           int max_iters, int *launched) {
    *launched = 0;
    KrylovWork &w = p->kw;
    const int64_t nodes = A.n / A.dpn;
    int sms = 0;
    MG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device));
    // nodes spread over every SM (the FP64 pipe binds), whole warps of them
    const int64_t spread = std::max(1, std::min(sms, kRMaxCtas));
    int64_t npc = (nodes + spread - 1) / spread;
    npc = (npc + 3) / 4 * 4;
    const int64_t smem = npc * A.dpn * 8 * (cg ? 6 : 10);
    if (smem > kRSmemMax) return MG_OK;
    // in registers where a CTA has at most one node per group of lanes and its rows fit
    const int lanes = A.dpn == 3 ? Shape<3>::RG : A.dpn == 2 ? Shape<2>::RG : Shape<1>::RG;
    const int cols = A.dpn == 3 ? Shape<3>::RG * Shape<3>::RB : A.dpn == 2 ? Shape<2>::RG * Shape<2>::RB : Shape<1>::RB;
    const bool reg = npc * lanes <= kRThreads && A.max_row <= cols;
    const unsigned grid = (unsigned)((nodes + npc - 1) / npc);
    ResidentKernel k = A.dpn == 3 ? pick<3>(cg, reg) : A.dpn == 2 ? pick<2>(cg, reg) : pick<1>(cg, reg);
    MG_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void *>(k), cudaFuncAttributeMaxDynamicSharedMemorySize, kRSmemMax));
    // slots: the partials, then the arrival counter (0 at every launch) and the error flag
    double *parts = static_cast<double *>(w.slots);
    unsigned *count = reinterpret_cast<unsigned *>(parts + 4 * kRMaxCtas);
    MG_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(unsigned), p->stream));
    ResidentArgs a{A.rowptr, A.cols, A.vals, w.dinv, nodes, (int)npc, d_x, w.r, w.z, w.p0, w.rh, w.v,
                   w.p1, w.t, w.state, parts, count, max_iters, w.slot_err};
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k), dim3(grid), dim3(kRThreads), args,
                                                      (size_t)smem, p->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();  // the device cannot hold the grid at once: the other form runs
        return MG_OK;
    }
    MG_CUDA_TRY(e);
    count_launches(1);
    *launched = 1;
    return MG_OK;
}

}  // namespace mg
