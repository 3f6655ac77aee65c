// matfree.cu -- mixed-precision matrix-free SIMP operator on the 5th-generation
// tensor cores, FP32 inner CG and FP64 iterative refinement.
//
// Operator: y = sum_e E_e P_e^T K0 P_e u on a structured HEX8 grid (every
// element shares the reference stiffness K0 of StructuralElement3D,
// src/elasticity/solid_element_3d.cpp:135-423, scaled by the SIMP modulus of
// examples/structural/example_6/example_6.cpp:100-137).  Dirichlet dofs are
// eliminated (identity rows, zero columns) as in the plain form; they are
// marked by a zero Jacobi inverse, which keeps r, z and p zero there.
//
// The CG operator runs on the tensor cores by columns of nodes (mf_col_kernel), the
// multigrid levels on the CUDA cores with the factored element stiffness
// (mf_fac_kernel), the small levels of a chain on one thread-block cluster, and the
// FP64 residual in double-float arithmetic (mf_residual64_kernel).  Every owned dof
// adds its elements' contributions in a fixed order: no atomics, no colouring, one
// global write per dof; tiles evaluate the elements of their one-element halo anew.
//
// Reductions are per problem and deterministic: every tile (chunk) writes a
// partial and the last tile (chunk) of a problem -- found with a per-problem
// counter -- sums that problem's partials in index order.  A problem's result
// is therefore bitwise independent of which other problems share the batch.
#include <cstdlib>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>
#include <utility>

#include "matfree.cuh"

namespace mg {

namespace {

constexpr int kThreads = 256;

template <int P>
struct Prec {
    static constexpr bool kTf32 = (P == MG_MIXED_TF32 || P == MG_MIXED_TF32X3);
    static constexpr bool kSplit = (P == MG_MIXED_TF32X3 || P == MG_MIXED_BF16X3);
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// UMMA shared-memory descriptor, no swizzle, K-major canonical layout:
// 8-row x 16-byte core matrices; LBO = byte step between core matrices along K,
// SBO = byte step between 8-row groups; version field = 1 (sm_100 family).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;  // base offset 0, LBO mode 0, layout type 0 (SWIZZLE_NONE)
}

// instruction descriptor: D F32, A/B K-major, N columns, M = 128
template <bool TF32, int N>
__host__ __device__ constexpr uint32_t umma_idesc() {
    return (1u << 4) |                   // D format F32
           ((TF32 ? 2u : 1u) << 7) |     // A: TF32 (kind::tf32) / BF16 (kind::f16)
           ((TF32 ? 2u : 1u) << 10) |    // B
           (((uint32_t)N >> 3) << 17) |  // N >> 3
           ((128u >> 4) << 24);          // M >> 4
}

template <bool TF32, int N>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                     uint32_t accumulate) {
    if (TF32) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(umma_idesc<TF32, N>()), "r"(accumulate));
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(umma_idesc<TF32, N>()), "r"(accumulate));
    }
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Programmatic dependent launch: let the next kernel of the stream be scheduled
// now, then wait until the previous kernel has finished and its writes are
// visible (a no-op without a programmatic dependency).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_trigger();
    pdl_wait();
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(mbar), "r"(phase)
        : "memory");
    return ok != 0;
}

// bounded wait: false after the iteration cap (the caller records the error)
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t phase) {
    for (int i = 0; i < (1 << 22); i++)
        if (mbar_try_wait(mbar, phase)) return true;
    return false;
}

// 3D TMA tile load global -> shared, completion on an mbarrier
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            int z, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(mbar)
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}

// libMesh HEX8 local node a -> corner bits
__host__ __device__ __forceinline__ void corner_bits(int a, int &dx, int &dy, int &dz) {
    dx = ((a + 1) >> 1) & 1;
    dy = (a >> 1) & 1;
    dz = (a >> 2) & 1;
}
__host__ __device__ __forceinline__ int corner_index(int dx, int dy, int dz) {
    return dz * 4 + (dy ? (dx ? 2 : 3) : (dx ? 1 : 0));
}

__device__ __forceinline__ int64_t dof_index(const MfProblem &P, int gx, int gy, int gz, int c) {
    return P.dof_off + ((int64_t)gz * P.NY + gy) * P.pitch + 3 * gx + c;
}

// --------------------------------------------------------------- block helpers
// The vector kernels end on FP64 sums that one thread or warp forms alone, and a dependent
// FP64 addition takes about 75 cycles: the sums are trees of the least depth.
static_assert(kThreads == 256, "sum_warps adds eight warps' sums");
__device__ __forceinline__ double sum_warps(const double *sh) {
    return ((sh[0] + sh[1]) + (sh[2] + sh[3])) + ((sh[4] + sh[5]) + (sh[6] + sh[7]));
}

__device__ __forceinline__ double block_sum(double v, double *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    return threadIdx.x == 0 ? sum_warps(sh) : 0.0;  // valid in thread 0
}

// FP32 warp sums, FP64 across the block's warps; valid in thread 0
__device__ __forceinline__ double block_sum_f(float v, double *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[w] = (double)v;
    __syncthreads();
    return threadIdx.x == 0 ? sum_warps(sh) : 0.0;
}

// fixed-order sum of part[begin .. begin+count) over the block; valid in thread 0
__device__ __forceinline__ double ordered_sum(const double *part, int begin, int count) {
    __shared__ double tree[kThreads];
    double s = 0.0;
    for (int i = threadIdx.x; i < count; i += kThreads) s += __ldcg(part + begin + i);
    if (count > 32) {
        __syncthreads();
        tree[threadIdx.x] = s;
        __syncthreads();
        for (int w = kThreads / 2; w > 32; w >>= 1) {
            if (threadIdx.x < w) tree[threadIdx.x] += tree[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x < 32) s = tree[threadIdx.x] + tree[threadIdx.x + 32];
    }
    if (threadIdx.x < 32) {
        int w = 16;
        while (w >= count && w > 0) w >>= 1;  // the lanes from count on hold zeros
        for (; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
    }
    return s;
}

__device__ __forceinline__ bool is_bad(double x) { return !isfinite(x); }

// ----------------------------------------------------------- column operator
// y = sum_e E_e P_e^T K0 P_e x by columns of owned nodes (kCX x kCY nodes in x,
// y; up to kCZ node planes in z), streamed plane by plane.  The A operand of
// the tensor-core MMA is never assembled: the halo nodes of each plane are
// converted once into 16-byte node records (x, y, z, 0 in TF32; x, y, z and five
// zeros in BF16), and the MMA reads them in place.  An element plane holds 8 x 16
// elements, one M = 128 tile: row r = ey * 8 + ex; the eight rows of a core
// matrix are eight x-consecutive elements (nodes 16 bytes apart), the 16 row
// groups are the 16 element rows (stride of a node row).  One MMA per corner
// pair (dx = 0, 1 at fixed dy, dz) uses K chunks 16 bytes apart (the node and
// its x-neighbour), so the element operator is 4 MMAs per product (3 products
// in the split forms) against four B tiles cut from K0.
//
// The cost of one tcgen05.mma (M = 128, K = 8 TF32) grows little with N up to
// 64 (46, 48, 64, 128 cycles for N = 32, 64, 128, 256, measured on the GB300), so
// the split forms issue the hi records against [K0_hi | K0_lo] as one N = 64 MMA
// and the lo records against K0_hi as an N = 32 MMA: 8 MMAs per element plane
// instead of 12.  The accumulator holds hi.K_hi + lo.K_hi in columns 0-31 and
// hi.K_lo in columns 32-63; the drain adds the two.
//
// Warp roles (no CTA-wide barrier inside the plane stream; every hand-off is an
// mbarrier with a bounded wait), two CTAs of 12 warps per SM:
//   warp 0      one thread issues the TMA loads of each node plane (z and, in the
//               CG step, p_old; the moduli of the element plane) into a ring;
//   warp 1      one thread issues the MMAs of element plane s once node planes s
//               and s+1 are converted, into one of four TMEM accumulators;
//   warps 2-7   convert a node plane into the operand records (hi and lo parts)
//               and an FP32 copy u of the owned nodes (with p = z + beta p_old
//               fused), plus the plane's moduli, into rings;
//   warps 8-11  drain: thread = element (TMEM lane), reads its 24 results, scales
//               by E_e, sums the corner results into nodes (x: warp shuffle, y:
//               shuffle and, at the warp's first row, the previous warp's last row
//               through shared memory; z: the top corners of plane s-1 carried in
//               registers) and writes node plane s of y (and p_new) -- every node
//               sum in a fixed order, deterministic and atomic-free.
// The column sequence is chosen by the TMA thread alone and travels with the data
// (a record per ring slot), ending with a sentinel plane.
constexpr int kColThreads = 384;
constexpr int kColCtas = 2;                   // CTAs per SM
constexpr int kCConvWarps = 6;                // warps 2-7
constexpr int kCDrain0 = 2 + kCConvWarps;     // first drain warp (8: TMEM lane quarter = warp % 4)
constexpr int kCPX = kCX + 2;                 // 9 nodes per plane row
constexpr int kCPY = kCY + 2;                 // 17 node rows per plane
constexpr int kCPN = kCPX * kCPY;             // 153 nodes per plane
constexpr int kCPB = kCPN * 16;               // 2448 bytes per converted plane (one part)
constexpr int kCRawX = 32;                    // TMA node box: 32 floats x 17 rows x 1 plane
constexpr int kCRawNode = kCRawX * kCPY * 4;  // 2176
constexpr int kCRawE = 12 * 16 * 4;           // E box: 12 elements x 16 rows x 1 plane = 768
constexpr int kCRawSlot = 2 * kCRawNode + kCRawE;  // 5120 (z, p_old, E)
constexpr int kCNR = 4;                       // TMA ring slots
constexpr int kCNC = 6;                       // operand-record ring slots (hi | lo)
constexpr int kCNU = 8;                       // u / E ring slots (the drain's inputs)
constexpr int kCNT = 4;                       // TMEM accumulators (64 columns each)
constexpr int kCTCols = 64;                   // TMEM columns per accumulator
constexpr int kCOwn = kCX * kCY;              // 105 owned nodes per plane
constexpr int kCUSlot = kCOwn * 16 + 128 * 4; // u of the owned nodes as (x, y, z, -) + 128 moduli = 2192
constexpr int kCConvFloats = kCPN * 3;        // 459 values per node plane
constexpr int kCConvThreads = 32 * kCConvWarps;
constexpr int kCConvRounds = (kCConvFloats + kCConvThreads - 1) / kCConvThreads;  // 3
constexpr int kCXch = 4 * 8 * 8;              // exchange slot: 4 warps x 8 lanes x (6 + 2 pad) floats

constexpr int kC_OffB = 0;                                          // 4 B tiles x 2 KB: [K_hi | K_lo]
constexpr int kC_OffConv = 8192;                                    // kCNC x (hi, lo) records
constexpr int kC_OffRaw = (kC_OffConv + kCNC * 2 * kCPB + 127) / 128 * 128;  // TMA ring
constexpr int kC_OffU = kC_OffRaw + kCNR * kCRawSlot;               // u / E ring
constexpr int kC_OffX = kC_OffU + kCNU * kCUSlot;                   // y-exchange, 2 slots
constexpr int kC_OffMeta = kC_OffX + 2 * kCXch * 4;                 // plane records (int4)
constexpr int kC_OffRed = kC_OffMeta + (kCNR + kCNC + kCNU) * 16;   // column partials [2][4]
constexpr int kC_OffBar = kC_OffRed + 64;                           // mbarriers
// barriers: raw full/empty, conv full/empty, u full/empty, tmem full/empty, xch[2], red[2], fin
constexpr int kCBarRawFull = 0, kCBarRawEmpty = kCBarRawFull + kCNR, kCBarConvFull = kCBarRawEmpty + kCNR,
              kCBarConvEmpty = kCBarConvFull + kCNC, kCBarUFull = kCBarConvEmpty + kCNC,
              kCBarUEmpty = kCBarUFull + kCNU, kCBarTFull = kCBarUEmpty + kCNU, kCBarTEmpty = kCBarTFull + kCNT,
              kCBarXch = kCBarTEmpty + kCNT, kCBarRed = kCBarXch + 2, kCBarFin = kCBarRed + 2,
              kCBarCount = kCBarFin + 1;
constexpr int kC_OffFlags = kC_OffBar + kCBarCount * 8;             // tmem slot, abort flag
constexpr int kColSmem = kC_OffFlags + 16;
static_assert(kC_OffRaw % 128 == 0 && kCRawSlot % 128 == 0 && kCRawNode % 128 == 0, "TMA destinations");
static_assert(kC_OffConv % 16 == 0 && kCPB % 16 == 0 && kC_OffU % 16 == 0 && kCUSlot % 16 == 0, "alignment");
static_assert(kC_OffMeta % 16 == 0 && kC_OffBar % 8 == 0, "alignment");
static_assert(kColCtas * (kColSmem + 1024) <= 228 * 1024, "CTAs per SM");
static_assert(kCNT * kCTCols * kColCtas <= 512, "TMEM columns of the CTAs on an SM");
static_assert(kColThreads == 32 * (kCDrain0 + 4), "warp roles");

// bounded mbarrier wait that also gives up when another role has set the CTA's
// abort flag; a wait that runs out of polls sets the flag
__device__ __forceinline__ bool col_wait(uint32_t mbar, uint32_t phase, volatile int *abort_flag) {
    for (int i = 0; i < (1 << 22); i++) {
        if (mbar_try_wait(mbar, phase)) return true;
        if ((i & 63) == 63 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}

// columns [taddr, taddr + 24) of the warp's 32 TMEM lanes, one wait for both loads
__device__ __forceinline__ void tmem_ld24(uint32_t taddr, float (&v)[24]) {
    uint32_t r[24];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23])
        : "r"(taddr + 16));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 24; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// This CTA's columns are order[offs[blockIdx.x]] ...; the input vector is tensor map `in_slot`.
// MODE 1: CG step, gathered u = z + beta p_old (z = in_slot, p_old = map 1 +
//         parity), p_new (owned) = u, q = A u, per-problem alpha = rz / (p.q).
// MODE 2: y = rhs - A x.   MODE 3: y = A x.   (Both 0 on Dirichlet dofs.)
// A wait that times out sets bit 1 (tensor-core hand-offs) or bit 2 (data
// hand-offs) of *err and ends the block after its copies and MMAs have landed.
template <int PREC, int MODE>
__global__ void __launch_bounds__(kColThreads, kColCtas) mf_col_kernel(
    const MfProblem *__restrict__ probs, const MfCol *__restrict__ cols, const int *__restrict__ order,
    const int *__restrict__ offs, int sel,
    const CUtensorMap *__restrict__ tmaps, int in_slot, int parity, const uint32_t *__restrict__ Bop2,
    const float *__restrict__ dinv, const float *__restrict__ rhs, float *__restrict__ p0,
    float *__restrict__ p1, float *__restrict__ y, MfState *states, double *__restrict__ col_part,
    int *err) {
    // the prologue (barriers, TMEM, the constant B tiles, the zeroed records) overlaps
    // the previous kernel; everything after pdl_wait may read its results
    pdl_trigger();
    using PR = Prec<PREC>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int4 *meta_raw = reinterpret_cast<int4 *>(smem + kC_OffMeta);
    int4 *meta_conv = meta_raw + kCNR;
    int4 *meta_u = meta_conv + kCNC;
    double *red = reinterpret_cast<double *>(smem + kC_OffRed);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + kC_OffFlags);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kC_OffFlags + 4);
    const uint32_t bar0 = smem_u32(smem + kC_OffBar);
    auto bar = [&](int i) -> uint32_t { return bar0 + 8u * (uint32_t)i; };
    float *p_new = (MODE == 1) ? (parity ? p0 : p1) : nullptr;

    if (tid == 0) {
        for (int k = 0; k < kCNR; k++) {
            mbar_init(bar(kCBarRawFull + k), 1);
            mbar_init(bar(kCBarRawEmpty + k), kCConvWarps);
        }
        for (int k = 0; k < kCNC; k++) {
            mbar_init(bar(kCBarConvFull + k), kCConvWarps);
            mbar_init(bar(kCBarConvEmpty + k), 1);  // an MMA commit
        }
        for (int k = 0; k < kCNU; k++) {
            mbar_init(bar(kCBarUFull + k), kCConvWarps);
            mbar_init(bar(kCBarUEmpty + k), 4);     // the four drain warps
        }
        for (int k = 0; k < kCNT; k++) {
            mbar_init(bar(kCBarTFull + k), 1);
            mbar_init(bar(kCBarTEmpty + k), 4);
        }
        for (int k = 0; k < 2; k++) {
            mbar_init(bar(kCBarXch + k), 4);
            mbar_init(bar(kCBarRed + k), 4);
        }
        mbar_init(bar(kCBarFin), 1);
        *abort_flag = 0;
    }
    if (warp == 1) tmem_alloc(smem_u32(tslot), kCNT * kCTCols);
    {
        // B tiles in global memory: [tf32 hi 1024 | tf32 lo 1024 | bf16 hi 1024 | bf16 lo 1024]
        // words, tile t at 256 t in each part; in shared memory tile t at 512 t words as
        // [hi 256 | lo 256]: N = 64 rows, the lo rows one SBO step after the hi rows
        const uint32_t *src = Bop2 + (PR::kTf32 ? 0 : 2048);
        uint32_t *dst = reinterpret_cast<uint32_t *>(smem + kC_OffB);
        for (int i = tid; i < 2048; i += kColThreads) {
            const int part = i >> 10, t = (i >> 8) & 3, w = i & 255;
            dst[t * 512 + part * 256 + w] = src[i];
        }
        // node records: the unused lanes stay 0 (B has zero rows there; 0 x NaN is NaN)
        uint32_t *conv = reinterpret_cast<uint32_t *>(smem + kC_OffConv);
        for (int i = tid; i < kCNC * 2 * kCPB / 4; i += kColThreads) conv[i] = 0u;
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    // the work lists and the column and problem tables are constant: read the first before the wait
    const int at0 = offs[blockIdx.x], at_end = offs[blockIdx.x + 1], ci0 = at0 < at_end ? order[at0] : -1;
    if (tid == 0 && ci0 >= 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(probs + cols[ci0].prob));
    pdl_wait();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            uint32_t k = 0;
            int last_issue[kCNR] = {-1, -1, -1, -1};
            auto usable = [&](int ci) {
                const MfProblem &Q = probs[cols[ci].prob];
                return !states[Q.root].done && !Q.bottom && (sel < 0 || sel == (Q.coarse < 0 ? 1 : 0));
            };
            bool ok = true;
            for (int at = at0; at < at_end && ok; at++) {
                const int ci = at == at0 ? ci0 : order[at];
                if (!usable(ci)) continue;
                const MfCol cl = cols[ci];
                const MfProblem &P = probs[cl.prob];
                const int x0 = cl.cx * kCX, y0 = cl.cy * kCY, z0 = cl.cz * P.col_z;
                const int z1 = min(z0 + P.col_z, P.NZ);
                const int S = z1 - z0 + 1;                      // element planes z0-1 .. z1-1
                const int xs = (3 * (x0 - 1)) & ~3, xe = (x0 - 1) & ~3;  // 16-byte aligned box starts
                const CUtensorMap *maps = tmaps + (size_t)cl.prob * kMapsPerProblem;
                for (int p = 0; p <= S; p++, k++) {
                    const int slot = (int)(k % kCNR);
                    if (!col_wait(bar(kCBarRawEmpty + slot), ((k / kCNR) & 1u) ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    meta_raw[slot] = make_int4(ci, p, S, 0);
                    uint8_t *raw = smem + kC_OffRaw + slot * kCRawSlot;
                    const uint32_t bytes = (MODE == 1 ? 2 : 1) * kCRawNode + (p < S ? kCRawE : 0);
                    mbar_expect_tx(bar(kCBarRawFull + slot), bytes);
                    tma_load_3d(smem_u32(raw), maps + in_slot, xs, y0 - 1, z0 - 1 + p, bar(kCBarRawFull + slot));
                    if (MODE == 1)
                        tma_load_3d(smem_u32(raw + kCRawNode), maps + 1 + parity, xs, y0 - 1, z0 - 1 + p,
                                    bar(kCBarRawFull + slot));
                    if (p < S)
                        tma_load_3d(smem_u32(raw + 2 * kCRawNode), maps + 3, xe, y0 - 1, z0 - 1 + p,
                                    bar(kCBarRawFull + slot));
                    last_issue[slot] = (int)k;
                }
            }
            if (ok) {
                // sentinel: no data, the stream ends
                const int slot = (int)(k % kCNR);
                if (col_wait(bar(kCBarRawEmpty + slot), ((k / kCNR) & 1u) ^ 1u, abort_flag)) {
                    meta_raw[slot] = make_int4(-1, 0, 0, 0);
                    mbar_arrive(bar(kCBarRawFull + slot));
                }
            }
            if (*abort_flag) {
                atomicOr(err, 2);
                // let the copies in flight land before the block exits
                for (int s = 0; s < kCNR; s++)
                    if (last_issue[s] >= 0) {
                        const uint32_t ph = ((uint32_t)last_issue[s] / kCNR) & 1u;
                        for (int i = 0; i < (1 << 22) && !mbar_try_wait(bar(kCBarRawFull + s), ph); i++) {
                        }
                    }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            const uint32_t b_base = smem_u32(smem + kC_OffB), conv_base = smem_u32(smem + kC_OffConv);
            uint32_t es = 0;
            for (uint32_t k = 0;; k++) {
                const int cs = (int)(k % kCNC);
                if (!col_wait(bar(kCBarConvFull + cs), (k / kCNC) & 1u, abort_flag)) break;
                const int4 m = meta_conv[cs];
                if (m.x < 0) break;
                if (m.y >= 1) {
                    // element plane m.y - 1 from node planes k - 1 (dz = 0) and k (dz = 1)
                    const int ts = (int)(es % kCNT);
                    if (!col_wait(bar(kCBarTEmpty + ts), ((es / kCNT) & 1u) ^ 1u, abort_flag)) break;
                    fence_after();
                    const uint32_t d = tmem + (uint32_t)ts * kCTCols;
                    const int cprev = (int)((k - 1) % kCNC);
#pragma unroll
                    for (int st4 = 0; st4 < 4; st4++) {
                        const int dy = st4 & 1, dz = st4 >> 1;
                        const uint32_t a = conv_base + (dz ? cs : cprev) * 2 * kCPB + dy * kCPX * 16;
                        const uint64_t bd = umma_desc(b_base + st4 * 2048, 128, 256);
                        if (PR::kSplit) {
                            // hi records against [K_hi | K_lo] (columns 0-63), lo records
                            // against K_hi (columns 0-31)
                            umma<PR::kTf32, 64>(d, umma_desc(a, 16, kCPX * 16), bd, st4 ? 1u : 0u);
                            umma<PR::kTf32, 32>(d, umma_desc(a + kCPB, 16, kCPX * 16), bd, 1u);
                        } else {
                            umma<PR::kTf32, 32>(d, umma_desc(a, 16, kCPX * 16), bd, st4 ? 1u : 0u);
                        }
                    }
                    umma_commit(bar(kCBarTFull + ts));
                    umma_commit(bar(kCBarConvEmpty + cprev));             // node plane k - 1 is done
                    if (m.y == m.z) umma_commit(bar(kCBarConvEmpty + cs)); // the column's last node plane
                    es++;
                }
            }
            // every MMA issued has completed before the accumulators are freed
            umma_commit(bar(kCBarFin));
            for (int i = 0; i < (1 << 22) && !mbar_try_wait(bar(kCBarFin), 0u); i++) {
            }
            if (*abort_flag) atomicOr(err, 1);
        }
    } else if (warp < kCDrain0) {
        // ------------------------------------------------------------ converters
        const int ct = tid - 64;
        // per round: raw-box float index (ox added), record word, word of u (owned nodes)
        int src[kCConvRounds], dst[kCConvRounds], udst[kCConvRounds];
#pragma unroll
        for (int j = 0; j < kCConvRounds; j++) {
            const int i = ct + kCConvThreads * j;
            const int row = i / 27, kk = i - 27 * row, nx = kk / 3;
            src[j] = (i < kCConvFloats) ? row * kCRawX + kk : -1;
            dst[j] = (row * kCPX + nx) * 4 + kk % 3;  // node n, component c: word 4 n + c
            const bool owned = nx >= 1 && nx <= kCX && row >= 1 && row <= kCY;
            udst[j] = owned ? ((row - 1) * kCX + nx - 1) * 4 + kk % 3 : -1;
        }
        float beta = 0.0f;
        int ox = 0, oe = 0;
        for (uint32_t k = 0;; k++) {
            const int rs = (int)(k % kCNR), cs = (int)(k % kCNC), us = (int)(k % kCNU);
            bool ok = col_wait(bar(kCBarRawFull + rs), (k / kCNR) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const int4 m = meta_raw[rs];
            ok = col_wait(bar(kCBarConvEmpty + cs), ((k / kCNC) & 1u) ^ 1u, abort_flag) &&
                 col_wait(bar(kCBarUEmpty + us), ((k / kCNU) & 1u) ^ 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (m.x >= 0) {
                if (m.y == 0) {
                    const MfCol cl = cols[m.x];
                    const int x0 = cl.cx * kCX;
                    ox = 3 * (x0 - 1) - ((3 * (x0 - 1)) & ~3);
                    oe = (x0 - 1) - ((x0 - 1) & ~3);
                    beta = (MODE == 1) ? (float)states[cl.prob].beta : 0.0f;
                }
                const float *rz = reinterpret_cast<const float *>(smem + kC_OffRaw + rs * kCRawSlot);
                const float *rp = rz + kCRawNode / 4;
                const float *re = rz + 2 * kCRawNode / 4;
                uint32_t *hi = reinterpret_cast<uint32_t *>(smem + kC_OffConv + cs * 2 * kCPB);
                uint32_t *lo = hi + kCPB / 4;
                float *u = reinterpret_cast<float *>(smem + kC_OffU + us * kCUSlot);
                // all loads first: the stores below cannot alias them, but the compiler
                // cannot tell, and would otherwise order each round after the last
                float vz[kCConvRounds], vp[kCConvRounds];
#pragma unroll
                for (int j = 0; j < kCConvRounds; j++) {
                    const int bo = (src[j] < 0 ? 0 : src[j]) + ox;
                    vz[j] = rz[bo];
                    vp[j] = (MODE == 1) ? rp[bo] : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < kCConvRounds; j++) {
                    if (src[j] < 0) continue;
                    const float v = (MODE == 1) ? fmaf(beta, vp[j], vz[j]) : vz[j];
                    if (MODE == 1 && udst[j] >= 0) u[udst[j]] = v;
                    if (PR::kTf32) {
                        const uint32_t h = to_tf32(v);
                        hi[dst[j]] = h;
                        if (PR::kSplit) lo[dst[j]] = __float_as_uint(v - __uint_as_float(h));
                    } else {
                        // BF16 record: halves x, y, z at 8 n + c
                        const int hw = (dst[j] >> 2) * 8 + (dst[j] & 3);
                        const __nv_bfloat16 h = __float2bfloat16_rn(v);
                        reinterpret_cast<__nv_bfloat16 *>(hi)[hw] = h;
                        if (PR::kSplit)
                            reinterpret_cast<__nv_bfloat16 *>(lo)[hw] = __float2bfloat16_rn(v - __bfloat162float(h));
                    }
                }
                if (m.y < m.z) {
                    float *Eu = u + kCOwn * 4;
                    for (int e = ct; e < 128; e += kCConvThreads) Eu[e] = re[(e >> 3) * 12 + oe + (e & 7)];
                }
                fence_async_smem();  // the records are read by the tensor core (async proxy)
            }
            __syncwarp();
            if (lane == 0) {
                if (warp == 2) {
                    meta_conv[cs] = m;
                    meta_u[us] = m;
                }
                mbar_arrive(bar(kCBarRawEmpty + rs));
                mbar_arrive(bar(kCBarConvFull + cs));
                mbar_arrive(bar(kCBarUFull + us));
            }
            if (m.x < 0) break;
        }
    } else {
        // ------------------------------------------------------------ drain
        const int dw = warp & 3;                   // TMEM lane quarter (warps 8-11)
        const int r = dw * 32 + lane, ex = lane & 7, ey = r >> 3;
        float *xch = reinterpret_cast<float *>(smem + kC_OffX);
        uint32_t es = 0, xk = 0, rk = 0;
        float top[3] = {0.0f, 0.0f, 0.0f}, part = 0.0f;
        MfProblem P{};
        int x0 = 0, y0 = 0, z0 = 0, prob = 0;
        bool own = false;
        for (uint32_t k = 0;; k++) {
            const int us = (int)(k % kCNU);
            bool ok = col_wait(bar(kCBarUFull + us), (k / kCNU) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const int4 m = meta_u[us];
            if (m.x < 0) break;
            const float *u = reinterpret_cast<const float *>(smem + kC_OffU + us * kCUSlot);
            if (m.y == 0) {
                const MfCol cl = cols[m.x];
                prob = cl.prob;
                P = probs[prob];
                x0 = cl.cx * kCX;
                y0 = cl.cy * kCY;
                z0 = cl.cz * P.col_z;
                own = ex >= 1 && ey >= 1 && x0 + ex - 1 < P.NX && y0 + ey - 1 < P.NY;
                part = 0.0f;
                top[0] = top[1] = top[2] = 0.0f;
            }
            if (m.y < m.z) {
                // element plane s = m.y: its accumulator, scaled by E_e
                const int ts = (int)(es % kCNT);
                ok = col_wait(bar(kCBarTFull + ts), (es / kCNT) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                fence_after();
                float v[24];
                {
                    const uint32_t ta = tmem + ((uint32_t)(dw * 32) << 16) + (uint32_t)ts * kCTCols;
                    tmem_ld24(ta, v);
                    if (PR::kSplit) {
                        float w[24];
                        tmem_ld24(ta + 32, w);
#pragma unroll
                        for (int i = 0; i < 24; i++) v[i] += w[i];
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kCBarTEmpty + ts));
                es++;
                const float e = u[kCOwn * 4 + r];
                // in-plane sums: A = row-ey corners of node (ex, ey), B = row-ey corners of
                // node (ex, ey + 1); [0] bottom corners (dz = 0), [1] top corners (dz = 1)
                float A[2][3], B[2][3];
#pragma unroll
                for (int dz = 0; dz < 2; dz++)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float a00 = e * v[3 * corner_index(0, 0, dz) + c];
                        const float a10 = e * v[3 * corner_index(1, 0, dz) + c];
                        const float a01 = e * v[3 * corner_index(0, 1, dz) + c];
                        const float a11 = e * v[3 * corner_index(1, 1, dz) + c];
                        A[dz][c] = a00 + __shfl_up_sync(0xffffffffu, a10, 1);
                        B[dz][c] = a01 + __shfl_up_sync(0xffffffffu, a11, 1);
                    }
                // B of the row below: within the warp by a shuffle, across warps through
                // shared memory (the previous warp's last row)
                float Bp[2][3];
#pragma unroll
                for (int dz = 0; dz < 2; dz++)
#pragma unroll
                    for (int c = 0; c < 3; c++) Bp[dz][c] = __shfl_up_sync(0xffffffffu, B[dz][c], 8);
                const int xs2 = (int)(xk & 1u);
                float *xw = xch + xs2 * kCXch;
                if (lane >= 24) {
#pragma unroll
                    for (int dz = 0; dz < 2; dz++)
#pragma unroll
                        for (int c = 0; c < 3; c++) xw[(dw * 8 + ex) * 8 + dz * 3 + c] = B[dz][c];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kCBarXch + xs2));
                ok = col_wait(bar(kCBarXch + xs2), (xk >> 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                xk++;
                if (lane < 8 && dw > 0) {
#pragma unroll
                    for (int dz = 0; dz < 2; dz++)
#pragma unroll
                        for (int c = 0; c < 3; c++) Bp[dz][c] = xw[((dw - 1) * 8 + ex) * 8 + dz * 3 + c];
                }
                // node plane m.y = bottom corners of element plane m.y + top corners of m.y - 1
                if (m.y >= 1 && own) {
                    const int gx = x0 + ex - 1, gy = y0 + ey - 1, gz = z0 - 1 + m.y;
                    const int64_t gd = dof_index(P, gx, gy, gz, 0);
                    float4 uv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (MODE == 1) uv = *reinterpret_cast<const float4 *>(u + ((ey - 1) * kCX + ex - 1) * 4);
                    const float un[3] = {uv.x, uv.y, uv.z};
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float acc = (A[0][c] + Bp[0][c]) + top[c];
                        if (MODE == 1) {
                            y[gd + c] = acc;
                            p_new[gd + c] = un[c];
                            part = fmaf(un[c], acc, part);
                        } else if (MODE == 2) {
                            y[gd + c] = (dinv[gd + c] == 0.0f) ? 0.0f : rhs[gd + c] - acc;
                        } else {
                            y[gd + c] = (dinv[gd + c] == 0.0f) ? 0.0f : acc;
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++) top[c] = A[1][c] + Bp[1][c];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kCBarUEmpty + us));
            if (MODE == 1 && m.y == m.z) {
                // column partial of p.q: FP32 within a warp, FP64 across the four warps
                float w = part;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
                const int rb = (int)(rk & 1u);
                if (lane == 0) {
                    red[rb * 4 + dw] = (double)w;
                    mbar_arrive(bar(kCBarRed + rb));
                }
                if (dw == 0) {
                    ok = col_wait(bar(kCBarRed + rb), (rk >> 1) & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    MfState *st = states + prob;
                    int last = 0;
                    if (lane == 0) {
                        const double sum = ((red[rb * 4] + red[rb * 4 + 1]) + red[rb * 4 + 2]) + red[rb * 4 + 3];
                        col_part[m.x] = sum;
                        __threadfence();
                        const unsigned tk = atomicAdd(&st->cnt_apply, 1u);
                        last = (tk + 1u == (unsigned)P.col_count);
                    }
                    last = __shfl_sync(0xffffffffu, last, 0);
                    if (last) {
                        __threadfence();
                        // eight independent loads in flight per lane, added in a fixed order
                        double s = 0.0;
                        for (int c0 = lane; c0 < P.col_count; c0 += 32 * 8) {
                            double pv[8];
#pragma unroll
                            for (int t = 0; t < 8; t++) {
                                const int c = c0 + 32 * t;
                                pv[t] = c < P.col_count ? __ldcg(col_part + P.col_begin + c) : 0.0;
                            }
                            s += ((pv[0] + pv[1]) + (pv[2] + pv[3])) + ((pv[4] + pv[5]) + (pv[6] + pv[7]));
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                        if (lane == 0) {
                            st->cnt_apply = 0;
                            st->pq = s;
                            if (is_bad(s)) { st->status = MG_ENAN; st->done = 1; }
                            else if (!(s > 0.0)) { st->status = MG_EBREAKDOWN; st->done = 1; }
                            else st->alpha = st->rz / s;
                        }
                    }
                }
                rk++;
            }
        }
        if (*abort_flag && lane == 0) atomicOr(err, 2);
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 1) tmem_dealloc(tmem, kCNT * kCTCols);
}

// ------------------------------------------------- factored CUDA-core operator
// y = sum_e E_e P_e^T K0 P_e x in FP32 on the CUDA cores with the factored
// element stiffness (hex8_factored.cuh: 2 x 72 butterfly additions + 45 FMA per
// element instead of 576 FMA), two elements per thread in packed FP32x2
// arithmetic.  A tile owns kFNX x kFNY nodes in x, y and P.fac_z node planes
// in z and streams through its element planes.  Warp w holds element rows 2w
// and 2w+1 of the kFEX x kFEY element plane around the owned nodes (lane = x;
// halo elements are recomputed by the neighbouring tiles).  The node planes
// (input, D^-1 and the per-mode node vectors) and the moduli plane arrive by
// TMA ahead of their use into a four-slot ring.
//
// The transform to sum/difference modes is a product of an x, y part, which
// belongs to a node plane, and a z part, which joins two planes.  So each node
// plane is gathered and transformed in x, y once, kept in registers, and met by
// the next plane in the z stage of the element plane between them; on the way
// back the z stage leaves a part for the plane below and one for the plane
// above, the two parts of a node plane are added in mode space, and one inverse
// x, y transform per node plane returns to the corners: two thirds of the
// butterflies, half the gathers, shuffles and exchanges of a form that treats
// each element plane by itself.  The corners are then summed into the owned
// nodes: along x with a warp shuffle (left element + right element), along y
// inside the thread (rows 2w, 2w+1) or through shared memory (row 2w+1 with the
// next warp's row 2w+2).  Every node's sum has the same fixed order
// (deterministic and independent of the tiling).  Bound by issue (44 % of its slots at
// 128x64x64) and by the start of a tile (tables and first planes, about 6,000 of 25,000
// cycles there); 16 warps per SM at 128 registers, no spills (D^-1 and the third plane are
// read behind the plane's barrier: read before it they spilled, and MODE 6 took 144 us
// where it takes 85).  MODE 2, 58 problems of 12.9 M dofs: 95 -> 84 us a launch, 66 with the
// tiles dealt by size (plan_fac_tiles); y = A x at 128x64x64 13.9 -> 12.2 us, at 192x96x96
// 31.6 -> 27.3 us.
constexpr int kFEX = 32, kFEY = 16;                // elements per tile plane
constexpr int kFNX = kFEX - 1, kFNY = kFEY - 1;    // owned nodes per tile plane
constexpr int kFPX = kFEX + 1, kFPY = kFEY + 1;    // tile node plane (with halo)
constexpr int kFThreads = 256;                     // 8 warps x 2 element rows
constexpr int kFMinZ = 1, kFMaxZ = 32;
constexpr int kFRing = 4;                          // 2 planes read, 2 in flight
constexpr int kFBoxX = 104;                        // TMA node box: 104 floats (3 kFPX + alignment) x kFPY rows
constexpr int kFPlaneF = 1792;                     // floats per node plane in the ring (7168 B, 128 B aligned)
constexpr int kFBoxE = 36;                         // TMA moduli box: 36 elements x kFEY rows
constexpr int kFModF = kFBoxE * kFEY;              // 576 floats
constexpr int kFXch = 3 * kFThreads;               // row exchange: 3 floats per thread
static_assert(kFBoxX * kFPY <= kFPlaneF && kFBoxX >= 3 + 3 * kFPX && kFBoxE >= 3 + kFEX, "boxes");
static_assert(kFThreads == 32 * (kFEY / 2) && kFEX == 32, "warp = element row pair, lane = x");
static_assert((kMaxSide + kFNX - 1) / kFNX <= 65536 && (kMaxSide + kFNY - 1) / kFNY <= 65536, "tile numbers");
// tensor maps per problem for this kernel: node vectors with the 104 x 17 x 1 box
// and the moduli with the 36 x 16 x 1 box
enum FacMap { kFMapMx = 0, kFMapMd, kFMapMy, kFMapMb, kFMapR, kFMapDinv, kFMapMr, kFMapZ, kFMapE, kFacMaps };
// node planes per ring slot: the input, D^-1 and (MODE 2, 5 rhs, MODE 4 r, MODE 6 the iterate)
__host__ __device__ constexpr int fac_planes(int mode) { return mode == 3 ? 2 : 3; }
__host__ __device__ constexpr int fac_slot(int mode) { return fac_planes(mode) * kFPlaneF + kFModF; }
__host__ __device__ constexpr int fac_smem(int mode) { return (kFRing * fac_slot(mode) + 2 * kFXch) * 4 + 128; }
// MODE 3: 72,832 B; MODE 2, 4, 5, 6: 101,504 B: two CTAs per SM

struct FacArgs {
    int in_map, b_map;  // tensor maps (FacMap) of the input and of the third node plane
    float *y;           // MODE 2, 3: output (MODE 2: nullable); MODE 4, 5: the new direction
    float *z;           // MODE 2: D^-1 times the output (nullable)
    float *r, *xs;      // MODE 4, 5: Chebyshev residual; MODE 4, 5, 6: iterate
    float c1, c2, inv_theta;
    int x0_zero;        // MODE 5, 6: the iterate starts at 0
};

// MODE 2: y = rhs - A x, z = D^-1 y.  MODE 3: y = A x.  (All 0 where dinv = 0.)
// MODE 4: one Chebyshev step on direction x = d: r -= A d; y = d' = c1 d +
//         c2 D^-1 r; xs += d' (mg_cheb_next_kernel's sequence, fused).
// MODE 5: the first two Chebyshev steps on rhs b from x = z = D^-1 b: d = z / theta,
//         xs (+)= d, r = b - A d, y = d' = c1 d + c2 D^-1 r, xs += d'
//         (mg_cheb_first_kernel's and mg_cheb_next_kernel's sequence, fused).
// MODE 6: the same two steps when no third follows: only xs changes, and with
//         D^-1 r = z - D^-1 A d the rhs is not needed either.
// The producers of a rhs write z beside it (the CG update, the restriction, MODE 2):
// formed here from b and D^-1 at every corner it took twice the shared loads of MODE 2 (a
// batch of 58 problems, 12.9 M dofs: 159 us a launch against 85 us for MODE 6).
// A TMA wait that exceeds its bound sets bit 4 of *err and ends the block.
template <int MODE>
__global__ void __launch_bounds__(kFThreads, 2) mf_fac_kernel(
    const MfProblem *__restrict__ probs, const MfCol *__restrict__ tiles, const int *__restrict__ offs, int sel,
    const FacK2 K, const CUtensorMap *__restrict__ fmaps, const MfState *__restrict__ states, const FacArgs A,
    int *err) {
    pdl_trigger();
    extern __shared__ __align__(128) float fsm[];
    __shared__ __align__(8) uint64_t bars[kFRing];
    constexpr int NP = fac_planes(MODE);
    // slot k: [input plane | D^-1 plane | third plane (NP = 3) | moduli]
    auto plane_of = [&](int slot, int part) { return fsm + slot * fac_slot(MODE) + part * kFPlaneF; };
    auto mod_of = [&](int slot) { return fsm + slot * fac_slot(MODE) + NP * kFPlaneF; };
    float(*sX)[3][kFThreads] = reinterpret_cast<float(*)[3][kFThreads]>(fsm + kFRing * fac_slot(MODE));
    const int tid = threadIdx.x, tx = tid & 31, w = tid >> 5;
    const uint32_t bar0 = smem_u32(&bars[0]);
    if (tid == 0)
        for (int k = 0; k < kFRing; k++) mbar_init(bar0 + 8 * k, 1);
    // the work lists, tile and problem tables and the tensor maps are constant: bring the first
    // tile's into the caches while the previous kernel drains, then wait for its results
    const int t_lo = offs[blockIdx.x], t_hi = offs[blockIdx.x + 1];  // this CTA's tiles
    if (tid == 0) {
        const int p0 = tiles[t_lo].prob;
        const char *line = reinterpret_cast<const char *>(probs + p0);
        asm volatile("prefetch.global.L1 [%0];" ::"l"(line));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(line + 128));
        const CUtensorMap *m0 = fmaps + (size_t)p0 * kFacMaps;
        auto prefetch = [&](int k) { asm volatile("prefetch.tensormap [%0];" ::"l"(m0 + k) : "memory"); };
        prefetch(A.in_map);
        prefetch(kFMapDinv);
        prefetch(kFMapE);
        if (NP == 3 && A.b_map >= 0) prefetch(A.b_map);
    }
    pdl_wait();
    __syncthreads();
    uint32_t phase = 0;   // bit k: parity of slot k's next completion
    uint32_t issued = 0;  // bit k: a load into slot k is outstanding (thread 0)
    bool failed = false;
    const bool third = MODE == 2 || MODE == 4 || MODE == 5 || (MODE == 6 && !A.x0_zero);
    const float2 neg1 = make_float2(-1.0f, -1.0f);
    for (int ti = t_lo; ti < t_hi && !failed; ti++) {
        const MfCol T = tiles[ti];
        const MfProblem P = probs[T.prob];
        if (states[P.root].done || P.bottom || (sel >= 0 && sel != (P.coarse < 0 ? 1 : 0))) continue;
        const int x0 = T.cx * kFNX, y0 = T.cy * kFNY, z0 = T.cz * P.fac_z;
        const int z1 = min(z0 + P.fac_z, P.NZ);
        const int S = z1 - z0 + 1;  // element planes z0-1 .. z1-1; node planes z0-1 .. z1
        // 16-byte aligned box starts and the offsets of the tile inside the boxes
        const int xs = (3 * (x0 - 1)) & ~3, ox = 3 * (x0 - 1) - xs;
        const int xe = (x0 - 1) & ~3, oe = (x0 - 1) - xe;
        const CUtensorMap *maps = fmaps + (size_t)T.prob * kFacMaps;
        const int64_t plane_stride = (int64_t)P.NY * P.pitch;
        const uint32_t bytes = (uint32_t)(((third ? 3 : 2) * kFBoxX * kFPY + kFModF) * 4);
        // node planes p (nz = z0 - 1 + p) and element plane p's moduli into slot p % kFRing
        auto issue = [&](int p) {
            const int slot = p % kFRing;
            const uint32_t bar = bar0 + 8 * slot;
            fence_async_smem();
            mbar_expect_tx(bar, bytes);
            tma_load_3d(smem_u32(plane_of(slot, 0)), maps + A.in_map, xs, y0 - 1, z0 - 1 + p, bar);
            tma_load_3d(smem_u32(plane_of(slot, 1)), maps + kFMapDinv, xs, y0 - 1, z0 - 1 + p, bar);
            if (third) tma_load_3d(smem_u32(plane_of(slot, 2)), maps + A.b_map, xs, y0 - 1, z0 - 1 + p, bar);
            tma_load_3d(smem_u32(mod_of(slot)), maps + kFMapE, xe, y0 - 1, z0 - 1 + p, bar);
        };
        // every thread waits for slot p's loads; false after the bound
        auto arrive = [&](int p) {
            const int slot = p % kFRing;
            const bool ok = mbar_wait_bounded(bar0 + 8 * slot, (phase >> slot) & 1u);
            phase ^= 1u << slot;
            if (tid == 0) issued &= ~(1u << slot);
            return ok;
        };
        // owned nodes: x = x0 + tx; rows y0 + 2w (row 2w+1 of the tile plane) and
        // y0 + 2w + 1 (row 2w+2, warps 0..6)
        const int gx = x0 + tx, gy1 = y0 + 2 * w, gy2 = gy1 + 1;
        const bool own1 = tx < kFNX && gx < P.NX && gy1 < P.NY;
        const bool own2 = tx < kFNX && w < kFEY / 2 - 1 && gx < P.NX && gy2 < P.NY;
        __syncthreads();  // the previous tile's readers of the ring and the exchange are done
        if (tid == 0) {
            for (int p = 0; p < 3 && p <= S; p++) {
                issue(p);
                issued |= 1u << (p % kFRing);
            }
        }
        bool ok = arrive(0);
        ok = arrive(1) && ok;
        // the xy modes (q = mx + 2 my) of node plane p at the element pair: element A = rows
        // 2w, 2w+1 of the plane in .x, B = rows 2w+1, 2w+2 in .y
        auto plane_modes = [&](int p, float2 (&m)[3][4]) {
            const float *n0 = plane_of(p % kFRing, 0) + ox;
            float nv[3][2][3];  // [row 2w + 0..2][bx][c]
#pragma unroll
            for (int r3 = 0; r3 < 3; r3++)
#pragma unroll
                for (int bx = 0; bx < 2; bx++) {
                    const int o = (2 * w + r3) * kFBoxX + 3 * (tx + bx);
#pragma unroll
                    for (int c = 0; c < 3; c++) nv[r3][bx][c] = n0[o + c];
                }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float2 sx[2], dx[2];  // [by]
#pragma unroll
                for (int by = 0; by < 2; by++) {
                    const float2 lo = make_float2(nv[by][0][c], nv[by + 1][0][c]);
                    const float2 hi = make_float2(nv[by][1][c], nv[by + 1][1][c]);
                    sx[by] = __fadd2_rn(lo, hi);
                    dx[by] = __ffma2_rn(lo, neg1, hi);  // hi - lo
                }
                m[c][0] = __fadd2_rn(sx[0], sx[1]);
                m[c][1] = __fadd2_rn(dx[0], dx[1]);
                m[c][2] = __ffma2_rn(sx[0], neg1, sx[1]);
                m[c][3] = __ffma2_rn(dx[0], neg1, dx[1]);
            }
        };
        float2 low[3][4], car[3][4];  // modes of node plane s; the top-face results of element plane s - 1 on it
        plane_modes(0, low);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int q = 0; q < 4; q++) car[c][q] = make_float2(0.0f, 0.0f);
        int64_t g1 = P.dof_off + ((int64_t)(z0 - 1) * P.NY + gy1) * P.pitch + 3 * gx;
        for (int s = 0; s < S; s++) {
            // element phase: the z stage of the transform joins node planes s and s + 1, the
            // result is split again into the plane below (completing node plane s together
            // with the carried results of the element plane below it) and the plane above
            float2 node[3][4];
            {
                float2 high[3][4], v[3][8];
                plane_modes(s + 1, high);
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        v[c][q] = __fadd2_rn(low[c][q], high[c][q]);
                        v[c][q + 4] = __ffma2_rn(low[c][q], neg1, high[c][q]);
                        low[c][q] = high[c][q];
                    }
                const float *Es = mod_of(s % kFRing) + oe + tx;
                const float2 e2 = make_float2(Es[2 * w * kFBoxE], Es[(2 * w + 1) * kFBoxE]);
                hex8_factored_khat2(K, e2, v);  // E = 0 (outside the grid) gives exact zeros
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        // mode 0 is zero
                        const float2 down = q ? __ffma2_rn(v[c][q + 4], neg1, v[c][q]) : __fmul2_rn(v[c][4], neg1);
                        const float2 up = q ? __fadd2_rn(v[c][q], v[c][q + 4]) : v[c][4];
                        node[c][q] = __fadd2_rn(car[c][q], down);
                        car[c][q] = up;
                    }
            }
            // node plane s (s >= 1; the halo plane 0 is the tile below's): back to the corners
            float2 xsum[3][2];  // [c][by]
            float(*X)[kFThreads] = sX[s & 1];
            if (s >= 1) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    float2 f[2][2];  // [by][bx]
                    const float2 y0 = __ffma2_rn(node[c][2], neg1, node[c][0]), y1 = __fadd2_rn(node[c][0], node[c][2]);
                    const float2 d0 = __ffma2_rn(node[c][3], neg1, node[c][1]), d1 = __fadd2_rn(node[c][1], node[c][3]);
                    f[0][0] = __ffma2_rn(d0, neg1, y0);
                    f[0][1] = __fadd2_rn(y0, d0);
                    f[1][0] = __ffma2_rn(d1, neg1, y1);
                    f[1][1] = __fadd2_rn(y1, d1);
                    // along x: node x0 + tx = corner dx = 1 of this lane's element + dx = 0 of the next lane's
#pragma unroll
                    for (int by = 0; by < 2; by++) {
                        float2 nb;
                        nb.x = __shfl_down_sync(0xffffffffu, f[by][0].x, 1);
                        nb.y = __shfl_down_sync(0xffffffffu, f[by][0].y, 1);
                        xsum[c][by] = __fadd2_rn(f[by][1], nb);
                    }
                    // along y: row 2w of this warp (element 2w at by = 0) goes to the warp above
                    X[c][tid] = xsum[c][0].x;
                }
            }
            // the next step's top plane (s + 2) has landed
            bool sok = true;
            if (s + 2 <= S) sok = arrive(s + 2);
            if (__syncthreads_or(!(sok && ok))) {
                failed = true;
                if (tid == 0) atomicOr(err, 4);
                break;
            }
            // plane s + 3 into the slot of plane s - 1, whose readers (the element phases of
            // steps s - 2, s - 1 and the node phase of step s - 1) are behind this barrier
            if (tid == 0 && s + 3 <= S) {
                issue(s + 3);
                issued |= 1u << ((s + 3) % kFRing);
            }
            if (s >= 1) {
                float nn[2][3];  // [row][c]: the operator at the owned nodes of node plane s
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    nn[0][c] = xsum[c][1].x + xsum[c][0].y;  // element 2w (by = 1) + 2w+1 (by = 0)
                    nn[1][c] = xsum[c][1].y + (w < kFEY / 2 - 1 ? X[c][tid + 32] : 0.0f);
                }
#pragma unroll
                for (int rr = 0; rr < 2; rr++) {
                    const bool own = rr ? own2 : own1;
                    if (!own) continue;
                    const int64_t g = g1 + (rr ? P.pitch : 0);
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float a = nn[rr][c];
                        // the input, D^-1 and the third plane at the node
                        const int o = ox + (2 * w + 1 + rr) * kFBoxX + 3 * (tx + 1) + c;
                        const float uu = plane_of(s % kFRing, 0)[o], dd = plane_of(s % kFRing, 1)[o];
                        const float bb = third ? plane_of(s % kFRing, 2)[o] : 0.0f;
                        if (MODE == 2) {
                            const float v = dd == 0.0f ? 0.0f : bb - a;
                            if (A.y) A.y[g + c] = v;
                            if (A.z) A.z[g + c] = dd * v;
                        } else if (MODE == 3) {
                            A.y[g + c] = dd == 0.0f ? 0.0f : a;
                        } else if (MODE == 4) {
                            const float rv = bb - (dd == 0.0f ? 0.0f : a);
                            const float dn2 = fmaf(A.c1, uu, A.c2 * dd * rv);
                            A.r[g + c] = rv;
                            A.y[g + c] = dn2;
                            A.xs[g + c] += dn2;
                        } else {
                            // the input is z: a is A z, so A d = a / theta
                            const float d0 = uu * A.inv_theta;
                            float dr;  // D^-1 r
                            if (MODE == 5) {
                                const float rv = dd == 0.0f ? bb : fmaf(-A.inv_theta, a, bb);
                                A.r[g + c] = rv;
                                dr = dd * rv;
                            } else {
                                dr = fmaf(-A.inv_theta * dd, a, uu);
                            }
                            const float dn2 = fmaf(A.c1, d0, A.c2 * dr);
                            if (MODE == 5) A.y[g + c] = dn2;
                            const float x0 = A.x0_zero ? 0.0f : MODE == 5 ? A.xs[g + c] : bb;
                            A.xs[g + c] = x0 + d0 + dn2;
                        }
                    }
                }
            }
            g1 += plane_stride;
        }
    }
    // after a failed wait, give the outstanding loads a bounded chance to land
    if (failed && tid == 0)
        for (int k = 0; k < kFRing; k++)
            if (issued & (1u << k)) (void)mbar_wait_bounded(bar0 + 8 * k, (phase >> k) & 1u);
    __syncthreads();
}

// ---------------------------------------------------------------- vector phase
// x += alpha p; r -= alpha q (r stays 0 on Dirichlet dofs, D^-1 = 0 there);
// z = D^-1 r; rz, rr -> beta, stop test.  float4 over 16-byte aligned chunks.
// mg = 1: z starts the multigrid V-cycle's first smoother; only rr (stop test) is
// reduced here and beta is formed after the V-cycle (mf_dot_rz_kernel).
__global__ void __launch_bounds__(kThreads) mf_update_kernel(
    const MfChunkDesc *__restrict__ chunks, int n_chunks, const MfProblem *__restrict__ probs,
    float *__restrict__ x, float *__restrict__ r, float *__restrict__ z,
    const float *__restrict__ p, const float *__restrict__ q, const float *__restrict__ dinv,
    MfState *states, double *__restrict__ chunk_part, int mg) {
    pdl_trigger();
    __shared__ double red_sh[kThreads / 32];
    __shared__ int sh_last;
    MfChunkDesc C = chunks[min((int)blockIdx.x, n_chunks - 1)];
    pdl_wait();
    for (int ci = blockIdx.x; ci < n_chunks; ci += gridDim.x) {
        if (ci != (int)blockIdx.x) C = chunks[ci];
        MfState *st = states + C.prob;
        if (st->done) continue;
        const float alpha = (float)st->alpha;
        float rz = 0.0f, rr = 0.0f;
#pragma unroll 4
        for (int64_t i = C.begin + 4 * threadIdx.x; i < C.end; i += 4 * kThreads) {
            const float4 pv = *reinterpret_cast<const float4 *>(p + i);
            const float4 qv = *reinterpret_cast<const float4 *>(q + i);
            const float4 dv = *reinterpret_cast<const float4 *>(dinv + i);
            float4 xv = *reinterpret_cast<const float4 *>(x + i);
            float4 rv = *reinterpret_cast<const float4 *>(r + i);
            xv.x = fmaf(alpha, pv.x, xv.x); xv.y = fmaf(alpha, pv.y, xv.y);
            xv.z = fmaf(alpha, pv.z, xv.z); xv.w = fmaf(alpha, pv.w, xv.w);
            rv.x = dv.x != 0.0f ? fmaf(-alpha, qv.x, rv.x) : 0.0f;
            rv.y = dv.y != 0.0f ? fmaf(-alpha, qv.y, rv.y) : 0.0f;
            rv.z = dv.z != 0.0f ? fmaf(-alpha, qv.z, rv.z) : 0.0f;
            rv.w = dv.w != 0.0f ? fmaf(-alpha, qv.w, rv.w) : 0.0f;
            const float4 zv = make_float4(dv.x * rv.x, dv.y * rv.y, dv.z * rv.z, dv.w * rv.w);
            *reinterpret_cast<float4 *>(x + i) = xv;
            *reinterpret_cast<float4 *>(r + i) = rv;
            *reinterpret_cast<float4 *>(z + i) = zv;
            rz = fmaf(rv.x, zv.x, fmaf(rv.y, zv.y, fmaf(rv.z, zv.z, fmaf(rv.w, zv.w, rz))));
            rr = fmaf(rv.x, rv.x, fmaf(rv.y, rv.y, fmaf(rv.z, rv.z, fmaf(rv.w, rv.w, rr))));
        }
        const double srz = mg ? 0.0 : block_sum_f(rz, red_sh);
        const double srr = block_sum_f(rr, red_sh);
        const MfProblem &P = probs[C.prob];
        if (threadIdx.x == 0) {
            if (!mg) chunk_part[ci] = srz;
            chunk_part[n_chunks + ci] = srr;
            __threadfence();
            const unsigned t = atomicAdd(&st->cnt_update, 1u);
            sh_last = (t == (unsigned)P.chunk_count - 1);
        }
        __syncthreads();
        if (sh_last) {
            const double trz = mg ? 0.0 : ordered_sum(chunk_part, P.chunk_begin, P.chunk_count);
            const double trr = ordered_sum(chunk_part + n_chunks, P.chunk_begin, P.chunk_count);
            if (threadIdx.x == 0) {
                st->cnt_update = 0;
                st->iter += 1;
                st->total_iter += 1;
                st->rr = trr;
                if (is_bad(trr) || (!mg && is_bad(trz))) { st->status = MG_ENAN; st->done = 1; }
                else {
                    if (!mg) {
                        st->beta = trz / st->rz;
                        st->rz = trz;
                    }
                    if (trr <= st->tol2) st->done = 1;
                    else if (st->iter >= st->maxit) { st->status = MG_ENOCONV; st->done = 1; }
                }
            }
        }
        __syncthreads();
    }
}

// r . z of the new residual and its preconditioned form: beta
__device__ __forceinline__ void finish_rz(MfState *st, double rz) {
    if (is_bad(rz) || !(rz > 0.0)) {
        // a preconditioner that is not positive on r: stop with breakdown
        st->status = is_bad(rz) ? MG_ENAN : MG_EBREAKDOWN;
        st->done = 1;
    } else {
        st->beta = st->first ? 0.0 : rz / st->rz;
        st->rz = rz;
        st->first = 0;
    }
}

// rz = r . z after the V-cycle
__global__ void __launch_bounds__(kThreads) mf_dot_rz_kernel(
    const MfChunkDesc *__restrict__ chunks, int n_chunks, const MfProblem *__restrict__ probs,
    const float *__restrict__ r, const float *__restrict__ z, MfState *states,
    double *__restrict__ chunk_part) {
    pdl_trigger();
    __shared__ double red_sh[kThreads / 32];
    __shared__ int sh_last;
    MfChunkDesc C = chunks[min((int)blockIdx.x, n_chunks - 1)];
    pdl_wait();
    for (int ci = blockIdx.x; ci < n_chunks; ci += gridDim.x) {
        if (ci != (int)blockIdx.x) C = chunks[ci];
        MfState *st = states + C.prob;
        if (st->done) continue;
        float rz = 0.0f;
#pragma unroll 4
        for (int64_t i = C.begin + 4 * threadIdx.x; i < C.end; i += 4 * kThreads) {
            const float4 rv = *reinterpret_cast<const float4 *>(r + i);
            const float4 zv = *reinterpret_cast<const float4 *>(z + i);
            rz = fmaf(rv.x, zv.x, fmaf(rv.y, zv.y, fmaf(rv.z, zv.z, fmaf(rv.w, zv.w, rz))));
        }
        const double srz = block_sum_f(rz, red_sh);
        const MfProblem &P = probs[C.prob];
        if (threadIdx.x == 0) {
            chunk_part[ci] = srz;
            __threadfence();
            const unsigned t = atomicAdd(&st->cnt_update, 1u);
            sh_last = (t == (unsigned)P.chunk_count - 1);
        }
        __syncthreads();
        if (sh_last) {
            const double trz = ordered_sum(chunk_part, P.chunk_begin, P.chunk_count);
            if (threadIdx.x == 0) {
                st->cnt_update = 0;
                finish_rz(st, trz);
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ multigrid kernels
// Chebyshev-Jacobi smoothing (first step): mr = rin; md = D^-1 rin / theta;
// mx = md (x0_zero) or mx + md.  Skips designs whose CG has stopped.
__global__ void __launch_bounds__(kThreads) mg_cheb_first_kernel(
    const MfChunkDesc *__restrict__ chunks, int lo, int hi, const MfProblem *__restrict__ probs,
    const MfState *states, const float *__restrict__ rin, float *__restrict__ mr,
    float *__restrict__ md, float *__restrict__ mx, const float *__restrict__ dinv,
    float inv_theta, int x0_zero, int sel) {
    pdl_enter();
    for (int ci = lo + blockIdx.x; ci < hi; ci += gridDim.x) {
        const MfChunkDesc C = chunks[ci];
        const MfProblem &Q = probs[C.prob];
        if (states[Q.root].done || Q.bottom || (sel >= 0 && sel != (Q.coarse < 0 ? 1 : 0))) continue;
#pragma unroll 4
        for (int64_t i = C.begin + 4 * threadIdx.x; i < C.end; i += 4 * kThreads) {
            const float4 rv = *reinterpret_cast<const float4 *>(rin + i);
            const float4 dv = *reinterpret_cast<const float4 *>(dinv + i);
            const float4 d = make_float4(dv.x * rv.x * inv_theta, dv.y * rv.y * inv_theta,
                                         dv.z * rv.z * inv_theta, dv.w * rv.w * inv_theta);
            float4 xv = x0_zero ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4 *>(mx + i);
            xv.x += d.x; xv.y += d.y; xv.z += d.z; xv.w += d.w;
            if (mr != rin) *reinterpret_cast<float4 *>(mr + i) = rv;
            *reinterpret_cast<float4 *>(md + i) = d;
            *reinterpret_cast<float4 *>(mx + i) = xv;
        }
    }
}

// Chebyshev step: mr -= A md (= my); md = c1 md + c2 D^-1 mr; mx += md
__global__ void __launch_bounds__(kThreads) mg_cheb_next_kernel(
    const MfChunkDesc *__restrict__ chunks, int lo, int hi, const MfProblem *__restrict__ probs,
    const MfState *states, const float *__restrict__ my, float *__restrict__ mr,
    float *__restrict__ md, float *__restrict__ mx, const float *__restrict__ dinv, float c1,
    float c2, int sel) {
    pdl_enter();
    for (int ci = lo + blockIdx.x; ci < hi; ci += gridDim.x) {
        const MfChunkDesc C = chunks[ci];
        const MfProblem &Q = probs[C.prob];
        if (states[Q.root].done || Q.bottom || (sel >= 0 && sel != (Q.coarse < 0 ? 1 : 0))) continue;
#pragma unroll 4
        for (int64_t i = C.begin + 4 * threadIdx.x; i < C.end; i += 4 * kThreads) {
            const float4 yv = *reinterpret_cast<const float4 *>(my + i);
            const float4 dv = *reinterpret_cast<const float4 *>(dinv + i);
            float4 rv = *reinterpret_cast<const float4 *>(mr + i);
            float4 d = *reinterpret_cast<const float4 *>(md + i);
            float4 xv = *reinterpret_cast<const float4 *>(mx + i);
            rv.x -= yv.x; rv.y -= yv.y; rv.z -= yv.z; rv.w -= yv.w;
            d.x = fmaf(c1, d.x, c2 * dv.x * rv.x); d.y = fmaf(c1, d.y, c2 * dv.y * rv.y);
            d.z = fmaf(c1, d.z, c2 * dv.z * rv.z); d.w = fmaf(c1, d.w, c2 * dv.w * rv.w);
            xv.x += d.x; xv.y += d.y; xv.z += d.z; xv.w += d.w;
            *reinterpret_cast<float4 *>(mr + i) = rv;
            *reinterpret_cast<float4 *>(md + i) = d;
            *reinterpret_cast<float4 *>(mx + i) = xv;
        }
    }
}

// The transfers run over the list of node blocks of the coarse problems that take part (a grid
// of the largest problem's blocks times the problems left most blocks of a mixed batch empty: 58
// problems, restriction from level 0 42 us a launch, 21 us from the list).
//
// restriction (transpose of trilinear interpolation) into the coarse problems:
// mb_c[I] = sum_d w(d) my_f[2I + d], d in {-1,0,1}^3, w = prod (1 - |d|/2);
// z_c = D^-1 mb_c
__global__ void __launch_bounds__(kNodeBlk) mg_restrict_kernel(const MfProblem *__restrict__ probs,
                                                          const MfNodeBlk *__restrict__ blks,
                                                          const MfState *states, const float *__restrict__ my,
                                                          float *__restrict__ mb, float *__restrict__ z,
                                                          const float *__restrict__ dinv) {
    pdl_trigger();
    const MfNodeBlk B = blks[blockIdx.x];
    const MfProblem C = probs[B.prob];
    const MfProblem F = probs[C.fine];
    pdl_wait();
    if (states[C.root].done) return;
    // one coarse node (3 dofs) per thread: its 27 fine neighbours' loads are all
    // issued before the sums (independent, predicated on the grid bounds)
    const int nn = C.NX * C.NY * C.NZ, n = B.node + threadIdx.x;
    if (n < nn) {
        const int I = n % C.NX, JK = n / C.NX, J = JK % C.NY, K = JK / C.NY;
        const int64_t o = C.dof_off + ((int64_t)K * C.NY + J) * C.pitch + 3 * I;
        float v[27][3];
#pragma unroll
        for (int q = 0; q < 27; q++) {
            const int dx = q % 3 - 1, dy = (q / 3) % 3 - 1, dz = q / 9 - 1;
            const int ii = 2 * I + dx, j = 2 * J + dy, k = 2 * K + dz;
            const bool in = ii >= 0 && ii < F.NX && j >= 0 && j < F.NY && k >= 0 && k < F.NZ;
            const float *src = my + F.dof_off + (in ? ((int64_t)k * F.NY + j) * F.pitch + 3 * ii : 0);
#pragma unroll
            for (int c = 0; c < 3; c++) v[q][c] = in ? src[c] : 0.0f;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            // the order of the sums: dz outermost, then dy, then dx (as the transpose of prolongation)
            float out = 0.0f;
#pragma unroll
            for (int q = 0; q < 27; q++) {
                const int dx = q % 3 - 1, dy = (q / 3) % 3 - 1, dz = q / 9 - 1;
                const float w = (dz ? 0.5f : 1.0f) * (dy ? 0.5f : 1.0f) * (dx ? 0.5f : 1.0f);
                out = fmaf(w, v[q][c], out);
            }
            const float dv = dinv[o + c];
            mb[o + c] = dv != 0.0f ? out : 0.0f;
            z[o + c] = dv * out;  // the smoother's start
        }
    }
}

// prolongation (trilinear) from the coarse problems into their fine ones:
// mx_f[i] += sum_I w mx_c[I] (skips Dirichlet dofs and padding).  One coarse node (I, J, K) per
// thread: it reads the cell's eight coarse nodes once and updates the fine nodes 2I..2I+1, 2J..2J+1,
// 2K..2K+1, each from its 1, 2, 4 or 8 parents; all loads are issued before the first sum.  Bound by
// DRAM and L2 (20 bytes a fine dof).  With a fine node per thread its up to eight parents were read
// for every node: 58 problems, level 0 (10.9 M dofs) 70 us a launch, 20 us by cells.
__global__ void __launch_bounds__(kNodeBlk) mg_prolong_kernel(const MfProblem *__restrict__ probs,
                                                         const MfNodeBlk *__restrict__ blks,
                                                         const MfState *states, float *mx,
                                                         const float *__restrict__ dinv) {
    pdl_trigger();
    const MfNodeBlk B = blks[blockIdx.x];
    const MfProblem C = probs[B.prob];
    const MfProblem F = probs[C.fine];
    const int n = B.node + threadIdx.x;
    const bool in = n < C.NX * C.NY * C.NZ;
    const int I = n % C.NX, JK = n / C.NX, J = JK % C.NY, K = JK / C.NY;
    pdl_wait();
    if (states[F.root].done || !in) return;
    const bool has_x = 2 * I + 1 < F.NX, has_y = 2 * J + 1 < F.NY, has_z = 2 * K + 1 < F.NZ;
    if (2 * I >= F.NX || 2 * J >= F.NY || 2 * K >= F.NZ) return;  // beyond an odd side
    float v[8][3];  // the cell's coarse nodes
    const float *src = mx + C.dof_off + ((int64_t)K * C.NY + J) * C.pitch + 3 * I;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const bool use = (!(q & 1) || has_x) && (!(q & 2) || has_y) && (!(q & 4) || has_z);
        const int64_t o = use ? ((int64_t)(q >> 2) * C.NY + ((q >> 1) & 1)) * C.pitch + 3 * (q & 1) : 0;
#pragma unroll
        for (int c = 0; c < 3; c++) v[q][c] = use ? src[o + c] : 0.0f;
    }
    // two neighbouring fine nodes are six floats from an even place on: three pairs, the last
    // pair and a half left out where the second node does not exist
    float m[4][6], d[4][6];
    const int64_t o0 = F.dof_off + ((int64_t)2 * K * F.NY + 2 * J) * F.pitch + 6 * I;
#pragma unroll
    for (int row = 0; row < 4; row++) {
        const bool use = (!(row & 1) || has_y) && (!(row & 2) || has_z);
        const int64_t o = o0 + (use ? ((int64_t)(row >> 1) * F.NY + (row & 1)) * F.pitch : 0);
#pragma unroll
        for (int h = 0; h < 3; h++) {
            if (has_x || h == 0) {
                const float2 mv = *reinterpret_cast<const float2 *>(mx + o + 2 * h);
                const float2 dv = *reinterpret_cast<const float2 *>(dinv + o + 2 * h);
                m[row][2 * h] = mv.x; m[row][2 * h + 1] = mv.y;
                d[row][2 * h] = dv.x; d[row][2 * h + 1] = dv.y;
            }
        }
        if (!has_x) { m[row][2] = mx[o + 2]; d[row][2] = dinv[o + 2]; }
    }
#pragma unroll
    for (int row = 0; row < 4; row++) {
        const int b = row & 1, a = row >> 1;
        if ((b && !has_y) || (a && !has_z)) continue;
        const int64_t o = o0 + ((int64_t)a * F.NY + b) * F.pitch;
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float w = (x ? 0.5f : 1.0f) * (b ? 0.5f : 1.0f) * (a ? 0.5f : 1.0f);
                float acc = 0.0f;
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if ((!(q & 1) || x) && (!(q & 2) || b) && (!(q & 4) || a)) acc = fmaf(w, v[q][c], acc);
                if (d[row][3 * x + c] != 0.0f) m[row][3 * x + c] += acc;
            }
        if (has_x) {
#pragma unroll
            for (int h = 0; h < 3; h++)
                *reinterpret_cast<float2 *>(mx + o + 2 * h) = make_float2(m[row][2 * h], m[row][2 * h + 1]);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) mx[o + c] = m[row][c];
        }
    }
}

// coarse moduli: E_c = 2 mean(E of the 8 children); the factor 2 is the
// element-size scaling of the 3D stiffness (K(2h) = 2 K(h)), so every level
// uses the fine-grid reference stiffness K0.  The last element of an odd direction
// reaches one fine element beyond the grid: those children count as void (0).
__global__ void mg_coarsen_kernel(const MfProblem *__restrict__ probs, int plo,
                                  float *__restrict__ E32) {
    const MfProblem C = probs[plo + blockIdx.y];
    const MfProblem F = probs[C.fine];
    const int64_t ne = (int64_t)C.nx * C.ny * C.nz;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int ex = (int)(e % C.nx), ey = (int)((e / C.nx) % C.ny), ez = (int)(e / ((int64_t)C.nx * C.ny));
        float s = 0.0f;
        for (int dz = 0; dz < 2; dz++)
            for (int dy = 0; dy < 2; dy++)
                for (int dx = 0; dx < 2; dx++)
                    if (2 * ex + dx < F.nx && 2 * ey + dy < F.ny && 2 * ez + dz < F.nz)
                        s += E32[F.elem_off + ((int64_t)(2 * ez + dz) * F.ny + 2 * ey + dy) * F.pitch_e + 2 * ex + dx];
        E32[C.elem_off + ((int64_t)ez * C.ny + ey) * C.pitch_e + ex] = 0.25f * s;
    }
}

// ------------------------------------------------------------- bottom V-cycle
// The small coarse levels of a design (from its chain head down to its coarsest
// grid) are solved in one launch, entirely in shared memory, in FP32 on the CUDA
// cores: the same Chebyshev-Jacobi smoothers, residuals, restriction and
// prolongation as the level-by-level launches above, without one launch per level
// operation (mg_bottom_cluster_kernel).
//
// Direct coarse solve: the coarsest grid of a bottom chain, when it has at most
// kCoarseDirectMax dofs, is solved exactly with the inverse of its assembled
// operator (FP32, formed on the device by mg_coarse_inverse_kernel) instead of a
// Chebyshev smoother of degree cdeg: one matrix-vector product instead of cdeg - 1
// operator applications, each a barrier round.  The operator is assembled from
// the level's moduli and K0 like the level operators (Dirichlet dofs: identity
// rows and zero columns), so the inverse is symmetric and the V-cycle stays a
// fixed symmetric preconditioner.
constexpr int kBottomSmemMax = 200 * 1024;
// Nodes of the largest level that a batched design's chain starts at; a design of any batch
// has the same chain.
constexpr int kBatchMaxHeadNodes = 1024;

struct BottomCheb {
    float inv_theta_s, inv_theta_c;
    float c1s[32], c2s[32], c1c[32], c2c[32];
};

// FP32 inverse of a chain's coarsest-grid operator (the direct coarse solve), one
// CTA per chain, formed whenever the chain's moduli change.  The operator is
// assembled from K0 and the level's moduli (one thread per row, the node's
// elements in a fixed order; Dirichlet rows and columns replaced by the identity;
// the upper triangle taken for both halves), padded to kCoarseDirectMax with the
// identity and inverted in place by the symmetric sweep operator (Goodnight,
// "A tutorial on the SWEEP operator", 1979): sweeping pivot k maps
// a_ij -> a_ij - a_ik a_kj / a_kk (i, j != k), a_ik -> a_ik / a_kk and
// a_kk -> -1 / a_kk; sweeping every pivot leaves -A^-1.  Each thread keeps a 6 x 6
// tile of the lower triangle in registers (the upper one is its mirror image, so
// the stored inverse is exactly symmetric and the V-cycle stays a fixed symmetric
// preconditioner).  A node's three pivots are swept between two barriers: every
// thread forms the second and third pivot row at its rows and columns from the
// three rows as they were before the node (the same operations in the same order
// as pivot by pivot).  Bound by the barriers and the chain of three reciprocals:
// 135 dofs 137 us with a barrier per pivot and both triangles kept, 76 us so.
// No pivoting: the pivots of a symmetric positive definite matrix are positive.  A
// pivot that is not (a singular or indefinite coarse operator) clears coarse_ok and
// the bottom kernel smooths that chain's coarsest grid instead.
constexpr int kCoarseTile = 6;
constexpr int kCoarseTiles = kCoarseDirectMax / kCoarseTile;
constexpr int kCoarseInvTiles = kCoarseTiles * (kCoarseTiles + 1) / 2;
constexpr int kCoarseInvThreads = (kCoarseInvTiles + 31) / 32 * 32;
constexpr int kCoarseMaxElems = 64;  // nodes <= kCoarseDirectMax / 3 = 48, so elements < 48
constexpr int kCoarsePitch = kCoarseDirectMax + 1;  // odd: a column's words lie in different banks
constexpr int kCoarseInvSmem =
    (kCoarseDirectMax * kCoarsePitch + 576 + kCoarseMaxElems + 7 * kCoarseDirectMax) * 4;
static_assert(kCoarseDirectMax % kCoarseTile == 0 && kCoarseTile % 3 == 0, "whole nodes per tile, whole tiles");

__global__ void __launch_bounds__(kCoarseInvThreads, 1) mg_coarse_inverse_kernel(
    const MfProblem *__restrict__ probs, const int *__restrict__ heads, const int *__restrict__ list,
    const float *__restrict__ E32, const float *__restrict__ dinv, const double *__restrict__ K0,
    const int64_t *__restrict__ coarse_off, float *__restrict__ coarse_inv, int *__restrict__ coarse_ok) {
    constexpr int NP = kCoarseDirectMax, T = kCoarseTile, LD = kCoarsePitch;
    extern __shared__ __align__(16) float sci[];
    float *sA = sci;              // assembled operator, rows of LD words
    float *sK = sA + NP * LD;     // K0 (576)
    float *sE = sK + 576;         // the level's moduli
    float *sv = sE + kCoarseMaxElems;  // three pivot rows, double-buffered (2 x 3 x NP)
    int *sfix = reinterpret_cast<int *>(sv + 6 * NP);
    const int h = list[blockIdx.x];
    const int64_t off = coarse_off[h];
    if (off < 0) return;
    int c = heads[h];
    while (probs[c].coarse >= 0) c = probs[c].coarse;
    const MfProblem C = probs[c];
    const int nd = 3 * C.NX * C.NY * C.NZ, ne = C.nx * C.ny * C.nz;
    if (nd > NP || ne > kCoarseMaxElems) {  // not a direct chain (the host never lists one)
        if (threadIdx.x == 0) coarse_ok[h] = 0;
        return;
    }
    const int tid = threadIdx.x;
    for (int i = tid; i < 576; i += kCoarseInvThreads) sK[i] = (float)K0[i];
    for (int e = tid; e < ne; e += kCoarseInvThreads) {
        const int ex = e % C.nx, ey = (e / C.nx) % C.ny, ez = e / (C.nx * C.ny);
        sE[e] = E32[C.elem_off + ((int64_t)ez * C.ny + ey) * C.pitch_e + ex];
    }
    for (int q = tid; q < nd; q += kCoarseInvThreads) {
        const int n = q / 3, cq = q - 3 * n;
        const int i = n % C.NX, j = (n / C.NX) % C.NY, k = n / (C.NX * C.NY);
        sfix[q] = dinv[dof_index(C, i, j, k, cq)] == 0.0f;
    }
    for (int i = tid; i < nd * LD; i += kCoarseInvThreads) sA[i] = 0.0f;
    __syncthreads();
    // a thread per row and column component
    for (int t = tid; t < 3 * nd; t += kCoarseInvThreads) {
        const int cb = t / nd, q = t - cb * nd;
        float *row = sA + q * LD + cb;
        const int n = q / 3, cq = q - 3 * n;
        const int i = n % C.NX, jj = (n / C.NX) % C.NY, k = n / (C.NX * C.NY);
        for (int a = 0; a < 8; a++) {
            int dx, dy, dz;
            corner_bits(a, dx, dy, dz);
            const int ex = i - dx, ey = jj - dy, ez = k - dz;
            if (ex < 0 || ey < 0 || ez < 0 || ex >= C.nx || ey >= C.ny || ez >= C.nz) continue;
            const float e = sE[ex + C.nx * (ey + C.ny * ez)];
#pragma unroll
            for (int bc = 0; bc < 8; bc++) {
                int bx, by, bz;
                corner_bits(bc, bx, by, bz);
                const int m = (ex + bx) + C.NX * ((ey + by) + C.NY * (ez + bz));
                row[3 * m] = fmaf(e, sK[(3 * a + cq) * 24 + 3 * bc + cb], row[3 * m]);
            }
        }
    }
    __syncthreads();
    // tile (ti, tj), tj <= ti, of the lower triangle, numbered row by row
    int ti = (int)((sqrtf(8.0f * tid + 1.0f) - 1.0f) * 0.5f);
    while (ti * (ti + 1) / 2 > tid) ti--;
    while ((ti + 1) * (ti + 2) / 2 <= tid) ti++;
    const int tj = tid - ti * (ti + 1) / 2, i0 = ti * T, j0 = tj * T;
    const bool mine = tid < kCoarseInvTiles;
    float2 a[T][T / 2];
#pragma unroll
    for (int r = 0; r < T; r++)
#pragma unroll
        for (int cc = 0; cc < T; cc++) {
            const int i = i0 + r, j = j0 + cc;
            float v = i == j ? 1.0f : 0.0f;
            if (mine && i < nd && j < nd && !sfix[i] && !sfix[j]) v = i <= j ? sA[i * LD + j] : sA[j * LD + i];
            (cc & 1 ? a[r][cc / 2].y : a[r][cc / 2].x) = v;
        }
    // the three rows from pivot k on into buffer `buf`: from the tiles of the row and, mirrored, of the column
    auto publish = [&](int k, int buf) {
        float *v = sv + buf * 3 * NP;
        const int kr = k - i0, kc = k - j0;
        if (!mine) return;
        if (kr == 0 || kr == 3) {
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int cc = 0; cc < T / 2; cc++) {
                    const float2 w = kr == 0 ? a[q][cc] : a[q + 3][cc];
                    v[q * NP + j0 + 2 * cc] = w.x;
                    v[q * NP + j0 + 2 * cc + 1] = w.y;
                }
        } else if (kc == 0 || kc == 3) {
#pragma unroll
            for (int r = 0; r < T; r++) {
                v[i0 + r] = kc == 0 ? a[r][0].x : a[r][1].y;
                v[NP + i0 + r] = kc == 0 ? a[r][0].y : a[r][2].x;
                v[2 * NP + i0 + r] = kc == 0 ? a[r][1].x : a[r][2].y;
            }
        }
    };
    publish(0, 0);
    __syncthreads();
    int ok = 1, cur = 0;
    for (int k = 0; k < nd; k += 3) {
        const float *v0 = sv + cur * 3 * NP, *v1 = v0 + NP, *v2 = v1 + NP;
        // the node's 3 x 3 block: its pivots, the same values in every thread (the exit is uniform)
        const float c01 = v0[k + 1], c02 = v0[k + 2];
        const float d0 = v0[k], p0 = 1.0f / d0;
        const float d1 = fmaf(-(c01 * c01), p0, v1[k + 1]), p1 = 1.0f / d1;
        const float c12 = fmaf(-(c01 * c02), p0, v1[k + 2]);
        const float d2 = fmaf(-(c12 * c12), p1, fmaf(-(c02 * c02), p0, v2[k + 2])), p2 = 1.0f / d2;
        if (!(d0 > 0.0f) || !isfinite(d0) || !(d1 > 0.0f) || !isfinite(d1) || !(d2 > 0.0f) || !isfinite(d2)) {
            ok = 0;
            break;
        }
        if (mine) {
            // the pivot rows at index i, each as it is when its pivot is swept
            auto rows_at = [&](int i, float &x0, float &x1, float &x2) {
                x0 = v0[i];
                x1 = i == k ? c01 * p0 : fmaf(-(c01 * x0), p0, v1[i]);
                x2 = i == k ? c02 * p0 : fmaf(-(c02 * x0), p0, v2[i]);
                x2 = i == k + 1 ? c12 * p1 : fmaf(-(c12 * x1), p1, x2);
            };
            // a swept row or column becomes v p: 0 - (-1 v) p, with the factor -1 at the swept
            // index and the tile's entries there set to 0 (few threads, in nearly every warp)
            const int kr = k - i0, kc = k - j0;
            float vi[3][T];
            float2 vj[3][T / 2];
#pragma unroll
            for (int r = 0; r < T; r++) {
                rows_at(i0 + r, vi[0][r], vi[1][r], vi[2][r]);
                vi[r % 3][r] = kr == r - r % 3 ? -1.0f : vi[r % 3][r];
            }
#pragma unroll
            for (int cc = 0; cc < T; cc++) {
                float x[3];
                rows_at(j0 + cc, x[0], x[1], x[2]);
                x[cc % 3] = kc == cc - cc % 3 ? -1.0f : x[cc % 3];
#pragma unroll
                for (int q = 0; q < 3; q++) (cc & 1 ? vj[q][cc / 2].y : vj[q][cc / 2].x) = x[q];
            }
            const bool swept = kr == 0 || kr == 3 || kc == 0 || kc == 3;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                if (swept) {
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        const int at = 3 * half + q;
                        if (kr == 3 * half)
#pragma unroll
                            for (int cc = 0; cc < T / 2; cc++) a[at][cc] = make_float2(0.0f, 0.0f);
                        if (kc == 3 * half)
#pragma unroll
                            for (int r = 0; r < T; r++) (at & 1 ? a[r][at / 2].y : a[r][at / 2].x) = 0.0f;
                    }
                }
                const float p = q == 0 ? p0 : q == 1 ? p1 : p2;
                const float2 np = make_float2(-p, -p);
#pragma unroll
                for (int r = 0; r < T; r++)
#pragma unroll
                    for (int cc = 0; cc < T / 2; cc++)
                        a[r][cc] = __ffma2_rn(__fmul2_rn(make_float2(vi[q][r], vi[q][r]), vj[q][cc]), np, a[r][cc]);
            }
        }
        cur ^= 1;
        if (k + 3 < nd) publish(k + 3, cur);
        __syncthreads();
    }
    if (tid == 0) coarse_ok[h] = ok;
    if (!ok || !mine) return;
    float *out = coarse_inv + off;
#pragma unroll
    for (int r = 0; r < T; r++)
#pragma unroll
        for (int cc = 0; cc < T; cc++) {
            const int i = i0 + r, j = j0 + cc;
            if (i >= nd || j >= nd) continue;
            const float w = cc & 1 ? a[r][cc / 2].y : a[r][cc / 2].x;
            out[i * nd + j] = -w;
            if (ti != tj) out[j * nd + i] = -w;
        }
}

// ------------------------------------------------- bottom V-cycle on a cluster
// A chain's V-cycle on a thread-block cluster of up to 16 CTAs: all 16 for a single
// design, whose chain can start at a larger level, for a small design at its own
// grid (the whole V-cycle and r.z are then one kernel; 16x8x8, solve with
// sensitivities: 2.80 -> 2.24 ms); in a batch as many as leave every chain its
// cluster at the same time.  CTA r owns the
// nodes [r chunk, (r + 1) chunk) of every level of the chain and keeps their x, b,
// r, d, y in its shared memory, with D^-1 of the nodes and the moduli of the
// elements around them; a phase reads other CTAs' nodes through distributed shared
// memory (mapa + ld.shared::cluster) and a cluster barrier (release / acquire)
// separates the phases.  Global memory is touched only at the start (rhs, tables)
// and at the end (the head's correction).  Every dof is computed by one thread in a
// fixed order whatever the cluster size, so the correction does not depend on it
// (r.z of a chain from the own grid does, in its rounding).  Batched chains: 58
// problems 68 us a launch with one CTA a chain, K0 and the operand both read from
// shared memory, 41 us with two.
constexpr int kClusterThreads = 512;
// Nodes of the largest level that a chain may start at, the design's own grid included: up to here
// the cluster's phases on 16 SMs beat the level kernels on all of them (us an iteration of single
// designs, chain from the own grid / level by level: 1,377 nodes 57.5 / 72.1, 3,509 78.5 / 80.6,
// 4,225 76.3 / 80.3, 4,913 77.6 / 83.0; 5,577 85.3 / 84.8).  The line also ends the search below the
// own grid, where the chain does not take r.z over and the two lie closer (chain from the level of these
// nodes / from the one below it: 1,377 112.6 / 122.1, 2,420 89.8 / 95.9, 3,312 98.9 / 98.5, 3,432
// 144.8 / 145.3, 3,549 99.9 / 99.0, 4,225 103.5 / 99.7).
constexpr int kClusterMaxHeadNodes = 5000;
constexpr int kClusterMax = 16;
constexpr int kClusterK0 = 576;  // K0 regrouped by the lanes' corners (floats)

__device__ __forceinline__ unsigned cluster_ctarank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_nctarank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// n / d for the level's small divisors by one rounded product (exact for every n
// of the level: the host checks each reciprocal against integer division)
__device__ __forceinline__ int cl_div(int n, float r) {
    return __float2int_rz(__fmul_rn(__fadd_rn(__int2float_rn(n), 0.5f), r));
}
__device__ __forceinline__ void cl_ijk(const ClusterLevel &L, int n, int &i, int &j, int &k) {
    k = cl_div(n, L.rNXY);
    const int rem = n - k * L.NXY;
    j = cl_div(rem, L.rNX);
    i = rem - j * L.NX;
}
// address in the cluster's shared memory of word `off` of CTA `rank`'s dynamic shared memory, and a
// load from it (volatile: the barriers between the phases order the loads, and loads that follow one
// another are in flight together)
__device__ __forceinline__ uint32_t cl_addr(const float *sm, int off, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(sm + off)), "r"(rank));
    return r;
}
__device__ __forceinline__ float cl_load(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// component c of node n of the vector whose slabs sit at offset `slab` in every CTA
__device__ __forceinline__ float cl_get(const float *sm, int slab, const ClusterLevel &L, int n, int c) {
    const int owner = cl_div(n, L.rchunk);
    return cl_load(cl_addr(sm, slab + (n - owner * L.chunk) * 3 + c, owner));
}

enum { kClX = 0, kClB, kClR, kClD, kClY };
__device__ __forceinline__ int cl_slab(const ClusterLevel &L, int v) { return L.s_vec + v * 3 * L.chunk; }

// One phase of the cluster V-cycle on level L: y = A in with eight lanes per node
// (lane dx + 2 dy + 4 dz forms the node's rows of the element node - d, the partial
// sums meet in a fixed xor butterfly), the elementwise update that follows it done by the lanes that
// hold each dof's sum, so that the phase needs no second barrier:
//   step 0, residual:             in = x;   r = b - y
//   step 1, first smoothing step: in = D^-1 rin theta (formed while staging rin);
//           r0 = rin, d0 = D^-1 r0 theta, x0 = d0 or x + d0, then the step-1 update
//   step 2, later smoothing step: in = d;   r -= y, d' = c1 d + c2 D^-1 r, x += d'
// (0 on Dirichlet dofs throughout).  The operand over the CTA's nodes and their
// one-layer halo (nodes n0 - H .. n1 - 1 + H, H = NX NY + NX + 1) is first staged
// in shared memory; no phase writes a slab that another CTA reads in it (the
// callers rotate r, d and y).
struct ClusterStep {
    int in, b, r_src, d_src, r_dst, d_dst, x;  // slabs (offsets in the CTA's shared memory)
    bool x0_zero, staged;                      // staged: the operand is in place already
    float inv_theta, c1, c2;
};

// The phases are short (one to four nodes a lane) and follow one another through a cluster barrier, so
// each is bound by its chain of dependent instructions, and what is the same in every phase is formed
// once, before the kernel waits for its predecessor: a lane's corner, and with it its 3 x 24 row block
// Kr of K0 (registers: 24 shared-memory loads a node and lane where there were 48); per level the
// cluster addresses that the staging reads and each node's elements (shared memory).  Inlined once
// per kind of phase: the V-cycle below is one loop over its phases.  With K0 and the operand both read
// from shared memory and the indices formed in every phase, 90x46x38 (a chain from 3,432 nodes) took
// 7.30 ms a solve with sensitivities where it takes 6.52, 64x32x32 (from 1,377) 7.21 and 6.91.
template <int STEP>
__device__ __forceinline__ void cl_step(const ClusterLevel &L, float *sm, const float (&Kr)[72], float *stage,
                                        const ClusterStep &S, int rank) {
    const int nn = L.NXY * L.NZ, NX = L.NX, NXY = L.NXY;
    const int n0 = rank * L.chunk, n1 = min(nn, n0 + L.chunk);
    const int H = NXY + NX + 1, nlo = max(0, n0 - H);
    const float *dinvL = sm + L.s_dinv, *EL = sm + L.s_E;
    if (n0 < n1 && !S.staged) {
        const int cnt = 3 * (min(nn, n1 + H) - nlo), slab = 4 * (S.in - L.s_vec);
        const int *addr = reinterpret_cast<const int *>(sm) + L.s_addr;
        // up to three words a thread in flight together: one round trip through the cluster's network
        for (int t = threadIdx.x; t < cnt; t += 3 * kClusterThreads) {
            const int t1 = t + kClusterThreads, t2 = t1 + kClusterThreads;
            float v0 = cl_load(addr[t] + slab), v1 = 0.0f, v2 = 0.0f;
            if (t1 < cnt) v1 = cl_load(addr[t1] + slab);
            if (t2 < cnt) v2 = cl_load(addr[t2] + slab);
            stage[t] = STEP == 1 ? dinvL[t] * v0 * S.inv_theta : v0;
            if (t1 < cnt) stage[t1] = STEP == 1 ? dinvL[t1] * v1 * S.inv_theta : v1;
            if (t2 < cnt) stage[t2] = STEP == 1 ? dinvL[t2] * v2 * S.inv_theta : v2;
        }
    }
    __syncthreads();
    const int *elems = reinterpret_cast<const int *>(sm) + L.s_elem;
    const int corner = threadIdx.x & 7, dx = corner & 1, dy = (corner >> 1) & 1, dz = corner >> 2;
    const int corner_u = 3 * (dx + NX * dy + NXY * dz), corner_e = dx + L.nx * (dy + L.ny * dz);
    const int own = n1 - n0;
    for (int w = (threadIdx.x >> 5) * 4; w < own; w += kClusterThreads / 8) {  // four nodes a warp
        const int n = w + ((threadIdx.x >> 3) & 3);
        const int el = n < own ? elems[n] : 0;
        const bool mine = n < own && corner < 3;
        const int lo = mine ? 3 * n + corner : 0;
        const float dn = dinvL[3 * (n0 - nlo) + lo];
        const float rv0 = sm[(STEP == 0 ? S.b : S.r_src) + lo];
        const float xv = STEP == 0 || (STEP == 1 && S.x0_zero) ? 0.0f : sm[S.x + lo];
        const float dv0 = STEP == 2 ? sm[S.d_src + lo] : 0.0f;
        float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
        if ((el >> corner) & 1) {
            const float e = EL[(el >> 8) - corner_e];
            const float *u0p = stage + 3 * (n0 - nlo + n) - corner_u;
            float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
#pragma unroll
            for (int bc = 0; bc < 8; bc++) {
                int bx, by, bz;
                corner_bits(bc, bx, by, bz);
                const float *u = u0p + 3 * (bx + NX * by + NXY * bz);
                const float *kb = Kr + 9 * bc;
                s0 = fmaf(kb[2], u[2], fmaf(kb[1], u[1], fmaf(kb[0], u[0], s0)));
                s1 = fmaf(kb[5], u[2], fmaf(kb[4], u[1], fmaf(kb[3], u[0], s1)));
                s2 = fmaf(kb[8], u[2], fmaf(kb[7], u[1], fmaf(kb[6], u[0], s2)));
            }
            a0 = e * s0;
            a1 = e * s1;
            a2 = e * s2;
        }
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, off);
            a1 += __shfl_xor_sync(0xffffffffu, a1, off);
            a2 += __shfl_xor_sync(0xffffffffu, a2, off);
        }
        if (mine) {
            const float y = dn == 0.0f ? 0.0f : (corner == 0 ? a0 : (corner == 1 ? a1 : a2));
            if (STEP == 0) {
                sm[S.r_dst + lo] = dn == 0.0f ? 0.0f : rv0 - y;
            } else {
                const float d0 = STEP == 1 ? dn * rv0 * S.inv_theta : dv0;
                const float x0 = STEP == 1 ? (S.x0_zero ? d0 : xv + d0) : xv;
                const float rv = rv0 - y;
                const float dv = fmaf(S.c1, d0, S.c2 * dn * rv);
                sm[S.r_dst + lo] = rv;
                sm[S.d_dst + lo] = dv;
                sm[S.x + lo] = x0 + dv;
            }
        }
    }
}

// Chebyshev-Jacobi smoothing of degree 1 for rhs rin: x (+)= D^-1 rin theta, no phase
__device__ __noinline__ void cl_smooth1(const ClusterLevel &L, float *sm, int rin, bool x0_zero,
                                        float inv_theta, int rank) {
    float *x = sm + cl_slab(L, kClX);
    const int nn = L.NXY * L.NZ;
    const int n0 = rank * L.chunk, nown = max(0, min(nn, n0 + L.chunk) - n0);
    const float *dinvL = sm + L.s_dinv + 3 * (n0 - max(0, n0 - (L.NXY + L.NX + 1)));
    for (int q = threadIdx.x; q < 3 * nown; q += kClusterThreads) {
        const float dv = dinvL[q] * sm[rin + q] * inv_theta;
        x[q] = x0_zero ? dv : x[q] + dv;
    }
    cluster_barrier();
}

// restriction: cluster address of the residual at fine neighbour `lane` (< 27) of coarse node n, 0 if none
__device__ __forceinline__ int cl_fine_addr(const float *sm, const ClusterLevel &F, const ClusterLevel &C, int n, int lane) {
    int I, J, K;
    cl_ijk(C, n, I, J, K);
    const int ii = 2 * I + lane % 3 - 1, jj = 2 * J + lane / 3 % 3 - 1, kk = 2 * K + lane / 9 - 1;
    if (lane >= 27 || ii < 0 || ii >= F.NX || jj < 0 || jj >= F.NY || kk < 0 || kk >= F.NZ) return 0;
    const int nf = ii + F.NX * (jj + F.NY * kk), owner = cl_div(nf, F.rchunk);
    return (int)cl_addr(sm, cl_slab(F, kClR) + 3 * (nf - owner * F.chunk), owner);
}

__global__ void __launch_bounds__(kClusterThreads, 1) mg_bottom_cluster_kernel(
    const ClusterChain *__restrict__ chains, MfState *states, const float *__restrict__ E32,
    const float *__restrict__ dinv, const float *__restrict__ rhs, float *__restrict__ mx, bool from_root,
    const float *__restrict__ k0f, const __grid_constant__ BottomCheb cc, int sdeg, int cdeg,
    const int64_t *__restrict__ coarse_off, const float *__restrict__ coarse_inv, const int *__restrict__ coarse_ok) {
    // D^-1, the moduli and the coarse inverse were formed before this graph ran
    // (activation); they are loaded while the preceding kernel finishes, the
    // head's rhs and the solver state only after it
    pdl_trigger();
    extern __shared__ __align__(16) float sm[];  // stage, per level: D^-1, E, slabs, tables
    __shared__ double s_rz[kClusterMax], s_red[kClusterThreads / 32];
    const int csize = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // (in shared memory: read by level from the constant bank, the tables slowed every phase)
    __shared__ ClusterChain ch;
    const int chain = blockIdx.x / csize;
    for (int i = threadIdx.x; i < (int)(sizeof(ClusterChain) / 4); i += kClusterThreads)
        reinterpret_cast<int *>(&ch)[i] = reinterpret_cast<const int *>(chains + chain)[i];
    __syncthreads();
    const int m = ch.m;
    int *smi = reinterpret_cast<int *>(sm);
    // D^-1 and E of every level (compact order) as far as this CTA's phases read them: its
    // nodes and their halo, the elements around its nodes.  Copied asynchronously: the round
    // trips of all levels overlap (one after another they took 9 to 12 thousand cycles).
    auto copy_word = [&](int off, const float *src) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(sm + off)), "l"(src) : "memory");
    };
    for (int l = 0; l < m; l++) {
        const ClusterLevel &L = ch.L[l];
        const int nn = L.NXY * L.NZ, H = L.NXY + L.NX + 1;
        if (l < m - 1) {  // where each warp's lanes read for its first coarse node (a CTA without
                          // nodes of this level may own coarse ones)
            const ClusterLevel &C = ch.L[l + 1];
            const int n = rank * C.chunk + warp;
            smi[L.s_fine + threadIdx.x] =
                n < min(C.NXY * C.NZ, (rank + 1) * C.chunk) ? cl_fine_addr(sm, L, C, n, lane) : 0;
        }
        const int n0 = rank * L.chunk, n1 = min(nn, n0 + L.chunk), nlo = max(0, n0 - H);
        if (n0 >= n1) continue;
        const int cnt = 3 * (min(nn, n1 + H) - nlo);
#pragma unroll 2
        for (int t = threadIdx.x; t < cnt; t += kClusterThreads) {
            const int n = nlo + t / 3, c = t - 3 * (t / 3);
            int i, j, k;
            cl_ijk(L, n, i, j, k);
            const int idx = (k * L.NY + j) * L.pitch + 3 * i + c;
            copy_word(L.s_dinv + t, dinv + L.dof_off + idx);
            if (l == 0) smi[ch.s_idx + t] = idx;
            const int owner = cl_div(n, L.rchunk);
            smi[L.s_addr + t] = (int)cl_addr(sm, L.s_vec + 3 * (n - owner * L.chunk) + c, owner);
        }
        const int nxy = L.nx * L.ny;
        const float rnx = 1.0f / (float)L.nx, rnxy = 1.0f / (float)nxy;  // exact quotients: fewer than 2^13 elements
        const int e1 = nxy * min(L.nz, cl_div(n1 - 1, L.rNXY) + 1);
        for (int e = nxy * max(0, cl_div(n0, L.rNXY) - 1) + threadIdx.x; e < e1; e += kClusterThreads) {
            const int ez = cl_div(e, rnxy), er = e - ez * nxy, ey = cl_div(er, rnx), ex = er - ey * L.nx;
            copy_word(L.s_E + e, E32 + L.elem_off + ((int64_t)ez * L.ny + ey) * L.pitch_e + ex);
        }
        for (int n = n0 + threadIdx.x; n < n1; n += kClusterThreads) {
            // the element at corner 0 and which of the eight lie in the grid
            int i, j, k;
            cl_ijk(L, n, i, j, k);
            const int mx = (i < L.nx ? 0x55 : 0) | (i > 0 ? 0xaa : 0);
            const int my = (j < L.ny ? 0x33 : 0) | (j > 0 ? 0xcc : 0);
            const int mz = (k < L.nz ? 0x0f : 0) | (k > 0 ? 0xf0 : 0);
            smi[L.s_elem + n - n0] = (i + L.nx * (j + L.ny * k)) << 8 | (mx & my & mz);
            if (l < m - 1) {  // its first parent among those this CTA stages, and which others it has
                const ClusterLevel &C = ch.L[l + 1];
                const int kc = (k >> 1) - (cl_div(n0, L.rNXY) >> 1);
                smi[L.s_par + n - n0] = ((i >> 1) + C.NX * (j >> 1) + C.NXY * kc) << 3 | (k & 1) << 2 | (j & 1) << 1 | (i & 1);
            }
        }
    }
    float Kr[72];  // rows of this lane's corner, [node][row][component]
    {
        const float4 *src = reinterpret_cast<const float4 *>(k0f + 72 * (threadIdx.x & 7));
#pragma unroll
        for (int i = 0; i < 18; i++) {
            const float4 v = __ldg(src + i);
            Kr[4 * i] = v.x; Kr[4 * i + 1] = v.y; Kr[4 * i + 2] = v.z; Kr[4 * i + 3] = v.w;
        }
    }
    // the direct solve's rows of this CTA (one warp per row), loaded now
    const ClusterLevel &Lc = ch.L[m - 1];
    const int64_t inv_off = coarse_ok[chain] ? coarse_off[chain] : -1;
    const int nnc = Lc.NXY * Lc.NZ, ndc = 3 * nnc;
    const int c0 = rank * Lc.chunk, crows = 3 * max(0, min(nnc, c0 + Lc.chunk) - c0);
    constexpr int kInvPer = (kCoarseDirectMax + 31) / 32;
    float inv[kInvPer];
#pragma unroll
    for (int t = 0; t < kInvPer; t++) {
        const int r = lane + 32 * t;
        inv[t] = (inv_off >= 0 && warp < crows && r < ndc)
                     ? __ldg(coarse_inv + inv_off + (int64_t)(3 * c0 + warp) * ndc + r)
                     : 0.0f;
    }
    const ClusterLevel &L0 = ch.L[0];
    const int own0 = rank * L0.chunk, nown0 = max(0, min(L0.NXY * L0.NZ, own0 + L0.chunk) - own0);
    const int *idx0 = smi + ch.s_idx + 3 * (own0 - max(0, own0 - (L0.NXY + L0.NX + 1)));  // of the own dofs
    rhs += L0.dof_off;
    mx += L0.dof_off;
    float *b0 = sm + cl_slab(L0, kClB);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    pdl_wait();
    // The first phase's operand comes from the rhs in global memory and not from other CTAs, with
    // the CTA's own rhs among it; loaded along with the state
    const bool first_staged = m > 1 ? sdeg >= 2 : inv_off < 0 && cdeg >= 2;
    {
        const int nlo = max(0, own0 - (L0.NXY + L0.NX + 1)), at = 3 * (own0 - nlo);
        const int cnt = nown0 ? 3 * (min(L0.NXY * L0.NZ, own0 + L0.chunk + L0.NXY + L0.NX + 1) - nlo) : 0;
        const float inv_theta = m > 1 ? cc.inv_theta_s : cc.inv_theta_c;
        const int *idx = smi + ch.s_idx;
        const int done = states[ch.root].done;
        float v[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int t = threadIdx.x + k * kClusterThreads;
            v[k] = t < cnt ? __ldcg(rhs + idx[t]) : 0.0f;
        }
        // the same state in every CTA of the cluster: all return, or none
        if (done) return;
        auto place = [&](int t, float w) {
            sm[ch.s_stage + t] = sm[L0.s_dinv + t] * w * inv_theta;
            if ((unsigned)(t - at) < (unsigned)(3 * nown0)) b0[t - at] = w;
        };
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (const int t = threadIdx.x + k * kClusterThreads; t < cnt) place(t, v[k]);
        for (int t = threadIdx.x + 3 * kClusterThreads; t < cnt; t += kClusterThreads) place(t, __ldcg(rhs + idx[t]));
    }
    if (!first_staged) cluster_barrier();
    // down the chain: smooth, residual, restrict; the coarsest grid; up: prolong, residual, smooth
    for (int it = 0; it < 2 * m - 1; it++) {
        const int l = it < m ? it : 2 * m - 2 - it;
        const bool down = it < m - 1, up = it >= m;
        const ClusterLevel &F = ch.L[l], &C = ch.L[min(l + 1, m - 1)];
        const int nnF = F.NXY * F.NZ, n0 = rank * F.chunk, nown = max(0, min(nnF, n0 + F.chunk) - n0);
        const float *dinvF = sm + F.s_dinv + 3 * (n0 - max(0, n0 - (F.NXY + F.NX + 1)));  // own dofs
        if (up) {
            // the coarse planes around the own nodes first (the address of a parent by itself, up to
            // eight a dof, cost more than this copy)
            const int kc0 = cl_div(n0, F.rNXY) >> 1, kc1 = min((cl_div(n0 + max(nown, 1) - 1, F.rNXY) + 1) >> 1, C.NZ - 1);
            float *stage = sm + ch.s_stage, *xF = sm + cl_slab(F, kClX);
            const int cnt = nown > 0 ? 3 * C.NXY * (kc1 - kc0 + 1) : 0;
            for (int t = threadIdx.x; t < cnt; t += kClusterThreads)
                stage[t] = cl_get(sm, cl_slab(C, kClX), C, C.NXY * kc0 + t / 3, t - 3 * (t / 3));
            __syncthreads();
            for (int q = threadIdx.x; q < 3 * nown; q += kClusterThreads) {
                if (dinvF[q] == 0.0f) continue;
                const int par = smi[F.s_par + q / 3], ox = par & 1, oy = (par >> 1) & 1, oz = (par >> 2) & 1;
                const float w = (ox ? 0.5f : 1.0f) * (oy ? 0.5f : 1.0f) * (oz ? 0.5f : 1.0f);
                const float *xc = stage + 3 * (par >> 3) + q % 3;
                float acc = 0.0f;
#pragma unroll
                for (int t = 0; t < 8; t++) {  // the 1, 2, 4 or 8 parents in a fixed order
                    const int a = t >> 2, bb = (t >> 1) & 1, cc2 = t & 1;
                    if ((a == 0 || oz) && (bb == 0 || oy) && (cc2 == 0 || ox))
                        acc = fmaf(w, xc[3 * (cc2 + C.NX * bb + C.NXY * a)], acc);
                }
                xF[q] += acc;
            }
            cluster_barrier();
        } else if (!down && inv_off >= 0) {
            // the coarsest grid by the stored inverse: one warp per own row, partial sums met by
            // a fixed xor butterfly; the first pass uses the rows loaded at the start
            float *bc = sm + ch.s_stage, *xc = sm + cl_slab(Lc, kClX);
            for (int r = threadIdx.x; r < ndc; r += kClusterThreads) bc[r] = cl_get(sm, cl_slab(Lc, kClB), Lc, r / 3, r % 3);
            __syncthreads();
            for (int w0 = 0; w0 < crows; w0 += kClusterThreads / 32) {
                const int w = w0 + warp;
                if (w >= crows) break;  // whole warps leave together
                float sacc = 0.0f;
#pragma unroll
                for (int t = 0; t < kInvPer; t++) {
                    const int r = lane + 32 * t;
                    if (r < ndc) {
                        const float a = w0 == 0 ? inv[t] : __ldg(coarse_inv + inv_off + (int64_t)(3 * c0 + w) * ndc + r);
                        sacc = fmaf(a, bc[r], sacc);
                    }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) sacc += __shfl_xor_sync(0xffffffffu, sacc, off);
                if (lane == 0) xc[w] = dinvF[w] == 0.0f ? 0.0f : sacc;
            }
            cluster_barrier();
            continue;
        }
        const bool coarsest = !down && !up;
        const int deg = coarsest ? cdeg : sdeg;
        const int n_smooth = max(deg, 1) - 1, n_steps = n_smooth + (coarsest ? 0 : 1);
        const float inv_theta = coarsest ? cc.inv_theta_c : cc.inv_theta_s;
        const int bF = cl_slab(F, kClB);
        int r = cl_slab(F, kClR), d = cl_slab(F, kClD), sp = cl_slab(F, kClY);
        if (deg <= 1 && !up) cl_smooth1(F, sm, bF, true, inv_theta, rank);
        for (int s = 0; s < n_steps; s++) {
            const bool residual = down ? s == n_smooth : (up && s == 0);
            const int k = up ? s : s + 1;  // smoothing step
            ClusterStep S;
            S.x = cl_slab(F, kClX);
            S.inv_theta = inv_theta;
            S.x0_zero = !up;
            S.staged = it == 0 && s == 0 && first_staged;
            S.r_dst = S.r_src = r;
            S.d_dst = S.d_src = d;
            if (residual) {
                S.in = S.x;
                S.b = bF;
                S.r_dst = cl_slab(F, kClR);
                if (up) r = S.r_dst;
                cl_step<0>(F, sm, Kr, sm + ch.s_stage, S, rank);
            } else {
                S.c1 = coarsest ? cc.c1c[k] : cc.c1s[k];
                S.c2 = coarsest ? cc.c2c[k] : cc.c2s[k];
                if (k == 1) {
                    // reads the rhs at the neighbours: where it is r (post-smoothing on the residual),
                    // the new residual goes to the spare slab
                    S.in = S.r_src = up ? r : bF;
                    if (up) {
                        S.r_dst = sp;
                        sp = r;
                        r = S.r_dst;
                    }
                    cl_step<1>(F, sm, Kr, sm + ch.s_stage, S, rank);
                } else {
                    // reads d at the neighbours: the new direction goes to the spare slab
                    S.in = d;
                    S.d_dst = sp;
                    sp = d;
                    d = S.d_dst;
                    cl_step<2>(F, sm, Kr, sm + ch.s_stage, S, rank);
                }
            }
            cluster_barrier();
        }
        if (deg <= 1 && up) cl_smooth1(F, sm, r, false, inv_theta, rank);
        if (down) {
            // one warp per coarse node: lane t < 27 takes fine neighbour t (all three
            // components), the weighted values meet in a fixed xor butterfly
            const int nnC = C.NXY * C.NZ, m0 = rank * C.chunk, m1 = min(nnC, m0 + C.chunk);
            const float *dinvC = sm + C.s_dinv + 3 * (m0 - max(0, m0 - (C.NXY + C.NX + 1)));
            float *bC = sm + cl_slab(C, kClB);
            const int dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
            const float w = (dz ? 0.5f : 1.0f) * (dy ? 0.5f : 1.0f) * (dx ? 0.5f : 1.0f);
            for (int n = m0 + warp; n < m1; n += kClusterThreads / 32) {
                const uint32_t a = n == m0 + warp ? smi[F.s_fine + threadIdx.x] : cl_fine_addr(sm, F, C, n, lane);
                float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f;
                if (a) {
                    v0 = w * cl_load(a);
                    v1 = w * cl_load(a + 4);
                    v2 = w * cl_load(a + 8);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    v0 += __shfl_xor_sync(0xffffffffu, v0, off);
                    v1 += __shfl_xor_sync(0xffffffffu, v1, off);
                    v2 += __shfl_xor_sync(0xffffffffu, v2, off);
                }
                if (lane < 3) {
                    const float v = lane == 0 ? v0 : (lane == 1 ? v1 : v2);
                    bC[3 * (n - m0) + lane] = dinvC[3 * (n - m0) + lane] != 0.0f ? v : 0.0f;
                }
            }
            cluster_barrier();
        }
    }
    // the head's correction over this CTA's nodes back to the padded global layout
    const float *x0 = sm + cl_slab(L0, kClX);
    float rz = 0.0f;
    for (int q = threadIdx.x; q < 3 * nown0; q += kClusterThreads) {
        mx[idx0[q]] = x0[q];
        rz = fmaf(b0[q], x0[q], rz);
    }
    if (!from_root) return;
    // the whole V-cycle ran here: r.z and beta too (as mf_dot_rz_kernel)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) rz += __shfl_xor_sync(0xffffffffu, rz, off);
    if (lane == 0) s_red[warp] = (double)rz;
    __syncthreads();
    if (warp == 0) {
        double s = lane < kClusterThreads / 32 ? s_red[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) {
            uint32_t at_first;  // the same word of the cluster's first CTA
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at_first) : "r"(smem_u32(s_rz + rank)));
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at_first), "d"(s) : "memory");
        }
    }
    cluster_barrier();
    if (rank == 0 && warp == 0) {
        double s = lane < csize ? s_rz[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) finish_rz(states + ch.root, s);
    }
}

// The kernels of the refinement phases act on the few problems that are in the phase; their
// blocks walk only those problems' parts (chunks, bricks).  A walk over every part, each
// behind its table and state reads, cost a batch of 58 problems about 1 us a part and block.
//
// Calls body(part index) for the parts [begin, end) that range(p) gives of the problems p < n
// with in_phase(p), spread over the grid; every one of the block's NT threads calls it.
// Every block numbers the parts for itself, so in_phase must not change while the kernel runs.
template <int NT, typename InPhase, typename Range, typename Body>
__device__ __forceinline__ void for_active_parts(int n, InPhase in_phase, Range range, Body body) {
    if (n == 1) {  // no tables: they cost a single 16x8x8 or 48x24x24 solve 2 %
        if (!in_phase(0)) return;
        int begin, end;
        range(0, begin, end);
        for (int i = begin + blockIdx.x; i < end; i += gridDim.x) body(i);
        return;
    }
    __shared__ int s_end[NT], s_begin[NT], s_warp[NT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int start = blockIdx.x;  // of this window's numbering
    for (int p0 = 0; p0 < n; p0 += NT) {
        const int p = p0 + threadIdx.x;
        const bool in = p < n && in_phase(p);
        if (!__syncthreads_or(in)) continue;  // also: the previous window's tables are no longer read
        int begin = 0, end = 0;
        if (in) range(p, begin, end);
        int sum = end - begin;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        if (lane == 31) s_warp[w] = sum;
        __syncthreads();
        for (int k = 0; k < w; k++) sum += s_warp[k];
        s_end[threadIdx.x] = sum;
        s_begin[threadIdx.x] = begin;
        __syncthreads();
        const int total = s_end[NT - 1];
        for (; start < total; start += gridDim.x) {
            int lo = 0, hi = NT - 1;  // the first problem whose parts end beyond start
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_end[mid] > start) hi = mid;
                else lo = mid + 1;
            }
            body(s_begin[lo] + start - (lo ? s_end[lo - 1] : 0));
        }
        start -= total;
    }
}

// inner CG start (problems in INIT): b = scale r64 (unit norm), x = 0, r = b,
// z = D^-1 r, p0 = p1 = 0; moves the problem to CG
__global__ void __launch_bounds__(kThreads) mf_inner_init_kernel(
    const MfChunkDesc *__restrict__ chunks, int n_chunks, const MfProblem *__restrict__ probs,
    const double *__restrict__ r64, float *__restrict__ x, float *__restrict__ r,
    float *__restrict__ z, float *__restrict__ p0, float *__restrict__ p1,
    const float *__restrict__ dinv, MfState *states, double *__restrict__ chunk_part,
    double inner_rtol2, int maxit, int n_fine) {
    pdl_enter();
    __shared__ double red_sh[kThreads / 32];
    __shared__ int sh_last;
    for_active_parts<kThreads>(n_fine, [&](int p) { return states[p].resid != 0; },
                     [&](int p, int &begin, int &end) {
                         begin = probs[p].chunk_begin;
                         end = begin + probs[p].chunk_count;
                     }, [&](int ci) {
        const MfChunkDesc C = chunks[ci];
        MfState *st = states + C.prob;
        if (st->phase != kPhaseInit) return;  // finished by its residual
        const double scale = st->scale;
        float rz = 0.0f, rr = 0.0f;
        for (int64_t i = C.begin + threadIdx.x; i < C.end; i += kThreads) {
            const float bi = dinv[i] != 0.0f ? (float)(r64[i] * scale) : 0.0f;
            x[i] = 0.0f;
            r[i] = bi;
            const float zi = dinv[i] * bi;
            z[i] = zi;
            p0[i] = 0.0f;  // either may be the first step's p_old
            p1[i] = 0.0f;
            rz = fmaf(bi, zi, rz);
            rr = fmaf(bi, bi, rr);
        }
        const double srz = block_sum_f(rz, red_sh);
        const double srr = block_sum_f(rr, red_sh);
        const MfProblem &P = probs[C.prob];
        if (threadIdx.x == 0) {
            chunk_part[ci] = srz;
            chunk_part[n_chunks + ci] = srr;
            __threadfence();
            const unsigned t = atomicAdd(&st->cnt_update, 1u);
            sh_last = (t == (unsigned)P.chunk_count - 1);
        }
        __syncthreads();
        if (sh_last) {
            const double trz = ordered_sum(chunk_part, P.chunk_begin, P.chunk_count);
            const double trr = ordered_sum(chunk_part + n_chunks, P.chunk_begin, P.chunk_count);
            if (threadIdx.x == 0) {
                st->cnt_update = 0;
                st->rz = trz;
                st->rr = trr;
                st->bb = trr;
                st->tol2 = inner_rtol2 * trr;
                st->beta = 0.0;
                st->iter = 0;
                st->maxit = maxit;
                st->status = 0;
                st->first = 1;
                st->done = (trr <= st->tol2 || trr == 0.0) ? 1 : 0;
                if (is_bad(trr)) { st->status = MG_ENAN; st->done = 1; }
                st->phase = kPhaseCG;
            }
        }
        __syncthreads();
    });
}

// a problem whose inner CG has just stopped and whose correction is usable
__device__ __forceinline__ bool inner_finished(const MfState *st) {
    return st->phase == kPhaseCG && st->done && (st->status == 0 || st->status == MG_ENOCONV);
}

// refinement update u += x / scale (x is 0 on Dirichlet dofs and padding) for
// the problems whose inner CG has stopped
__global__ void __launch_bounds__(kThreads) mf_refine_kernel(
    const MfChunkDesc *__restrict__ chunks, const MfProblem *__restrict__ probs, int n_fine,
    const float *__restrict__ x, double *__restrict__ u64, const MfState *states) {
    pdl_enter();
    for_active_parts<kThreads>(n_fine, [&](int p) { return inner_finished(states + p); },
                     [&](int p, int &begin, int &end) {
                         begin = probs[p].chunk_begin;
                         end = begin + probs[p].chunk_count;
                     }, [&](int ci) {
        const MfChunkDesc C = chunks[ci];
        const double inv = 1.0 / states[C.prob].scale;
        for (int64_t i = C.begin + threadIdx.x; i < C.end; i += kThreads)
            u64[i] = fma((double)x[i], inv, u64[i]);
    });
}

// Whether a solve's time is up, by the device's own clock: its budget runs from the first look, which is
// behind the first kernels of its first loop body.  Called by one thread of the loop's deciding kernels,
// so that a loop of 64 bodies overruns its limit by one body and not by the rest of a launch.  c: *clock,
// loaded with the kernel's other words (one after another, the loads cost 0.3 us a body: 16x8x8 0.4 %).
__device__ __forceinline__ bool time_is_up(MfLoopClock *clock, const MfLoopClock &c) {
    if (c.budget_ns <= 0) return false;
    int64_t now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (c.start_ns == 0) clock->start_ns = now;
    return now - (c.start_ns ? c.start_ns : now) >= c.budget_ns;
}

// after the refinement update: a stopped inner CG sends its problem back to the
// FP64 residual, or ends it on a breakdown / NaN (one block).  LOOP: the last kernel of a
// while-loop body; the loop goes on while a problem is unfinished, no wait has timed out, the
// solve has time left and fewer than `limit` bodies have run since the launch (loop[0]).  loop[1] counts all
// bodies, of nested loops those inside (mf_gate_kernel) and loop[2] those around them.
constexpr int kPhaseThreads = 256;
template <bool LOOP>
__global__ void __launch_bounds__(kPhaseThreads) mf_phase_kernel(MfState *states, int n_fine,
                                                                 cudaGraphConditionalHandle handle, int *loop,
                                                                 int limit, bool nested, const int *err,
                                                                 MfLoopClock *clock) {
    pdl_enter();
    int active = 0, bodies = 0, failed = 0;
    MfLoopClock c{0, 0};
    if (LOOP && threadIdx.x == 0) {
        bodies = loop[0] + 1;
        failed = *err;
        c = *clock;
    }
    for (int i = threadIdx.x; i < n_fine; i += kPhaseThreads) {
        MfState *st = states + i;
        if (st->phase == kPhaseCG && st->done) {
            if (st->status != 0 && st->status != MG_ENOCONV) {
                st->ref_status = st->status;
                st->ref_done = 1;
                st->phase = kPhaseFin;
            } else {
                st->refine += 1;
                st->status = 0;
                st->u_zero = 0;  // u has been corrected
                st->phase = kPhaseResid;
            }
        }
        st->resid = st->phase == kPhaseResid;
        active |= st->phase != kPhaseFin;
    }
    if (LOOP) {
        active = __syncthreads_or(active);
        if (threadIdx.x == 0) {
            const bool more = active && bodies < limit && failed == 0 && !time_is_up(clock, c);
            loop[0] = more ? bodies : 0;
            loop[nested ? 2 : 1] += 1;
            cudaGraphSetConditional(handle, more ? 1u : 0u);
        }
    }
}

// The CG loop of a single problem inside its refinement loop goes on while its inner CG does
// (count: the last kernel of a body; else before the loop).
__global__ void mf_gate_kernel(const MfState *states, cudaGraphConditionalHandle handle, int *loop, int limit,
                               bool count, const int *err, MfLoopClock *clock) {
    pdl_enter();
    const MfLoopClock c = *clock;
    const int bodies = loop[0] + (count ? 1 : 0), all = loop[1] + 1, failed = *err;
    const bool active = states[0].phase == kPhaseCG && !states[0].done;
    if (count) {
        loop[0] = bodies;
        loop[1] = all;
    }
    const bool up = time_is_up(clock, c);
    const bool more = active && bodies < limit && failed == 0 && !up;
    cudaGraphSetConditional(handle, more ? 1u : 0u);
}

// FP64 outer residual r = f - K u (double-float arithmetic, factored element
// stiffness, hex8_factored.cuh), per-problem ||r||^2 -> scale.  A tile owns
// kROwnX x kROwnY nodes in x, y (to the end of the side in the last tile) and
// P.res_z node planes, evaluates the kREX x kREY elements around them, a thread
// each, and streams through the element layers as mf_fac_kernel does: the x, y part
// of the transform belongs to a node plane and is formed once for the two layers
// that meet there, and the results of the two layers are added in mode space before
// one inverse x, y transform per node plane.  Its four corner values go to shared
// memory, from where every owned node adds those of its four elements in a fixed
// order (deterministic, atomic-free).  u's planes arrive by asynchronous copies two
// layers ahead and are split into double-floats once per tile.
// Bound by the FP32 pipe (an addition of two double-floats is 11 instructions):
// 128x64x64 169 us with bricks of 8^3 nodes that evaluated 1.9 elements for each one
// and 24 corner values apiece, 102 us so; the z overlap and the tiles' edges leave 1.3.
constexpr int kROwnX = 16, kROwnY = 8;
constexpr int kREX = kROwnX + 1, kREY = kROwnY + 1;   // elements per tile layer
constexpr int kRNX = kREX + 1, kRNY = kREY + 1;       // nodes per tile plane
constexpr int kRThreads = 160;                        // 153 elements, 153 nodes at most
constexpr int kRPlane = 3 * kRNX * kRNY;              // 540 words of a node plane
constexpr int kRLoads = (kRPlane + kRThreads - 1) / kRThreads;
constexpr int kRMaxZ = 12;
constexpr int kResidSmem = (2 * kRPlane + 2 * kRPlane + 2 * 12 * kRThreads) * 8;  // planes, raw planes, exchange
static_assert(kREX * kREY <= kRThreads, "one element and one node per thread");
static_assert((kMaxSide + kROwnX - 1) / kROwnX <= 32768 && (kMaxSide + kROwnY - 1) / kROwnY <= 32768, "tile numbers");

// block sum of kRThreads threads; valid in thread 0
__device__ __forceinline__ double resid_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    return threadIdx.x == 0 ? ((sh[0] + sh[1]) + (sh[2] + sh[3])) + sh[4] : 0.0;
}
static_assert(kRThreads == 5 * 32, "resid_sum adds five warps");

__global__ void __launch_bounds__(kRThreads, 3) mf_residual64_kernel(
    const MfProblem *__restrict__ probs, const MfBrick *__restrict__ bricks, int n_bricks,
    const dfloat *__restrict__ Edf, const uint8_t *__restrict__ node_fix,
    const double *__restrict__ u64, const double *__restrict__ f64, const __grid_constant__ FacK<dfloat> K,
    double *__restrict__ r64, MfState *states, double *__restrict__ brick_part, double rtol2,
    int max_ref, int n_fine) {
    pdl_enter();
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ double red_sh[kRThreads / 32];
    __shared__ int sh_last;
    dfloat *planes = reinterpret_cast<dfloat *>(smem);                // [2][kRPlane]
    double *raws = reinterpret_cast<double *>(planes + 2 * kRPlane);  // [2][kRPlane]
    dfloat *xchg = reinterpret_cast<dfloat *>(raws + 2 * kRPlane);    // [2][12][kRThreads]
    const int tid = threadIdx.x;
    const bool active = tid < kREX * kREY;
    const int tx = active ? tid % kREX : 0, ty = active ? tid / kREX : 0;  // of the thread's element and node
    for_active_parts<kRThreads>(n_fine, [&](int p) { return states[p].resid != 0; },
                     [&](int p, int &begin, int &end) {
                         begin = probs[p].brick_begin;
                         end = begin + probs[p].brick_count;
                     }, [&](int bi) {
        const MfBrick br = bricks[bi];
        const MfProblem &P = probs[br.prob];
        MfState *st = states + br.prob;
        const bool need_ff = st->ff64 == 0.0;  // first residual of a solve: also ||f||^2
        const bool u_zero = st->u_zero != 0;    // cold start: r = f, no operator pass
        const int NX = P.NX, NY = P.NY, NZ = P.NZ, nx = P.nx, ny = P.ny, nz = P.nz, pitch = P.pitch;
        const int gx0 = br.bx * kROwnX, gy0 = br.by * kROwnY, z0 = br.bz * P.res_z, z1 = min(z0 + P.res_z, NZ);
        const int ownx = gx0 + kROwnX >= nx ? NX - gx0 : kROwnX, owny = gy0 + kROwnY >= ny ? NY - gy0 : kROwnY;
        const int S = z1 - z0 + 1;  // element layers z0 - 1 .. z1 - 1; node planes z0 - 1 .. z1
        const uint8_t *fix = node_fix + P.node_off;
        const double *u = u64 + P.dof_off;
        // node plane p (z0 - 1 + p): the words of this thread, copied into raw buffer p & 1, and
        // split from there (0 beyond the grid and on Dirichlet dofs) into plane buffer p & 1
        auto word = [&](int k, int p, int &t, int &gx, int64_t &line, int &c) {
            t = tid + k * kRThreads;
            const int row = t / (3 * kRNX), col = t - row * (3 * kRNX), i = col / 3;
            const int gy = gy0 - 1 + row, gz = z0 - 1 + p;
            gx = gx0 - 1 + i;
            c = col - 3 * i;
            line = (int64_t)gz * NY + gy;
            return t < kRPlane && (unsigned)gx < (unsigned)NX && (unsigned)gy < (unsigned)NY && (unsigned)gz < (unsigned)NZ;
        };
        auto load = [&](int p, unsigned (&fb)[kRLoads]) {  // fb: 1 where the word is 0
#pragma unroll
            for (int k = 0; k < kRLoads; k++) {
                int t, gx, c;
                int64_t line;
                fb[k] = 1;
                if (word(k, p, t, gx, line, c)) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(raws + (p & 1) * kRPlane + t)),
                                 "l"(u + line * pitch + 3 * gx + c) : "memory");
                    fb[k] = (unsigned)fix[line * NX + gx] >> c;
                }
            }
        };
        auto split = [&](int p, const unsigned (&fb)[kRLoads]) {
#pragma unroll
            for (int k = 0; k < kRLoads; k++) {
                const int t = tid + k * kRThreads;
                if (t >= kRPlane) continue;
                planes[(p & 1) * kRPlane + t] = fb[k] & 1 ? df_zero() : df_split(raws[(p & 1) * kRPlane + t]);
            }
        };
        // the element's modulus in layer s
        const int gex = gx0 - 1 + tx, gey = gy0 - 1 + ty;
        const bool in_grid = active && (unsigned)gex < (unsigned)nx && (unsigned)gey < (unsigned)ny;
        const dfloat *Ecol = Edf + P.elem_off + (in_grid ? (int64_t)gey * P.pitch_e + gex : 0);
        const int64_t Elayer = (int64_t)ny * P.pitch_e;
        auto modulus = [&](int s) {
            const int k = z0 - 1 + s;
            return in_grid && s < S && k >= 0 && k < nz ? Ecol[k * Elayer] : df_zero();
        };
        // x, y modes (q = mx + 2 my) of plane p at the element
        auto modes = [&](int p, int c, dfloat (&m)[4]) {
            const dfloat *n0 = planes + (p & 1) * kRPlane + 3 * (ty * kRNX + tx) + c;
            const dfloat a = n0[0], b = n0[3], cc = n0[3 * kRNX], d = n0[3 * kRNX + 3];
            const dfloat s0 = a + b, s1 = cc + d, d0 = b - a, d1 = d - cc;
            m[0] = s0 + s1;
            m[1] = d0 + d1;
            m[2] = s1 - s0;
            m[3] = d1 - d0;
        };
        unsigned fb[kRLoads];
        dfloat low[3][4], car[3][4], e = df_zero();  // modes of plane s; results of layer s - 1 on it
        if (!u_zero) {
            unsigned fb1[kRLoads];
            load(0, fb);
            load(1, fb1);
            e = modulus(0);
            asm volatile("cp.async.wait_all;" ::: "memory");
            split(0, fb);
            split(1, fb1);
            load(2, fb);  // a tile has two layers at least
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 3; c++) {
                modes(0, c, low[c]);
#pragma unroll
                for (int q = 0; q < 4; q++) car[c][q] = df_zero();
            }
            __syncthreads();  // plane 0 is read; plane 2 takes its buffer in the first layer
        }
        const bool own = active && tx < ownx && ty < owny;
        const int64_t line0 = (int64_t)(z0 - 1) * NY + gy0 + ty, fix0 = line0 * NX + gx0 + tx;
        const int64_t g0 = P.dof_off + line0 * pitch + 3 * (gx0 + tx);
        double part = 0.0, fpart = 0.0;
        for (int s = 0; s < S; s++) {
            dfloat *X = xchg + (s & 1) * 12 * kRThreads;
            if (!u_zero) {
                const dfloat e_next = modulus(s + 1);
                dfloat v[3][8];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    dfloat high[4];
                    modes(s + 1, c, high);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (q) v[c][q] = low[c][q] + high[q];  // mode 0 has no part in the result
                        v[c][q + 4] = high[q] - low[c][q];
                        low[c][q] = high[q];
                    }
                }
                hex8_factored_khat_df(K, e, v);
                e = e_next;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    dfloat node[4];  // plane s: the layer below's part and this layer's
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        node[q] = q ? car[c][q] + (v[c][q] - v[c][q + 4]) : car[c][0] - v[c][4];
                        car[c][q] = q ? v[c][q] + v[c][q + 4] : v[c][4];
                    }
                    if (s >= 1) {  // back to the corners; plane 0 is the tile below's
                        const dfloat y0 = node[0] - node[2], y1 = node[0] + node[2];
                        const dfloat d0 = node[1] - node[3], d1 = node[1] + node[3];
                        X[(4 * c) * kRThreads + tid] = y0 - d0;  // corner bx + 2 by
                        X[(4 * c + 1) * kRThreads + tid] = y0 + d0;
                        X[(4 * c + 2) * kRThreads + tid] = y1 - d1;
                        X[(4 * c + 3) * kRThreads + tid] = y1 + d1;
                    }
                }
                // plane s + 2 into the buffer of plane s, whose readers are behind the last barrier
                if (s + 2 <= S) {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    split(s + 2, fb);
                    if (s + 3 <= S) load(s + 3, fb);
                }
            }
            double fv[3] = {0.0, 0.0, 0.0};
            const int64_t g = g0 + (int64_t)s * NY * pitch;
            uint8_t fixed = 0;
            if (s >= 1 && own) {
                fixed = fix[fix0 + (int64_t)s * NY * NX];
#pragma unroll
                for (int c = 0; c < 3; c++) fv[c] = f64[g + c];
            }
            __syncthreads();
            if (s >= 1 && own) {
                // the node is corner (0, 0) of element (tx + 1, ty + 1), ...; the tile's last node
                // of a side has no element beyond it
                const bool right = tx + 1 < kREX, back = ty + 1 < kREY;
                const dfloat *Xn = X + tid;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    double yv = 0.0;
                    if (!u_zero) {
                        dfloat y = Xn[(4 * c + 3) * kRThreads];
                        if (right) y += Xn[(4 * c + 2) * kRThreads + 1];
                        if (back) y += Xn[(4 * c + 1) * kRThreads + kREX];
                        if (right && back) y += Xn[(4 * c) * kRThreads + kREX + 1];
                        yv = df_to(y);
                    }
                    double rv = fv[c] - yv;
                    if ((fixed >> c) & 1) rv = 0.0;
                    r64[g + c] = rv;
                    part = fma(rv, rv, part);
                    if (need_ff) fpart = fma(fv[c], fv[c], fpart);
                }
            }
        }
        const double s = resid_sum(part, red_sh);
        const double sf = need_ff ? resid_sum(fpart, red_sh) : 0.0;
        if (tid == 0) {
            brick_part[bi] = s;
            brick_part[n_bricks + bi] = sf;
            __threadfence();
            const unsigned t = atomicAdd(&st->cnt_res, 1u);
            sh_last = (t == (unsigned)P.brick_count - 1);
        }
        __syncthreads();  // also: the tile's last reads of the buffers are done
        if (sh_last) {
            auto total = [&](const double *v) {
                double w = 0.0;
                for (int i = tid; i < P.brick_count; i += kRThreads) w += __ldcg(v + P.brick_begin + i);
                return resid_sum(w, red_sh);
            };
            const double rr = total(brick_part);
            const double ff = need_ff ? total(brick_part + n_bricks) : 0.0;
            if (tid == 0) {
                st->cnt_res = 0;
                if (need_ff) st->ff64 = ff > 0.0 ? ff : -1.0;  // -1: zero load (u = 0)
                st->rr64 = rr;
                st->scale = rr > 0.0 ? 1.0 / sqrt(rr) : 1.0;
                st->phase = kPhaseFin;
                st->ref_done = 1;
                if (st->ff64 < 0.0) st->rr64 = 0.0;
                else if (is_bad(rr)) st->ref_status = MG_ENAN;
                else if (rr <= rtol2 * st->ff64) st->ref_status = 0;
                else if (st->refine >= max_ref) st->ref_status = MG_ENOCONV;
                else { st->ref_done = 0; st->phase = kPhaseInit; }
            }
        }
        __syncthreads();
    });
}

// Jacobi inverse of the mixed operator: 1 / sum_e E_e K0[3a+c][3a+c];
// 0 on Dirichlet dofs and padding (marks them for the vector kernels).  Blocks of some 2,048
// words, whole grid rows (j, k), from a list of all problems; a thread per word.  (A grid of the
// largest problem's blocks times the problems, 64-bit divisions and K0 converted from FP64 in
// every thread: 58 designs with their levels 536 us, 131 us so.)  runs > 0: the blocks are those of the
// runs [first, first + size) of the list: run_end[r] counts the blocks of the runs up to r, run_first
// follows it (every other of 58 16x8x8 designs started and ended: 1,007 us with a launch a run, 721 so).
__host__ __device__ constexpr int diag_rows(int pitch) { return pitch >= 2048 ? 1 : 2048 / pitch; }
__global__ void __launch_bounds__(256) mf_diag_kernel(const MfProblem *__restrict__ probs,
                                                      const MfNodeBlk *__restrict__ blks, int runs,
                                                      const int *__restrict__ run_end,
                                                      const float *__restrict__ E32, const uint8_t *__restrict__ node_fix,
                                                      const double *__restrict__ K0, float *__restrict__ dinv) {
    __shared__ float sk[24];  // the diagonal of K0
    __shared__ int s_blk;
    if (threadIdx.x < 24) sk[threadIdx.x] = (float)K0[25 * threadIdx.x];
    if (runs == 0 && threadIdx.x == 0) s_blk = blockIdx.x;
    for (int r = threadIdx.x; r < runs; r += 256) {
        const int lo = r ? run_end[r - 1] : 0, at = (int)blockIdx.x - lo;
        if (at >= 0 && (int)blockIdx.x < run_end[r]) s_blk = run_end[runs + r] + at;
    }
    __syncthreads();
    const MfNodeBlk B = blks[s_blk];
    const MfProblem &P = probs[B.prob];
    const int NX = P.NX, NY = P.NY, nx = P.nx, ny = P.ny, nz = P.nz, pitch = P.pitch;
    const int row1 = min(B.node + diag_rows(pitch), NY * P.NZ);
    const float *E = E32 + P.elem_off;
    const uint8_t *fix = node_fix + P.node_off;
    float *out = dinv + P.dof_off;
    for (int i = threadIdx.x; i < (row1 - B.node) * pitch; i += 256) {
        const int row = B.node + i / pitch, xin = i % pitch;
        float v = 0.0f;
        if (xin < 3 * NX) {
            const int gx = xin / 3, c = xin - 3 * gx, gy = row % NY, gz = row / NY;
            // FP32 (the Jacobi inverse is stored in FP32; GB300's FP64 pipe issues two
            // DFMA per cycle per SM), the node's elements in a fixed order
            float d = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
                const int ex = gx - dx, ey = gy - dy, ez = gz - dz;
                if (ex < 0 || ey < 0 || ez < 0 || ex >= nx || ey >= ny || ez >= nz) continue;
                d = fmaf(E[((int64_t)ez * ny + ey) * P.pitch_e + ex], sk[3 * corner_index(dx, dy, dz) + c], d);
            }
            const bool fixed = (fix[(int64_t)row * NX + gx] >> c) & 1;
            v = (fixed || d == 0.0f) ? 0.0f : 1.0f / d;
        }
        out[(int64_t)row * pitch + xin] = v;
    }
}

// compliance adjoint sensitivity dC/drho_e = -dE_e u_e^T K0 u_e, written
// unpadded (element order x-fastest) at dc + out_off[prob]
// dc_e = -dE_e u_e^T K0 u_e for the listed problems, in the factored form:
// u_e^T K0 u_e = u~^T (Khat / 64) u~ with u~ the sum/difference modes of u_e (72
// butterfly additions, 45 + 21 products instead of the 600 of the dense product),
// in double-float arithmetic on the FP32 pipes (48-bit significand; GB300's FP64
// pipe issues two DFMA per cycle per SM) from the FP64 u and Khat, the final
// product with dE_e in FP64
__global__ void mf_sens_kernel(const MfProblem *__restrict__ probs, int n_probs,
                               const double *__restrict__ dE64, const uint8_t *__restrict__ node_fix,
                               const double *__restrict__ u64, FacK<dfloat> K,
                               const int64_t *__restrict__ out_off, double *__restrict__ dc) {
    const int pi = blockIdx.y;
    if (pi >= n_probs) return;
    const MfProblem P = probs[pi];
    if (out_off[pi] < 0) return;  // not part of this evaluation
    const int64_t ne = (int64_t)P.nx * P.ny * P.nz;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int ex = (int)(e % P.nx), ey = (int)((e / P.nx) % P.ny), ez = (int)(e / ((int64_t)P.nx * P.ny));
        dfloat v[3][8];  // component c at lexicographic corner b = bx + 2 by + 4 bz
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const int bx = b & 1, by = (b >> 1) & 1, bz = b >> 2;
            const int64_t gn = (ex + bx) + (int64_t)P.NX * ((ey + by) + (int64_t)P.NY * (ez + bz));
            const uint8_t fx = node_fix[P.node_off + gn];
            const double *u = u64 + dof_index(P, ex + bx, ey + by, ez + bz, 0);
#pragma unroll
            for (int c = 0; c < 3; c++) v[c][b] = ((fx >> c) & 1) ? df_zero() : df_split(u[c]);
        }
        hex8_factored_forward(v);
        dfloat yh[3][8];
        hex8_factored_khat(K, v, yh);
        dfloat s = df_zero();
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int m = 1; m < 8; m++) s = fma_t(v[c][m], yh[c][m], s);
        dc[out_off[pi] + e] = -dE64[P.elem_off + ((int64_t)ez * P.ny + ey) * P.pitch_e + ex] * df_to(s);
    }
}

// per-chunk partial of a.b; host sums each problem's chunks in order
__global__ void mf_dot_chunks_kernel(const MfChunkDesc *__restrict__ chunks, int n_chunks,
                                     const double *__restrict__ a, const double *__restrict__ b,
                                     double *__restrict__ part) {
    __shared__ double red_sh[kThreads / 32];
    for (int ci = blockIdx.x; ci < n_chunks; ci += gridDim.x) {
        const MfChunkDesc C = chunks[ci];
        double s = 0.0;
        for (int64_t i = C.begin + threadIdx.x; i < C.end; i += kThreads) s = fma(a[i], b[i], s);
        const double t = block_sum(s, red_sh);
        if (threadIdx.x == 0) part[ci] = t;
        __syncthreads();
    }
}

// unpadded element array (x-fastest) -> padded FP32, double-float (the outer
// residual's moduli) and FP64 (dE/drho) tables of problem P
__global__ void pack_elems_kernel(const MfProblem *__restrict__ probs, int pi,
                                  const double *__restrict__ E, const double *__restrict__ dE,
                                  float *__restrict__ E32, dfloat *__restrict__ Edf,
                                  double *__restrict__ dE64) {
    const MfProblem P = probs[pi];
    const int64_t ne = (int64_t)P.nx * P.ny * P.nz;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t ex = e % P.nx, row = e / P.nx;
        const int64_t o = P.elem_off + row * P.pitch_e + ex;
        if (E) {
            Edf[o] = df_from(E[e]);
            E32[o] = (float)E[e];
        }
        if (dE) dE64[o] = dE[e];
    }
}

// padded <-> unpadded node-interleaved FP64 vectors of problem P
__global__ void unpack_vec_kernel(const MfProblem *__restrict__ probs, int pi,
                                  double *__restrict__ padded, double *__restrict__ flat,
                                  int to_flat) {
    const MfProblem P = probs[pi];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n_dofs;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = i / (3 * P.NX), xin = i - row * 3 * P.NX;
        const int64_t o = P.dof_off + row * P.pitch + xin;
        if (to_flat) flat[i] = padded[o];
        else padded[o] = flat[i];
    }
}

__global__ void fill_f32_kernel(float *__restrict__ a, const float *__restrict__ mask, float v,
                                int64_t n) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = (mask[i] != 0.0f) ? v : 0.0f;
}

inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// B tiles of the column operator: tile t = dy + 2 dz holds the K0 columns of the
// corners (0, dy, dz) and (1, dy, dz) (K chunk dx: x, y, z, 0 in TF32; x, y, z
// and five zeros in BF16) for the 32 N rows n = 3 a + c (libMesh corner a; rows
// 24..31 zero), in the no-swizzle K-major layout: core matrix (n / 8, dx) at
// ((n / 8) * 2 + dx) * 128 bytes.  [tf32 hi | tf32 lo | bf16 hi | bf16 lo], 1024
// words each.
void pack_b_columns(const double *K0, std::vector<uint32_t> &out) {
    auto tf32_round = [](float x) -> float {
        uint32_t u;
        memcpy(&u, &x, 4);
        if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;  // nearest, ties away
        float r;
        memcpy(&r, &u, 4);
        return r;
    };
    auto bf16_bits = [](float x) -> uint32_t {
        uint32_t u;
        memcpy(&u, &x, 4);
        return ((u + 0x7fffu + ((u >> 16) & 1u)) >> 16) & 0xffffu;  // nearest even
    };
    auto bits_of = [](uint32_t h) -> float {
        const uint32_t u = h << 16;
        float r;
        memcpy(&r, &u, 4);
        return r;
    };
    auto fbits = [](float x) -> uint32_t {
        uint32_t u;
        memcpy(&u, &x, 4);
        return u;
    };
    out.assign(4096, 0u);
    for (int t = 0; t < 4; t++) {
        const int dy = t & 1, dz = t >> 1;
        for (int n = 0; n < 32; n++)
            for (int dx = 0; dx < 2; dx++) {
                const int a = corner_index(dx, dy, dz);
                const int core = (n / 8) * 2 + dx;
                for (int c = 0; c < 3; c++) {
                    const double v = (n < 24) ? K0[n * 24 + 3 * a + c] : 0.0;
                    // TF32: 4 words per row
                    const int w = t * 256 + core * 32 + (n % 8) * 4 + c;
                    const float h = tf32_round((float)v);
                    out[w] = fbits(h);
                    out[1024 + w] = fbits(tf32_round((float)(v - (double)h)));
                    // BF16: 8 halves per row (x, y, z, 0, 0, 0, 0, 0)
                    const int wb = 2048 + t * 256 + core * 32 + (n % 8) * 4 + c / 2;
                    const uint32_t hb = bf16_bits((float)v);
                    const uint32_t lb = bf16_bits((float)(v - (double)bits_of(hb)));
                    out[wb] |= hb << (16 * (c & 1));
                    out[1024 + wb] |= lb << (16 * (c & 1));
                }
            }
    }
}

// Launch with programmatic dependent launch (the kernel starts with pdl_enter):
// the launch latency of the solver step's kernels overlaps their predecessors.
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// launch_pdl with a thread-block cluster of csize CTAs along x
template <typename... KArgs, typename... Args>
void launch_cluster_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int csize, cudaStream_t s,
                        Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)csize;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

struct ApplyArgs {
    int level, in_slot, parity;
    const float *rhs;
    float *y;
    int sel = -1;  // -1 every problem; 0 problems with a coarser level; 1 those without
};

template <int PREC, int MODE>
void launch_apply(MfBatch &b, const ApplyArgs &a) {
    if (!b.lvl_col_ctas[a.level]) return;
    launch_pdl(mf_col_kernel<PREC, MODE>, b.lvl_col_ctas[a.level], kColThreads, kColSmem, b.stream, 
        b.probs, b.cols, b.col_order, b.col_offs + b.lvl_col_off[a.level], a.sel, b.tmaps, a.in_slot, a.parity, b.Bop2, b.dinv,
        a.rhs, b.p0, b.p1, a.y, b.states, b.col_part, b.err);
}

template <int MODE>
void launch_apply_prec(MfBatch &b, int prec, const ApplyArgs &a) {
    switch (prec) {
        case MG_MIXED_TF32: launch_apply<MG_MIXED_TF32, MODE>(b, a); break;
        case MG_MIXED_BF16: launch_apply<MG_MIXED_BF16, MODE>(b, a); break;
        case MG_MIXED_TF32X3: launch_apply<MG_MIXED_TF32X3, MODE>(b, a); break;
        default: launch_apply<MG_MIXED_BF16X3, MODE>(b, a); break;
    }
}

// the factored kernel's tensor map of a batch vector
int fac_map_of(const MfBatch &b, const float *v) {
    if (v == b.mx) return kFMapMx;
    if (v == b.md) return kFMapMd;
    if (v == b.my) return kFMapMy;
    if (v == b.mb) return kFMapMb;
    if (v == b.r) return kFMapR;
    if (v == b.mr) return kFMapMr;
    if (v == b.z) return kFMapZ;
    return -1;
}

template <int MODE>
void launch_fac(MfBatch &b, int l, int sel, const FacArgs &a) {
    if (a.in_map < 0 || ((MODE == 2 || MODE == 4 || MODE == 5) && a.b_map < 0)) {
        b.enqueue_error = MG_EINVAL;  // reported by the caller of the enqueue
        return;
    }
    if (!b.lvl_fac_ctas[l]) return;
    launch_pdl(mf_fac_kernel<MODE>, b.lvl_fac_ctas[l], kFThreads, fac_smem(MODE), b.stream, b.probs, b.fac_tiles,
               b.fac_offs + b.lvl_fac_off[l], sel, b.fac2, b.fac_maps, b.states, a, b.err);
}

// level operator of the multigrid, y = A x (MODE 3) or rhs - A x (MODE 2; z, nullable: D^-1 y,
// the factored operator only), on level l: the factored CUDA-core operator (fac) or the
// tensor-core column operator in precision prec (x is the vector of map in_slot there)
template <int MODE>
void launch_level_op(MfBatch &b, bool fac, int prec, int l, int in_slot, const float *x, const float *rhs,
                     float *y, int sel, float *z = nullptr) {
    if (fac) {
        launch_fac<MODE>(b, l, sel,
                         FacArgs{fac_map_of(b, x), rhs ? fac_map_of(b, rhs) : -1, y, z, nullptr, nullptr, 0.0f, 0.0f,
                                 0.0f, 0});
    } else {
        ApplyArgs a{l, in_slot, 0, rhs, y, sel};
        launch_apply_prec<MODE>(b, prec, a);
    }
}

// CG step on the level-0 columns (z from map in_slot)
void launch_cg_apply(MfBatch &b, int prec, int in_slot, int parity) {
    ApplyArgs a{0, in_slot, parity, nullptr, b.q};
    launch_apply_prec<1>(b, prec, a);
}

template <int PREC>
int set_apply_attrs() {
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kColSmem));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kColSmem));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, kColSmem));
    // all of the unified L1/shared storage as shared memory: two CTAs per SM
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 1>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 2>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_col_kernel<PREC, 3>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    return MG_OK;
}

int configure_kernels() {
    static bool done = false;
    if (done) return MG_OK;
    MG_TRY(set_apply_attrs<MG_MIXED_TF32>());
    MG_TRY(set_apply_attrs<MG_MIXED_BF16>());
    MG_TRY(set_apply_attrs<MG_MIXED_TF32X3>());
    MG_TRY(set_apply_attrs<MG_MIXED_BF16X3>());
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_residual64_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, kResidSmem));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_fac_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, fac_smem(2)));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_fac_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, fac_smem(3)));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_fac_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, fac_smem(4)));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_fac_kernel<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, fac_smem(5)));
    MG_CUDA_TRY(cudaFuncSetAttribute(mf_fac_kernel<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, fac_smem(6)));
    MG_CUDA_TRY(cudaFuncSetAttribute(mg_coarse_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kCoarseInvSmem));
    MG_CUDA_TRY(cudaFuncSetAttribute(mg_bottom_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    MG_CUDA_TRY(cudaFuncSetAttribute(mg_bottom_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kBottomSmemMax));
    done = true;
    return MG_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_fn(EncodeTiledFn *fn) {
    static EncodeTiledFn cached = nullptr;
    if (!cached) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        MG_CUDA_TRY(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                                     cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !p) {
            set_error("cuTensorMapEncodeTiled unavailable");
            return MG_ECUDA;
        }
        cached = reinterpret_cast<EncodeTiledFn>(p);
    }
    *fn = cached;
    return MG_OK;
}

int make_map(EncodeTiledFn fn, CUtensorMap *m, void *base, uint64_t d0, uint64_t d1, uint64_t d2,
             uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1, uint32_t b2) {
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
        return MG_ECUDA;
    }
    return MG_OK;
}

void launch_update(MfBatch &b, float *pnew, bool mg) {
    const int n0 = b.lvl_chunk_hi[0];
    launch_pdl(mf_update_kernel, std::max(1, std::min(n0, b.vec_grid)), kThreads, 0, b.stream, 
        b.chunks, n0, b.probs, b.x, b.r, b.z, pnew, b.q, b.dinv, b.states, b.chunk_part, mg ? 1 : 0);
}

// Jacobi inverse of n blocks: of the list from `first` on, or of `runs` runs of it
int launch_diag(MfBatch &b, int first, int n, int runs = 0, const int *run_end = nullptr) {
    mf_diag_kernel<<<n, 256, 0, b.stream>>>(b.probs, b.diag_blks + first, runs, run_end, b.E32, b.node_fix, b.K0, b.dinv);
    MG_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return MG_OK;
}

int compute_diag(MfBatch &b) {
    MG_TRY(launch_diag(b, 0, b.diag_at.back()));
    return MG_OK;  // the operator-only paths need no coarse inverse; activation forms it
}

// Jacobi inverse of the listed level-0 problems and all their coarse levels, and
// the inverse of the coarsest grid of their direct chains; nothing waits on the host
int compute_diag_list(MfBatch &b, const std::vector<int> &level0) {
    std::vector<int> list;  // the chains, then the runs of blocks (ends, firsts)
    if (level0.empty()) return MG_OK;
    for (size_t h = 0; h < b.h_heads.size(); h++)
        if (b.h_coarse_off[h] >= 0 && std::find(level0.begin(), level0.end(), b.h_head_root[h]) != level0.end())
            list.push_back((int)h);
    const int n_inv = (int)list.size();
    // the blocks of a problem and its coarse levels are neighbours in the list, as are those of
    // neighbouring problems
    std::vector<int> probs(level0), first, end;
    std::sort(probs.begin(), probs.end());
    int n = 0;
    for (size_t k = 0; k < probs.size(); k++) {
        const int lo = b.diag_at[probs[k]], hi = b.diag_at[probs[k] + 1];
        if (k && probs[k] == probs[k - 1]) continue;
        n += hi - lo;
        if (k && probs[k] == probs[k - 1] + 1) {
            end.back() = n;
        } else {
            first.push_back(lo);
            end.push_back(n);
        }
    }
    const int runs = first.size() > 1 ? (int)first.size() : 0;
    if (runs) {
        list.insert(list.end(), end.begin(), end.end());
        list.insert(list.end(), first.begin(), first.end());
    }
    if (!list.empty()) {
        // the pinned staging buffer: the previous call's copy must have read it
        if (b.stage_pending) MG_CUDA_TRY(cudaEventSynchronize(b.stage_ev));
        memcpy(b.stage_host, list.data(), list.size() * sizeof(int));
        MG_CUDA_TRY(cudaMemcpyAsync(b.start_list, b.stage_host, list.size() * sizeof(int), cudaMemcpyHostToDevice, b.stream));
        MG_CUDA_TRY(cudaEventRecord(b.stage_ev, b.stream));
        b.stage_pending = true;
    }
    MG_TRY(launch_diag(b, runs ? 0 : first[0], n, runs, b.start_list + n_inv));
    if (n_inv) {
        mg_coarse_inverse_kernel<<<(unsigned)n_inv, kCoarseInvThreads, kCoarseInvSmem, b.stream>>>(
            b.probs, b.heads, b.start_list, b.E32, b.dinv, b.K0, b.coarse_off, b.coarse_inv,
            b.coarse_ok);
        MG_CUDA_TRY(cudaGetLastError());
        count_launches(1);
    }
    return MG_OK;
}

}  // namespace

// ----------------------------------------------------------------------- host
void hex8_box_stiffness(double hx, double hy, double hz, double nu, double K[576]) {
    // same quadrature as the FP64 element kernel: 2x2x2 Gauss, E = 1
    const double gp = 0.57735026918962576451;
    const double lam = nu / (1.0 - nu - 2.0 * nu * nu), mu = 1.0 / (2.0 * (1.0 + nu));
    double S[8][8][9];
    memset(S, 0, sizeof(S));
    for (int q = 0; q < 8; q++) {
        const double xi = (q & 1) ? gp : -gp, eta = (q >> 1 & 1) ? gp : -gp, zeta = (q >> 2 & 1) ? gp : -gp;
        const double w = (hx * hy * hz) / 8.0;  // det J, unit weights
        double g[8][3];
        for (int a = 0; a < 8; a++) {
            int dx, dy, dz;
            corner_bits(a, dx, dy, dz);
            const double sx = dx ? 1 : -1, sy = dy ? 1 : -1, sz = dz ? 1 : -1;
            const double fx = 0.5 * (1 + sx * xi), fy = 0.5 * (1 + sy * eta), fz = 0.5 * (1 + sz * zeta);
            g[a][0] = 0.5 * sx * fy * fz * (2.0 / hx);
            g[a][1] = 0.5 * sy * fx * fz * (2.0 / hy);
            g[a][2] = 0.5 * sz * fx * fy * (2.0 / hz);
        }
        for (int a = 0; a < 8; a++)
            for (int b = 0; b < 8; b++)
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) S[a][b][i * 3 + j] += w * g[a][i] * g[b][j];
    }
    for (int a = 0; a < 8; a++)
        for (int b = 0; b < 8; b++) {
            const double *s = S[a][b];
            const double tr = s[0] + s[4] + s[8];
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++)
                    K[(3 * a + i) * 24 + 3 * b + j] = lam * s[i * 3 + j] + mu * s[j * 3 + i] + (i == j ? mu * tr : 0.0);
        }
}

// shared-memory layout of the cluster bottom kernel for clusters of cs CTAs: per
// chain its level table (nodes per CTA, offsets of D^-1, E and the CTA's slabs);
// returns the dynamic shared memory (bytes) of the largest chain
int64_t cluster_layout(const MfBatch &b, int cs, std::vector<ClusterChain> &chains) {
    chains.assign(b.h_heads.size(), ClusterChain{});
    int64_t most = 0;
    for (size_t h = 0; h < b.h_heads.size(); h++) {
        ClusterChain &ch = chains[h];
        ch.root = b.h_head_root[h];
        int m = 0;
        int64_t stage = 0;
        for (int t = b.h_heads[h]; t >= 0 && m < kBottomMaxLevels; t = b.h_probs[t].coarse, m++) {
            const MfProblem &T = b.h_probs[t];
            ClusterLevel &L = ch.L[m];
            L.NX = T.NX; L.NY = T.NY; L.NZ = T.NZ;
            L.nx = T.nx; L.ny = T.ny; L.nz = T.nz;
            L.pitch = T.pitch; L.pitch_e = T.pitch_e;
            L.dof_off = T.dof_off; L.elem_off = T.elem_off;
            const int nn = T.NX * T.NY * T.NZ, H = T.NX * T.NY + T.NX + 1;
            int64_t staged = 0;  // words staged by one CTA
            L.chunk = (nn + cs - 1) / cs;
            L.NXY = T.NX * T.NY;
            L.rNX = 1.0f / (float)T.NX;
            L.rNXY = 1.0f / (float)L.NXY;
            L.rchunk = 1.0f / (float)L.chunk;
            // the device divides by one rounded product: check it for every node
            auto fdiv = [](int n, float r) { return (int)(((float)n + 0.5f) * r); };
            for (int n = 0; n < nn; n++)
                if (fdiv(n, L.rNXY) != n / L.NXY || fdiv(n, L.rchunk) != n / L.chunk ||
                    (n < L.NXY && fdiv(n, L.rNX) != n / T.NX))
                    return -1;
            for (int r = 0; r < cs; r++) {
                const int n0 = r * L.chunk, n1 = std::min(nn, n0 + L.chunk);
                if (n0 < n1) staged = std::max<int64_t>(staged, 3LL * (std::min(nn, n1 + H) - std::max(0, n0 - H)));
            }
            staged = (staged + 3) / 4 * 4;
            stage = std::max(stage, staged);
            if (m > 0) {  // prolongation to the level above stages the coarse planes around its nodes
                const ClusterLevel &F = ch.L[m - 1];
                const int nf = F.NXY * F.NZ;
                for (int n0 = 0; n0 < nf; n0 += F.chunk) {
                    const int k0 = n0 / F.NXY >> 1;
                    const int k1 = std::min(((std::min(nf, n0 + F.chunk) - 1) / F.NXY + 1) >> 1, T.NZ - 1);
                    stage = std::max<int64_t>(stage, 3LL * L.NXY * (k1 - k0 + 1));
                }
            }
            stage = std::max<int64_t>(stage, 3LL * nn <= kCoarseDirectMax ? 3LL * nn : 0);  // rhs of a direct solve
            L.s_dinv = (int)staged;  // words, until the offsets are given below
        }
        ch.m = m;
        int64_t off = 0;
        auto take = [&](int64_t words) {
            const int at = (int)off;
            off += (words + 3) / 4 * 4;
            return at;
        };
        ch.s_stage = take(stage);
        ch.s_idx = take(m > 0 ? ch.L[0].s_dinv : 0);
        for (int l = 0; l < m; l++) {
            ClusterLevel &L = ch.L[l];
            const int staged = L.s_dinv;
            L.s_dinv = take(staged);
            L.s_addr = take(staged);
            L.s_E = take((int64_t)L.nx * L.ny * L.nz);
            L.s_vec = take(15LL * L.chunk);
            L.s_elem = take(L.chunk);
            L.s_par = take(L.chunk);
            L.s_fine = take(kClusterThreads);
        }
        most = std::max(most, off * 4);
    }
    return most;
}

// Work of unequal size dealt to the CTAs of a grid: the largest first, each to the CTA with the
// least so far (Graham's longest-processing-time rule), equal ones in their order.  order: the
// pieces CTA by CTA; offs: where each CTA's begin (ctas + 1 entries).  Returns the largest load.
int deal_work(const std::vector<int> &cost, int ctas, std::vector<int> &order, std::vector<int> &offs) {
    std::vector<int> by(cost.size());
    for (size_t i = 0; i < by.size(); i++) by[i] = (int)i;
    std::stable_sort(by.begin(), by.end(), [&](int a, int c) { return cost[a] > cost[c]; });
    std::vector<std::vector<int>> own(ctas);
    typedef std::pair<int, int> Load;  // (load, CTA)
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
    for (int c = 0; c < ctas; c++) heap.push(Load(0, c));
    int most = 0;
    for (int i : by) {
        const Load l = heap.top();
        heap.pop();
        own[l.second].push_back(i);
        most = std::max(most, l.first + cost[i]);
        heap.push(Load(l.first + cost[i], l.second));
    }
    order.clear();
    offs.assign(1, 0);
    for (int c = 0; c < ctas; c++) {
        order.insert(order.end(), own[c].begin(), own[c].end());
        offs.push_back((int)order.size());
    }
    return most;
}

// Tiles of the factored operator, by level: kFNX x kFNY owned nodes, fac_z node planes.  A tile
// costs its planes, one element layer more, and about two layers for its start (tables, first
// loads).  The depth (at most kFMaxZ, the same rule for all problems of the level) is the one
// whose tiles, dealt out, leave the least to the busiest CTA.  With the deepest tiles dealt round
// robin, the busiest CTA had 96 layers where the mean is 49 (58 problems of 16x8x8 to 96x48x48) and
// 69 where it is 34 (two of 192x96x96); MODE 2 on level 0 took 86 and 73 us there, dealt so 66 and 56.
void plan_fac_tiles(MfBatch &b, int ctas) {
    b.h_fac_tiles.clear();
    b.h_fac_offs.clear();
    b.lvl_fac_off.clear();
    b.lvl_fac_ctas.clear();
    for (int l = 0; l < b.n_levels; l++) {
        auto depth = [](const MfProblem &P, int cap) {
            const int parts = std::min(32767, (P.NZ + cap - 1) / cap);  // tile numbers are 16 bits
            return (P.NZ + parts - 1) / parts;
        };
        auto tiles_of = [&](int cap, std::vector<MfCol> &tiles, std::vector<int> &cost) {
            tiles.clear();
            cost.clear();
            for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++) {
                const MfProblem &P = b.h_probs[pi];
                if (P.bottom) continue;  // solved inside its chain
                const int tx = (P.NX + kFNX - 1) / kFNX, ty = (P.NY + kFNY - 1) / kFNY, z = depth(P, cap);
                for (int k = 0; k * z < P.NZ; k++)
                    for (int j = 0; j < ty; j++)
                        for (int i = 0; i < tx; i++) {
                            tiles.push_back(MfCol{pi, (uint16_t)i, (uint16_t)j, (uint16_t)k, 0});
                            cost.push_back(std::min(z, P.NZ - k * z) + 3);
                        }
            }
        };
        std::vector<MfCol> tiles;
        std::vector<int> cost, order, offs;
        int best = 0, best_cap = kFMaxZ;
        int64_t layers = 0;
        for (int cap = kFMaxZ; cap >= kFMinZ; cap = cap > 16 ? cap - 8 : cap > 8 ? cap - 2 : cap - 1) {
            tiles_of(cap, tiles, cost);
            layers = 0;
            for (int c : cost) layers += c;
            if (best && layers >= (int64_t)best * ctas) break;  // shallower tiles only add layers
            const int most = deal_work(cost, ctas, order, offs);
            if (!best || most < best) {
                best = most;
                best_cap = cap;
            }
        }
        tiles_of(best_cap, tiles, cost);
        const int used = (int)std::min<int64_t>(ctas, (int64_t)tiles.size());
        deal_work(cost, used, order, offs);
        for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++) b.h_probs[pi].fac_z = depth(b.h_probs[pi], best_cap);
        const int base = (int)b.h_fac_tiles.size();
        b.lvl_fac_off.push_back((int)b.h_fac_offs.size());
        b.lvl_fac_ctas.push_back(used);
        for (int o : offs) b.h_fac_offs.push_back(base + o);
        for (int i : order) b.h_fac_tiles.push_back(tiles[i]);
    }
}

// The columns of the tensor-core operator, by level, dealt out in the same way (58 problems, round
// robin: 209 layers on the busiest CTA where the mean is 156, 180 us a launch; dealt so 165).  Their numbers, by which the partial
// sums of p.q are kept, stay those of their problem.
void plan_cols(MfBatch &b, int ctas) {
    b.h_col_order.clear();
    b.h_col_offs.clear();
    b.lvl_col_off.clear();
    b.lvl_col_ctas.clear();
    for (int l = 0; l < b.n_levels; l++) {
        std::vector<int> cols, cost, order, offs;
        for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++) {
            const MfProblem &P = b.h_probs[pi];
            for (int c = P.col_begin; c < P.col_begin + P.col_count && !P.bottom; c++) {
                cols.push_back(c);
                cost.push_back(std::min(P.col_z, P.NZ - b.h_cols[c].cz * P.col_z) + 1);
            }
        }
        const int used = std::min<int>(ctas, (int)cols.size()), base = (int)b.h_col_order.size();
        deal_work(cost, used, order, offs);
        b.lvl_col_off.push_back((int)b.h_col_offs.size());
        b.lvl_col_ctas.push_back(used);
        for (int o : offs) b.h_col_offs.push_back(base + o);
        for (int i : order) b.h_col_order.push_back(cols[i]);
    }
}

int mf_batch_init(MfBatch &b, const std::vector<MfProblem> &shapes, double hx, double hy,
                  double hz, double nu, cudaStream_t stream, int max_levels, bool bottom_cluster) {
    MG_TRY(configure_kernels());
    EncodeTiledFn enc = nullptr;
    MG_TRY(encode_fn(&enc));
    int dev = 0, sms = 0;
    MG_CUDA_TRY(cudaGetDevice(&dev));
    MG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    b.stream = stream;
    b.hx = hx; b.hy = hy; b.hz = hz; b.nu = nu;
    // level 0: the designs; then every design's coarse levels, ordered by level
    b.n_fine = (int)shapes.size();
    b.h_probs.clear();
    for (size_t i = 0; i < shapes.size(); i++) {
        MfProblem P = shapes[i];
        P.level = 0;
        P.root = (int)i;
        P.coarse = -1;
        P.fine = -1;
        b.h_probs.push_back(P);
    }
    b.lvl_prob_lo.assign(1, 0);
    b.lvl_prob_hi.assign(1, b.n_fine);
    for (int lev = 1; lev < std::max(1, std::min(max_levels, kMaxLevels)); lev++) {
        const int lo = b.lvl_prob_lo.back(), hi = b.lvl_prob_hi.back();
        const int start = (int)b.h_probs.size();
        for (int f = lo; f < hi; f++) {
            const MfProblem F = b.h_probs[f];
            if (!mg_coarsens(F.nx, F.ny, F.nz)) continue;
            MfProblem C{};
            C.nx = (F.nx + 1) / 2; C.ny = (F.ny + 1) / 2; C.nz = (F.nz + 1) / 2;
            C.level = lev;
            C.root = F.root;
            C.fine = f;
            C.coarse = -1;
            // a load case sharing its design's moduli shares the coarse moduli too
            C.share_elems = (F.share_elems >= 0) ? b.h_probs[F.share_elems].coarse : -1;
            b.h_probs[f].coarse = (int)b.h_probs.size();
            b.h_probs.push_back(C);
        }
        if ((int)b.h_probs.size() == start) break;
        b.lvl_prob_lo.push_back(start);
        b.lvl_prob_hi.push_back((int)b.h_probs.size());
    }
    b.n_levels = (int)b.lvl_prob_lo.size();
    b.n_probs = (int)b.h_probs.size();
    int64_t dof = 0, el = 0, nd = 0;
    int nb = 0, nc = 0;
    b.h_bricks.clear();
    b.h_chunks.clear();
    b.h_cols.clear();
    for (size_t pi = 0; pi < b.h_probs.size(); pi++) {
        MfProblem &P = b.h_probs[pi];
        if (P.nx <= 0 || P.ny <= 0 || P.nz <= 0 || P.nx >= kMaxSide || P.ny >= kMaxSide || P.nz >= kMaxSide) {
            set_error("bad grid %dx%dx%d", P.nx, P.ny, P.nz);
            return MG_EINVAL;
        }
        P.NX = P.nx + 1; P.NY = P.ny + 1; P.NZ = P.nz + 1;
        P.pitch = (3 * P.NX + 3) / 4 * 4;
        P.pitch_e = (P.nx + 3) / 4 * 4;
        P.n_dofs = (int64_t)P.NX * P.NY * P.NZ * 3;
        P.n_pad = (int64_t)P.pitch * P.NY * P.NZ;
        if (P.share_elems >= 0 && P.share_elems < (int)pi) {
            const MfProblem &S = b.h_probs[P.share_elems];
            if (S.nx != P.nx || S.ny != P.ny || S.nz != P.nz) {
                set_error("shared element tables need equal grids");
                return MG_EINVAL;
            }
            P.elem_off = S.elem_off;
        } else {
            P.share_elems = -1;
            P.elem_off = el;
            el += (int64_t)P.pitch_e * P.ny * P.nz;
        }
        P.dof_off = dof;
        P.node_off = nd;
        dof += P.n_pad;
        nd += (int64_t)P.NX * P.NY * P.NZ;
        // tiles of the FP64 residual: as deep as one wave of resident tiles allows, up to kRMaxZ
        // node planes (a layer more is evaluated than planes are owned).  In a batch several
        // problems form their residual in the same step: an eighth of the slots each, whatever
        // the others are (the tiles decide the order of the sum ||r||^2)
        const int bx = (P.nx + kROwnX - 1) / kROwnX, by = (P.ny + kROwnY - 1) / kROwnY;
        const int64_t res_slots = bottom_cluster ? 3LL * sms : 3LL * sms / 8;
        const int64_t res_per = std::max<int64_t>(1, res_slots / ((int64_t)bx * by));
        P.res_z = (int)std::max<int64_t>((P.NZ + 32766) / 32767, std::min<int64_t>(kRMaxZ, (P.NZ + res_per - 1) / res_per));
        const int bz = (P.NZ + P.res_z - 1) / P.res_z;
        P.brick_begin = nb;
        P.brick_count = bx * by * bz;
        for (int k = 0; k < bz; k++)
            for (int j = 0; j < by; j++)
                for (int i = 0; i < bx; i++)
                    b.h_bricks.push_back(MfBrick{(int)pi, (int16_t)i, (int16_t)j, (int16_t)k, 0});
        nb += P.brick_count;
        // Columns of the tensor-core operator: as deep as one wave of resident columns allows, up
        // to kCZ node planes; a second, partial wave would double the launch's time.  A single
        // small grid's columns are as short as the slots allow, one plane and two element layers
        // at the least: 16x8x8 54.8 us an iteration with four planes at least, 52.4 with one;
        // 48x24x24 108.3 and 106.1.  In a batch a design takes a quarter of the slots, eight planes
        // at least and equal columns where they make one wave, whatever the batch holds: the columns
        // decide the order of its p.q.  ms a solve (the slots divided by the level's designs / half /
        // a quarter / a sixth of them): 58 problems 44.2 / 44.6 / 44.3 / 44.2, sixteen 32x16x16
        // 7.75 / 7.56 / 7.56 / 7.55, one 48x24x24 3.36 / 3.51 / 3.50 / 3.57, one 64x32x32 5.62 /
        // 5.79 / 6.06 / 6.07.
        const int cx = (P.NX + kCX - 1) / kCX, cy = (P.NY + kCY - 1) / kCY;
        const int64_t slots = kColCtas * (int64_t)sms;
        const int64_t col_per = std::max<int64_t>(1, (bottom_cluster ? slots : slots / 4) / ((int64_t)cx * cy));
        P.col_z = (int)std::min<int64_t>(kCZ, std::max<int64_t>(bottom_cluster ? 1 : 8, (P.NZ + col_per - 1) / col_per));
        const int col_parts = (P.NZ + P.col_z - 1) / P.col_z;
        if (!bottom_cluster && (int64_t)cx * cy * col_parts <= slots) P.col_z = (P.NZ + col_parts - 1) / col_parts;
        const int cz = (P.NZ + P.col_z - 1) / P.col_z;
        P.col_begin = (int)b.h_cols.size();
        P.col_count = cx * cy * cz;
        for (int k = 0; k < cz; k++)
            for (int j = 0; j < cy; j++)
                for (int i = 0; i < cx; i++)
                    b.h_cols.push_back(MfCol{(int)pi, (uint16_t)i, (uint16_t)j, (uint16_t)k, 0});
        int chunk = kMinChunk;
        while (chunk < kMaxChunk && P.n_pad > (int64_t)chunk * (bottom_cluster ? 8 * sms : 8 * sms / 16)) chunk *= 2;
        P.chunk_begin = nc;
        P.chunk_count = (int)((P.n_pad + chunk - 1) / chunk);
        for (int c = 0; c < P.chunk_count; c++) {
            MfChunkDesc C;
            C.prob = (int)pi;
            C.pad = 0;
            C.begin = P.dof_off + (int64_t)c * chunk;
            C.end = std::min(P.dof_off + P.n_pad, C.begin + chunk);
            b.h_chunks.push_back(C);
        }
        nc += P.chunk_count;
    }
    b.n_bricks = nb;
    b.n_chunks = nc;
    b.n_cols = (int)b.h_cols.size();
    b.lvl_brick_hi.clear(); b.lvl_chunk_lo.clear(); b.lvl_chunk_hi.clear();
    for (int l = 0; l < b.n_levels; l++) {
        const MfProblem &A = b.h_probs[b.lvl_prob_lo[l]], &Z = b.h_probs[b.lvl_prob_hi[l] - 1];
        b.lvl_brick_hi.push_back(Z.brick_begin + Z.brick_count);
        b.lvl_chunk_lo.push_back(A.chunk_begin);
        b.lvl_chunk_hi.push_back(Z.chunk_begin + Z.chunk_count);
    }
    b.n_pad = dof;
    b.n_elem_pad = el;
    b.n_nodes = nd;
    // bottom chains: for every design, the first level below the finest with at most
    // kBatchMaxHeadNodes nodes whose tables fit one CTA; for a single design (bottom_cluster)
    // the first with at most kClusterMaxHeadNodes, the finest included, whose tables some
    // cluster can hold.  The tables hold a halo of NX NY nodes on each side, so a flat
    // design's wide levels do not fit: 80x64x4 starts at its third level (from the second
    // 16 CTAs need 209 KB each, from the third 54).  Larger levels run level by level on the
    // whole GPU; without any chain a solve of 80x64x4 took 74.4 ms, so 38.1 (34x34x3: 25.1, 11.4).
    int64_t inv_floats = 0;
    {
        const bool single = bottom_cluster && b.n_fine == 1;
        b.h_heads.clear();
        b.h_head_root.clear();
        b.bottom_smem = 0;
        b.bottom_cluster = 0;
        b.chains_from_root = false;
        for (MfProblem &T : b.h_probs) T.bottom = 0;
        // The chains of b.h_heads on the largest clusters (16 CTAs: non-portable size) that the
        // device can place for all of them at once, one CTA a chain where there are more chains
        // than that; false: none that holds the tables.  MASTGPU_BOTTOM_CLUSTER caps the cluster
        // (1, 2, 4, 8 or 16 CTAs): a test knob, the correction does not depend on the cluster size
        int cap = kClusterMax;
        if (const char *env = std::getenv("MASTGPU_BOTTOM_CLUSTER")) cap = std::max(1, std::min(kClusterMax, std::atoi(env)));
        int first = 1;
        while (first * 2 <= cap) first *= 2;
        auto place = [&] {
            for (int cs = first; cs >= 1; cs /= 2) {
                if (cs > 1 && (int64_t)b.h_heads.size() * cs > sms) continue;
                std::vector<ClusterChain> chains;
                const int64_t smem = cluster_layout(b, cs, chains);
                if (smem < 0 || smem > kBottomSmemMax) continue;
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3((unsigned)(cs * b.h_heads.size()));
                cfg.blockDim = dim3(kClusterThreads);
                cfg.dynamicSmemBytes = smem;
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = (unsigned)cs;
                attr[0].val.clusterDim.y = 1;
                attr[0].val.clusterDim.z = 1;
                cfg.attrs = attr;
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, mg_bottom_cluster_kernel, &cfg) == cudaSuccess &&
                    n >= (cs > 1 ? (int)b.h_heads.size() : 1)) {
                    b.bottom_cluster = cs;
                    b.bottom_smem = (int)smem;
                    b.h_cl_chains.swap(chains);
                    return true;
                }
                cudaGetLastError();  // clear the failed query
            }
            return false;
        };
        for (int r = 0; r < b.n_fine; r++)
            for (int q = single && b.h_probs[r].coarse >= 0 ? r : b.h_probs[r].coarse; q >= 0; q = b.h_probs[q].coarse) {
                const MfProblem &Hd = b.h_probs[q];
                const int64_t head_nodes = (int64_t)Hd.NX * Hd.NY * Hd.NZ;
                int64_t depth = 0, words = 6 * head_nodes;  // at most what cluster_layout gives one CTA
                for (int t = q; t >= 0; t = b.h_probs[t].coarse, depth++) {
                    const MfProblem &T = b.h_probs[t];
                    words += 23LL * T.NX * T.NY * T.NZ + (int64_t)T.nx * T.ny * T.nz + kClusterThreads + 32;
                }
                if (depth > kBottomMaxLevels || head_nodes > (single ? kClusterMaxHeadNodes : kBatchMaxHeadNodes)) continue;
                // a batched chain fits one CTA, in whatever batch (a long thin design's levels shrink slowly)
                if (!single && 4 * words > kBottomSmemMax) continue;
                b.h_heads.push_back(q);
                b.h_head_root.push_back(r);
                if (single && !place()) {
                    b.h_heads.clear();
                    b.h_head_root.clear();
                    continue;
                }
                b.chains_from_root = q == r;
                break;
            }
        if (!single && !b.h_heads.empty()) place();
        if (!b.bottom_cluster) {
            b.h_heads.clear();
            b.h_head_root.clear();
            b.chains_from_root = false;
        }
        // the problems of the chains; direct coarse solves where the coarsest grid is small enough
        b.h_coarse_off.assign(b.h_heads.size(), -1);
        for (size_t h = 0; h < b.h_heads.size(); h++) {
            int c = b.h_heads[h];
            for (int t = c; t >= 0; t = b.h_probs[t].coarse) {
                b.h_probs[t].bottom = t != b.h_head_root[h];
                c = t;
            }
            const MfProblem &C = b.h_probs[c];
            const int64_t nd = 3LL * C.NX * C.NY * C.NZ;
            if (nd <= kCoarseDirectMax) {
                b.h_coarse_off[h] = inv_floats;
                inv_floats += nd * nd;
            }
        }
    }
    plan_fac_tiles(b, 2 * sms);  // two factored-operator CTAs per SM
    plan_cols(b, kColCtas * sms);
    // node blocks of the transfers, by level: the coarse problems whose fine one is not inside a
    // bottom chain
    {
        std::vector<MfNodeBlk> blks;
        b.lvl_blk_lo.clear();
        b.lvl_blk_hi.clear();
        for (int l = 0; l < b.n_levels; l++) {
            b.lvl_blk_lo.push_back((int)blks.size());
            for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++) {
                const MfProblem &P = b.h_probs[pi];
                if (P.fine < 0 || b.h_probs[P.fine].bottom) continue;
                for (int n = 0; n < P.NX * P.NY * P.NZ; n += kNodeBlk) blks.push_back(MfNodeBlk{pi, n});
            }
            b.lvl_blk_hi.push_back((int)blks.size());
        }
        MG_TRY(dev_alloc_n(&b.node_blks, std::max<size_t>(1, blks.size())));
        if (!blks.empty())
            MG_CUDA_TRY(cudaMemcpyAsync(b.node_blks, blks.data(), blks.size() * sizeof(MfNodeBlk),
                                        cudaMemcpyHostToDevice, b.stream));
        MG_CUDA_TRY(cudaStreamSynchronize(b.stream));  // blks is a host temporary
    }
    MG_TRY(dev_alloc_n(&b.coarse_off, std::max<size_t>(1, b.h_coarse_off.size())));
    MG_TRY(dev_alloc_n(&b.coarse_inv, (size_t)std::max<int64_t>(1, inv_floats)));
    MG_TRY(dev_alloc_n(&b.coarse_ok, std::max<size_t>(1, b.h_coarse_off.size())));
    b.res_grid = std::max(1, std::min(nb, 3 * sms));    // FP64 residual: three CTAs per SM
    b.vec_grid = std::max(1, std::min(nc, 8 * sms));
    MG_TRY(dev_alloc_n(&b.probs, b.h_probs.size()));
    MG_TRY(dev_alloc_n(&b.bricks, b.h_bricks.size()));
    MG_TRY(dev_alloc_n(&b.cols, b.h_cols.size()));
    MG_TRY(dev_alloc_n(&b.col_order, b.h_col_order.size()));
    MG_TRY(dev_alloc_n(&b.col_offs, b.h_col_offs.size()));
    MG_TRY(dev_alloc_n(&b.col_part, b.h_cols.size()));
    MG_TRY(dev_alloc_n(&b.fac_tiles, std::max<size_t>(1, b.h_fac_tiles.size())));
    MG_TRY(dev_alloc_n(&b.fac_offs, b.h_fac_offs.size()));
    MG_TRY(dev_alloc_n(&b.Bop2, 4096));
    MG_TRY(dev_alloc_n(&b.chunks, b.h_chunks.size()));
    static_assert(sizeof(MfLoopClock) <= sizeof(MfState) && alignof(MfLoopClock) <= alignof(MfState), "clock slot");
    MG_TRY(dev_alloc_n(&b.states, (size_t)b.n_probs + 1));
    b.clock = reinterpret_cast<MfLoopClock *>(b.states + b.n_probs);
    MG_TRY(dev_alloc_n(&b.tmaps, (size_t)b.n_probs * kMapsPerProblem));
    MG_TRY(dev_alloc_n(&b.fac_maps, (size_t)b.n_probs * kFacMaps));
    MG_CUDA_TRY(cudaMallocHost(reinterpret_cast<void **>(&b.states_host), b.n_probs * sizeof(MfState)));
    MG_TRY(dev_alloc_n(&b.E32, (size_t)el + 4));
    MG_TRY(dev_alloc_n(&b.Edf, (size_t)el + 4));
    MG_TRY(dev_alloc_n(&b.dE64, (size_t)el + 4));
    MG_TRY(dev_alloc_n(&b.node_fix, (size_t)nd));
    float **f32s[] = {&b.x, &b.r, &b.z, &b.p0, &b.p1, &b.q, &b.dinv,
                      &b.mb, &b.mx, &b.md, &b.my, &b.mr};
    for (float **v : f32s) MG_TRY(dev_alloc_n(v, (size_t)dof));
    MG_TRY(dev_alloc_n(&b.u64, (size_t)dof));
    MG_TRY(dev_alloc_n(&b.r64, (size_t)dof));
    MG_TRY(dev_alloc_n(&b.f64, (size_t)dof));
    MG_TRY(dev_alloc_n(&b.brick_part, (size_t)2 * nb));  // operator partials | ||f||^2 partials
    MG_TRY(dev_alloc_n(&b.chunk_part, (size_t)2 * nc));
    MG_TRY(dev_alloc_n(&b.err, kErrWords));
    MG_CUDA_TRY(cudaMallocHost(&b.err_host, kErrWords * sizeof(int)));
    b.loop_bodies = b.loop_outer = 0;
    {
        std::vector<MfNodeBlk> blks;
        b.diag_at.assign(1, 0);
        for (int r = 0; r < b.n_fine; r++) {
            for (int q = r; q >= 0; q = b.h_probs[q].coarse)
                for (int row = 0; row < b.h_probs[q].NY * b.h_probs[q].NZ; row += diag_rows(b.h_probs[q].pitch))
                    blks.push_back(MfNodeBlk{q, row});
            b.diag_at.push_back((int)blks.size());
        }
        MG_TRY(dev_alloc_n(&b.diag_blks, blks.size()));
        MG_CUDA_TRY(cudaMemcpyAsync(b.diag_blks, blks.data(), blks.size() * sizeof(MfNodeBlk), cudaMemcpyHostToDevice,
                                    b.stream));
        MG_CUDA_TRY(cudaStreamSynchronize(b.stream));  // blks is a host temporary
    }
    const size_t start_words = b.h_heads.size() + 2 * (size_t)b.n_fine;
    MG_TRY(dev_alloc_n(&b.start_list, start_words));
    MG_TRY(dev_alloc_n(&b.sens_offs, (size_t)std::max(1, b.n_fine)));
    MG_CUDA_TRY(cudaMallocHost(&b.sens_offs_host, (size_t)std::max(1, b.n_fine) * sizeof(int64_t)));
    MG_CUDA_TRY(cudaMallocHost(&b.stage_host, start_words * sizeof(int)));
    MG_CUDA_TRY(cudaEventCreateWithFlags(&b.stage_ev, cudaEventDisableTiming));
    MG_TRY(dev_alloc_n(&b.heads, std::max<size_t>(1, b.h_heads.size())));
    MG_TRY(dev_alloc_n(&b.K0, 576));
    double K0[576];
    hex8_box_stiffness(hx, hy, hz, nu, K0);
    if (!hex8_factored_build(K0, b.fac64, b.fac32)) return MG_EINVAL;
    for (int k = 0; k < kFacN; k++) b.facdf.v[k] = dfloat_of(b.fac64.v[k]);
    for (int k = 0; k < kFacN; k++) b.fac2.v[k] = make_float2(b.fac32.v[k], b.fac32.v[k]);
    // Gershgorin bound of D^-1 A: every assembled row is a positive combination
    // of K0 rows, so max_i sum_j |K0_ij| / K0_ii bounds it on every level
    b.cheb_lmax = 0.0;
    for (int i = 0; i < 24; i++) {
        double sabs = 0.0;
        for (int j = 0; j < 24; j++) sabs += fabs(K0[i * 24 + j]);
        b.cheb_lmax = std::max(b.cheb_lmax, sabs / K0[i * 24 + i]);
    }
    // tensor maps: z, p0, p1, E, debug x per problem
    std::vector<CUtensorMap> maps(b.n_probs * kMapsPerProblem);
    for (int pi = 0; pi < b.n_probs; pi++) {
        const MfProblem &P = b.h_probs[pi];
        float *vecs[5] = {b.z, b.p0, b.p1, b.mx, b.md};
        const int slot[5] = {0, 1, 2, 4, 5};
        // column operator: one node plane {32 floats, 17 rows} / element plane {12, 16}
        for (int k = 0; k < 5; k++)
            MG_TRY(make_map(enc, &maps[pi * kMapsPerProblem + slot[k]], vecs[k] + P.dof_off,
                            3 * (uint64_t)P.NX, P.NY, P.NZ, (uint64_t)P.pitch * 4,
                            (uint64_t)P.pitch * P.NY * 4, kCRawX, kCPY, 1));
        MG_TRY(make_map(enc, &maps[pi * kMapsPerProblem + 3], b.E32 + P.elem_off, P.nx, P.ny, P.nz,
                        (uint64_t)P.pitch_e * 4, (uint64_t)P.pitch_e * P.ny * 4, 12, 16, 1));
    }
    // factored level operator: node planes {104 floats, 17 rows}, moduli planes {36, 16}
    std::vector<CUtensorMap> fmaps((size_t)b.n_probs * kFacMaps);
    for (int pi = 0; pi < b.n_probs; pi++) {
        const MfProblem &P = b.h_probs[pi];
        float *vecs[kFMapE] = {b.mx, b.md, b.my, b.mb, b.r, b.dinv, b.mr, b.z};
        for (int k = 0; k < kFMapE; k++)
            MG_TRY(make_map(enc, &fmaps[(size_t)pi * kFacMaps + k], vecs[k] + P.dof_off, 3 * (uint64_t)P.NX, P.NY,
                            P.NZ, (uint64_t)P.pitch * 4, (uint64_t)P.pitch * P.NY * 4, kFBoxX, kFPY, 1));
        MG_TRY(make_map(enc, &fmaps[(size_t)pi * kFacMaps + kFMapE], b.E32 + P.elem_off, P.nx, P.ny, P.nz,
                        (uint64_t)P.pitch_e * 4, (uint64_t)P.pitch_e * P.ny * 4, kFBoxE, kFEY, 1));
    }
    cudaStream_t s = b.stream;
    MG_CUDA_TRY(cudaMemcpyAsync(b.tmaps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.fac_maps, fmaps.data(), fmaps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.probs, b.h_probs.data(), b.h_probs.size() * sizeof(MfProblem), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.bricks, b.h_bricks.data(), b.h_bricks.size() * sizeof(MfBrick), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.cols, b.h_cols.data(), b.h_cols.size() * sizeof(MfCol), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.col_order, b.h_col_order.data(), b.h_col_order.size() * sizeof(int),
                                cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.col_offs, b.h_col_offs.data(), b.h_col_offs.size() * sizeof(int),
                                cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.fac_tiles, b.h_fac_tiles.data(), b.h_fac_tiles.size() * sizeof(MfCol),
                                cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.fac_offs, b.h_fac_offs.data(), b.h_fac_offs.size() * sizeof(int),
                                cudaMemcpyHostToDevice, s));
    {
        std::vector<uint32_t> bop2;
        pack_b_columns(K0, bop2);
        MG_CUDA_TRY(cudaMemcpyAsync(b.Bop2, bop2.data(), bop2.size() * 4, cudaMemcpyHostToDevice, s));
        MG_CUDA_TRY(cudaStreamSynchronize(s));  // bop2 is a host temporary
    }
    MG_CUDA_TRY(cudaMemcpyAsync(b.chunks, b.h_chunks.data(), b.h_chunks.size() * sizeof(MfChunkDesc), cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemcpyAsync(b.K0, K0, 576 * 8, cudaMemcpyHostToDevice, s));
    if (b.bottom_cluster) {
        // K0 in FP32, the three rows of the corner (dx, dy, dz) at 72 (dx + 2 dy + 4 dz) as
        // [node][row][component]
        std::vector<float> k0f(kClusterK0);
        for (int i = 0; i < kClusterK0; i++) {
            const int lex = i / 72, bc = i % 72 / 9, r = i % 9 / 3, c = i % 3;
            const int a = corner_index(lex & 1, (lex >> 1) & 1, lex >> 2);
            k0f[i] = (float)K0[(3 * a + r) * 24 + 3 * bc + c];
        }
        MG_TRY(dev_alloc_n(&b.cl_k0, (size_t)kClusterK0));
        MG_CUDA_TRY(cudaMemcpyAsync(b.cl_k0, k0f.data(), k0f.size() * 4, cudaMemcpyHostToDevice, s));
        MG_TRY(dev_alloc_n(&b.cl_chains, b.h_cl_chains.size()));
        MG_CUDA_TRY(cudaMemcpyAsync(b.cl_chains, b.h_cl_chains.data(), b.h_cl_chains.size() * sizeof(ClusterChain),
                                    cudaMemcpyHostToDevice, s));
        MG_CUDA_TRY(cudaStreamSynchronize(s));  // k0f is a host temporary
    }
    if (!b.h_coarse_off.empty()) {
        MG_CUDA_TRY(cudaMemcpyAsync(b.coarse_off, b.h_coarse_off.data(), b.h_coarse_off.size() * sizeof(int64_t),
                                    cudaMemcpyHostToDevice, s));
        MG_CUDA_TRY(cudaMemsetAsync(b.coarse_ok, 0, b.h_coarse_off.size() * sizeof(int), s));
    }
    if (!b.h_heads.empty())
        MG_CUDA_TRY(cudaMemcpyAsync(b.heads, b.h_heads.data(), b.h_heads.size() * sizeof(int),
                                    cudaMemcpyHostToDevice, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.states, 0, (b.n_probs + 1) * sizeof(MfState), s));
    MG_CUDA_TRY(cudaMemsetAsync(b.err, 0, kErrWords * sizeof(int), s));
    MG_CUDA_TRY(cudaMemsetAsync(b.u64, 0, dof * 8, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.r64, 0, dof * 8, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.f64, 0, dof * 8, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.node_fix, 0, nd, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.E32, 0, (el + 4) * 4, s));
    MG_CUDA_TRY(cudaMemsetAsync(b.Edf, 0, (el + 4) * sizeof(dfloat), s));
    MG_CUDA_TRY(cudaMemsetAsync(b.dE64, 0, (el + 4) * 8, s));
    float *zero_vecs[] = {b.x, b.r, b.z, b.p0, b.p1, b.q, b.dinv, b.mb, b.mx, b.md, b.my, b.mr};
    for (float *v : zero_vecs) MG_CUDA_TRY(cudaMemsetAsync(v, 0, dof * 4, s));
    MG_CUDA_TRY(cudaStreamSynchronize(s));
    return MG_OK;
}

void mf_batch_free(MfBatch &b) {
    if (b.stream) cudaStreamSynchronize(b.stream);
    if (b.graph) cudaGraphExecDestroy(b.graph);
    void *ptrs[] = {b.probs, b.bricks, b.chunks, b.states, b.tmaps, b.E32, b.Edf, b.dE64,
                    b.node_fix, b.x, b.r, b.z, b.p0, b.p1, b.q, b.dinv, b.u64, b.r64,
                    b.f64, b.brick_part, b.chunk_part, b.err, b.K0, b.mb, b.mx, b.md,
                    b.my, b.mr, b.diag_blks, b.start_list, b.heads, b.cols, b.col_order, b.col_offs, b.col_part, b.Bop2, b.fac_tiles, b.fac_offs, b.fac_maps, b.node_blks,
                    b.coarse_off, b.coarse_inv, b.coarse_ok, b.cl_k0, b.cl_chains, b.sens_offs};
    for (void *q : ptrs) dev_free(q);
    if (b.stage_host) cudaFreeHost(b.stage_host);
    if (b.sens_offs_host) cudaFreeHost(b.sens_offs_host);
    if (b.stage_ev) cudaEventDestroy(b.stage_ev);
    if (b.states_host) cudaFreeHost(b.states_host);
    if (b.err_host) cudaFreeHost(b.err_host);
    b = MfBatch();
}

int mf_batch_set_bc(MfBatch &b, int i, const uint8_t *node_fix_host, const double *f_host) {
    if (i < 0 || i >= b.n_probs) return MG_EINVAL;
    const MfProblem &P = b.h_probs[i];
    const int64_t nn = (int64_t)P.NX * P.NY * P.NZ;
    cudaStream_t s = b.stream;
    if (node_fix_host) {
        MG_CUDA_TRY(cudaMemcpyAsync(b.node_fix + P.node_off, node_fix_host, nn, cudaMemcpyHostToDevice, s));
        // coarse levels: a coarse node is constrained where its fine node (2I,2J,2K) is; the
        // last node of an odd direction lies beyond the grid and takes the last fine node's
        std::vector<uint8_t> fine(node_fix_host, node_fix_host + nn), coarse;
        for (int f = i; b.h_probs[f].coarse >= 0; f = b.h_probs[f].coarse) {
            const MfProblem &F = b.h_probs[f], &C = b.h_probs[F.coarse];
            coarse.assign((size_t)C.NX * C.NY * C.NZ, 0);
            for (int K = 0; K < C.NZ; K++)
                for (int J = 0; J < C.NY; J++)
                    for (int I = 0; I < C.NX; I++)
                        coarse[I + (size_t)C.NX * (J + (size_t)C.NY * K)] =
                            fine[std::min(2 * I, F.nx) +
                                 (size_t)F.NX * (std::min(2 * J, F.ny) + (size_t)F.NY * std::min(2 * K, F.nz))];
            MG_CUDA_TRY(cudaMemcpyAsync(b.node_fix + C.node_off, coarse.data(), coarse.size(),
                                        cudaMemcpyHostToDevice, s));
            MG_CUDA_TRY(cudaStreamSynchronize(s));
            fine.swap(coarse);
        }
    }
    if (f_host) {
        std::vector<double> pad(P.n_pad, 0.0);
        for (int64_t row = 0; row < (int64_t)P.NY * P.NZ; row++)
            memcpy(pad.data() + row * P.pitch, f_host + row * 3 * P.NX, 3 * P.NX * sizeof(double));
        MG_CUDA_TRY(cudaMemcpyAsync(b.f64 + P.dof_off, pad.data(), P.n_pad * 8, cudaMemcpyHostToDevice, s));
        MG_CUDA_TRY(cudaStreamSynchronize(s));  // pad is a host temporary
    }
    if (node_fix_host) MG_CUDA_TRY(cudaStreamSynchronize(s));
    return MG_OK;
}

int mf_batch_set_moduli(MfBatch &b, int i, const double *E_dev, const double *dE_dev) {
    if (i < 0 || i >= b.n_probs) return MG_EINVAL;
    const MfProblem &P = b.h_probs[i];
    const int64_t ne = (int64_t)P.nx * P.ny * P.nz;
    pack_elems_kernel<<<std::min(blocks_for(ne, 256), 4096u), 256, 0, b.stream>>>(
        b.probs, i, E_dev, dE_dev, b.E32, b.Edf, b.dE64);
    MG_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    if (E_dev)
        for (int f = i; b.h_probs[f].coarse >= 0; f = b.h_probs[f].coarse) {
            const int c = b.h_probs[f].coarse;
            const MfProblem &C = b.h_probs[c];
            const int64_t nc = (int64_t)C.nx * C.ny * C.nz;
            dim3 grid(std::min(blocks_for(nc, 256), 4096u), 1);
            mg_coarsen_kernel<<<grid, 256, 0, b.stream>>>(b.probs, c, b.E32);
            MG_CUDA_TRY(cudaGetLastError());
            count_launches(1);
        }
    return MG_OK;
}

int mf_batch_get_u(MfBatch &b, int i, double *u_dev) {
    const MfProblem &P = b.h_probs[i];
    unpack_vec_kernel<<<std::min(blocks_for(P.n_dofs, 256), 4096u), 256, 0, b.stream>>>(
        b.probs, i, b.u64, u_dev, 1);
    MG_CUDA_TRY(cudaGetLastError());
    return MG_OK;
}

int mf_batch_set_u(MfBatch &b, int i, const double *u_dev) {
    const MfProblem &P = b.h_probs[i];
    unpack_vec_kernel<<<std::min(blocks_for(P.n_dofs, 256), 4096u), 256, 0, b.stream>>>(
        b.probs, i, b.u64, const_cast<double *>(u_dev), 0);
    MG_CUDA_TRY(cudaGetLastError());
    return MG_OK;
}

int mf_apply(MfBatch &b, int precision, const double *x_host, double *y_host, int prob) {
    MG_TRY(compute_diag(b));
    const MfProblem &P = b.h_probs[prob];
    std::vector<float> pad(P.n_pad, 0.0f);
    for (int64_t row = 0; row < (int64_t)P.NY * P.NZ; row++)
        for (int64_t k = 0; k < 3 * P.NX; k++) pad[row * P.pitch + k] = (float)x_host[row * 3 * P.NX + k];
    MG_CUDA_TRY(cudaMemcpyAsync(b.mx + P.dof_off, pad.data(), P.n_pad * 4, cudaMemcpyHostToDevice, b.stream));
    MG_CUDA_TRY(cudaMemsetAsync(b.states, 0, b.n_probs * sizeof(MfState), b.stream));
    if (precision == MG_OPERATOR_FACTORED_FP32) {
        launch_fac<3>(b, P.level, -1,
                      FacArgs{kFMapMx, -1, b.my, nullptr, nullptr, nullptr, 0.0f, 0.0f, 0.0f, 0});
    } else {
        ApplyArgs a{P.level, 4, 0, nullptr, b.my};
        launch_apply_prec<3>(b, precision, a);
    }
    MG_CUDA_TRY(cudaGetLastError());
    MG_CUDA_TRY(cudaMemcpyAsync(pad.data(), b.my + P.dof_off, P.n_pad * 4, cudaMemcpyDeviceToHost, b.stream));
    MG_CUDA_TRY(cudaStreamSynchronize(b.stream));
    int herr = 0;
    MG_CUDA_TRY(cudaMemcpy(&herr, b.err, sizeof(int), cudaMemcpyDeviceToHost));
    if (herr) {
        set_error("tensor-core pipeline wait exceeded its bound (error flag %d)", herr);
        return MG_ETIMEDOUT;
    }
    for (int64_t row = 0; row < (int64_t)P.NY * P.NZ; row++)
        for (int64_t k = 0; k < 3 * P.NX; k++) y_host[row * 3 * P.NX + k] = pad[row * P.pitch + k];
    return MG_OK;
}

// enqueue `reps` CG-mode operator launches on the level-0 bricks (timing hook; no sync)
int mf_launch_apply(MfBatch &b, int precision, int reps) {
    MG_TRY(compute_diag(b));
    MG_CUDA_TRY(cudaMemsetAsync(b.states, 0, b.n_probs * sizeof(MfState), b.stream));
    // nonzero search direction (zero on Dirichlet dofs) so every launch does the full work
    fill_f32_kernel<<<blocks_for(b.n_pad, 256), 256, 0, b.stream>>>(b.z, b.dinv, 1.0f, b.n_pad);
    if (precision == MG_OPERATOR_FACTORED_FP32) {
        // the multigrid level operator y = A x on level 0 (mx, my)
        fill_f32_kernel<<<blocks_for(b.n_pad, 256), 256, 0, b.stream>>>(b.mx, b.dinv, 1.0f, b.n_pad);
        for (int i = 0; i < reps; i++) launch_level_op<3>(b, true, 0, 0, 4, b.mx, nullptr, b.my, -1);
    } else {
        for (int i = 0; i < reps; i++) launch_cg_apply(b, precision, 0, i & 1);
    }
    MG_CUDA_TRY(cudaGetLastError());
    count_launches(reps + 2);
    return MG_OK;
}

namespace {

// precision of the multigrid smoothers: the single-product form of the family
int mg_precision(int prec) {
    return (prec == MG_MIXED_BF16 || prec == MG_MIXED_BF16X3) ? MG_MIXED_BF16 : MG_MIXED_TF32;
}

// Chebyshev coefficients for degree `deg` on [lmax/30, lmax]
struct Cheb {
    float inv_theta;
    float c1[32], c2[32];
};
Cheb cheb_coeffs(double lmax, int deg) {
    Cheb c{};
    const double lmin = lmax / 30.0, theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
    const double sigma = theta / delta;
    double rho = 1.0 / sigma;
    c.inv_theta = (float)(1.0 / theta);
    for (int k = 1; k < deg && k < 32; k++) {
        const double rn = 1.0 / (2.0 * sigma - rho);
        c.c1[k] = (float)(rn * rho);
        c.c2[k] = (float)(2.0 * rn / delta);
        rho = rn;
    }
    return c;
}

// one Chebyshev smoothing pass of degree deg on level l: mx (+)= S(rin), on the
// level's problems selected by sel (see ApplyArgs)
long long enqueue_smooth(MfBatch &b, bool fac, int prec, int l, const float *rin, int x0_zero, int deg,
                         const Cheb &cc, int sel) {
    const int clo = b.lvl_chunk_lo[l], chi = b.lvl_chunk_hi[l];
    const int grid = std::max(1, std::min(chi - clo, b.vec_grid));
    if (fac && deg >= 2) {
        // fused, from z = D^-1 rin (in b.z): the first two steps in one launch, then one launch
        // per step, the direction alternating md / my (md is never rin)
        if (deg == 2) {
            launch_fac<6>(b, l, sel,
                          FacArgs{kFMapZ, kFMapMx, nullptr, nullptr, nullptr, b.mx, cc.c1[1], cc.c2[1], cc.inv_theta,
                                  x0_zero});
            return 1;
        }
        launch_fac<5>(b, l, sel,
                      FacArgs{kFMapZ, fac_map_of(b, rin), b.md, nullptr, b.mr, b.mx, cc.c1[1], cc.c2[1], cc.inv_theta,
                              x0_zero});
        float *din = b.md, *dout = b.my;
        long long n = 1;
        for (int k = 2; k < deg; k++) {
            launch_fac<4>(b, l, sel,
                          FacArgs{fac_map_of(b, din), kFMapMr, dout, nullptr, b.mr, b.mx, cc.c1[k], cc.c2[k], 0.0f, 0});
            std::swap(din, dout);
            n += 1;
        }
        return n;
    }
    launch_pdl(mg_cheb_first_kernel, grid, kThreads, 0, b.stream, b.chunks, clo, chi, b.probs, b.states, rin,
                                                          b.mr, b.md, b.mx, b.dinv, cc.inv_theta, x0_zero, sel);
    long long n = 1;
    for (int k = 1; k < deg; k++) {
        launch_level_op<3>(b, fac, prec, l, 5, b.md, nullptr, b.my, sel);
        launch_pdl(mg_cheb_next_kernel, grid, kThreads, 0, b.stream, b.chunks, clo, chi, b.probs, b.states, b.my,
                                                             b.mr, b.md, b.mx, b.dinv, cc.c1[k], cc.c2[k], sel);
        n += 2;
    }
    return n;
}

// V-cycle z = M r on every design at once (level-0 rhs = CG residual r, z = mx).
// A problem whose own coarsest grid is level l gets the coarse-grid smoother
// (degree cdeg) there, whatever the depth of the other problems, so that each
// problem's preconditioner does not depend on the batch it is solved in.  The
// small levels of each chain (MfProblem::bottom) are done by one launch
// (mg_bottom_cluster_kernel) between the down and the up sweep.
long long enqueue_vcycle(MfBatch &b, bool fac, int prec, int sdeg, int cdeg) {
    const Cheb cs = cheb_coeffs(b.cheb_lmax, sdeg), cc = cheb_coeffs(b.cheb_lmax, cdeg);
    const int L = b.n_levels;
    auto any_level = [&](int l) {  // some problem of level l is solved level by level
        if (l == 0 && b.chains_from_root) return false;
        for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++)
            if (!b.h_probs[pi].bottom) return true;
        return false;
    };
    auto own_coarsest = [&](int l) {  // ... and has no coarser level
        for (int pi = b.lvl_prob_lo[l]; pi < b.lvl_prob_hi[l]; pi++)
            if (!b.h_probs[pi].bottom && b.h_probs[pi].coarse < 0) return true;
        return false;
    };
    long long n = 0;
    for (int l = 0; l < L - 1; l++) {
        if (!any_level(l)) continue;
        const float *rin = (l == 0) ? b.r : b.mb;
        n += enqueue_smooth(b, fac, prec, l, rin, 1, sdeg, cs, 0);
        launch_level_op<2>(b, fac, prec, l, 4, b.mx, rin, b.my, 0);  // my = rin - A mx
        if (const int blks = b.lvl_blk_hi[l + 1] - b.lvl_blk_lo[l + 1])
            launch_pdl(mg_restrict_kernel, blks, kNodeBlk, 0, b.stream, b.probs, b.node_blks + b.lvl_blk_lo[l + 1],
                       b.states, b.my, b.mb, b.z, b.dinv);
        n += 2;
        if (own_coarsest(l)) n += enqueue_smooth(b, fac, prec, l, rin, 1, cdeg, cc, 1);
    }
    if (any_level(L - 1)) n += enqueue_smooth(b, fac, prec, L - 1, L == 1 ? b.r : b.mb, 1, cdeg, cc, -1);
    if (!b.h_heads.empty()) {
        BottomCheb bc{};
        bc.inv_theta_s = cs.inv_theta;
        bc.inv_theta_c = cc.inv_theta;
        for (int k = 0; k < 32; k++) {
            bc.c1s[k] = cs.c1[k]; bc.c2s[k] = cs.c2[k];
            bc.c1c[k] = cc.c1[k]; bc.c2c[k] = cc.c2[k];
        }
        launch_cluster_pdl(mg_bottom_cluster_kernel, (unsigned)(b.h_heads.size() * b.bottom_cluster),
                           kClusterThreads, b.bottom_smem, b.bottom_cluster, b.stream, b.cl_chains, b.states, b.E32,
                           b.dinv, b.chains_from_root ? b.r : b.mb, b.mx, b.chains_from_root, b.cl_k0, bc, sdeg, cdeg,
                           b.coarse_off, b.coarse_inv, b.coarse_ok);
        n += 1;
    }
    for (int l = L - 2; l >= 0; l--) {
        if (!any_level(l)) continue;
        const float *rin = (l == 0) ? b.r : b.mb;
        if (const int blks = b.lvl_blk_hi[l + 1] - b.lvl_blk_lo[l + 1])
            launch_pdl(mg_prolong_kernel, blks, kNodeBlk, 0, b.stream, b.probs, b.node_blks + b.lvl_blk_lo[l + 1],
                       b.states, b.mx, b.dinv);
        // my = rin - A mx; the fused smoother starts from z = D^-1 my (and of degree 2 needs no more)
        const bool from_z = fac && sdeg >= 2;
        launch_level_op<2>(b, fac, prec, l, 4, b.mx, rin, from_z && sdeg == 2 ? nullptr : b.my, 0,
                           from_z ? b.z : nullptr);
        n += 2 + enqueue_smooth(b, fac, prec, l, b.my, 0, sdeg, cs, 0);
    }
    return n;
}

// One solver step over every problem of the batch; each kernel acts only on the
// problems in its phase, so problems advance independently:
//   FP64 residual + stop test (RESID) | inner CG start (INIT) |
//   [multigrid z = M r, rz, beta] | p, q = A p, alpha | x, r, stop test |
//   u += d of stopped inner solves | phase transitions.
constexpr int kLoopBodies = 64;  // bodies of one loop launch at most

// the residual and the start of the inner CG
long long enqueue_refine_begin(MfBatch &b, const MfSolveParams &prm) {
    const int n0 = b.lvl_chunk_hi[0], nb0 = b.lvl_brick_hi[0];
    const int vg0 = std::max(1, std::min(n0, b.vec_grid));
    const int maxit = prm.max_iterations > 0 ? prm.max_iterations : 100000;
    const int max_ref = prm.max_refinements > 0 ? prm.max_refinements : 30;
    launch_pdl(mf_residual64_kernel, std::max(1, std::min(nb0, b.res_grid)), kRThreads, kResidSmem, b.stream,
        b.probs, b.bricks, nb0, b.Edf, b.node_fix, b.u64, b.f64, b.facdf, b.r64, b.states,
        b.brick_part, prm.rtol * prm.rtol, max_ref, b.n_fine);
    launch_pdl(mf_inner_init_kernel, vg0, kThreads, 0, b.stream,
        b.chunks, n0, b.probs, b.r64, b.x, b.r, b.z, b.p0, b.p1, b.dinv, b.states, b.chunk_part,
        prm.inner_rtol * prm.inner_rtol, maxit, b.n_fine);
    return 2;
}

// one iteration of the inner CG
long long enqueue_cg(MfBatch &b, const MfSolveParams &prm, int parity) {
    const int n0 = b.lvl_chunk_hi[0];
    const int vg0 = std::max(1, std::min(n0, b.vec_grid));
    const bool use_mg = prm.mg && b.n_levels > 1;
    long long n = 2;
    float *pnew = parity ? b.p0 : b.p1;
    if (use_mg) {
        const int sdeg = prm.smooth_deg > 0 ? prm.smooth_deg : 2;
        const int cdeg = prm.coarse_deg > 0 ? prm.coarse_deg : 8;
        n += enqueue_vcycle(b, prm.mg_operator == 0, mg_precision(prm.precision), sdeg, cdeg);
        if (!b.chains_from_root) {
            launch_pdl(mf_dot_rz_kernel, vg0, kThreads, 0, b.stream, b.chunks, n0, b.probs, b.r, b.mx, b.states,
                       b.chunk_part);
            n += 1;
        }
        launch_cg_apply(b, prm.precision, 4, parity);  // p = z + beta p_old, q = A p, alpha
        launch_update(b, pnew, true);                  // x, r, stop test
    } else {
        launch_cg_apply(b, prm.precision, 0, parity);
        launch_update(b, pnew, false);                 // also z = D^-1 r, beta
    }
    return n;
}

// the refinement update and the phase transitions; loop_end: the end of a while loop's body on
// that handle (nullable)
long long enqueue_refine_end(MfBatch &b, const cudaGraphConditionalHandle *loop_end, bool nested) {
    const int vg0 = std::max(1, std::min(b.lvl_chunk_hi[0], b.vec_grid));
    if (nested)  // behind a loop, not behind a kernel: no programmatic launch
        mf_refine_kernel<<<vg0, kThreads, 0, b.stream>>>(b.chunks, b.probs, b.n_fine, b.x, b.u64, b.states);
    else
        launch_pdl(mf_refine_kernel, vg0, kThreads, 0, b.stream, b.chunks, b.probs, b.n_fine, b.x, b.u64, b.states);
    if (loop_end)
        launch_pdl(mf_phase_kernel<true>, 1, kPhaseThreads, 0, b.stream, b.states, b.n_fine, *loop_end, b.err + 1,
                   kLoopBodies, nested, b.err, b.clock);
    else
        launch_pdl(mf_phase_kernel<false>, 1, kPhaseThreads, 0, b.stream, b.states, b.n_fine,
                   cudaGraphConditionalHandle{}, nullptr, 0, false, nullptr, nullptr);
    return 2;
}

// a while node in graph g behind deps; its body graph
cudaError_t add_while(cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps, cudaGraphConditionalHandle &handle,
                      cudaGraphNode_t &node, cudaGraph_t &body) {
    cudaError_t e = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = handle;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    e = cudaGraphAddNode(&node, g, deps.empty() ? nullptr : deps.data(), nullptr, deps.size(), &np);
    if (e == cudaSuccess) body = np.conditional.phGraph_out[0];
    return e;
}

// what `enqueue` launches, captured into graph g behind deps; last: the nodes it ends on
template <typename Enqueue>
cudaError_t capture_into(cudaStream_t s, cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps, Enqueue enqueue,
                         std::vector<cudaGraphNode_t> *last = nullptr) {
    cudaError_t e = cudaStreamBeginCaptureToGraph(s, g, deps.empty() ? nullptr : deps.data(), nullptr, deps.size(),
                                                  cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    enqueue();
    if (last) {
        cudaStreamCaptureStatus status;
        const cudaGraphNode_t *nodes = nullptr;
        size_t n = 0;
        e = cudaStreamGetCaptureInfo(s, &status, nullptr, nullptr, &nodes, nullptr, &n);
        if (e == cudaSuccess && status == cudaStreamCaptureStatusActive) last->assign(nodes, nodes + n);
    }
    cudaGraph_t captured = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(s, &captured);  // the same graph as g
    return e != cudaSuccess ? e : e2;
}

// CUDA graph of `chunk` solver steps (even: the p0/p1 roles alternate per step),
// cached per parameter set; with `loop` the steps are the body of a while loop that the
// device ends, else they run once per launch.  A solve to completion that returned to the
// host after every two steps spent 20 us a round trip on it (16x8x8 2.60 -> 2.24 ms looped,
// 48x24x24 4.64 -> 4.26, 128x64x64 8.21 -> 7.83); the request loop launches single bodies,
// between which it admits requests.  A single problem's CG steps loop inside its refinement
// loop, so that they do not launch the refinement's four kernels each time to find nothing to do
// (1.4 to 2.9 us apiece: 90x46x38 6.59 -> 6.51 ms, 64x32x32 BF16X3 6.63 -> 6.59);
// the problems of a batch are in different phases.
int build_step_graph(MfBatch &b, const MfSolveParams &prm, int chunk, bool loop) {
    const std::vector<double> key = {(double)prm.precision, (double)chunk, (double)prm.mg,
                                     (double)prm.smooth_deg, (double)prm.coarse_deg, prm.rtol,
                                     prm.inner_rtol, (double)prm.max_iterations,
                                     (double)prm.max_refinements, (double)b.vec_grid,
                                     (double)prm.mg_operator, loop ? (b.n_fine == 1 ? 2.0 : 1.0) : 0.0};
    if (b.graph && b.graph_key == key) return MG_OK;
    if (b.graph) {
        cudaGraphExecDestroy(b.graph);
        b.graph = nullptr;
    }
    cudaGraph_t g = nullptr;
    MG_CUDA_TRY(cudaGraphCreate(&g, 0));
    const bool nested = loop && b.n_fine == 1;
    cudaGraph_t body = g, inner = nullptr;
    cudaGraphConditionalHandle handle{}, inner_handle{};
    cudaGraphNode_t node;
    cudaError_t e = loop ? add_while(g, {}, handle, node, body) : cudaSuccess;
    long long n = 0, n_outer = 0;
    b.enqueue_error = 0;
    if (e == cudaSuccess && nested) {
        // the refinement's start and the first decision; the CG loop; the refinement's end.  The
        // inner loop's handle belongs to the outer body, so its node is made before the capture
        // of what sets it, and the edge to it afterwards.
        std::vector<cudaGraphNode_t> last;
        e = add_while(body, {}, inner_handle, node, inner);
        if (e == cudaSuccess)
            e = capture_into(b.stream, body, {}, [&] {
                n_outer += enqueue_refine_begin(b, prm);
                launch_pdl(mf_gate_kernel, 1, 1, 0, b.stream, b.states, inner_handle, b.err + 1, kLoopBodies, false, b.err,
                           b.clock);
                n_outer += 1;
            }, &last);
        for (size_t k = 0; k < last.size() && e == cudaSuccess; k++)
            e = cudaGraphAddDependencies(body, &last[k], &node, nullptr, 1);
        if (e == cudaSuccess)
            e = capture_into(b.stream, inner, {}, [&] {
                for (int it = 0; it < chunk; it++) n += enqueue_cg(b, prm, it & 1);
                launch_pdl(mf_gate_kernel, 1, 1, 0, b.stream, b.states, inner_handle, b.err + 1, kLoopBodies, true, b.err,
                           b.clock);
                n += 1;
            });
        if (e == cudaSuccess)
            e = capture_into(b.stream, body, {node}, [&] { n_outer += enqueue_refine_end(b, &handle, true); });
    } else if (e == cudaSuccess) {
        e = capture_into(b.stream, body, {}, [&] {
            for (int it = 0; it < chunk; it++) {
                n += enqueue_refine_begin(b, prm);
                n += enqueue_cg(b, prm, it & 1);
                n += enqueue_refine_end(b, loop && it == chunk - 1 ? &handle : nullptr, false);
            }
        });
    }
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        set_error("graph capture: %s", cudaGetErrorString(e));
        return MG_ECUDA;
    }
    if (b.enqueue_error) {
        cudaGraphDestroy(g);
        set_error("factored level operator: a vector without a tensor map");
        return b.enqueue_error;
    }
    e = cudaGraphInstantiate(&b.graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        b.graph = nullptr;
        set_error("graph instantiate: %s", cudaGetErrorString(e));
        return MG_ECUDA;
    }
    b.graph_key = key;
    b.graph_launches = n;
    b.graph_outer = n_outer;
    return MG_OK;
}

}  // namespace

// FP64 iterative refinement around FP32 tensor-core CG, per problem:
//   r = f - K u (FP64);  stop when ||r|| <= rtol ||f||;
//   solve A d = r / ||r|| with FP32 CG to inner_rtol (Jacobi or multigrid
//   V-cycle preconditioned);  u += ||r|| d.
// The phases run on the device (build_step_graph); the host only relaunches the
// step graph until every active problem has finished.
int mf_batch_prepare(MfBatch &b, const MfSolveParams &prm, bool loop) {
    const bool use_mg = prm.mg && b.n_levels > 1;
    // launch shape of the vector kernels (captured in the graph)
    int dev = 0, sms = 0;
    MG_CUDA_TRY(cudaGetDevice(&dev));
    MG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int per_sm = prm.vec_blocks_per_sm > 0 ? std::min(prm.vec_blocks_per_sm, 64) : 8;
    const int vg = std::max(1, std::min(b.n_chunks, per_sm * sms));
    if (vg != b.vec_grid) {
        b.vec_grid = vg;
        if (b.graph) cudaGraphExecDestroy(b.graph);
        b.graph = nullptr;
    }
    const int chunk = prm.graph_chunk > 0 ? (prm.graph_chunk + 1) / 2 * 2 : (use_mg ? 2 : 16);
    MfSolveParams p2 = prm;
    p2.mg = use_mg ? 1 : 0;
    return build_step_graph(b, p2, chunk, loop);
}

int mf_batch_reset_states(MfBatch &b, double budget_s) {
    std::vector<MfState> init(b.n_probs + 1);  // and the loop's clock behind the states
    memset(init.data(), 0, init.size() * sizeof(MfState));
    for (int i = 0; i < b.n_probs; i++) {
        init[i].done = 1;
        init[i].ref_done = 1;
        init[i].phase = kPhaseFin;
    }
    MfLoopClock clock{0, 0};
    if (budget_s > 0) clock.budget_ns = (int64_t)std::max(1.0, std::min(budget_s * 1e9, 9e18));
    memcpy(&init[b.n_probs], &clock, sizeof(clock));
    MG_CUDA_TRY(cudaMemcpyAsync(b.states, init.data(), init.size() * sizeof(MfState), cudaMemcpyHostToDevice,
                                b.stream));
    MG_CUDA_TRY(cudaStreamSynchronize(b.stream));  // init is a host temporary
    memcpy(b.states_host, init.data(), b.n_probs * sizeof(MfState));
    return MG_OK;
}

int mf_batch_activate(MfBatch &b, const std::vector<int> &level0, bool warm_start) {
    for (int i : level0)
        if (i < 0 || i >= b.n_fine) return MG_EINVAL;
    MG_TRY(compute_diag_list(b, level0));
    for (int i : level0) {
        const MfProblem &P = b.h_probs[i];
        if (!warm_start) MG_CUDA_TRY(cudaMemsetAsync(b.u64 + P.dof_off, 0, P.n_pad * 8, b.stream));
        // the pinned host mirror entry is the staging buffer; the next
        // read_states (later in stream order) overwrites it
        MfState &h = b.states_host[i];
        memset(&h, 0, sizeof(MfState));
        h.done = 1;
        h.phase = kPhaseResid;  // its first residual pass also forms ||f||^2
        h.resid = 1;
        h.u_zero = warm_start ? 0 : 1;
        MG_CUDA_TRY(cudaMemcpyAsync(b.states + i, &h, sizeof(MfState), cudaMemcpyHostToDevice, b.stream));
    }
    return MG_OK;
}

int mf_batch_step_begin(MfBatch &b) {
    if (!b.graph) {
        set_error("mf_batch_step before mf_batch_prepare");
        return MG_EINVAL;
    }
    MG_CUDA_TRY(cudaGraphLaunch(b.graph, b.stream));
    // only the level-0 problems have a solver state
    MG_CUDA_TRY(cudaMemcpyAsync(b.states_host, b.states, b.n_fine * sizeof(MfState), cudaMemcpyDeviceToHost,
                                b.stream));
    MG_CUDA_TRY(cudaMemcpyAsync(b.err_host, b.err, kErrWords * sizeof(int), cudaMemcpyDeviceToHost, b.stream));
    return MG_OK;
}

int mf_batch_step_end(MfBatch &b) {
    MG_CUDA_TRY(cudaStreamSynchronize(b.stream));
    // a loop launch reports the bodies it has run
    count_launches(b.graph_launches * (b.graph_key.back() != 0.0 ? b.err_host[2] - b.loop_bodies : 1) +
                   b.graph_outer * (b.err_host[3] - b.loop_outer));
    b.loop_bodies = b.err_host[2];
    b.loop_outer = b.err_host[3];
    if (*b.err_host) {
        set_error("tensor-core pipeline wait exceeded its bound (error flag %d)", *b.err_host);
        return MG_ETIMEDOUT;
    }
    return MG_OK;
}

int mf_batch_finish(MfBatch &b, int i) {
    // a zero load gives u = 0 (the residual pass marks it with ||f||^2 = -1)
    if (b.states_host[i].ff64 < 0.0)
        MG_CUDA_TRY(cudaMemsetAsync(b.u64 + b.h_probs[i].dof_off, 0, b.h_probs[i].n_pad * 8, b.stream));
    return b.states_host[i].ref_status;
}

int mf_batch_solve(MfBatch &b, const MfSolveParams &prm, bool warm_start) {
    const double t0 = wall_time();
    MG_TRY(mf_batch_prepare(b, prm, true));
    // the time left, or none: the loop ends within a body of it
    MG_TRY(mf_batch_reset_states(b, prm.timeout_s > 0 ? std::max(1e-9, prm.timeout_s - (wall_time() - t0)) : 0.0));
    std::vector<int> act;
    for (int i = 0; i < b.n_fine; i++)
        if (!prm.active || prm.active[i]) act.push_back(i);
    MG_TRY(mf_batch_activate(b, act, warm_start));
    for (;;) {
        MG_TRY(mf_batch_step_begin(b));
        MG_TRY(mf_batch_step_end(b));
        bool all_done = true;
        for (int i : act) all_done &= b.states_host[i].phase == kPhaseFin;
        if (all_done) break;
        if (prm.timeout_s > 0 && wall_time() - t0 > prm.timeout_s) {
            set_error("mixed solve exceeded %.1f s", prm.timeout_s);
            return MG_ETIMEDOUT;
        }
    }
    int rc = MG_OK;
    for (int i : act) {
        const int st = mf_batch_finish(b, i);
        if (st != 0 && rc == MG_OK) rc = st;
    }
    return rc;
}

// compliance f.u per design (host) and dC/drho (unpadded, designs back to back
// in problem order at dc_unpadded_dev) from the resident solutions
int mf_batch_compliance(MfBatch &b, double *compliance_host, double *dc_unpadded_dev,
                        const uint8_t *active) {
    cudaStream_t s = b.stream;
    const int n0 = b.lvl_chunk_hi[0];
    if (compliance_host) {
        mf_dot_chunks_kernel<<<std::max(1, std::min(n0, b.vec_grid)), kThreads, 0, s>>>(
            b.chunks, n0, b.f64, b.u64, b.chunk_part);
        MG_CUDA_TRY(cudaGetLastError());
        std::vector<double> part(n0);
        MG_CUDA_TRY(cudaMemcpyAsync(part.data(), b.chunk_part, n0 * 8, cudaMemcpyDeviceToHost, s));
        MG_CUDA_TRY(cudaStreamSynchronize(s));
        for (int i = 0; i < b.n_fine; i++) {
            const MfProblem &P = b.h_probs[i];
            double c = 0;
            for (int k = 0; k < P.chunk_count; k++) c += part[P.chunk_begin + k];
            compliance_host[i] = c;
        }
    }
    if (dc_unpadded_dev) {
        // output offsets through the batch's pinned staging (free again when this returns)
        int64_t *offs = b.sens_offs_host;
        int64_t o = 0, max_ne = 1;
        for (int i = 0; i < b.n_fine; i++) {
            const MfProblem &P = b.h_probs[i];
            offs[i] = (active && !active[i]) ? -1 : o;  // -1: leave this problem's output
            o += (int64_t)P.nx * P.ny * P.nz;
            max_ne = std::max<int64_t>(max_ne, (int64_t)P.nx * P.ny * P.nz);
        }
        MG_CUDA_TRY(cudaMemcpyAsync(b.sens_offs, offs, b.n_fine * 8, cudaMemcpyHostToDevice, s));
        dim3 grid(std::max(1u, std::min(blocks_for(max_ne, 128), 4096u)), b.n_fine);
        mf_sens_kernel<<<grid, 128, 0, s>>>(b.probs, b.n_fine, b.dE64, b.node_fix, b.u64, b.facdf,
                                            b.sens_offs, dc_unpadded_dev);
        cudaError_t e = cudaGetLastError();
        cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("sensitivity kernel: %s", cudaGetErrorString(e));
            return MG_ECUDA;
        }
    }
    return MG_OK;
}

// ----------------------------------------------------- single-problem mixed path
struct MatfreeWork {
    MfBatch batch;
};

namespace {

int matfree_setup(mg_problem *p) {
    if (p->mf) return MG_OK;
    if (p->physics != MG_PHYSICS_ELASTICITY_HEX8 || p->grid_nx <= 0 || p->grid_ny <= 0 ||
        p->grid_nz <= 0 || (int64_t)p->grid_nx * p->grid_ny * p->grid_nz != p->n_elems) {
        set_error("the mixed form needs the structured HEX8 grid (grid dims)");
        return MG_ENOTSUP;
    }
    const int nx = p->grid_nx, ny = p->grid_ny, nz = p->grid_nz;
    // the grid must be uniform: coords(i,j,k) = (i hx, j hy, k hz) + origin
    const double *c = p->h_coords.data();
    const int64_t NX = nx + 1, NY = ny + 1;
    const double hx = c[3] - c[0], hy = c[NX * 3 + 1] - c[1], hz = c[NX * NY * 3 + 2] - c[2];
    for (int64_t n = 0; n < p->n_nodes; n++) {
        const int64_t i = n % NX, j = (n / NX) % NY, k = n / (NX * NY);
        if (fabs(c[n * 3] - (c[0] + i * hx)) > 1e-9 * (1 + fabs(hx) * nx) ||
            fabs(c[n * 3 + 1] - (c[1] + j * hy)) > 1e-9 * (1 + fabs(hy) * ny) ||
            fabs(c[n * 3 + 2] - (c[2] + k * hz)) > 1e-9 * (1 + fabs(hz) * nz)) {
            set_error("mesh is not a uniform structured grid");
            return MG_ENOTSUP;
        }
    }
    for (int64_t e = 0; e < p->n_elems; e++) {
        const int64_t i = e % nx, j = (e / nx) % ny, k = e / ((int64_t)nx * ny);
        if (p->h_conn[e * 8] != (int32_t)(i + NX * (j + NY * k))) {
            set_error("connectivity is not the libMesh grid numbering");
            return MG_ENOTSUP;
        }
    }
    MatfreeWork *w = new MatfreeWork();
    MfProblem P{};
    P.nx = nx; P.ny = ny; P.nz = nz;
    P.share_elems = -1;
    int rc = mf_batch_init(w->batch, {P}, hx, hy, hz, p->mat.nu, p->stream, kMaxLevels, true);
    if (rc == MG_OK) {
        std::vector<uint8_t> nf(p->n_nodes, 0);
        for (int64_t n = 0; n < p->n_nodes; n++)
            for (int cc = 0; cc < 3; cc++)
                if (p->h_fixed[n * 3 + cc]) nf[n] |= (uint8_t)(1u << cc);
        rc = mf_batch_set_bc(w->batch, 0, nf.data(), p->h_F.data());
    }
    if (rc != MG_OK) {
        mf_batch_free(w->batch);
        delete w;
        return rc;
    }
    p->mf = w;
    return MG_OK;
}

}  // namespace

int matfree_solve(mg_problem *p, const mg_solve_opts &o, mg_solve_report *rep, bool x_zero) {
    MG_TRY(matfree_setup(p));
    MfBatch &b = p->mf->batch;
    MG_TRY(mf_batch_set_moduli(b, 0, p->d_E, p->d_dE));
    if (!x_zero) {
        MG_TRY(mf_batch_set_u(b, 0, p->d_X));
        count_launches(1);
    }
    MfSolveParams prm;
    prm.precision = o.precision;
    prm.rtol = o.rtol;
    prm.inner_rtol = o.inner_rtol > 0 ? o.inner_rtol : 1e-4;
    prm.max_iterations = o.max_iterations;
    prm.max_refinements = o.max_refinements;
    prm.graph_chunk = o.graph_chunk;
    prm.timeout_s = o.timeout_s;
    prm.mg = (o.preconditioner == MG_PC_MULTIGRID) ? 1 : 0;
    prm.smooth_deg = o.smooth_degree;
    prm.coarse_deg = o.coarse_degree;
    prm.vec_blocks_per_sm = o.vec_blocks_per_sm;
    prm.mg_operator = o.smoother_operator == MG_SMOOTHER_TENSOR ? 1 : 0;
    // from 0 (activation clears u): the first residual is f without an operator pass
    int rc = mf_batch_solve(b, prm, !x_zero);
    MG_TRY(mf_batch_get_u(b, 0, p->d_X));
    count_launches(1);
    MG_CUDA_TRY(cudaStreamSynchronize(p->stream));
    const MfState &h = b.states_host[0];
    if (rep) {
        rep->newton_iterations = 1;
        rep->krylov_iterations = h.total_iter;
        rep->refinements = h.refine;
        rep->relres = h.ff64 > 0.0 ? sqrt(h.rr64 / h.ff64) : 0.0;
        rep->residual_norm = sqrt(h.rr64);
    }
    return rc;
}

int matfree_apply_debug(mg_problem *p, int precision, const double *x_host, double *y_host) {
    MG_TRY(matfree_setup(p));
    MfBatch &b = p->mf->batch;
    MG_TRY(mf_batch_set_moduli(b, 0, p->d_E, p->d_dE));
    return mf_apply(b, precision, x_host, y_host, 0);
}

// dC/drho from the resident solution with the shared K0 (FP64)
int matfree_sensitivity(mg_problem *p, double *dc_host) {
    MG_TRY(matfree_setup(p));
    MfBatch &b = p->mf->batch;
    MG_TRY(mf_batch_set_moduli(b, 0, p->d_E, p->d_dE));
    MG_TRY(mf_batch_set_u(b, 0, p->d_X));
    MG_TRY(mf_batch_compliance(b, nullptr, p->d_elem_out));
    MG_CUDA_TRY(cudaMemcpyAsync(dc_host, p->d_elem_out, p->n_elems * 8, cudaMemcpyDeviceToHost, p->stream));
    MG_CUDA_TRY(cudaStreamSynchronize(p->stream));
    return MG_OK;
}

int matfree_compliance_resident(mg_problem *p, double *compliance) {
    MG_TRY(matfree_setup(p));
    MfBatch &b = p->mf->batch;
    double c = 0.0;
    MG_TRY(mf_batch_compliance(b, &c, p->d_elem_out));
    count_launches(2);
    if (compliance) *compliance = c;
    return MG_OK;
}

int matfree_launch_apply(mg_problem *p, int precision, int reps) {
    MG_TRY(matfree_setup(p));
    MfBatch &b = p->mf->batch;
    MG_TRY(mf_batch_set_moduli(b, 0, p->d_E, p->d_dE));
    return mf_launch_apply(b, precision, reps);
}

void matfree_free(mg_problem *p) {
    if (!p->mf) return;
    mf_batch_free(p->mf->batch);
    delete p->mf;
    p->mf = nullptr;
}

}  // namespace mg
