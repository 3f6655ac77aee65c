// filter.cu -- the density filter of MAST::FilterBase on the GPU (mg_filter_*).
//
// MAST (src/level_set/filter_base.cpp) filters the design field with
// normalised hat weights: point i takes w_ij = (r - d_ij) / sum_k (r - d_ik)
// over all points j within distance r (`_init` :378-437, `_init2` :275-359);
// compute_filtered_values (:58-95) forms sum_j w_ij x_j for design-variable
// points and passes the others through.  The design-gradient chain rule of the
// topology-optimisation loop (examples/structural/example_6/example_6.cpp:
// 661-697, where the filtered unit perturbations become the density
// sensitivities) is the transpose: dq/dx = F^T dq/dx_filtered.
//
// Two layouts:
//   * structured grids: the element centroids form a lattice, so the weights
//     are one stencil of integer offsets, applied with the per-point normalisation
//     (which only differs near the boundary) precomputed: with mirrored offsets
//     folded together where it is a ball of cells, else one point per thread;
//   * arbitrary points: the neighbour lists are found on the host with a
//     bucket grid of cell size r and stored as a CSR matrix and its transpose;
//     FP64 CSR products apply F and F^T.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <unordered_map>
#include <vector>

#include "mg_internal.h"

namespace mg {
namespace {

inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

struct StencilArgs {
    int nx, ny, nz;       // grid (nz = 1 in 2D)
    int n_off;
    const int *ox, *oy, *oz;
    const double *w;      // r - d per offset
};

// S_e = sum of the in-domain stencil weights; stores 1 / S_e
__global__ void stencil_norm_kernel(StencilArgs a, double *__restrict__ inv_s) {
    const int64_t n = (int64_t)a.nx * a.ny * a.nz;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e % a.nx), j = (int)((e / a.nx) % a.ny), k = (int)(e / ((int64_t)a.nx * a.ny));
        double s = 0.0;
        for (int o = 0; o < a.n_off; o++) {
            const int ii = i + a.ox[o], jj = j + a.oy[o], kk = k + a.oz[o];
            if (ii < 0 || jj < 0 || kk < 0 || ii >= a.nx || jj >= a.ny || kk >= a.nz) continue;
            s += a.w[o];
        }
        inv_s[e] = 1.0 / s;
    }
}

// forward: out_e = dv_e ? sum_o w_o in_{e+o} / S_e : in_e
// transpose: out_f = (dv_f ? 0 : in_f) + sum_o w_o [dv_{f+o}] in_{f+o} / S_{f+o}
// (the stencil is symmetric, so the transpose gathers over the same offsets)
__global__ void stencil_apply_kernel(StencilArgs a, const double *__restrict__ inv_s,
                                     const uint8_t *__restrict__ dv, const double *__restrict__ in,
                                     double *__restrict__ out, int transpose) {
    const int64_t n = (int64_t)a.nx * a.ny * a.nz;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e % a.nx), j = (int)((e / a.nx) % a.ny), k = (int)(e / ((int64_t)a.nx * a.ny));
        const bool is_dv = !dv || dv[e];
        if (!transpose && !is_dv) {
            out[e] = in[e];
            continue;
        }
        double acc = 0.0;
        for (int o = 0; o < a.n_off; o++) {
            const int ii = i + a.ox[o], jj = j + a.oy[o], kk = k + a.oz[o];
            if (ii < 0 || jj < 0 || kk < 0 || ii >= a.nx || jj >= a.ny || kk >= a.nz) continue;
            const int64_t f = ii + (int64_t)a.nx * (jj + (int64_t)a.ny * kk);
            if (!transpose) acc = fma(a.w[o], in[f], acc);
            else if (!dv || dv[f]) acc = fma(a.w[o], in[f] * inv_s[f], acc);
        }
        out[e] = transpose ? (is_dv ? acc : acc + in[e]) : acc * inv_s[e];
    }
}

// The same stencil where it is a ball of up to kFoldMax cells.  The weights depend on |a|, |b|, |c| only, so values at
// mirrored offsets are added before they are multiplied: along x into F_a = v(x - a) +
// v(x + a), along y into G_ab = F_a(y - b) + F_a(y + b), and the plane sums P_c = sum_ab
// w_abc G_ab go to the outputs at z - c and z + c.  For a radius of 2.5 cells that is 32 FP64
// operations a point instead of 81, on a GPU whose FP64 pipe (two DFMA per cycle and SM)
// binds the filter.  A block of 32 x 4 points marches through a chunk of z planes; the
// outputs still open sit in registers, the next plane is fetched while one is folded.
// Microseconds at 128x64x64, one point per thread -> folded: radius 1.5 25 -> 25 (transpose
// 43 -> 29), 2.5 86 -> 60 (166 -> 72), 3.5 184 -> 107 (358 -> 125); 32x16x16 with 2.5 cells 14.5 ->
// 8.4 (16.6 -> 10.5).  Larger radii and uneven spacings keep the form above.
constexpr int kFoldX = 32, kFoldY = 4, kFoldMax = 3;  // kFoldMax: most cells of the radius

struct FoldWeights {
    double w[(kFoldMax + 1) * (kFoldMax + 1) * (kFoldMax + 1)];  // [c][b][a]
};

// A: cells of the radius; D: the stencil is a^2 + b^2 + c^2 <= D (known to the compiler: with
// a test per weight the sums became chains of single instructions, twice the time)
template <int A, int D>
__global__ void __launch_bounds__(kFoldX * kFoldY) stencil_fold_kernel(
    int nx, int ny, int nz, int zc, const FoldWeights W, const double *__restrict__ inv_s,
    const uint8_t *__restrict__ dv, const double *__restrict__ in, double *__restrict__ out, int transpose) {
    constexpr int H = kFoldY + 2 * A, NR = (H + kFoldY - 1) / kFoldY;  // rows of a plane, per warp
    __shared__ double F[2][A + 1][H][kFoldX];                          // F_0 = v; double-buffered
    auto weight = [&](int c, int b, int a) { return W.w[(c * (kFoldMax + 1) + b) * (kFoldMax + 1) + a]; };
    auto inside = [](int c, int b, int a) { return a * a + b * b + c * c <= D; };
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * kFoldX, y0 = blockIdx.y * kFoldY, z0 = blockIdx.z * zc, z1 = min(z0 + zc, nz);
    const int x = x0 + tx, y = y0 + ty;
    const bool own = x < nx && y < ny;
    const int64_t plane = (int64_t)nx * ny, col = x + (int64_t)nx * y;
    // a warp's rows: lane = x, and the row's 2 A halo points (A left, then A right) in lanes 0 .. 2 A - 1
    const int xh = tx < A ? x0 - A + tx : x0 + kFoldX + tx - A;
    const bool in_x = x < nx, in_h = tx < 2 * A && xh >= 0 && xh < nx;
    auto value = [&](int64_t e) { return !transpose ? in[e] : (!dv || dv[e]) ? in[e] * inv_s[e] : 0.0; };
    auto fetch = [&](int p, double (&v)[NR], double (&h)[NR]) {
#pragma unroll
        for (int k = 0; k < NR; k++) {
            const int r = ty + k * kFoldY, j = y0 - A + r;
            const bool row = r < H && j >= 0 && j < ny && p >= 0 && p < nz;
            const int64_t e = (int64_t)nx * j + plane * p;
            v[k] = row && in_x ? value(e + x) : 0.0;
            h[k] = row && in_h ? value(e + xh) : 0.0;
        }
    };
    double acc[2 * A + 1], v[NR], h[NR];  // acc[j]: the output plane p - A + j
#pragma unroll
    for (int j = 0; j <= 2 * A; j++) acc[j] = 0.0;
    fetch(z0 - A, v, h);
    for (int p = z0 - A; p < z1 + A; p++) {
        const bool live = p >= 0 && p < nz;  // uniform
        // what the output completed by this plane needs, fetched before the arithmetic
        const int z = p - A;
        const bool emit = own && z >= z0;
        const int64_t eo = emit ? col + plane * z : 0;
        const bool is_dv = !emit || !dv || dv[eo];
        const double so = emit && !transpose ? inv_s[eo] : 0.0, keep = emit && dv ? in[eo] : 0.0;
        double(*Fp)[H][kFoldX] = F[p & 1];
        if (live) {
#pragma unroll
            for (int k = 0; k < NR; k++) {
                const int r = ty + k * kFoldY;
                if (r >= H) break;  // whole warps
                Fp[0][r][tx] = v[k];
#pragma unroll
                for (int a = 1; a <= A; a++) {
                    // v(x - a): the halo's lane A + x - a where x < a; v(x + a) likewise
                    const double l = __shfl_sync(0xffffffffu, v[k], (tx - a) & 31),
                                 lh = __shfl_sync(0xffffffffu, h[k], (A + tx - a) & 31),
                                 g = __shfl_sync(0xffffffffu, v[k], (tx + a) & 31),
                                 gh = __shfl_sync(0xffffffffu, h[k], (A + tx + a - kFoldX) & 31);
                    Fp[a][r][tx] = (tx < a ? lh : l) + (tx + a >= kFoldX ? gh : g);
                }
            }
        }
        if (p + 1 < z1 + A) fetch(p + 1, v, h);
        __syncthreads();
        if (live) {
            double G[A + 1][A + 1];  // [b][a]
#pragma unroll
            for (int b = 0; b <= A; b++)
#pragma unroll
                for (int a = 0; a <= A; a++) {
                    if (!inside(0, b, a)) continue;  // then no plane uses it
                    G[b][a] = Fp[a][ty + A - b][tx];
                    if (b) G[b][a] += Fp[a][ty + A + b][tx];
                }
#pragma unroll
            for (int c = 0; c <= A; c++) {
                // planes outside the chunk take nothing from this one
                const bool below = p - c >= z0 && p - c < z1, above = c && p + c >= z0 && p + c < z1;
                if (!(below || above)) continue;
                double P = 0.0;
#pragma unroll
                for (int b = 0; b <= A; b++)
#pragma unroll
                    for (int a = 0; a <= A; a++)
                        if (inside(c, b, a)) P = fma(weight(c, b, a), G[b][a], P);
                if (below) acc[A - c] += P;
                if (above) acc[A + c] += P;
            }
        }
        if (emit) out[eo] = transpose ? (is_dv ? acc[0] : acc[0] + keep) : (is_dv ? acc[0] * so : keep);
#pragma unroll
        for (int j = 0; j < 2 * A; j++) acc[j] = acc[j + 1];
        acc[2 * A] = 0.0;
    }
}

// y_i = (pass_i ? x_i : 0) + sum_k vals_k x_cols_k (one warp per row)
__global__ void csr_filter_kernel(int64_t n, const int64_t *__restrict__ rowptr, const int32_t *__restrict__ cols,
                                  const double *__restrict__ vals, const uint8_t *__restrict__ pass,
                                  const uint8_t *__restrict__ gate, const double *__restrict__ x,
                                  double *__restrict__ y) {
    const int lane = threadIdx.x & 31;
    for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n;
         row += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        double acc = 0.0;
        for (int64_t k = rowptr[row] + lane; k < rowptr[row + 1]; k += 32) {
            const int32_t c = cols[k];
            if (!gate || gate[c]) acc = fma(vals[k], x[c], acc);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) y[row] = (pass && pass[row]) ? x[row] + acc : acc;
    }
}

}  // namespace
}  // namespace mg

using namespace mg;

struct mg_filter {
    cudaStream_t stream = nullptr;
    int64_t n = 0, nnz = 0;
    bool grid = false;
    StencilArgs st{};
    FoldWeights fold{};
    int fold_a = 0, fold_d = 0, fold_zc = 0;  // the folded form's shape (fold_a = 0: not used), planes per block
    int *d_ox = nullptr, *d_oy = nullptr, *d_oz = nullptr;
    double *d_w = nullptr, *d_inv_s = nullptr;
    uint8_t *d_dv = nullptr, *d_not_dv = nullptr;
    // points: F (rows: filtered points) and F^T, normalised weights
    int64_t *d_rp = nullptr, *d_rpt = nullptr;
    int32_t *d_c = nullptr, *d_ct = nullptr;
    double *d_v = nullptr, *d_vt = nullptr;
    double *d_in = nullptr, *d_out = nullptr;  // staging for host buffers
};

namespace mg {
namespace {

template <class T>
int upload(T **dst, const T *src, size_t n, cudaStream_t s) {
    MG_TRY(dev_alloc_n(dst, std::max<size_t>(n, 1)));
    if (n) MG_CUDA_TRY(cudaMemcpyAsync(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice, s));
    return MG_OK;
}

int finish_create(mg_filter *f, const uint8_t *dv) {
    MG_TRY(dev_alloc_n(&f->d_in, (size_t)f->n));
    MG_TRY(dev_alloc_n(&f->d_out, (size_t)f->n));
    if (dv) {
        MG_TRY(upload(&f->d_dv, dv, (size_t)f->n, f->stream));
        std::vector<uint8_t> nd((size_t)f->n);
        for (int64_t i = 0; i < f->n; i++) nd[i] = dv[i] ? 0 : 1;
        MG_TRY(upload(&f->d_not_dv, nd.data(), nd.size(), f->stream));
        MG_CUDA_TRY(cudaStreamSynchronize(f->stream));
    }
    return MG_OK;
}

// z planes per block of the folded form.  A plane of a block takes the FP64 pipe for
// kFoldCycles per warp instruction (counted from the stencil) and about kFoldLatency cycles
// more before its results are there (barrier, shared memory, one chain of sums), which only
// other blocks of the SM can fill; a halo plane is partial work.  The cheapest choice by that
// model: 128x64x64 with 2.5 cells takes 16 planes, two blocks on most SMs.
constexpr double kFoldCycles = 18.0, kFoldLatency = 2500.0;

int fold_chunk(const mg_filter *f, int sms) {
    const int A = f->fold_a, nz = f->st.nz;
    int pairs = 0, products = 0;
    for (int c = 0; c <= A; c++)
        for (int b = 0; b <= A; b++)
            for (int a = 0; a <= A; a++)
                if (a * a + b * b + c * c <= f->fold_d) {
                    products++;
                    pairs += c == 0;
                }
    const double work = kFoldCycles * (A * (kFoldY + 2 * A) + kFoldY * (pairs - A - 1 + products + 2 * A + 2));
    const int64_t tiles = (int64_t)((f->st.nx + kFoldX - 1) / kFoldX) * ((f->st.ny + kFoldY - 1) / kFoldY);
    int best = 1;
    double least = 1e300;
    for (int zc = 1; zc <= nz; zc++) {
        const int64_t rounds = (tiles * ((nz + zc - 1) / zc) + sms - 1) / sms;
        const double cost = (zc + 1.2 * A) * std::max(rounds * work, work + kFoldLatency);
        if (cost < least) {
            least = cost;
            best = zc;
        }
    }
    return best;
}

template <int A, int D>
void launch_fold(const mg_filter *f, const double *in, double *out, int transpose, cudaStream_t s) {
    const StencilArgs &a = f->st;
    const dim3 grid((a.nx + kFoldX - 1) / kFoldX, (a.ny + kFoldY - 1) / kFoldY, (a.nz + f->fold_zc - 1) / f->fold_zc);
    stencil_fold_kernel<A, D><<<grid, dim3(kFoldX, kFoldY), 0, s>>>(a.nx, a.ny, a.nz, f->fold_zc, f->fold, f->d_inv_s,
                                                                    f->d_dv, in, out, transpose);
}

// the squared radii (in cells) between which a ball of cells changes, up to kFoldMax cells
constexpr int kFoldBalls[] = {1, 2, 3, 4, 5, 6, 8, 9, 10, 11, 12, 13, 14};

void dispatch_fold(const mg_filter *f, const double *in, double *out, int transpose, cudaStream_t s) {
    switch (f->fold_d) {
        case 1: launch_fold<1, 1>(f, in, out, transpose, s); break;
        case 2: launch_fold<1, 2>(f, in, out, transpose, s); break;
        case 3: launch_fold<1, 3>(f, in, out, transpose, s); break;
        case 4: launch_fold<2, 4>(f, in, out, transpose, s); break;
        case 5: launch_fold<2, 5>(f, in, out, transpose, s); break;
        case 6: launch_fold<2, 6>(f, in, out, transpose, s); break;
        case 8: launch_fold<2, 8>(f, in, out, transpose, s); break;
        case 9: launch_fold<3, 9>(f, in, out, transpose, s); break;
        case 10: launch_fold<3, 10>(f, in, out, transpose, s); break;
        case 11: launch_fold<3, 11>(f, in, out, transpose, s); break;
        case 12: launch_fold<3, 12>(f, in, out, transpose, s); break;
        case 13: launch_fold<3, 13>(f, in, out, transpose, s); break;
        case 14: launch_fold<3, 14>(f, in, out, transpose, s); break;
    }
}

// The folded form's shape for a stencil of offsets (a, b, c) with weights w, or none: the
// offsets have to be exactly those of a ball of cells (2D grids: a disc).
void plan_fold(mg_filter *f, const std::vector<int> &ox, const std::vector<int> &oy, const std::vector<int> &oz,
               const std::vector<double> &w, bool flat) {
    int far = 0;
    for (size_t o = 0; o < w.size(); o++) far = std::max(far, ox[o] * ox[o] + oy[o] * oy[o] + oz[o] * oz[o]);
    // 2D: the smallest ball whose disc holds the stencil (the planes above and below are empty)
    for (int d : kFoldBalls) {
        if (d < far) continue;
        size_t count = 0;
        for (int c = flat ? 0 : -kFoldMax; c <= (flat ? 0 : kFoldMax); c++)
            for (int b = -kFoldMax; b <= kFoldMax; b++)
                for (int a = -kFoldMax; a <= kFoldMax; a++) count += a * a + b * b + c * c <= d;
        if (count != w.size()) continue;
        f->fold_d = d;
        f->fold_a = d < 4 ? 1 : d < 9 ? 2 : 3;
        for (size_t o = 0; o < w.size(); o++)
            if (ox[o] >= 0 && oy[o] >= 0 && oz[o] >= 0)
                f->fold.w[(oz[o] * (kFoldMax + 1) + oy[o]) * (kFoldMax + 1) + ox[o]] = w[o];
        return;
    }
}

int run(mg_filter *f, const double *in, double *out, int transpose, cudaStream_t s) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        MG_CUDA_TRY(cudaGetDevice(&dev));
        MG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    }
    if (f->grid && f->fold_a) {
        if (!f->fold_zc) f->fold_zc = fold_chunk(f, sms);
        dispatch_fold(f, in, out, transpose, s);
    } else if (f->grid) {
        const unsigned g = std::min(blocks_for(f->n, 256), (unsigned)(8 * sms));
        stencil_apply_kernel<<<g, 256, 0, s>>>(f->st, f->d_inv_s, f->d_dv, in, out, transpose);
    } else {
        const unsigned g = std::min(blocks_for(f->n * 32, 256), 65535u);
        // F holds unit rows for non-design points; F^T holds the design rows'
        // entries only, plus the pass-through of non-design points
        if (!transpose)
            csr_filter_kernel<<<g, 256, 0, s>>>(f->n, f->d_rp, f->d_c, f->d_v, nullptr, nullptr, in, out);
        else
            csr_filter_kernel<<<g, 256, 0, s>>>(f->n, f->d_rpt, f->d_ct, f->d_vt, f->d_not_dv, nullptr, in, out);
    }
    MG_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return MG_OK;
}

}  // namespace
}  // namespace mg

extern "C" {

int mg_filter_create_grid(int32_t nx, int32_t ny, int32_t nz, double hx, double hy, double hz, double radius,
                          const uint8_t *dv_mask, mg_filter **out) {
    if (!out) return MG_EINVAL;
    *out = nullptr;
    const int NZ = nz > 0 ? nz : 1;
    if (nx <= 0 || ny <= 0 || nz < 0 || !(radius > 0.0) || !(hx > 0.0) || !(hy > 0.0) || (nz > 0 && !(hz > 0.0))) {
        set_error("mg_filter_create_grid: bad grid or radius");
        return MG_EINVAL;
    }
    // stencil: integer offsets within the radius (weight r - d, 0 at d = r kept out)
    std::vector<int> ox, oy, oz;
    std::vector<double> w;
    const int ax = (int)floor(radius / hx), ay = (int)floor(radius / hy), az = nz > 0 ? (int)floor(radius / hz) : 0;
    if ((int64_t)(2 * ax + 1) * (2 * ay + 1) * (2 * az + 1) > 1 << 20) {
        set_error("mg_filter_create_grid: radius spans too many elements");
        return MG_EINVAL;
    }
    for (int c = -az; c <= az; c++)
        for (int b = -ay; b <= ay; b++)
            for (int a = -ax; a <= ax; a++) {
                const double d = sqrt((a * hx) * (a * hx) + (b * hy) * (b * hy) + (c * hz) * (c * hz));
                if (d <= radius && radius - d > 0.0) {
                    ox.push_back(a);
                    oy.push_back(b);
                    oz.push_back(c);
                    w.push_back(radius - d);
                }
            }
    mg_filter *f = new mg_filter();
    auto fail = [&](int rc) {
        mg_filter_destroy(f);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete f;
        set_error("cudaStreamCreate failed (no usable GPU?)");
        return MG_ECUDA;
    }
    f->grid = true;
    f->n = (int64_t)nx * ny * NZ;
    f->nnz = (int64_t)w.size();
    int rc;
    if ((rc = upload(&f->d_ox, ox.data(), ox.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_oy, oy.data(), oy.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_oz, oz.data(), oz.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_w, w.data(), w.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = dev_alloc_n(&f->d_inv_s, (size_t)f->n)) != MG_OK) return fail(rc);
    f->st = StencilArgs{nx, ny, NZ, (int)w.size(), f->d_ox, f->d_oy, f->d_oz, f->d_w};
    if (ny <= kFoldY * 65535 && NZ <= 65535) plan_fold(f, ox, oy, oz, w, NZ == 1);
    stencil_norm_kernel<<<std::min(blocks_for(f->n, 256), 4096u), 256, 0, f->stream>>>(f->st, f->d_inv_s);
    count_launches(1);
    if (cudaGetLastError() != cudaSuccess) return fail(MG_ECUDA);
    if ((rc = finish_create(f, dv_mask)) != MG_OK) return fail(rc);
    if (cudaStreamSynchronize(f->stream) != cudaSuccess) return fail(MG_ECUDA);
    *out = f;
    return MG_OK;
}

int mg_filter_create_points(int64_t n, int32_t dim, const double *xyz, double radius, const uint8_t *dv_mask,
                            mg_filter **out) {
    if (!out) return MG_EINVAL;
    *out = nullptr;
    if (n <= 0 || n > INT32_MAX || dim < 1 || dim > 3 || !xyz || !(radius > 0.0)) {
        set_error("mg_filter_create_points: bad points or radius");
        return MG_EINVAL;
    }
    for (int64_t i = 0; i < n * dim; i++)
        if (!isfinite(xyz[i])) {
            set_error("mg_filter_create_points: non-finite coordinate");
            return MG_EINVAL;
        }
    // bucket grid of cell size r: neighbours lie in the 3^dim surrounding cells
    double lo[3] = {0, 0, 0};
    for (int c = 0; c < dim; c++) {
        lo[c] = xyz[c];
        for (int64_t i = 0; i < n; i++) lo[c] = std::min(lo[c], xyz[i * dim + c]);
    }
    auto cell_of = [&](int64_t i, int c) { return (int64_t)floor((xyz[i * dim + c] - lo[c]) / radius); };
    auto key = [](int64_t a, int64_t b, int64_t c) { return (a * 73856093LL) ^ (b * 19349663LL) ^ (c * 83492791LL); };
    std::unordered_map<int64_t, std::vector<int32_t>> buckets;
    buckets.reserve((size_t)n);
    for (int64_t i = 0; i < n; i++)
        buckets[key(cell_of(i, 0), dim > 1 ? cell_of(i, 1) : 0, dim > 2 ? cell_of(i, 2) : 0)].push_back((int32_t)i);
    std::vector<int64_t> rp((size_t)n + 1, 0);
    std::vector<int32_t> cols;
    std::vector<double> vals;
    std::vector<std::pair<int32_t, double>> row;
    for (int64_t i = 0; i < n; i++) {
        row.clear();
        const int64_t ci = cell_of(i, 0), cj = dim > 1 ? cell_of(i, 1) : 0, ck = dim > 2 ? cell_of(i, 2) : 0;
        double sum = 0.0;
        for (int64_t dk = (dim > 2 ? -1 : 0); dk <= (dim > 2 ? 1 : 0); dk++)
            for (int64_t dj = (dim > 1 ? -1 : 0); dj <= (dim > 1 ? 1 : 0); dj++)
                for (int64_t di = -1; di <= 1; di++) {
                    auto it = buckets.find(key(ci + di, cj + dj, ck + dk));
                    if (it == buckets.end()) continue;
                    for (int32_t j : it->second) {
                        double d2 = 0.0;
                        for (int c = 0; c < dim; c++) {
                            const double t = xyz[i * dim + c] - xyz[(int64_t)j * dim + c];
                            d2 += t * t;
                        }
                        const double d = sqrt(d2);
                        if (d <= radius && radius - d > 0.0) {
                            row.push_back({j, radius - d});
                            sum += radius - d;
                        }
                    }
                }
        std::sort(row.begin(), row.end());
        row.erase(std::unique(row.begin(), row.end(),
                              [](const std::pair<int32_t, double> &a, const std::pair<int32_t, double> &b) {
                                  return a.first == b.first;
                              }),
                  row.end());
        // recompute the sum over the unique neighbours (hash collisions may repeat a bucket)
        sum = 0.0;
        for (auto &p : row) sum += p.second;
        const bool is_dv = !dv_mask || dv_mask[i];
        if (is_dv)
            for (auto &p : row) {
                cols.push_back(p.first);
                vals.push_back(p.second / sum);
            }
        else {  // a non-design point keeps its value: unit row
            cols.push_back((int32_t)i);
            vals.push_back(1.0);
        }
        rp[i + 1] = (int64_t)cols.size();
    }
    // F^T restricted to design rows (the non-design identity is added by the kernel)
    std::vector<int64_t> rpt((size_t)n + 1, 0);
    std::vector<int64_t> cnt((size_t)n, 0);
    for (int64_t i = 0; i < n; i++)
        if (!dv_mask || dv_mask[i])
            for (int64_t k = rp[i]; k < rp[i + 1]; k++) cnt[cols[k]]++;
    for (int64_t j = 0; j < n; j++) rpt[j + 1] = rpt[j] + cnt[j];
    std::vector<int32_t> ct((size_t)rpt[n]);
    std::vector<double> vt((size_t)rpt[n]);
    std::vector<int64_t> pos(rpt.begin(), rpt.end() - 1);
    for (int64_t i = 0; i < n; i++)
        if (!dv_mask || dv_mask[i])
            for (int64_t k = rp[i]; k < rp[i + 1]; k++) {
                const int64_t p = pos[cols[k]]++;
                ct[p] = (int32_t)i;
                vt[p] = vals[k];
            }
    mg_filter *f = new mg_filter();
    auto fail = [&](int rc) {
        mg_filter_destroy(f);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete f;
        set_error("cudaStreamCreate failed (no usable GPU?)");
        return MG_ECUDA;
    }
    f->n = n;
    f->nnz = (int64_t)cols.size();
    int rc;
    if ((rc = upload(&f->d_rp, rp.data(), rp.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_c, cols.data(), cols.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_v, vals.data(), vals.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_rpt, rpt.data(), rpt.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_ct, ct.data(), ct.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = upload(&f->d_vt, vt.data(), vt.size(), f->stream)) != MG_OK) return fail(rc);
    if ((rc = finish_create(f, dv_mask)) != MG_OK) return fail(rc);
    if (cudaStreamSynchronize(f->stream) != cudaSuccess) return fail(MG_ECUDA);
    *out = f;
    return MG_OK;
}

int mg_filter_info(const mg_filter *f, int64_t *n, int64_t *nnz) {
    if (!f) return MG_EINVAL;
    if (n) *n = f->n;
    if (nnz) *nnz = f->nnz;
    return MG_OK;
}

int mg_filter_apply_device(mg_filter *f, const double *in_dev, double *out_dev, int32_t transpose, void *stream) {
    if (!f || !in_dev || !out_dev || in_dev == out_dev) return MG_EINVAL;
    cudaStream_t s = stream ? (cudaStream_t)stream : f->stream;
    return run(f, in_dev, out_dev, transpose, s);
}

int mg_filter_apply(mg_filter *f, const double *in, double *out, int32_t transpose) {
    if (!f || !in || !out) return MG_EINVAL;
    MG_CUDA_TRY(cudaMemcpyAsync(f->d_in, in, f->n * 8, cudaMemcpyHostToDevice, f->stream));
    MG_TRY(run(f, f->d_in, f->d_out, transpose, f->stream));
    MG_CUDA_TRY(cudaMemcpyAsync(out, f->d_out, f->n * 8, cudaMemcpyDeviceToHost, f->stream));
    MG_CUDA_TRY(cudaStreamSynchronize(f->stream));
    return MG_OK;
}

void mg_filter_destroy(mg_filter *f) {
    if (!f) return;
    if (f->stream) cudaStreamSynchronize(f->stream);
    void *p[] = {f->d_ox, f->d_oy, f->d_oz, f->d_w, f->d_inv_s, f->d_dv, f->d_not_dv, f->d_rp, f->d_rpt,
                 f->d_c, f->d_ct, f->d_v, f->d_vt, f->d_in, f->d_out};
    for (void *q : p) dev_free(q);
    if (f->stream) cudaStreamDestroy(f->stream);
    delete f;
}

}  // extern "C"
