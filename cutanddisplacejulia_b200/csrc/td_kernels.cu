// TD pair kernels for sm_100a (FP64 CUDA-core work; no tensor-core shape).
//
// Work decomposition: one thread per observation point, one block per
// (128-point tile, chunk of triangles).  The block stages the triangles'
// precomputed records (TriDev; the full-space and frame-only ones eight at a
// time) in shared memory; every thread reads each as a broadcast, evaluates its
// pair and writes the pair's outputs
// (consecutive threads = consecutive rows of a column-major M x N influence
// matrix, so every store is coalesced).
//
// Output modes:
//   OUT_INF   18 strain and / or 9 displacement influence matrices (TD overload
//             src/TD.jl:135-216)
//   OUT_SUM   per-chunk partial sums over triangles of strain (6) and
//             displacement (3) (TD summing overload src/TD.jl:219-410); a
//             second kernel adds the chunks in index order (deterministic)
//   OUT_TRAC  9 traction influence matrices, strain converted in registers
//             (ConvertStrainInfMatsToTraction, src/CalculateInfluenceMatrices3D.jl:73-114)
//   OUT_AMAT  the 3N x 3N system matrix -[Atn;Atss;Atds] (src/SlipCalculator3D.jl:13-16)
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "td_device.cuh"
#include "td_kernels.h"

namespace cad {

// ------------------------------------------------------------ setup kernel
__global__ void td_setup_kernel(const double* __restrict__ P1, const double* __restrict__ P2,
                                const double* __restrict__ P3, int64_t N, const double* __restrict__ Dss,
                                const double* __restrict__ Dds, const double* __restrict__ Dn, int64_t slip_stride,
                                double nu, int hs, int sides, TriDev* __restrict__ out)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= N) return;
    TriDev& t = out[j];
    const double a[3] = {P1[j], P1[j + N], P1[j + 2 * N]};
    const double b[3] = {P2[j], P2[j + N], P2[j + 2 * N]};
    const double c[3] = {P3[j], P3[j + N], P3[j + 2 * N]};
    build_triangle(a, b, c, Dss ? Dss[j * slip_stride] : 1.0, Dds ? Dds[j * slip_stride] : 1.0,
                   Dn ? Dn[j * slip_stride] : 1.0, nu, hs != 0, t, sides != 0);
}

// ------------------------------------------------ half-space argument check
// flag |= 1 when any vertex or observation z > 0 (src/TD.jl:606-619).
// With nz set, the observation z is Z - 1e-12 nz (collocation points from
// midpoints and normals, as SetupCollationPoints forms them).  horizontal (may
// be null) |= 1 when a triangle is exactly horizontal.
__global__ void hs_check_kernel(const double* __restrict__ Z, const double* __restrict__ nz, int64_t M,
                                const double* __restrict__ P1, const double* __restrict__ P2,
                                const double* __restrict__ P3, int64_t N, int* __restrict__ flag,
                                int* __restrict__ horizontal)
{
    int bad = 0, level = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < M + N; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < M) bad |= (nz ? Z[i] - nz[i] * 1e-12 : Z[i]) > 0.0;
        else {
            const int64_t j = i - M;
            bad |= (P1[j + 2 * N] > 0.0) | (P2[j + 2 * N] > 0.0) | (P3[j + 2 * N] > 0.0);
            if (horizontal) {   // the normal exactly vertical, as build_frame forms it
                double a[3], b[3], n[3];
                for (int c = 0; c < 3; ++c) {
                    a[c] = sub_rn(P2[j + c * N], P1[j + c * N]);
                    b[c] = sub_rn(P3[j + c * N], P1[j + c * N]);
                }
                cross3_rn(a, b, n);
                const double nn = norm3_rn(n[0], n[1], n[2]);
                level |= n[0] / nn == 0.0 && n[1] / nn == 0.0;
            }
        }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
    if (horizontal && __syncthreads_or(level) && threadIdx.x == 0) atomicOr(horizontal, 1);
}

// ---------------------------------------------------- collocation points
// obs = incentre - 1e-12 * normal (SetupCollationPoints,
// src/CalculateInfluenceMatrices3D.jl:52-71) and the strike / dip directions
// of every element (CalculateSSandDSDirs, src/CalculateSSandDSDirs.jl:417-481).
__global__ void colloc_kernel(const double* __restrict__ normals, const double* __restrict__ mid, int64_t N,
                              double* __restrict__ X, double* __restrict__ Y, double* __restrict__ Z,
                              double* __restrict__ dirs /* 9 x N: n, ss, ds */)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double cx = normals[i], cy = normals[i + N], cz = normals[i + 2 * N];
    X[i] = mid[i] - cx * 1e-12;
    Y[i] = mid[i + N] - cy * 1e-12;
    Z[i] = mid[i + 2 * N] - cz * 1e-12;
    const double inv = 1.0 / sqrt(cx * cx + cy * cy);
    double ss[3] = {-(cy * inv), cx * inv, 0.0};
    const double dsz = cos(acos(cz) - M_PI / 2.0);
    double L = sin(acos(dsz));
    if (cz < 0.0) L = -L;
    const double a = atan2(cy, cx);
    double ds[3] = {-(cos(a) * L), -(sin(a) * L), dsz};
    if (cx == 0.0 && cy == 0.0) {
        ds[0] = -1.0; ds[1] = 0.0; ds[2] = 0.0;
        ss[0] = 0.0; ss[1] = cz < 1.0 ? -1.0 : 1.0; ss[2] = 0.0;
    }
    dirs[i] = cx; dirs[i + N] = cy; dirs[i + 2 * N] = cz;
    for (int k = 0; k < 3; ++k) { dirs[i + (3 + k) * N] = ss[k]; dirs[i + (6 + k) * N] = ds[k]; }
}

// Unit-mode strain -> (Tn, Tss, Tds) on the element with normal n, strike ss,
// dip ds (Hooke, CalculateNormalTraction3D!, TractionVectorCartesianComponents3D!,
// CalculateTractionInChosenDirection3D!).
template <typename R>
__device__ __forceinline__ void strain_to_traction(const R e[6], R lam, R G2, const R n[3], const R ss[3],
                                                   const R ds[3], R out[3])
{
    const R cons = lam * (e[0] + e[1] + e[2]);
    const R Sxx = G2 * e[0] + cons, Syy = G2 * e[1] + cons, Szz = G2 * e[2] + cons;
    const R Sxy = G2 * e[3], Sxz = G2 * e[4], Syz = G2 * e[5];
    const R cx = n[0], cy = n[1], cz = n[2];
    const R two = R(2.0);
    out[0] = Sxx * (cx * cx) + Syy * (cy * cy) + Szz * (cz * cz) + two * Sxy * (cx * cy) + two * Syz * (cy * cz) +
             two * Sxz * (cz * cx);
    const R Tx = Sxx * cx + Sxy * cy + Sxz * cz;
    const R Ty = Sxy * cx + Syy * cy + Syz * cz;
    const R Tz = Sxz * cx + Syz * cy + Szz * cz;
    // traction projected onto the plane: t - (t.n) n
    const R tn = Tx * cx + Ty * cy + Tz * cz;
    const R px = Tx - tn * cx, py = Ty - tn * cy, pz = Tz - tn * cz;
    out[1] = px * ss[0] + py * ss[1] + pz * ss[2];
    out[2] = px * ds[0] + py * ds[1] + pz * ds[2];
}

// ------------------------------------------------------------- pair kernel
enum EdgeKind { EDGE_NONE = 0, EDGE_FSC = 1, EDGE_FULL = 2 };
// record values a pair kernel stages per triangle, and triangles staged between
// two barriers (the small records 8 at a time)
__host__ __device__ constexpr int pair_words(bool hs, int edge) { return hs ? (edge ? kTriWordsImg : kTriWordsHS) : kTriWordsFS; }
__host__ __device__ constexpr int pair_stage(bool hs, int edge, bool one) { return one || (hs && !edge) ? 1 : 8; }

// NEAR: rewrite only the triangles whose centroid lies within the near
// radius of some point of the block (the FP64 pass of the mixed assembly).
// LIST (OUT_AMAT only): incremental re-assembly through a.tri_list /
// a.obs_list into a system of a.Ntot elements.
// MINB > 1: compiled for MINB resident blocks per SM (fewer registers per
// thread, more warps to hide the FP64 latency, some spilling) -- a launch
// shape the autotuner may pick for the half-space system matrix.
// EDGE (half space, but for the full-space sums): the staged record is the
// two frames only.
//   EDGE_FSC: the free-surface corrections are left to per-edge work.
//   OUT_AMAT, OUT_TRAC (strain) and OUT_INF: they come from the per-edge maps
//   a.fscG (side_map_kernel).  OUT_SUM: they are left out here, and
//   side_sum_kernel adds each edge's once.
//   EDGE_FULL: so is the whole strain (real, image and correction), which
//   depends on the triangles' sides alone; the pair only combines its three
//   sides' maps (tractions already for OUT_AMAT and OUT_TRAC).  OUT_SUM (full
//   space too): the displacement's solid angles; side_sum_kernel or
//   segment_sum_kernel adds the rest.  Points on a side become NaN.
template <bool HS, bool STRAIN, bool DISP, int OUT, bool NEAR = false, bool LIST = false, int MINB = 1,
          int EDGE = EDGE_NONE>
__global__ void __launch_bounds__(kPairThreads, MINB) td_pair_kernel(PairArgs a)
{
    static_assert(EDGE == EDGE_NONE || (!HS && EDGE == EDGE_FULL && OUT == OUT_SUM) || (HS && !LIST && !NEAR &&
                            (((OUT == OUT_AMAT || OUT == OUT_TRAC) && STRAIN && !DISP) || OUT == OUT_SUM ||
                             OUT == OUT_INF)),
                  "shared edges: HS system matrix, traction or influence fields, or sums only");
    constexpr bool EDGE_MAPS = EDGE != EDGE_NONE && OUT != OUT_SUM;
    constexpr bool EDGE_TRAC = EDGE == EDGE_FULL && (OUT == OUT_AMAT || OUT == OUT_TRAC);
    // values per (edge, point) in the maps: strain 18 (tractions 9), then displacement 9
    constexpr int64_t kQ = EDGE_TRAC ? 9 : (STRAIN ? 18 : 0) + (DISP ? 9 : 0);
    extern __shared__ double smem[];
    constexpr int words = pair_words(HS, EDGE);
    constexpr int stage = pair_stage(HS, EDGE, NEAR || LIST);
    const int64_t i = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const bool active = i < a.M;
    // LIST: this thread's point (system row) and the full system's size
    const int64_t io = (LIST && a.obs_list && active) ? (int64_t)a.obs_list[i] : i;
    const int64_t NS = LIST ? a.Ntot : a.N;
    const int64_t MD = (LIST || EDGE_MAPS) ? a.Ntot : a.M;
    double X = 0.0, Y = 0.0, Z = 0.0;
    if (active) { X = a.X[io]; Y = a.Y[io]; Z = a.Z[io]; }
    const int64_t j0 = (int64_t)blockIdx.y * a.tri_chunk;
    const int64_t j1 = min(a.N, j0 + a.tri_chunk);
    // row stride of the M x N output fields: a block of an Ntot-point system
    // with the edge maps
    const int64_t MR = EDGE_MAPS ? MD : a.M;
    const int64_t MN = MR * a.N;
    double sumE[6] = {0, 0, 0, 0, 0, 0}, sumU[3] = {0, 0, 0};
    double n[3] = {0, 0, 0}, ss[3] = {0, 0, 0}, ds[3] = {0, 0, 0};
    if ((OUT == OUT_TRAC || OUT == OUT_AMAT) && active) {
        for (int k = 0; k < 3; ++k) {
            n[k] = a.dirs[io + k * MD];
            ss[k] = a.dirs[io + (3 + k) * MD];
            ds[k] = a.dirs[io + (6 + k) * MD];
        }
    }
    const double near_r2 = NEAR ? a.near[3 * a.N] : 0.0;
    for (int64_t j = j0; j < j1; ++j) {
        const int slot = (int)(j - j0) % stage;
        if (NEAR) {
            bool nr = false;
            if (active) {
                const double dx = X - a.near[j], dy = Y - a.near[j + a.N], dz = Z - a.near[j + 2 * a.N];
                nr = dx * dx + dy * dy + dz * dz < near_r2;
            }
            if (!__syncthreads_or(nr)) continue;   // also the barrier before restaging
        } else if (slot == 0) {
            __syncthreads();
        }
        const int64_t jt = (LIST && a.tri_list) ? (int64_t)a.tri_list[j] : j;   // system column
        if (slot == 0) {   // the next records (`stage` of them, but for lists one) into shared memory
            const int n = (int)min((int64_t)stage, j1 - j);
            for (int k = 0; k < n; ++k) {
                const double* src = reinterpret_cast<const double*>(a.tri + jt + k);
                for (int w = threadIdx.x; w < words; w += kPairThreads) smem[k * words + w] = src[w];
            }
            __syncthreads();
        }
        if (!active) continue;
        const TriDev& t = *reinterpret_cast<const TriDev*>(smem + slot * words);
        if constexpr (EDGE_TRAC) {
            double S[9];
            sum_side_maps<9>(a.fscG + i, a.M, 9 * a.M, a.side_edge + 3 * jt, S);
            const bool nan = pair_on_side(t, X, Y, Z);
            const double* axes[3] = {t.real.Vn, t.real.Vs, t.real.Vd};
            const double slip[3] = {t.Dn, t.Dss, t.Dds};
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    double tr = slip[m] * (axes[m][0] * S[r] + axes[m][1] * S[3 + r] + axes[m][2] * S[6 + r]);
                    if (nan) tr = qnan<double>();
                    if (OUT == OUT_TRAC) a.trac[(3 * m + r) * MN + i + MR * j] = tr;
                    else a.A[(int64_t)(r * MD + io) + a.lda * (int64_t)(m * NS + jt)] = -tr;
                }
            continue;
        }
        if constexpr (OUT == OUT_SUM && EDGE == EDGE_FULL) {
            static_assert(DISP, "strain alone leaves the pairs to on_side_kernel");
            pair_angle<HS, STRAIN>(t, X, Y, Z, sumE, sumU);
            continue;
        } else if constexpr (OUT == OUT_SUM && (!HS || EDGE != EDGE_NONE)) {
            pair_net<HS, STRAIN, DISP>(t, X, Y, Z, sumE, sumU);
            continue;
        }
        if (STRAIN) {
            double E[3][6];
            if constexpr (EDGE_MAPS && EDGE == EDGE_FULL)
                pair_strain_full(t, X, Y, Z, a.fscG + i, a.M, kQ * a.M, a.side_edge + 3 * jt, E);
            else if constexpr (EDGE_MAPS)
                pair_strain_edges(t, X, Y, Z, a.fscG + i, a.M, kQ * a.M, a.side_edge + 3 * jt, E);
            else
                pair_strain<HS>(t, X, Y, Z, E);
            if (OUT == OUT_INF) {
#pragma unroll
                for (int m = 0; m < 3; ++m)
#pragma unroll
                    for (int k = 0; k < 6; ++k) a.strain[(6 * m + k) * MN + i + MR * j] = E[m][k];
            } else if (OUT == OUT_SUM) {
#pragma unroll
                for (int k = 0; k < 6; ++k) sumE[k] += (E[0][k] + E[1][k]) + E[2][k];
            } else {
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    double tr[3];
                    strain_to_traction(E[m], a.lambda, 2.0 * a.G, n, ss, ds, tr);
                    if (OUT == OUT_TRAC) {
#pragma unroll
                        for (int r = 0; r < 3; ++r) a.trac[(3 * m + r) * MN + i + MR * j] = tr[r];
                    } else {
#pragma unroll
                        for (int r = 0; r < 3; ++r)
                            a.A[(int64_t)(r * MD + io) + a.lda * (int64_t)(m * NS + jt)] = -tr[r];
                    }
                }
            }
        }
        if (DISP) {
            double U[3][3];
            if constexpr (EDGE_MAPS)
                pair_disp_edges(t, X, Y, Z, a.fscG + i + (STRAIN ? 18 : 0) * a.M, a.M, kQ * a.M, a.side_edge + 3 * jt,
                                U);
            else
                pair_disp<HS>(t, X, Y, Z, U);
            if (OUT == OUT_INF) {
#pragma unroll
                for (int m = 0; m < 3; ++m)
#pragma unroll
                    for (int c = 0; c < 3; ++c) a.disp[(3 * m + c) * MN + i + MR * j] = U[m][c];
            } else if (OUT == OUT_SUM) {
#pragma unroll
                for (int c = 0; c < 3; ++c) sumU[c] += (U[0][c] + U[1][c]) + U[2][c];
            }
        }
    }
    if (OUT == OUT_SUM && active) {
        double* p = a.partial + (int64_t)blockIdx.y * 9 * a.M;
#pragma unroll
        for (int k = 0; k < 6; ++k) p[k * a.M + i] = sumE[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) p[(6 + c) * a.M + i] = sumU[c];
    }
}

// The triangles' share of strain sums whose sides are taken per mesh edge: NaN
// at points on a side or vertex (HS: or on the mirror image's), 0 elsewhere.
// A point can be on a side only where its offset from the plane, in unfused
// arithmetic, is exactly 0; the rest of the test runs only there.  Each thread
// takes four points: with one, the six values of a plane that every thread
// reads from shared memory bound it (2013 x 20 000: 129 us, now 37).
constexpr int kMarkStage = 32, kMarkPts = 4;
template <bool HS>
__global__ void __launch_bounds__(kPairThreads) on_side_kernel(PairArgs a)
{
    constexpr int F = HS ? 2 : 1;
    __shared__ __align__(16) double s_plane[kMarkStage][F][6];   // P2, Vn
    const int64_t i0 = (int64_t)blockIdx.x * (kPairThreads * kMarkPts) + threadIdx.x;
    double X[kMarkPts], Y[kMarkPts], Z[kMarkPts];
    bool nan[kMarkPts];
#pragma unroll
    for (int q = 0; q < kMarkPts; ++q) {
        const int64_t i = min(i0 + q * kPairThreads, a.M - 1);
        X[q] = a.X[i];
        Y[q] = a.Y[i];
        Z[q] = a.Z[i];
        nan[q] = false;
    }
    const int64_t j0 = (int64_t)blockIdx.y * a.tri_chunk;
    const int64_t j1 = min(a.N, j0 + a.tri_chunk);
    for (int64_t jb = j0; jb < j1; jb += kMarkStage) {
        const int nt = (int)min((int64_t)kMarkStage, j1 - jb);
        __syncthreads();
        for (int w = threadIdx.x; w < nt * F * 6; w += kPairThreads) {
            const int k = w / (F * 6), f = w / 6 % F, c = w % 6;
            const Frame& fr = f ? a.tri[jb + k].image : a.tri[jb + k].real;
            s_plane[k][f][c] = c < 3 ? fr.P2[c] : fr.Vn[c - 3];
        }
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < nt; ++k) {
            unsigned in = 0u;
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const double* p = s_plane[k][f];
#pragma unroll
                for (int q = 0; q < kMarkPts; ++q) {
                    const double x = dot3_rn(p[3], p[4], p[5], sub_rn(X[q], p[0]), sub_rn(Y[q], p[1]), sub_rn(Z[q], p[2]));
                    in |= x == 0.0 ? 1u << q : 0u;
                }
            }
            if (in) {
                const TriDev& t = a.tri[jb + k];
#pragma unroll
                for (int q = 0; q < kMarkPts; ++q)
                    if ((in >> q) & 1u)
                        nan[q] = nan[q] || (HS ? pair_on_side(t, X[q], Y[q], Z[q])
                                               : on_side_or_vertex(t.real, X[q], Y[q], Z[q]));
            }
        }
    }
    double* p = a.partial + (int64_t)blockIdx.y * 9 * a.M;
#pragma unroll
    for (int q = 0; q < kMarkPts; ++q) {
        const int64_t i = i0 + q * kPairThreads;
        if (i < a.M)
#pragma unroll
            for (int k = 0; k < 6; ++k) p[k * a.M + i] = nan[q] ? qnan<double>() : 0.0;
    }
}

static cudaError_t launch_on_side(const PairArgs& a, bool hs, cudaStream_t st)
{
    constexpr int pts = kPairThreads * kMarkPts;
    const dim3 grid((unsigned)((a.M + pts - 1) / pts), (unsigned)((a.N + a.tri_chunk - 1) / a.tri_chunk));
    if (hs) on_side_kernel<true><<<grid, kPairThreads, 0, st>>>(a);
    else on_side_kernel<false><<<grid, kPairThreads, 0, st>>>(a);
    return cudaGetLastError();
}

// Adds the per-chunk partial sums in chunk order: out[f][i] = sum_c partial[c][f][i].
__global__ void sum_chunks_kernel(const double* __restrict__ partial, int64_t nchunk, int64_t M, int fields_mask,
                                  double* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= M || !((fields_mask >> f) & 1)) return;
    double s = 0.0;
    for (int64_t c = 0; c < nchunk; ++c) s += partial[(c * 9 + f) * M + i];
    out[f * M + i] = s;
}

// As sum_chunks_kernel, with strain fields (0-5) and displacement fields
// (6-8) written to two separate outputs (6 x M and 3 x M).
__global__ void sum_chunks_split_kernel(const double* __restrict__ partial, int64_t nchunk, int64_t M,
                                        int fields_mask, double* __restrict__ strain_out,
                                        double* __restrict__ disp_out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= M || !((fields_mask >> f) & 1)) return;
    double s = 0.0;
    for (int64_t c = 0; c < nchunk; ++c) s += partial[(c * 9 + f) * M + i];
    if (f < 6) strain_out[f * M + i] = s;
    else disp_out[(f - 6) * M + i] = s;
}

// TD_sum (src/TD_sum.jl:1-41): sum the three modes, then across the N columns.
// in: nf*3 matrices M x N (field f of mode m at in + (m*nf + f)*M*N), out: nf x M.
__global__ void td_sum_kernel(const double* __restrict__ in, int64_t M, int64_t N, int nf, double* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= M) return;
    const int64_t MN = M * N;
    double s = 0.0;
    for (int64_t j = 0; j < N; ++j) {
        const int64_t o = i + M * j;
        s += (in[(0 * nf + f) * MN + o] + in[(1 * nf + f) * MN + o]) + in[(2 * nf + f) * MN + o];
    }
    out[f * M + i] = s;
}

// ------------------------------------------------------- fixed elements
// Splice of CalculateInfluenceMatrices3D with fixed elements (ConcatInfMats,
// PutDispInfsIntoInfMat, src/CalculateInfluenceMatrices3D.jl:145-199): field
// f's row i is the displacement influence disp[f] (nfix x N) of fixed row
// fixrow[i] when i is fixed (fixrow[i] >= 0), else the traction influence
// trac[f] (N x N); only the columns freecol[0..nf) are kept.  amat = 0:
// out + f * N * nf holds field f (N x nf, column-major); amat = 1: out is the
// system A (3N x 3nf, lda) = -[[F0 F3 F6]; [F1 F4 F7]; [F2 F5 F8]].
__global__ void splice_fixed_kernel(const double* __restrict__ trac, const double* __restrict__ disp, int64_t N,
                                    int64_t nfix, const int* __restrict__ fixrow, const int* __restrict__ freecol,
                                    int64_t nf, int amat, double* __restrict__ out, int64_t lda)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t jf = blockIdx.y;
    const int f = blockIdx.z;
    if (i >= N || jf >= nf) return;
    const int64_t j = freecol[jf];
    const int fr = fixrow[i];
    const double v = fr >= 0 ? disp[(int64_t)f * nfix * N + fr + nfix * j] : trac[(int64_t)f * N * N + i + N * j];
    if (!amat) {
        out[(int64_t)f * N * nf + i + N * jf] = v;
    } else {
        const int m = f / 3, r = f % 3;   // field 3m + r: slip mode m (column block), traction row r
        out[(r * N + i) + lda * (m * nf + jf)] = -v;
    }
}

// out[k] = (X, Y, Z)[idx[k]] as three SoA arrays of length n
__global__ void gather_points_kernel(const double* __restrict__ X, const double* __restrict__ Y,
                                     const double* __restrict__ Z, const int* __restrict__ idx, int64_t n,
                                     double* __restrict__ out)
{
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t i = idx[k];
    out[k] = X[i];
    out[k + n] = Y[i];
    out[k + 2 * n] = Z[i];
}

// ----------------------------------------------- mixed-precision assembly
// Centroids of the triangles (near + [0, 3N)) and the squared near-field
// radius (near[3N]) = (factor x mean edge length)^2; one block, fixed
// summation order.
__global__ void __launch_bounds__(1024) near_setup_kernel(const double* __restrict__ P1, const double* __restrict__ P2,
                                                          const double* __restrict__ P3, int64_t N, double factor,
                                                          double* __restrict__ near)
{
    __shared__ double s_sum[1024];
    double acc = 0.0;
    for (int64_t j = threadIdx.x; j < N; j += blockDim.x) {
        double e = 0.0;
        for (int c = 0; c < 3; ++c) near[j + c * N] = (P1[j + c * N] + P2[j + c * N] + P3[j + c * N]) / 3.0;
        const double* P[3] = {P1, P2, P3};
        for (int v = 0; v < 3; ++v) {
            const double* p = P[v];
            const double* q = P[(v + 1) % 3];
            const double dx = q[j] - p[j], dy = q[j + N] - p[j + N], dz = q[j + 2 * N] - p[j + 2 * N];
            e += sqrt(dx * dx + dy * dy + dz * dz);
        }
        acc += e;
    }
    s_sum[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) s_sum[threadIdx.x] += s_sum[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double r = factor * (N > 0 ? s_sum[0] / (3.0 * (double)N) : 0.0);
        near[3 * N] = r * r;
    }
}

// FP32 copy of the first `words` values of each triangle record (records
// `stride` values apart in both copies): element-wise, then the origins' low
// parts (an FP32 record keeps each origin as hi + lo).
__global__ void tri_to_f32_kernel(const double* __restrict__ in, int64_t N, int words, int stride,
                                  float* __restrict__ out)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N * words) return;
    const int64_t j = i / words;
    const int w = (int)(i - j * words);
    const int64_t at = j * stride + w;
    constexpr int kReal = (int)((offsetof(TriDev, real) + offsetof(Frame, P2lo)) / sizeof(double));
    constexpr int kImage = (int)((offsetof(TriDev, image) + offsetof(Frame, P2lo)) / sizeof(double));
    constexpr int kSide0 = (int)((offsetof(TriDev, side) + offsetof(FscSide, PAlo)) / sizeof(double));
    constexpr int kSideW = (int)(sizeof(FscSide) / sizeof(double));
    bool lo = (w >= kReal && w < kReal + 3) || (w >= kImage && w < kImage + 3);
    for (int sd = 0; sd < 3; ++sd) lo = lo || (w >= kSide0 + sd * kSideW && w < kSide0 + sd * kSideW + 3);
    if (lo) {
        const double hi = in[at - 3];
        out[at] = (float)(hi - (double)(float)hi);
    } else {
        out[at] = (float)in[at];
    }
}

// Far-field pass: the system-matrix kernel with FP32 records and FP32
// arithmetic (coordinates relative to each origin formed in FP64).
template <bool HS>
__global__ void __launch_bounds__(kPairThreads) td_pair_f32_kernel(PairArgs a)
{
    extern __shared__ float smem32[];
    constexpr int words = HS ? kTriWordsHS : kTriWordsFS;
    const TriDevT<float>& t = *reinterpret_cast<const TriDevT<float>*>(smem32);
    const int64_t i = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const bool active = i < a.M;
    double X = 0.0, Y = 0.0, Z = 0.0;
    if (active) { X = a.X[i]; Y = a.Y[i]; Z = a.Z[i]; }
    const int64_t j0 = (int64_t)blockIdx.y * a.tri_chunk;
    const int64_t j1 = min(a.N, j0 + a.tri_chunk);
    float n[3] = {0, 0, 0}, ss[3] = {0, 0, 0}, ds[3] = {0, 0, 0};
    if (active) {
        for (int k = 0; k < 3; ++k) {
            n[k] = (float)a.dirs[i + k * a.M];
            ss[k] = (float)a.dirs[i + (3 + k) * a.M];
            ds[k] = (float)a.dirs[i + (6 + k) * a.M];
        }
    }
    const float* recs = reinterpret_cast<const float*>(a.tri32);
    const float lam = (float)a.lambda, G2 = (float)(2.0 * a.G);
    for (int64_t j = j0; j < j1; ++j) {
        __syncthreads();
        const float* src = recs + j * (int64_t)kTriWordsHS;   // records keep the FP64 stride
        for (int w = threadIdx.x; w < words; w += kPairThreads) smem32[w] = src[w];
        __syncthreads();
        if (!active) continue;
        float E[3][6];
        pair_strain<HS>(t, X, Y, Z, E);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            float tr[3];
            strain_to_traction(E[m], lam, G2, n, ss, ds, tr);
#pragma unroll
            for (int r = 0; r < 3; ++r) a.A[(int64_t)(r * a.N + i) + a.lda * (int64_t)(m * a.N + j)] = -(double)tr[r];
        }
    }
}

// ------------------------------------------------------------ launchers
template <bool HS, bool STRAIN, bool DISP, int OUT, int MINB = 1>
static cudaError_t launch_pair(const PairArgs& a, cudaStream_t st)
{
    const size_t smem = (size_t)pair_words(HS, EDGE_NONE) * pair_stage(HS, EDGE_NONE, false) * sizeof(double);
    auto kern = td_pair_kernel<HS, STRAIN, DISP, OUT, false, false, MINB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t ntile = (a.M + kPairThreads - 1) / kPairThreads;
    const int64_t nchunk = (a.N + a.tri_chunk - 1) / a.tri_chunk;
    if (ntile == 0 || nchunk == 0) return cudaSuccess;
    dim3 grid((unsigned)ntile, (unsigned)nchunk);
    kern<<<grid, kPairThreads, smem, st>>>(a);
    return cudaGetLastError();
}

#define CAD_DISPATCH_FLAGS(OUTK)                                                              \
    if (hs) {                                                                                 \
        if (strain && disp) return launch_pair<true, true, true, OUTK>(a, st);                \
        if (strain) return launch_pair<true, true, false, OUTK>(a, st);                       \
        if (disp) return launch_pair<true, false, true, OUTK>(a, st);                         \
    } else {                                                                                  \
        if (strain && disp) return launch_pair<false, true, true, OUTK>(a, st);               \
        if (strain) return launch_pair<false, true, false, OUTK>(a, st);                      \
        if (disp) return launch_pair<false, false, true, OUTK>(a, st);                        \
    }                                                                                         \
    return cudaSuccess;

cudaError_t launch_td_pairs(const PairArgs& a, int out, bool hs, bool strain, bool disp, cudaStream_t st)
{
    switch (out) {
        case OUT_INF: { CAD_DISPATCH_FLAGS(OUT_INF) }
        case OUT_SUM: { CAD_DISPATCH_FLAGS(OUT_SUM) }
        case OUT_TRAC:
            if (hs) return launch_pair<true, true, false, OUT_TRAC>(a, st);
            return launch_pair<false, true, false, OUT_TRAC>(a, st);
        case OUT_AMAT:
            if (hs) {
                if (a.min_blocks == 3) return launch_pair<true, true, false, OUT_AMAT, 3>(a, st);
                if (a.min_blocks == 4) return launch_pair<true, true, false, OUT_AMAT, 4>(a, st);
                return launch_pair<true, true, false, OUT_AMAT>(a, st);
            }
            return launch_pair<false, true, false, OUT_AMAT>(a, st);
    }
    return cudaErrorInvalidValue;
}

// ------------------------------------------------ shared-edge half space
// One mesh edge's free-surface record (geometry only) per thread; edge e's
// endpoints PA, PB at pts[6 e ..].
__global__ void edge_setup_kernel(const double* __restrict__ pts, int64_t E, double nu, FscSide* __restrict__ out)
{
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= E) return;
    const double PA[3] = {pts[6 * e], pts[6 * e + 1], pts[6 * e + 2]};
    const double PB[3] = {pts[6 * e + 3], pts[6 * e + 4], pts[6 * e + 5]};
    build_side_geom(PA, PB, nu, out[e]);
}

// G[(e * Q + q) M + i] = value q of edge e's maps at point i: the strain map
// (18 values, KIND EDGE_FSC the free-surface correction, EDGE_FULL the whole
// strain) or, TRAC, the whole strain as tractions on the point's element (9),
// then the correction's displacement map (9) when DISP.  Block = 128 points x
// a chunk of edges, 8 edge records staged in shared memory at a time.
constexpr int kEdgeStage = 8;
struct SideMapArgs {
    const FscSide* edges;
    int64_t E, echunk;
    const double *X, *Y, *Z;
    int64_t M;
    double* G;
    const double* dirs;   // TRAC: the points' element axes (row stride dirs_ld), elastic constants
    int64_t dirs_ld;
    double lambda, G2;
};
// The whole strain is built for three resident blocks per SM.
template <int KIND, bool DISP, bool TRAC>
__global__ void __launch_bounds__(kPairThreads, KIND == EDGE_FULL && !DISP ? 3 : 1) side_map_kernel(const SideMapArgs a)
{
    extern __shared__ double smem[];
    const int64_t i = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const bool active = i < a.M;
    const int64_t M = a.M;
    double* __restrict__ G = a.G + i;
    double x = 0.0, y = 0.0, z = 0.0;
    double n[3] = {0, 0, 0}, ss[3] = {0, 0, 0}, ds[3] = {0, 0, 0};
    if (active) {
        x = a.X[i];
        y = a.Y[i];
        z = a.Z[i];
        if (TRAC)
            for (int k = 0; k < 3; ++k) {
                n[k] = a.dirs[i + k * a.dirs_ld];
                ss[k] = a.dirs[i + (3 + k) * a.dirs_ld];
                ds[k] = a.dirs[i + (6 + k) * a.dirs_ld];
            }
    }
    const int64_t e0 = (int64_t)blockIdx.y * a.echunk;
    const int64_t e1 = min(a.E, e0 + a.echunk);
    constexpr int64_t Q = (TRAC ? 9 : KIND != EDGE_NONE ? 18 : 0) + (DISP ? 9 : 0);
    for (int64_t eb = e0; eb < e1; eb += kEdgeStage) {
        const int ne = (int)min((int64_t)kEdgeStage, e1 - eb);
        __syncthreads();
        const double* src = reinterpret_cast<const double*>(a.edges + eb);
        for (int w = threadIdx.x; w < ne * kSideWords; w += kPairThreads) smem[w] = src[w];
        __syncthreads();
        if (!active) continue;
#pragma unroll 1
        for (int k = 0; k < ne; ++k) {
            const FscSide& s = reinterpret_cast<const FscSide*>(smem)[k];
            const int64_t e = eb + k;
            if constexpr (TRAC) {
                double W[3][3];
                side_traction_map(s, x, y, z, a.lambda, a.G2, n, ss, ds, W);
#pragma unroll
                for (int q = 0; q < 9; ++q) G[(e * Q + q) * M] = W[q / 3][q % 3];
            } else if (KIND != EDGE_NONE) {
                double Gm[3][6];
                if (KIND == EDGE_FSC && s.skip != 0.0) {
#pragma unroll
                    for (int q = 0; q < 18; ++q) Gm[q / 6][q % 6] = 0.0;
                } else {
                    side_strain_map<KIND == EDGE_FULL>(s, x, y, z, Gm);
                }
#pragma unroll
                for (int q = 0; q < 18; ++q) G[(e * Q + q) * M] = Gm[q / 6][q % 6];
            }
            if (DISP) {
                double Gu[3][3];
                if (s.skip != 0.0) {
#pragma unroll
                    for (int q = 0; q < 9; ++q) Gu[q / 3][q % 3] = 0.0;
                } else {
                    fsc_disp_map(s, x, y, z, Gu);
                }
                constexpr int64_t q0 = Q - 9;
#pragma unroll
                for (int q = 0; q < 9; ++q) G[(e * Q + q0 + q) * M] = Gu[q / 3][q % 3];
            }
        }
    }
}

size_t edge_record_bytes() { return sizeof(FscSide); }

cudaError_t launch_assemble_edges(PairArgs a, int out_kind, bool strain, bool disp, bool full,
                                  const double* edge_pts, int64_t E, const int* side_edge, void* edge_rec, double* G, int64_t Mc, double nu,
                                  cudaStream_t st, int64_t* launches)
{
    if (out_kind == OUT_AMAT || out_kind == OUT_TRAC) {
        strain = true;
        disp = false;
    } else if (out_kind != OUT_INF || !(strain || disp)) {
        return cudaErrorInvalidValue;
    }
    if (a.M == 0 || a.N == 0) return cudaSuccess;
    if (E > 0) {
        edge_setup_kernel<<<(unsigned)((E + 31) / 32), 32, 0, st>>>(edge_pts, E, nu, (FscSide*)edge_rec);
        if (launches) ++*launches;
        if (cudaError_t e = cudaGetLastError()) return e;
    }
    using PairKernel = void (*)(PairArgs);
    using MapKernel = void (*)(SideMapArgs);
    PairKernel pk;
    MapKernel ek;
    const bool trac = out_kind != OUT_INF;
    if (trac && full) {
        // (the maps' loads bound the system matrix of 10 000 triangles: 4.4 ms at
        // three resident blocks, 4.0 at five)
        pk = out_kind == OUT_TRAC ? td_pair_kernel<true, true, false, OUT_TRAC, false, false, 1, EDGE_FULL>
                                  : td_pair_kernel<true, true, false, OUT_AMAT, false, false, 5, EDGE_FULL>;
        ek = side_map_kernel<EDGE_FULL, false, true>;
    } else if (trac) {
        pk = out_kind == OUT_TRAC ? td_pair_kernel<true, true, false, OUT_TRAC, false, false, 1, EDGE_FSC>
                                  : td_pair_kernel<true, true, false, OUT_AMAT, false, false, 1, EDGE_FSC>;
        ek = side_map_kernel<EDGE_FSC, false, false>;
    } else if (strain && disp) {
        pk = full ? td_pair_kernel<true, true, true, OUT_INF, false, false, 1, EDGE_FULL>
                  : td_pair_kernel<true, true, true, OUT_INF, false, false, 1, EDGE_FSC>;
        ek = full ? side_map_kernel<EDGE_FULL, true, false> : side_map_kernel<EDGE_FSC, true, false>;
    } else if (strain) {
        pk = full ? td_pair_kernel<true, true, false, OUT_INF, false, false, 1, EDGE_FULL>
                  : td_pair_kernel<true, true, false, OUT_INF, false, false, 1, EDGE_FSC>;
        ek = full ? side_map_kernel<EDGE_FULL, false, false> : side_map_kernel<EDGE_FSC, false, false>;
    } else {
        pk = td_pair_kernel<true, false, true, OUT_INF, false, false, 1, EDGE_FSC>;
        ek = side_map_kernel<EDGE_NONE, true, false>;
    }
    const size_t psmem = (size_t)pair_words(true, EDGE_FSC) * pair_stage(true, EDGE_FSC, false) * sizeof(double);
    const size_t esmem = (size_t)kSideWords * kEdgeStage * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(pk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ek, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)esmem);
    if (e != cudaSuccess) return e;
    const int64_t echunk_max = a.min_blocks == 1 ? 96 : 32;
    for (int64_t c0 = 0; c0 < a.M; c0 += Mc) {
        const int64_t mc = a.M - c0 < Mc ? a.M - c0 : Mc;
        const unsigned tiles = (unsigned)((mc + kPairThreads - 1) / kPairThreads);
        if (E > 0) {
            // small maps: fewer edges per block, so that every SM has its three
            // blocks four times over (900 triangles x 1111 points: 174 us in 135
            // blocks of 96 edges on 148 SMs, now 101)
            int64_t echunk = tiles * E / (148 * 12) / kEdgeStage * kEdgeStage;
            echunk = echunk < kEdgeStage ? kEdgeStage : echunk < echunk_max ? echunk : echunk_max;
            const SideMapArgs m{(const FscSide*)edge_rec, E, echunk, a.X + c0, a.Y + c0, a.Z + c0, mc, G,
                                a.dirs ? a.dirs + c0 : nullptr, a.M, a.lambda, 2.0 * a.G};
            ek<<<dim3(tiles, (unsigned)((E + echunk - 1) / echunk)), kPairThreads, esmem, st>>>(m);
            if (launches) ++*launches;
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        PairArgs b = a;
        b.X = a.X + c0;
        b.Y = a.Y + c0;
        b.Z = a.Z + c0;
        b.dirs = a.dirs ? a.dirs + c0 : nullptr;
        b.A = a.A ? a.A + c0 : nullptr;
        b.trac = a.trac ? a.trac + c0 : nullptr;
        b.strain = a.strain ? a.strain + c0 : nullptr;
        b.disp = a.disp ? a.disp + c0 : nullptr;
        b.M = mc;
        b.Ntot = a.M;   // the output fields' row stride
        b.fscG = G;
        b.side_edge = side_edge;
        pk<<<dim3(tiles, (unsigned)((a.N + a.tri_chunk - 1) / a.tri_chunk)), kPairThreads, psmem, st>>>(b);
        if (launches) ++*launches;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Net Burgers vector of a mesh edge: the signed sum over the triangle sides on
// it (list[0 .. n) = +-(triangle + 1), in no fixed order) of Dn Vn + Dss Vs +
// Dds Vd, the same bits whatever the order.
// A few sides are sorted into triangle order, then side order, by one thread.
__device__ __forceinline__ void net_burgers(int* __restrict__ list, int n, const TriDev* __restrict__ tri, double B[3])
{
    for (int i = 1; i < n; ++i) {
        const int v = list[i];
        int j = i;
        for (; j > 0 && (abs(list[j - 1]) > abs(v) || (abs(list[j - 1]) == abs(v) && list[j - 1] < v)); --j)
            list[j] = list[j - 1];
        list[j] = v;
    }
    B[0] = B[1] = B[2] = 0.0;
    for (int k = 0; k < n; ++k) {
        const int c = list[k];
        const TriDev& t = tri[(c > 0 ? c : -c) - 1];
        const double sg = c > 0 ? 1.0 : -1.0;
        const double slip[3] = {t.Dn, t.Dss, t.Dds};
        if (slip[0] == 0.0 && slip[1] == 0.0 && slip[2] == 0.0) continue;
        const double* axes[3] = {t.real.Vn, t.real.Vs, t.real.Vd};
        for (int m = 0; m < 3; ++m)
            for (int i = 0; i < 3; ++i) B[i] = add_rn(B[i], sg * mul_rn(axes[m][i], slip[m]));
    }
}

// Many sides (one patch listed with many slips) are summed by the block without
// sorting: each term is cut into multiples of three units, the first such that
// n terms add up exactly in double, each next finer by the bits that are left, so
// that no order of the additions shows (the reproducible sums of Demmel and
// Nguyen, 2013).  What is cut off is below n^4 2^-154 of the largest term.
constexpr int kBurgersThreads = 256, kBurgersWarps = kBurgersThreads / 32;
__device__ __forceinline__ void side_term(int c, const TriDev* __restrict__ tri, double v[3])
{
    const TriDev& t = tri[(c > 0 ? c : -c) - 1];
    const double sg = c > 0 ? 1.0 : -1.0;
    const double a = sg * t.Dn, b = sg * t.Dss, d = sg * t.Dds;
    const bool none = a == 0.0 && b == 0.0 && d == 0.0;   // (its axes may be none)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double x = dot3_rn(t.real.Vn[i], t.real.Vs[i], t.real.Vd[i], a, b, d);
        v[i] = none ? 0.0 : x;
    }
}
// (every thread of the block; s_red: 9 kBurgersWarps doubles; B in every thread)
__device__ __noinline__ void net_burgers_block(const int* __restrict__ list, int n, const TriDev* __restrict__ tri,
                                               double* s_red, double B[3])
{
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double big[3] = {0.0, 0.0, 0.0}, v[3];
    for (int k = threadIdx.x; k < n; k += kBurgersThreads) {
        side_term(list[k], tri, v);
        for (int i = 0; i < 3; ++i) big[i] = fmax(big[i], fabs(v[i]));
    }
    __syncthreads();   // s_red is free
    for (int i = 0; i < 3; ++i) {
        for (int d = 16; d; d >>= 1) big[i] = fmax(big[i], __shfl_xor_sync(full, big[i], d));
        if (lane == 0) s_red[3 * warp + i] = big[i];
    }
    __syncthreads();
    for (int w = 0; w < kBurgersWarps; ++w)
        for (int i = 0; i < 3; ++i) big[i] = fmax(big[i], s_red[3 * w + i]);
    const int bits = 33 - __clz(n);   // n < 2^(bits - 1)
    // at[i][q]: a term plus this, less this, is the term in units of its last place
    double at[3][3], sum[3][3] = {};
    for (int i = 0; i < 3; ++i)
        for (int q = 0; q < 3; ++q)
            at[i][q] = big[i] > 0.0 ? scalbn(1.5, ilogb(big[i]) + 1 + bits + q * (bits - 53)) : 0.0;
    for (int k = threadIdx.x; k < n; k += kBurgersThreads) {
        side_term(list[k], tri, v);
        for (int i = 0; i < 3; ++i)
            for (int q = 0; q < 3; ++q) {
                const double u = sub_rn(add_rn(v[i], at[i][q]), at[i][q]);
                sum[i][q] = add_rn(sum[i][q], u);
                v[i] = sub_rn(v[i], u);
            }
    }
    __syncthreads();
    for (int i = 0; i < 3; ++i)
        for (int q = 0; q < 3; ++q) {
            for (int d = 16; d; d >>= 1) sum[i][q] = add_rn(sum[i][q], __shfl_xor_sync(full, sum[i][q], d));
            if (lane == 0) s_red[9 * warp + 3 * i + q] = sum[i][q];
        }
    __syncthreads();
    for (int i = 0; i < 3; ++i) {
        double t[3] = {0.0, 0.0, 0.0};
        for (int w = 0; w < kBurgersWarps; ++w)
            for (int q = 0; q < 3; ++q) t[q] = add_rn(t[q], s_red[9 * w + 3 * i + q]);
        B[i] = add_rn(t[0], add_rn(t[1], t[2]));
    }
}

// The net Burgers vector of edge e = 32 blockIdx.x + lane to each lane of warp 0
// (none where e >= E); the other warps help with long lists only.  A list goes to
// the block where one thread's sort of it would take more than some microseconds:
// sorted by one thread, the five edges of two neighbours listed 100 000 times would
// take 2.5e9 dependent moves in memory each; at 300 points the whole call takes 3.7 ms.
constexpr int kSortedSides = 32;
__device__ __forceinline__ void edge_burgers(int64_t e, int64_t E, const int* __restrict__ ptr,
                                             const int* __restrict__ cnt, int* __restrict__ sides,
                                             const TriDev* __restrict__ tri, double B[3])
{
    __shared__ int s_first[32], s_n[32];
    __shared__ double s_red[9 * kBurgersWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    B[0] = B[1] = B[2] = 0.0;
    int n = 0;
    if (warp == 0) {
        const int first = e < E ? ptr[e] : 0;
        n = e < E ? cnt[e] : 0;
        s_first[lane] = first;
        s_n[lane] = n;
        if (n <= kSortedSides) net_burgers(sides + first, n, tri, B);
    }
    if (!__syncthreads_or(n > kSortedSides)) return;
    for (int q = 0; q < 32; ++q) {
        if (s_n[q] <= kSortedSides) continue;
        double S[3];
        net_burgers_block(sides + s_first[q], s_n[q], tri, s_red, S);
        if (threadIdx.x == q)
            for (int i = 0; i < 3; ++i) B[i] = S[i];
    }
}

// Each half-space edge's record for its net Burgers vector.
__global__ void __launch_bounds__(kBurgersThreads) edge_burgers_kernel(const double* __restrict__ pts, int64_t E, const int* __restrict__ ptr,
                                    const int* __restrict__ cnt, int* __restrict__ sides,
                                    const TriDev* __restrict__ tri, double nu, FscSide* __restrict__ out)
{
    const int64_t e = blockIdx.x * (int64_t)32 + (threadIdx.x & 31);
    double B[3];
    edge_burgers(e, E, ptr, cnt, sides, tri, B);
    if (e >= E || threadIdx.x >= 32) return;
    const double PA[3] = {pts[6 * e], pts[6 * e + 1], pts[6 * e + 2]};
    const double PB[3] = {pts[6 * e + 3], pts[6 * e + 4], pts[6 * e + 5]};
    build_side_burgers(PA, PB, B, nu, out[e]);
}

// Each full-space edge's; the number of edges is read on the device (count).
__global__ void __launch_bounds__(kBurgersThreads) segment_burgers_kernel(const double* __restrict__ pts, const int* __restrict__ count,
                                       const int* __restrict__ ptr, const int* __restrict__ cnt,
                                       int* __restrict__ sides, const TriDev* __restrict__ tri, double K8,
                                       SegRec* __restrict__ out)
{
    const int64_t e = blockIdx.x * (int64_t)32 + (threadIdx.x & 31), E = *count;
    double B[3];
    edge_burgers(e, E, ptr, cnt, sides, tri, B);
    if (e >= E || threadIdx.x >= 32) return;
    const double PA[3] = {pts[6 * e], pts[6 * e + 1], pts[6 * e + 2]};
    const double PB[3] = {pts[6 * e + 3], pts[6 * e + 4], pts[6 * e + 5]};
    build_segment(PA, PB, B, K8, out[e]);
}

// partial[(blockIdx.y * 9 + f) M + i] = the full-space strain (f 0-5) and the
// segments' displacement (f 6-8) at point i of the edges of chunk blockIdx.y of
// gridDim.y, summed in edge order (kSegStage records staged in shared memory at
// a time).  FP64 bound, 141 FP64 instructions per (edge, point) against about 490
// per (triangle, point) side by side: strain of 2013 triangles (3072 edges) at
// 20 000 points 670 us where the pairs took 1430 (two points per thread: 682).
constexpr int kSegStage = 16;
template <bool STRAIN, bool DISP>
__global__ void __launch_bounds__(kPairThreads) segment_sum_kernel(const SegRec* __restrict__ edges,
                                                                   const int* __restrict__ count,
                                                                   const double* __restrict__ X,
                                                                   const double* __restrict__ Y,
                                                                   const double* __restrict__ Z, int64_t M,
                                                                   double* __restrict__ partial)
{
    __shared__ __align__(16) double smem[kSegStage * kSegWords];
    const int64_t i = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const bool active = i < M;
    double x = 0.0, y = 0.0, z = 0.0;
    if (active) { x = X[i]; y = Y[i]; z = Z[i]; }
    double sE[6] = {}, sU[3] = {};
    const int64_t E = *count, echunk = (E + gridDim.y - 1) / gridDim.y;
    const int64_t e0 = min(E, (int64_t)blockIdx.y * echunk), e1 = min(E, e0 + echunk);
    for (int64_t eb = e0; eb < e1; eb += kSegStage) {
        const int ne = (int)min((int64_t)kSegStage, e1 - eb);
        __syncthreads();
        const double* src = reinterpret_cast<const double*>(edges + eb);
        for (int w = threadIdx.x; w < ne * kSegWords; w += kPairThreads) smem[w] = src[w];
        // edges without slip add nothing, also where 0 x the point's integrals is no
        // 0; beside one with slip, whose field is no number there either, they may
        // (a test of every edge costs 1 %)
        if (!__syncthreads_or(threadIdx.x < ne && edges[eb + threadIdx.x].slips != 0.0) || !active) continue;
#pragma unroll 1
        for (int k = 0; k < ne; ++k)
            segment_sum<STRAIN, DISP>(reinterpret_cast<const SegRec*>(smem)[k], x, y, z, sE, sU);
    }
    if (!active) return;
    double* p = partial + (int64_t)blockIdx.y * 9 * M;
#pragma unroll
    for (int k = 0; k < 6; ++k) p[k * M + i] = sE[k];
#pragma unroll
    for (int c = 0; c < 3; ++c) p[(6 + c) * M + i] = sU[c];
}

// partial[(blockIdx.y * 9 + f) M + i] = the strain (f 0-5; STRAIN EDGE_FSC: the
// free-surface correction, EDGE_FULL: all of it) and the correction's
// displacement (f 6-8; EDGE_FULL: all but the solid angles) at point i of the edges of chunk blockIdx.y, summed in
// edge order (8 edge records staged in shared memory at a time).  FP64 bound,
// 1122 FP64 instructions per (edge, point); three resident blocks per SM are worth
// the spills (208 bytes stored, 208 loaded; strain and displacement of 15 150 edges
// at 10 000 points, the real and image segments' displacement included: 14.5 ms at
// two blocks and 66 % of the pipe, 13.6 and 71 % at three).  The triangles' solid angles take 2.7 ms more; with the segments'
// displacement taken side by side the pairs took 7.3.
template <int STRAIN, bool DISP>
__global__ void __launch_bounds__(kPairThreads, STRAIN == EDGE_NONE ? 4 : STRAIN == EDGE_FSC && DISP ? 2 : 3)
side_sum_kernel(const FscSide* __restrict__ edges, int64_t E, int64_t echunk, const double* __restrict__ X,
                const double* __restrict__ Y, const double* __restrict__ Z, int64_t M, double* __restrict__ partial)
{
    extern __shared__ double smem[];
    const int64_t i = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const bool active = i < M;
    double x = 0.0, y = 0.0, z = 0.0;
    if (active) { x = X[i]; y = Y[i]; z = Z[i]; }
    double Es[3][6] = {}, Us[3][3] = {};
    const int64_t e0 = (int64_t)blockIdx.y * echunk;
    const int64_t e1 = min(E, e0 + echunk);
    for (int64_t eb = e0; eb < e1; eb += kEdgeStage) {
        const int ne = (int)min((int64_t)kEdgeStage, e1 - eb);
        __syncthreads();
        const double* src = reinterpret_cast<const double*>(edges + eb);
        for (int w = threadIdx.x; w < ne * kSideWords; w += kPairThreads) smem[w] = src[w];
        __syncthreads();
        if (!active) continue;
#pragma unroll 1
        for (int k = 0; k < ne; ++k) {
            const FscSide& s = reinterpret_cast<const FscSide*>(smem)[k];
            if constexpr (STRAIN == EDGE_FULL) {
                if (s.skip != 2.0) side_sum_full<DISP>(s, x, y, z, Es[0], Us[0]);
                continue;
            }
            if (s.skip != 0.0) continue;
            if (STRAIN == EDGE_FSC) fsc_strain(s, x, y, z, 0.0, 0.0, 1.0, Es);
            if (DISP) fsc_disp(s, x, y, z, 0.0, 0.0, 1.0, Us);
        }
    }
    if (!active) return;
    double* p = partial + (int64_t)blockIdx.y * 9 * M;
#pragma unroll
    for (int k = 0; k < 6; ++k) p[k * M + i] = STRAIN ? Es[0][k] : 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) p[(6 + c) * M + i] = DISP ? Us[0][c] : 0.0;
}

cudaError_t launch_td_sum_edges(PairArgs a, bool strain, bool disp, bool full, const EdgeArrays& ed, int64_t E,
                                void* edge_rec, double nu, int64_t echunk, double* edge_partial, cudaStream_t st, int64_t* launches)
{
    if (a.M == 0 || a.N == 0 || !(strain || disp)) return cudaSuccess;
    const size_t psmem = (size_t)pair_words(true, EDGE_FSC) * pair_stage(true, EDGE_FSC, false) * sizeof(double);
    const size_t esmem = (size_t)kSideWords * kEdgeStage * sizeof(double);
    const unsigned tiles = (unsigned)((a.M + kPairThreads - 1) / kPairThreads);
    auto pairs = [&](auto kern) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem);
        if (e != cudaSuccess) return e;
        kern<<<dim3(tiles, (unsigned)((a.N + a.tri_chunk - 1) / a.tri_chunk)), kPairThreads, psmem, st>>>(a);
        if (launches) ++*launches;
        return cudaGetLastError();
    };
    auto sums = [&](auto kern) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)esmem);
        if (e != cudaSuccess) return e;
        kern<<<dim3(tiles, (unsigned)((E + echunk - 1) / echunk)), kPairThreads, esmem, st>>>(
            (const FscSide*)edge_rec, E, echunk, a.X, a.Y, a.Z, a.M, edge_partial);
        if (launches) ++*launches;
        return cudaGetLastError();
    };
    cudaError_t e;
    if (strain && disp)
        e = full ? pairs(td_pair_kernel<true, true, true, OUT_SUM, false, false, 1, EDGE_FULL>)
                 : pairs(td_pair_kernel<true, true, true, OUT_SUM, false, false, 1, EDGE_FSC>);
    else if (strain && full) {
        e = launch_on_side(a, true, st);
        if (launches) ++*launches;
    } else if (strain)
        e = pairs(td_pair_kernel<true, true, false, OUT_SUM, false, false, 1, EDGE_FSC>);
    else
        e = pairs(td_pair_kernel<true, false, true, OUT_SUM, false, false, 1, EDGE_FSC>);
    if (e != cudaSuccess || E == 0) return e;
    edge_burgers_kernel<<<(unsigned)((E + 31) / 32), kBurgersThreads, 0, st>>>(ed.pts, E, ed.ptr, ed.cnt, ed.sides, a.tri, nu,
                                                                   (FscSide*)edge_rec);
    if (launches) ++*launches;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (strain && disp) return full ? sums(side_sum_kernel<EDGE_FULL, true>) : sums(side_sum_kernel<EDGE_FSC, true>);
    if (strain) return full ? sums(side_sum_kernel<EDGE_FULL, false>) : sums(side_sum_kernel<EDGE_FSC, false>);
    return sums(side_sum_kernel<EDGE_NONE, true>);
}

cudaError_t launch_td_sum_segments(PairArgs a, bool strain, bool disp, const EdgeArrays& ed, void* seg_rec, double nu,
                                   int64_t nechunk, double* edge_partial, cudaStream_t st, int64_t* launches)
{
    if (a.M == 0 || a.N == 0 || !(strain || disp)) return cudaSuccess;
    const size_t psmem = (size_t)pair_words(false, EDGE_FULL) * pair_stage(false, EDGE_FULL, false) * sizeof(double);
    const unsigned tiles = (unsigned)((a.M + kPairThreads - 1) / kPairThreads);
    SegRec* rec = (SegRec*)seg_rec;
    const double K8 = 0.5 * kInv4Pi / (1.0 - nu);
    segment_burgers_kernel<<<(unsigned)((3 * a.N + 31) / 32), kBurgersThreads, 0, st>>>(ed.pts, ed.count, ed.ptr, ed.cnt, ed.sides,
                                                                           a.tri, K8, rec);
    auto pairs = [&](auto kern) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem);
        if (e != cudaSuccess) return e;
        kern<<<dim3(tiles, (unsigned)((a.N + a.tri_chunk - 1) / a.tri_chunk)), kPairThreads, psmem, st>>>(a);
        return cudaGetLastError();
    };
    cudaError_t e;
    if (strain && disp) e = pairs(td_pair_kernel<false, true, true, OUT_SUM, false, false, 1, EDGE_FULL>);
    else if (strain) e = launch_on_side(a, false, st);
    else e = pairs(td_pair_kernel<false, false, true, OUT_SUM, false, false, 1, EDGE_FULL>);
    if (e != cudaSuccess) return e;
    const dim3 grid(tiles, (unsigned)nechunk);
    auto sums = [&](auto kern) { kern<<<grid, kPairThreads, 0, st>>>(rec, ed.count, a.X, a.Y, a.Z, a.M, edge_partial); };
    if (strain && disp) sums(segment_sum_kernel<true, true>);
    else if (strain) sums(segment_sum_kernel<true, false>);
    else sums(segment_sum_kernel<false, true>);
    *launches += 3;
    return cudaGetLastError();
}

size_t segment_record_bytes() { return sizeof(SegRec); }

cudaError_t launch_splice_fixed(const double* trac, const double* disp, int64_t N, int64_t nfix, const int* fixrow,
                                const int* freecol, int64_t nf, bool amat, double* out, int64_t lda, cudaStream_t st)
{
    if (N == 0 || nf == 0) return cudaSuccess;
    dim3 grid((unsigned)((N + 127) / 128), (unsigned)nf, 9);
    splice_fixed_kernel<<<grid, 128, 0, st>>>(trac, disp, N, nfix, fixrow, freecol, nf, amat ? 1 : 0, out, lda);
    return cudaGetLastError();
}

cudaError_t launch_gather_points(const double* X, const double* Y, const double* Z, const int* idx, int64_t n,
                                 double* out, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    gather_points_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(X, Y, Z, idx, n, out);
    return cudaGetLastError();
}

cudaError_t launch_assemble_mixed(PairArgs a, bool hs, const double* P1, const double* P2, const double* P3,
                                  double near_factor, void* tri32, double* near, cudaStream_t st, int64_t* launches)
{
    if (a.N == 0 || a.M == 0) return cudaSuccess;
    near_setup_kernel<<<1, 1024, 0, st>>>(P1, P2, P3, a.N, near_factor, near);
    const int words = hs ? kTriWordsHS : kTriWordsFS;
    const int64_t total = a.N * words;
    tri_to_f32_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(reinterpret_cast<const double*>(a.tri), a.N,
                                                                         words, kTriWordsHS, (float*)tri32);
    *launches += 2;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    a.tri32 = tri32;
    a.near = near;
    const int64_t ntile = (a.M + kPairThreads - 1) / kPairThreads;
    const int64_t nchunk = (a.N + a.tri_chunk - 1) / a.tri_chunk;
    dim3 grid((unsigned)ntile, (unsigned)nchunk);
    {
        auto kern = hs ? td_pair_f32_kernel<true> : td_pair_f32_kernel<false>;
        const size_t smem = (size_t)words * sizeof(float);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<grid, kPairThreads, smem, st>>>(a);
        ++*launches;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    {
        auto kern = hs ? td_pair_kernel<true, true, false, OUT_AMAT, true>
                       : td_pair_kernel<false, true, false, OUT_AMAT, true>;
        const size_t smem = (size_t)words * sizeof(double);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<grid, kPairThreads, smem, st>>>(a);
        ++*launches;
    }
    return cudaGetLastError();
}

size_t tri_record_bytes_f32() { return sizeof(TriDevT<float>); }

cudaError_t launch_assemble_update(PairArgs a, bool hs, const int* list, int64_t k, cudaStream_t st,
                                   int64_t* launches)
{
    if (k == 0 || a.N == 0) return cudaSuccess;
    const int words = hs ? kTriWordsHS : kTriWordsFS;
    const size_t smem = (size_t)words * sizeof(double);
    auto kern = hs ? td_pair_kernel<true, true, false, OUT_AMAT, false, true>
                   : td_pair_kernel<false, true, false, OUT_AMAT, false, true>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t Ntot = a.N;
    a.Ntot = Ntot;
    // columns of the listed triangles, every point
    PairArgs c = a;
    c.tri_list = list;
    c.obs_list = nullptr;
    c.M = Ntot;
    c.N = k;
    c.tri_chunk = k < 8 ? k : 8;
    dim3 gc((unsigned)((Ntot + kPairThreads - 1) / kPairThreads), (unsigned)((k + c.tri_chunk - 1) / c.tri_chunk));
    kern<<<gc, kPairThreads, smem, st>>>(c);
    // rows of the listed points, every triangle
    PairArgs r = a;
    r.tri_list = nullptr;
    r.obs_list = list;
    r.M = k;
    r.N = Ntot;
    r.tri_chunk = 8;
    dim3 gr((unsigned)((k + kPairThreads - 1) / kPairThreads), (unsigned)((Ntot + 7) / 8));
    kern<<<gr, kPairThreads, smem, st>>>(r);
    *launches += 2;
    return cudaGetLastError();
}

cudaError_t launch_td_setup(const double* P1, const double* P2, const double* P3, int64_t N, const double* Dss,
                            const double* Dds, const double* Dn, int64_t slip_stride, double nu, bool hs,
                            TriDev* out, cudaStream_t st, bool sides)
{
    if (N == 0) return cudaSuccess;
    const int bs = 32;   // a thread's chain bounds it: spread over the SMs
    td_setup_kernel<<<(unsigned)((N + bs - 1) / bs), bs, 0, st>>>(P1, P2, P3, N, Dss, Dds, Dn, slip_stride, nu,
                                                                  hs ? 1 : 0, sides ? 1 : 0, out);
    return cudaGetLastError();
}

cudaError_t launch_hs_check(const double* Z, int64_t M, const double* P1, const double* P2, const double* P3,
                            int64_t N, int* flag, cudaStream_t st, const double* nz, bool clear, int* horizontal)
{
    cudaError_t e = clear ? cudaMemsetAsync(flag, 0, sizeof(int), st) : cudaSuccess;
    if (e != cudaSuccess || M + N == 0) return e;
    const int bs = 256;
    int64_t nb = (M + N + bs - 1) / bs;
    if (nb > 1184) nb = 1184;
    hs_check_kernel<<<(unsigned)nb, bs, 0, st>>>(Z, nz, M, P1, P2, P3, N, flag, horizontal);
    return cudaGetLastError();
}

cudaError_t launch_colloc(const double* normals, const double* mid, int64_t N, double* X, double* Y, double* Z,
                          double* dirs, cudaStream_t st)
{
    if (N == 0) return cudaSuccess;
    const int bs = 128;
    colloc_kernel<<<(unsigned)((N + bs - 1) / bs), bs, 0, st>>>(normals, mid, N, X, Y, Z, dirs);
    return cudaGetLastError();
}

cudaError_t launch_sum_chunks(const double* partial, int64_t nchunk, int64_t M, int fields_mask, double* out,
                              cudaStream_t st)
{
    if (M == 0) return cudaSuccess;
    const int bs = 256;
    dim3 grid((unsigned)((M + bs - 1) / bs), 9);
    sum_chunks_kernel<<<grid, bs, 0, st>>>(partial, nchunk, M, fields_mask, out);
    return cudaGetLastError();
}

cudaError_t launch_sum_chunks_split(const double* partial, int64_t nchunk, int64_t M, int fields_mask,
                                    double* strain_out, double* disp_out, cudaStream_t st)
{
    if (M == 0) return cudaSuccess;
    const int bs = 256;
    dim3 grid((unsigned)((M + bs - 1) / bs), 9);
    sum_chunks_split_kernel<<<grid, bs, 0, st>>>(partial, nchunk, M, fields_mask, strain_out, disp_out);
    return cudaGetLastError();
}

cudaError_t launch_td_sum(const double* in, int64_t M, int64_t N, int nf, double* out, cudaStream_t st)
{
    if (M == 0) return cudaSuccess;
    const int bs = 256;
    dim3 grid((unsigned)((M + bs - 1) / bs), (unsigned)nf);
    td_sum_kernel<<<grid, bs, 0, st>>>(in, M, N, nf, out);
    return cudaGetLastError();
}

}  // namespace cad
