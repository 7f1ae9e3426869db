// Mesh-edge table on the device: an open-addressing hash table keyed by the two
// end points of a side (whichever way it runs, compared bit for bit, -0.0 taken
// as 0.0).  The table holds side numbers; the smallest side number of a key
// represents its edge, so the numbering does not depend on the order in which
// threads insert.  A few passes over 3 N sides of ~2-4 us each at 30 000 sides,
// latency-bound, in place of a device-to-host copy of the vertices and a host
// hash map (about 5 ms at 10 000 triangles, 0.3 ms at 900).
#include "edges.h"

namespace cad {

namespace {

constexpr int kThreads = 256;

struct Ends {
    long long v[6];
};

__device__ __forceinline__ Ends side_ends(const double* __restrict__ P1, const double* __restrict__ P2,
                                          const double* __restrict__ P3, int64_t N, int k)
{
    const int j = k / 3, s = k - 3 * j;
    const double* a = s == 0 ? P1 : s == 1 ? P2 : P3;
    const double* b = s == 0 ? P2 : s == 1 ? P3 : P1;
    Ends e;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        e.v[c] = __double_as_longlong(a[j + c * N] + 0.0);   // + 0.0 turns -0.0 into 0.0
        e.v[3 + c] = __double_as_longlong(b[j + c * N] + 0.0);
    }
    return e;
}

__device__ __forceinline__ bool runs_along(const Ends& a, const Ends& b)
{
    bool eq = true;
#pragma unroll
    for (int c = 0; c < 6; ++c) eq = eq && a.v[c] == b.v[c];
    return eq;
}
__device__ __forceinline__ bool same_edge(const Ends& a, const Ends& b)
{
    bool rev = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) rev = rev && a.v[c] == b.v[3 + c] && a.v[3 + c] == b.v[c];
    return rev || runs_along(a, b);
}

__device__ __forceinline__ unsigned edge_hash(const Ends& e)
{
    unsigned long long h[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        unsigned long long x = 0x9e3779b97f4a7c15ull;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x ^= (unsigned long long)e.v[3 * p + c];
            x *= 0xff51afd7ed558ccdull;
            x ^= x >> 32;
        }
        h[p] = x;
    }
    unsigned long long s = h[0] + h[1];   // the same for both directions
    s *= 0xc4ceb9fe1a85ec53ull;
    return (unsigned)(s >> 32);
}

// Every side enters its slot; the slot keeps the smallest side of its edge.
// The table has at least twice as many slots as there are sides, so a free
// slot is always met.
__global__ void __launch_bounds__(kThreads) edge_insert_kernel(const double* __restrict__ P1,
                                                               const double* __restrict__ P2,
                                                               const double* __restrict__ P3, int64_t N,
                                                               int* __restrict__ table, unsigned mask)
{
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= 3 * N) return;
    const Ends me = side_ends(P1, P2, P3, N, k);
    unsigned slot = edge_hash(me) & mask;
    for (unsigned probe = 0; probe <= mask; ++probe, slot = (slot + 1) & mask) {
        const int cur = atomicCAS(table + slot, -1, k);
        if (cur == -1) return;
        if (same_edge(me, side_ends(P1, P2, P3, N, cur))) {
            atomicMin(table + slot, k);
            return;
        }
    }
}

// rep[k]: the side that represents k's edge; block_first[b]: representatives
// in block b of sides.
__global__ void __launch_bounds__(kThreads) edge_find_kernel(const double* __restrict__ P1,
                                                             const double* __restrict__ P2,
                                                             const double* __restrict__ P3, int64_t N,
                                                             const int* __restrict__ table, unsigned mask,
                                                             int* __restrict__ rep, int* __restrict__ block_first)
{
    const int k = blockIdx.x * kThreads + threadIdx.x;
    int r = -1;
    if (k < 3 * N) {
        const Ends me = side_ends(P1, P2, P3, N, k);
        unsigned slot = edge_hash(me) & mask;
        for (unsigned probe = 0; probe <= mask; ++probe, slot = (slot + 1) & mask) {
            const int cur = table[slot];
            if (cur == k || (cur >= 0 && same_edge(me, side_ends(P1, P2, P3, N, cur)))) {
                r = cur;
                break;
            }
        }
        if (r < 0) r = k;
        rep[k] = r;
    }
    const int n = __syncthreads_count(k < 3 * N && r == k);
    if (threadIdx.x == 0) block_first[blockIdx.x] = n;
}

// Exclusive prefix sums of n block counts in place; the total to count[0].
__global__ void __launch_bounds__(1024) edge_scan_kernel(int* __restrict__ v, int n, int* __restrict__ count)
{
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + threadIdx.x;
        const int x = i < n ? v[i] : 0;
        int s = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += y;
        }
        if (lane == 31) s_warp[warp] = s;
        __syncthreads();
        int w = s_warp[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        const int before = warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0;
        const int total = __shfl_sync(0xffffffffu, w, 31);
        if (i < n) v[i] = base + before + s - x;
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) count[0] = base;
}

// Edge numbers of the representatives, their end points, and zeroed counters.
__global__ void __launch_bounds__(kThreads) edge_number_kernel(const double* __restrict__ P1,
                                                               const double* __restrict__ P2,
                                                               const double* __restrict__ P3, int64_t N,
                                                               const int* __restrict__ rep,
                                                               const int* __restrict__ block_first,
                                                               int* __restrict__ number, double* __restrict__ pts,
                                                               int* __restrict__ cnt)
{
    __shared__ int s_warp[kThreads / 32];
    const int k = blockIdx.x * kThreads + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool first = k < 3 * N && rep[k] == k;
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    if (!first) return;
    int e = block_first[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) e += s_warp[w];
    number[k] = e;
    if (cnt) cnt[e] = 0;
    const Ends me = side_ends(P1, P2, P3, N, k);
#pragma unroll
    for (int c = 0; c < 6; ++c) pts[6 * (int64_t)e + c] = __longlong_as_double(me.v[c]);
}

// Every side's signed edge number (and the number of sides on each edge).
__global__ void __launch_bounds__(kThreads) edge_code_kernel(const double* __restrict__ P1,
                                                             const double* __restrict__ P2,
                                                             const double* __restrict__ P3, int64_t N,
                                                             const int* __restrict__ rep,
                                                             const int* __restrict__ number, int* __restrict__ code,
                                                             int* __restrict__ cnt)
{
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= 3 * N) return;
    const int r = rep[k], e = number[r];
    const bool along = r == k || runs_along(side_ends(P1, P2, P3, N, k), side_ends(P1, P2, P3, N, r));
    code[k] = along ? e + 1 : -(e + 1);
    if (cnt) atomicAdd(cnt + e, 1);
}

// Room for each edge's sides, taken from one counter (the segments' order does
// not matter); the counts restart as fill positions.
__global__ void __launch_bounds__(kThreads) edge_room_kernel(const int* __restrict__ count, int* __restrict__ cnt,
                                                             int* __restrict__ ptr, int* __restrict__ fill,
                                                             int* __restrict__ total)
{
    const int e = blockIdx.x * kThreads + threadIdx.x;
    if (e >= count[0]) return;
    ptr[e] = atomicAdd(total, cnt[e]);
    fill[e] = 0;
}
__global__ void __launch_bounds__(kThreads) edge_sides_kernel(const int* __restrict__ code, int64_t N,
                                                              const int* __restrict__ ptr, int* __restrict__ fill,
                                                              int* __restrict__ sides)
{
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= 3 * N) return;
    const int c = code[k], e = (c > 0 ? c : -c) - 1, t = k / 3 + 1;
    sides[ptr[e] + atomicAdd(fill + e, 1)] = c > 0 ? t : -t;
}

int64_t table_slots(int64_t N)
{
    int64_t t = 64;
    while (t < 6 * N) t *= 2;
    return t;
}

}  // namespace

bool edge_table_fits(int64_t N) { return 6 * N <= int64_t(1) << 31; }

size_t edge_work_ints(int64_t N)
{
    return (size_t)table_slots(N) + 9 * (size_t)N + (size_t)(3 * N + kThreads - 1) / kThreads + 2;
}

cudaError_t launch_edge_table(const double* P1, const double* P2, const double* P3, int64_t N, const EdgeArrays& a,
                              bool lists, cudaStream_t st, int64_t* launches)
{
    if (N <= 0) return cudaMemsetAsync(a.count, 0, sizeof(int), st);
    if (!edge_table_fits(N)) return cudaErrorInvalidValue;
    const unsigned slots = (unsigned)table_slots(N);
    const unsigned nb = (unsigned)((3 * N + kThreads - 1) / kThreads);
    int* table = a.work;
    int* rep = table + (size_t)slots;
    int* number = rep + 3 * N;
    int* fill = number + 3 * N;
    int* block_first = fill + 3 * N;
    int* total = block_first + nb;
    if (cudaError_t e = cudaMemsetAsync(table, 0xff, (size_t)slots * sizeof(int), st)) return e;
    edge_insert_kernel<<<nb, kThreads, 0, st>>>(P1, P2, P3, N, table, slots - 1);
    edge_find_kernel<<<nb, kThreads, 0, st>>>(P1, P2, P3, N, table, slots - 1, rep, block_first);
    edge_scan_kernel<<<1, 1024, 0, st>>>(block_first, (int)nb, a.count);
    edge_number_kernel<<<nb, kThreads, 0, st>>>(P1, P2, P3, N, rep, block_first, number, a.pts,
                                                lists ? a.cnt : nullptr);
    edge_code_kernel<<<nb, kThreads, 0, st>>>(P1, P2, P3, N, rep, number, a.code, lists ? a.cnt : nullptr);
    *launches += 5;
    if (lists) {
        if (cudaError_t e = cudaMemsetAsync(total, 0, sizeof(int), st)) return e;
        edge_room_kernel<<<nb, kThreads, 0, st>>>(a.count, a.cnt, a.ptr, fill, total);
        edge_sides_kernel<<<nb, kThreads, 0, st>>>(a.code, N, a.ptr, fill, a.sides);
        *launches += 2;
    }
    return cudaGetLastError();
}

}  // namespace cad
