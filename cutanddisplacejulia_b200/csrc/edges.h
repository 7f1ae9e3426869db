// Mesh-edge table of a triangle list, built on the device (edges.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace cad {

// The distinct sides (edges) of N triangles.  Side s of triangle j (number
// 3 j + s) runs P1->P2, P2->P3, P3->P1.  Edges are numbered in the order in
// which the sides first meet them, and run the way that first side does.
struct EdgeArrays {
    double* pts;   // 6 per edge: its end points (room for 3 N edges)
    int* code;     // 3 per triangle: +(edge + 1), or -(edge + 1) for a side running against its edge
    int* ptr;      // per edge: first entry in sides (sums only)
    int* cnt;      // per edge: number of sides on it (sums only)
    int* sides;    // +-(triangle + 1) of the sides on each edge, in no particular order (sums only)
    int* work;     // edge_work_ints(N) ints
    int* count;    // device: [0] number of edges
};

size_t edge_work_ints(int64_t N);
// Whether the table of N triangles can be built: its slots (a power of two, at
// least two per side) are counted in 32 bits.  Larger lists stay per side.
bool edge_table_fits(int64_t N);

// Fills pts, code and count[0] (and ptr, cnt, sides with lists = true) from
// the vertex lists (N x 3 column-major); edge_table_fits(N).
cudaError_t launch_edge_table(const double* P1, const double* P2, const double* P3, int64_t N, const EdgeArrays& a,
                              bool lists, cudaStream_t st, int64_t* launches);

}  // namespace cad
