// fedg_two.cuh -- kernels whose threads carry the same node of two consecutive elements in packed pairs: the
// elements of a thread, their neighbours, and the layout of a field in shared memory.  Mesh: any struct
// with NeX, NeY, NeZ.
#pragma once
#include "fedg_p2.cuh"

namespace fedg {
namespace {

// position of node (i, row = j + N1 k): rows permuted so that one column of neighbouring rows falls on
// different banks
template <int N1>
__device__ __forceinline__ int two_at(int i, int row) {
  if (N1 == 8) i ^= row & 7;
  if (N1 == 4) i ^= (row >> 1) & 3;
  return row * N1 + i;
}

// blocks per SM that make up `total` threads
constexpr int two_minb(int threads, int total) { return total / ((threads + 31) / 32 * 32); }

// the thread's (first) node in elements e[0] and e[1] (e[1] = e[0] where the last element has no partner, or with SOLO
// none has one)
struct TwoIdx {
  int e[2], ex[2], ey[2], ez[2], nxy, p, i, j, k;
  bool valid, both;
};
template <int N1, int PPB, int NT, bool SOLO = false, class Mesh>
__device__ __forceinline__ TwoIdx two_idx(const Mesh& op, int Ne, int& pair) {
  constexpr int NF = N1 * N1;
  TwoIdx x;
  pair = threadIdx.x / NT;
  x.p = threadIdx.x - pair * NT;
  const int e0 = (SOLO ? 1 : 2) * (blockIdx.x * PPB + pair);
  x.valid = e0 < Ne;
  x.both = !SOLO && e0 + 1 < Ne;
  x.nxy = op.NeX * op.NeY;
  x.i = x.p % N1;
  x.j = (x.p / N1) % N1;
  x.k = x.p / NF;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    x.e[m] = x.valid ? (x.both ? e0 + m : e0) : 0;
    x.ez[m] = x.e[m] / x.nxy;
    x.ey[m] = (x.e[m] - x.ez[m] * x.nxy) / op.NeX;
    x.ex[m] = x.e[m] - x.ez[m] * x.nxy - x.ey[m] * op.NeX;
  }
  return x;
}
// the neighbour across face dir (0 x, 1 y, 2 z) on the lower (up = 0) or upper side; -1 at a lid
template <class Mesh>
__device__ __forceinline__ int two_nbr(const Mesh& op, const TwoIdx& x, int m, int dir, int up) {
  const int e = x.e[m];
  if (dir == 0) return up ? (x.ex[m] < op.NeX - 1 ? e + 1 : e - (op.NeX - 1)) : (x.ex[m] > 0 ? e - 1 : e + op.NeX - 1);
  if (dir == 1)
    return up ? (x.ey[m] < op.NeY - 1 ? e + op.NeX : e - (op.NeY - 1) * op.NeX)
              : (x.ey[m] > 0 ? e - op.NeX : e + (op.NeY - 1) * op.NeX);
  return up ? (x.ez[m] < op.NeZ - 1 ? e + x.nxy : -1) : (x.ez[m] > 0 ? e - x.nxy : -1);
}
// node (i, j, k) of face node ab on side `s` (0 lower, 1 upper) of direction dir
template <int N1>
__device__ __forceinline__ void two_face_node(int dir, int s, int ab, int& i, int& row) {
  const int a = ab % N1, b = ab / N1, w = s * (N1 - 1);
  i = dir == 0 ? w : a;
  row = dir == 0 ? a + N1 * b : (dir == 1 ? w + N1 * b : b + N1 * w);
}

}  // namespace
}  // namespace fedg
