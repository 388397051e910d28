// Line classes: the lines of a problem have few distinct sequences of coefficients (a layered specimen with
// some flaws has one per layer and flaw pattern), so the step keeps one table per distinct line and a class per line
// instead of two values per voxel.  At 65x512x512 that takes 16 of the y sweep's 32 bytes per voxel and 16 of the z
// sweep's 40 out of its HBM traffic.  Lines are compared bit for bit: the step's arithmetic does not change.
#include <algorithm>

#include "hs2g_internal.cuh"

namespace hs2g {
namespace {

constexpr int kTh = 256;

__device__ __forceinline__ unsigned long long mix(unsigned long long h, double v) {
  h = (h ^ (unsigned long long)__double_as_longlong(v)) * 0x9E3779B97F4A7C15ull;
  return h ^ (h >> 29);
}

// the line's hash goes into an open-addressing table; slot[l]: where; owner[slot]: the smallest line with that hash
__global__ void hash_lines_kernel(LineGrid g, unsigned long long* keys, int* owner, int64_t mask, int* slot) {
  const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= g.lines()) return;
  int64_t p = g.base(l);
  unsigned long long h = 1;
  for (int64_t r = 0; r < g.n; ++r, p += g.rst) h = mix(mix(h, g.a[p]), g.b[p]);
  if (h == 0) h = 1;
  int64_t e = (int64_t)(h >> 17) & mask;
  for (;; e = (e + 1) & mask) {  // the table has twice as many entries as there are lines
    const unsigned long long k = atomicCAS(keys + e, 0ull, h);
    if (k == 0ull || k == h) break;
  }
  slot[l] = (int)e;
  atomicMin(owner + e, (int)l);
}
// one class per owning line
__global__ void number_lines_kernel(int64_t lines, const int* owner, const int* slot, int* id, int* rep, int* count,
                                    int max_class) {
  const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= lines || owner[slot[l]] != (int)l) return;
  const int c = atomicAdd(count, 1);
  if (c < max_class) rep[c] = (int)l;
  id[slot[l]] = c;
}
// classes per line, each line checked against its class's line (a clash of hashes clears *same)
__global__ void assign_lines_kernel(LineGrid g, const int* slot, const int* id, const int* rep, int32_t* cls, int* same) {
  const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= g.lines()) return;
  const int c = id[slot[l]];
  cls[l] = c;
  int64_t p = g.base(l), q = g.base(rep[c]);
  bool eq = true;
  for (int64_t r = 0; r < g.n; ++r, p += g.rst, q += g.rst)
    eq &= __double_as_longlong(g.a[p]) == __double_as_longlong(g.a[q]) &&
          __double_as_longlong(g.b[p]) == __double_as_longlong(g.b[q]);
  if (!eq) *same = 0;
}
__global__ void gather_lines_kernel(LineGrid g, const int* rep, int64_t nclass, int64_t mid, double* ta, double* tb) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nclass * g.n) return;
  int64_t r = t % g.n;
  if (mid >= 0 && r > mid) r = mid + g.n - r;
  const int64_t p = g.base(rep[t / g.n]) + r * g.rst;
  ta[t] = g.a[p];
  tb[t] = g.b[p];
}

}  // namespace

size_t LineJob::scratch_bytes(int64_t lines) {
  const ClassTable t(lines);
  return t.bytes() + sizeof(int) * (size_t)max_class(lines) + 256;
}

cudaError_t LineJob::begin(unsigned char* scratch, cudaStream_t s) {
  const int64_t lines = grid.lines();
  table = ClassTable(lines);
  rep = reinterpret_cast<int*>(table.place(scratch));
  cudaError_t e = table.clear(s);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((lines + kTh - 1) / kTh);
  hash_lines_kernel<<<blocks, kTh, 0, s>>>(grid, table.keys, table.owner, table.cap - 1, table.slot);
  number_lines_kernel<<<blocks, kTh, 0, s>>>(lines, table.owner, table.slot, table.id, rep, table.count,
                                             (int)max_class(lines));
  return cudaGetLastError();
}

cudaError_t LineJob::finish(int64_t nclass, LineTables* out, cudaStream_t s) {
  *out = LineTables{};
  const int64_t lines = grid.lines(), n = grid.n;
  if (nclass > max_class(lines)) return cudaSuccess;
  unsigned char* m = nullptr;
  const size_t half = sizeof(double) * (size_t)(nclass * n);
  cudaError_t e = cudaMalloc(&m, 2 * half + sizeof(int32_t) * lines);
  if (e == cudaErrorMemoryAllocation) {  // no room for the tables: the arrays stay
    cudaGetLastError();
    return cudaSuccess;
  }
  if (e != cudaSuccess) return e;
  out->a = reinterpret_cast<double*>(m);
  out->b = reinterpret_cast<double*>(m + half);
  out->cls = reinterpret_cast<int32_t*>(m + 2 * half);
  out->nclass = nclass;
  out->bytes = 2 * half + sizeof(int32_t) * lines;
  assign_lines_kernel<<<(unsigned)((lines + kTh - 1) / kTh), kTh, 0, s>>>(grid, table.slot, table.id, rep, out->cls,
                                                                         table.count + 1);
  gather_lines_kernel<<<(unsigned)((nclass * n + kTh - 1) / kTh), kTh, 0, s>>>(grid, rep, nclass, mid, out->a, out->b);
  return cudaGetLastError();
}

}  // namespace hs2g
