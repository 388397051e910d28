// Line classes: the y and z lines of a problem have few distinct sequences of coefficients (a layered specimen with
// some flaws has one per layer and flaw pattern), so the step keeps one table per distinct line and a class per line
// instead of two values per voxel.  At 65x512x512 that takes 16 of the y sweep's 32 bytes per voxel and 16 of the z
// sweep's 40 out of its HBM traffic.  Lines are compared bit for bit: the step's arithmetic does not change.
#include <algorithm>

#include "hs2g_internal.cuh"

namespace hs2g {
namespace {

constexpr int kTh = 256;

struct LineGrid {
  const double* a;
  const double* b;
  int64_t outer, nx, ost, n, rst;  // line (o, i): rows r at o*ost + r*rst + i
  __device__ int64_t lines() const { return outer * nx; }
  __device__ int64_t base(int64_t l) const { return (l / nx) * ost + l % nx; }
};

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
__global__ void gather_lines_kernel(LineGrid g, const int* rep, int64_t nclass, double* ta, double* tb) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nclass * g.n) return;
  const int64_t p = g.base(rep[t / g.n]) + (t % g.n) * g.rst;
  ta[t] = g.a[p];
  tb[t] = g.b[p];
}

}  // namespace

cudaError_t classify_lines(const double* a, const double* b, int64_t outer, int64_t nx, int64_t ost, int64_t n,
                           int64_t rst, LineTables* out, cudaStream_t s) {
  *out = LineTables{};
  const int64_t lines = outer * nx;
  // Worth it when the tables are an eighth of the arrays: the classes of a warp's 16 lines then cost it no more
  // than reading the arrays would.
  const int64_t max_class = std::max<int64_t>(1, lines / 8);
  if (lines >= ((int64_t)1 << 30)) return cudaSuccess;
  int64_t cap = 64;
  while (cap < 2 * lines) cap *= 2;
  const LineGrid g{a, b, outer, nx, ost, n, rst};
  unsigned long long* keys = nullptr;
  int *ints = nullptr, host[2] = {0, 1};
  int32_t* cls = nullptr;
  // ints: owner[cap], id[cap], slot[lines], rep[max_class], {count, same}
  cudaError_t e = cudaMalloc(&keys, sizeof(*keys) * cap);
  if (e == cudaSuccess) e = cudaMalloc(&ints, sizeof(int) * (2 * cap + lines + max_class + 2));
  if (e == cudaSuccess) e = cudaMalloc(&cls, sizeof(int32_t) * lines);
  int *owner = ints, *id = ints + cap, *slot = id + cap, *rep = slot + lines, *count = rep + max_class;
  const unsigned blocks = (unsigned)((lines + kTh - 1) / kTh);
  if (e == cudaSuccess) e = cudaMemsetAsync(keys, 0, sizeof(*keys) * cap, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(owner, 0x7f, sizeof(int) * cap, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(count, host, sizeof host, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    hash_lines_kernel<<<blocks, kTh, 0, s>>>(g, keys, owner, cap - 1, slot);
    number_lines_kernel<<<blocks, kTh, 0, s>>>(lines, owner, slot, id, rep, count, (int)max_class);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, count, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  const int64_t nclass = host[0];
  if (e == cudaSuccess && nclass <= max_class) {
    e = cudaMalloc(&out->a, sizeof(double) * nclass * n);
    if (e == cudaSuccess) e = cudaMalloc(&out->b, sizeof(double) * nclass * n);
    if (e == cudaSuccess) {
      assign_lines_kernel<<<blocks, kTh, 0, s>>>(g, slot, id, rep, cls, count + 1);
      gather_lines_kernel<<<(unsigned)((nclass * n + kTh - 1) / kTh), kTh, 0, s>>>(g, rep, nclass, out->a, out->b);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host + 1, count + 1, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && host[1]) {
      out->cls = cls;
      out->nclass = nclass;
      cls = nullptr;
    } else {
      cudaFree(out->a);
      cudaFree(out->b);
      out->a = out->b = nullptr;
    }
  }
  cudaFree(keys);
  cudaFree(ints);
  cudaFree(cls);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

}  // namespace hs2g
