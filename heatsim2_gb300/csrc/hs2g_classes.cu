// Line classes: the lines of a problem have few distinct sequences of coefficients (a layered specimen with
// some flaws has one per layer and flaw pattern), so the step keeps one table per distinct line and a class per line
// instead of two values per voxel.  At 65x512x512 that takes 16 of the y sweep's 32 bytes per voxel and 16 of the z
// sweep's 40 out of its HBM traffic.  Lines are compared bit for bit: the step's arithmetic does not change.
//
// The search is part of setting a problem up, where a small problem waits for each launch and a long line for each
// dependent load: the three axes share their launches, a line's rows are spread over 8 or 32 threads, and the lines of a
// warp that are alike go to the table as one.  The search and the blocks' (hs2g_compile.cu), with a thread per line, an
// atomic per line and launches per axis: 153 us in 16 launches at 20x40x40, 4.3 ms at 64x4096x4; so 46 us in 7, and 0.53 ms.
#include <algorithm>

#include "hs2g_internal.cuh"

namespace hs2g {
namespace {

constexpr int kTh = 256;

__device__ __forceinline__ unsigned long long mix(unsigned long long h, double v) {
  h = (h ^ (unsigned long long)__double_as_longlong(v)) * 0x9E3779B97F4A7C15ull;
  return h ^ (h >> 29);
}

// The CTA's axis, and this thread's line of it and share of the line's rows (r0, r0 + dr, ...).  A CTA takes `per` lines;
// neighbouring threads take neighbouring rows of an x line, neighbouring lines otherwise.
struct Share {
  int axis, line;  // line within the CTA
  int64_t l;
  int r0, dr;
};
__device__ __forceinline__ Share share_of(const LineSearch& s) {
  Share w;
  w.axis = (int)blockIdx.x >= s.first_cta[1] ? ((int)blockIdx.x >= s.first_cta[2] ? 2 : 1) : 0;
  const int per = s.per[w.axis];
  w.dr = kTh / per;
  const bool rows = s.grid[w.axis].rst == 1;
  w.line = rows ? threadIdx.x / w.dr : threadIdx.x % per;
  w.r0 = rows ? threadIdx.x % w.dr : threadIdx.x / per;
  w.l = (int64_t)((int)blockIdx.x - s.first_cta[w.axis]) * per + w.line;
  return w;
}

// a line's hash, a sum over its rows, goes into an open-addressing table; slot[l]: where; owner[slot]: the smallest line
// with that hash
__global__ void __launch_bounds__(kTh) hash_lines_kernel(LineSearch s) {
  __shared__ unsigned long long part[kTh];
  const Share w = share_of(s);
  const LineGrid& g = s.grid[w.axis];
  const int64_t lines = g.lines();
  unsigned long long h = 0;
  if (w.l < lines) {
    const int64_t p = g.base(w.l);
#pragma unroll 4
    for (int64_t r = w.r0; r < g.n; r += w.dr)
      h += mix(mix((unsigned long long)(r + 1) * 0xD6E8FEB86659FD93ull, g.a[p + r * g.rst]), g.b[p + r * g.rst]);
  }
  const int per = s.per[w.axis];
  part[w.r0 * per + w.line] = h;
  __syncthreads();
  const int lane = threadIdx.x;
  if (lane >= per) return;
  const int64_t l = (int64_t)((int)blockIdx.x - s.first_cta[w.axis]) * per + lane;
  h = 0;
  for (int r = 0; r < w.dr; ++r) h += part[r * per + lane];
  h = (h ^ (h >> 32)) * 0x9E3779B97F4A7C15ull;
  s.table[w.axis].insert_all(per == 32 ? 0xffffffffu : (1u << per) - 1, l >= lines ? 0 : h ? h : 1, (int)l);
}
// a number for each owner; for a line's, the line
__global__ void __launch_bounds__(kTh) number_kernel(LineSearch s, ClassTable blocks) {
  int64_t l = blockIdx.x * (int64_t)kTh + threadIdx.x;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const ClassTable& t = s.table[a];
    if (l >= 0 && l < t.n && t.owner[t.slot[l]] == (int)l) {
      const int c = atomicAdd(t.count, 1);
      if (c < (int)LineSearch::max_class(t.n)) s.rep[a][c] = (int)l;
      t.id[t.slot[l]] = c;
    }
    l -= t.n;
  }
  if (l >= 0 && l < blocks.n && blocks.owner[blocks.slot[l]] == (int)l)
    blocks.id[blocks.slot[l]] = atomicAdd(blocks.count, 1);
}
// classes per line, each line checked against its class's line (a clash of hashes is noted in count[1])
__global__ void __launch_bounds__(kTh) assign_lines_kernel(LineSearch s) {
  const Share w = share_of(s);
  const LineGrid& g = s.grid[w.axis];
  if (w.l >= g.lines()) return;
  const ClassTable& t = s.table[w.axis];
  const int c = t.id[t.slot[w.l]];
  if (w.r0 == 0) s.cls[w.axis][w.l] = c;
  const int64_t p = g.base(w.l), q = g.base(s.rep[w.axis][c]);
  bool eq = true;
#pragma unroll 4
  for (int64_t r = w.r0; r < g.n; r += w.dr)
    eq &= __double_as_longlong(g.a[p + r * g.rst]) == __double_as_longlong(g.a[q + r * g.rst]) &&
          __double_as_longlong(g.b[p + r * g.rst]) == __double_as_longlong(g.b[q + r * g.rst]);
  if (!eq) t.count[1] = 1;
}
// the tables; blockIdx.y: the axis
__global__ void __launch_bounds__(kTh) gather_lines_kernel(LineSearch s) {
  const int a = blockIdx.y;
  const LineGrid& g = s.grid[a];
  const int64_t t = blockIdx.x * (int64_t)kTh + threadIdx.x;
  if (t >= s.nclass[a] * g.n) return;
  const int64_t c = t / g.n;
  int64_t r = t - c * g.n;
  if (s.mid[a] >= 0 && r > s.mid[a]) r = s.mid[a] + g.n - r;
  const int64_t p = g.base(s.rep[a][c]) + r * g.rst;
  s.ta[a][t] = g.a[p];
  s.tb[a][t] = g.b[p];
}

// CTAs of the axes that still count
unsigned share_ctas(LineSearch& s) {
  int64_t n = 0;
  for (int a = 0; a < 3; ++a) {
    s.per[a] = (s.grid[a].rst == 1 ? s.grid[a].n > 16 : s.grid[a].n >= 1024) ? 8 : 32;
    s.first_cta[a] = (int)n;
    n += (s.table[a].n + s.per[a] - 1) / s.per[a];
  }
  return (unsigned)n;
}

size_t up256(size_t n) { return (n + 255) & ~size_t(255); }
// Lays the four tables out in the scratch (null: only counts): all counts and keys, which start at 0, then all owners,
// which start above every number, then the rest.  Returns the bytes; zeros, owners: the bytes of the first two parts.
size_t place(unsigned char* at, LineSearch& s, ClassTable& blocks, size_t& zeros, size_t& owners) {
  ClassTable* t[4] = {&s.table[0], &s.table[1], &s.table[2], &blocks};
  size_t n = 256;
  for (int k = 0; k < 4; ++k) {
    t[k]->count = reinterpret_cast<int*>(at) + 2 * k;
    t[k]->keys = reinterpret_cast<unsigned long long*>(at + n);
    n += sizeof(unsigned long long) * (size_t)t[k]->cap();
  }
  zeros = n = up256(n);
  for (int k = 0; k < 4; ++k) {
    t[k]->owner = reinterpret_cast<int*>(at + n);
    n += sizeof(int) * (size_t)t[k]->cap();
  }
  owners = n - zeros;
  for (int k = 0; k < 4; ++k) {
    t[k]->id = reinterpret_cast<int*>(at + n);
    t[k]->slot = t[k]->id + t[k]->cap();
    n += sizeof(int) * (size_t)(t[k]->cap() + t[k]->n);
    if (k < 3) {
      s.rep[k] = reinterpret_cast<int*>(at + n);
      n += sizeof(int) * (size_t)LineSearch::max_class(t[k]->n);
    }
  }
  return up256(n);
}

}  // namespace

size_t LineSearch::scratch_bytes(const int64_t (&lines)[3], int64_t nblocks) {
  LineSearch s{};
  ClassTable blocks(nblocks);
  for (int a = 0; a < 3; ++a) s.table[a] = ClassTable(lines[a]);
  size_t zeros, owners;
  return place(nullptr, s, blocks, zeros, owners);
}

cudaError_t LineSearch::begin(unsigned char* scratch, ClassTable& blocks, cudaStream_t st) {
  size_t zeros, owners;
  place(scratch, *this, blocks, zeros, owners);
  cudaError_t e = cudaMemsetAsync(scratch, 0, zeros, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(scratch + zeros, 0x7f, owners, st);
  if (e != cudaSuccess) return e;
  const unsigned ctas = share_ctas(*this);
  if (ctas) hash_lines_kernel<<<ctas, kTh, 0, st>>>(*this);
  return cudaGetLastError();
}

cudaError_t LineSearch::number(const ClassTable& blocks, cudaStream_t st) {
  const int64_t n = table[0].n + table[1].n + table[2].n + blocks.n;
  if (n) number_kernel<<<(unsigned)((n + kTh - 1) / kTh), kTh, 0, st>>>(*this, blocks);
  return cudaGetLastError();
}

size_t LineSearch::choose(const int (&classes)[3]) {
  size_t bytes = 0;
  for (int a = 0; a < 3; ++a) {
    nclass[a] = classes[a];
    if (nclass[a] > max_class(table[a].n)) table[a].n = 0;  // the arrays stay
    if (table[a].n) bytes += up256(table_bytes(a));
  }
  return bytes;
}

cudaError_t LineSearch::finish(unsigned char* m, LineTables (&out)[3], cudaStream_t st) {
  int64_t most = 0;
  for (int a = 0; a < 3; ++a) {
    out[a] = LineTables{};
    if (!table[a].n) {
      nclass[a] = 0;
      continue;
    }
    const int64_t entries = nclass[a] * grid[a].n;
    out[a].a = ta[a] = reinterpret_cast<double*>(m);
    out[a].b = tb[a] = ta[a] + entries;
    out[a].cls = cls[a] = reinterpret_cast<int32_t*>(tb[a] + entries);
    out[a].nclass = nclass[a];
    out[a].bytes = table_bytes(a);
    m += up256(out[a].bytes);
    most = std::max(most, entries);
  }
  const unsigned ctas = share_ctas(*this);
  if (!ctas) return cudaSuccess;
  assign_lines_kernel<<<ctas, kTh, 0, st>>>(*this);
  gather_lines_kernel<<<dim3((unsigned)((most + kTh - 1) / kTh), 3), kTh, 0, st>>>(*this);
  return cudaGetLastError();
}

}  // namespace hs2g
