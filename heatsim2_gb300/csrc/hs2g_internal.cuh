// Internal declarations shared by the hs2g translation units (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/hs2g.h"

namespace hs2g {

// Grid dimensions; voxel p = (k*ny + j)*nx + i.
struct Dims {
  int64_t nz, ny, nx;
  __host__ __device__ int64_t nvox() const { return nz * ny * nx; }
  __host__ __device__ int64_t nxy() const { return ny * nx; }
};

constexpr int64_t kSMs = 152;  // of a GB300.  Launch shapes fill them; nothing is wrong where there are more or fewer

// middle column of the two-ended x elimination
__host__ __device__ inline int64_t x_mid(int64_t nx) { return (nx - 1) / 2; }

// Per-voxel coefficients of the scaled delta-form Douglas step.
//   stage 0 (x lines):  right-hand side wc*T + wxl*T[i-1] + wxh*T[i+1] + wyl*T[j-1] + wyh*T[j+1] + wzl*T[k-1]
//                       + wzh*T[k+1] + wq*Q, the line recurrences with a0, b0 to W0          (hs2g_x.cuh)
//   stage 1 (y lines):  the recurrences with a1, b1 from W0 to W1                            (hs2g_pair.cuh)
//   stage 2 (z lines):  the same with a2, b2 from W1 to dT;  T' = T + dT
// In FP64 every line is eliminated from both ends towards a middle row; the FP32 batch goes one way.  The line
// coefficients are stored negated, as the recurrences' multiply-adds take them.
// The stage-0 stencil coefficients come in blocks of 32 columns of an x-line (x-line L = k*ny + j, chunk ch), so that
// a warp reads one contiguous stream; equal blocks are kept once (bidx[L*nchunks + ch], null when there are too many
// distinct ones).  Lines whose coefficients are equal bit for bit share a table (cls0 per x-line, cls1 per y line
// (k, i) at k*nx + i, cls2 per z line (j, i) at j*nx + i); a null class array: values in voxel order with row pitch px.
struct Coeffs {
  double* xb;
  int32_t* bidx;
  int64_t nchunks;
  // Row pitch of the arrays the line solves copy 16 bytes at a time (W0, W1 and the line coefficients): nx, or nx rounded
  // up so that the rows start on 16-byte boundaries (an odd nx gets one pad column).  All other arrays have pitch nx.
  int64_t px;
  double* a0;
  double* b0;
  double* a1;
  double* b1;
  double* a2;
  double* b2;
  int32_t* cls0;
  int32_t* cls1;
  int32_t* cls2;
};

// The distinct lines of an axis: a[c*n + r], b[c*n + r] per class and row, cls[line]; cls is null when there are too
// many.
struct LineTables {
  double* a = nullptr;
  double* b = nullptr;
  int32_t* cls = nullptr;
  int64_t nclass = 0;
  size_t bytes = 0;
};
// Stencil blocks of a problem: the distinct ones with an index per (line, chunk), or all of them (bidx null).
struct XBlocks {
  void* pool = nullptr;
  int32_t* bidx = nullptr;
  int64_t count = 0;
  size_t bytes = 0;
};

// An open-addressing table over n things, by 64-bit hash: keys, the smallest thing of each key, the number it gets,
// each thing's slot, and {count of numbers, 1 once two different things were found under one key}.
struct ClassTable {
  int64_t n = 0;
  unsigned long long* keys = nullptr;
  int *owner = nullptr, *id = nullptr, *slot = nullptr, *count = nullptr;
  __host__ __device__ ClassTable(int64_t things = 0) : n(things) {}
  __host__ __device__ int64_t cap() const {  // at least twice as many entries as things
    int64_t c = 64;
    while (c < 2 * n) c *= 2;
    return c;
  }
  // the slot of hash h (not 0), thing l among its owners.  (Read before each atomic: of many things alike all but the
  // first few find what they would write.)
  __device__ __forceinline__ int insert(unsigned long long h, int l) const {
    const int64_t mask = cap() - 1;
    int64_t e = (int64_t)(h >> 17) & mask;
    for (;; e = (e + 1) & mask) {
      unsigned long long k = *(volatile unsigned long long*)(keys + e);
      if (k == 0ull) k = atomicCAS(keys + e, 0ull, h);
      if (k == 0ull || k == h) break;
    }
    if (*(volatile int*)(owner + e) > l) atomicMin(owner + e, l);
    return (int)e;
  }
  // the slots of the things of a warp's lanes (mask: lanes 0 .. some; things ascending, h 0: none), those alike as one
  __device__ __forceinline__ void insert_all(unsigned mask, unsigned long long h, int l) const {
    const int lane = threadIdx.x & 31, leader = __ffs(__match_any_sync(mask, h)) - 1;
    int e = 0;
    if (lane == leader && h) e = insert(h, l);
    e = __shfl_sync(mask, e, leader);
    if (h) slot[l] = e;
  }
};

// lines (o, i), i fastest, with row r at o*ost + r*rst + i of a and b
struct LineGrid {
  const double* a;
  const double* b;
  int64_t outer, nx, ost, n, rst;
  __host__ __device__ int64_t lines() const { return outer * nx; }
  __device__ int64_t base(int64_t l) const {  // (the search numbers lines in 32 bits)
    const unsigned o = (unsigned)l / (unsigned)nx;
    return o * ost + ((unsigned)l - o * (unsigned)nx);
  }
};
// Finding the line classes of the three axes (hs2g_classes.cu); grid, table[a].n (0: no search on that axis) and mid are
// the caller's.  begin queues the hashing (and clears the blocks' table beside the lines'), number the numbering of both;
// the caller reads the counts (2 ints per table from table[0].count on) and waits; choose takes the axes worth tables and
// returns the bytes of these, finish queues them and the check that sets count[1] on a clash of hashes.  mid >= 0: the rows
// above mid are tabulated last first (row r at position mid + n - r).
struct LineSearch {
  LineGrid grid[3];
  int64_t mid[3];
  ClassTable table[3];
  int* rep[3];  // a line of each class
  int per[3], first_cta[3];
  int64_t nclass[3];
  int32_t* cls[3];
  double *ta[3], *tb[3];
  // Worth it when the tables are an eighth of the arrays: they stay in cache, and where neighbouring lines are of one class,
  // as in a layered specimen, a warp reads one row for its sixteen.  At the worst, all neighbours different, us per sweep
  // from tables of 1/64, 1/16 and 1/8 of the lines, in brackets from the arrays: 64x256x512 x 186, 212, 212 [190], y 38
  // [67], z 83 [63]; 37x192x210 x 42, 44, 45 [52], y 20 [19], z 22 [23].
  __host__ __device__ static int64_t max_class(int64_t lines) { return lines / 8 > 1 ? lines / 8 : 1; }
  static size_t scratch_bytes(const int64_t (&lines)[3], int64_t nblocks);
  cudaError_t begin(unsigned char* scratch, ClassTable& blocks, cudaStream_t s);
  cudaError_t number(const ClassTable& blocks, cudaStream_t s);
  size_t table_bytes(int a) const {
    return 2 * sizeof(double) * (size_t)(nclass[a] * grid[a].n) + sizeof(int32_t) * (size_t)table[a].n;
  }
  size_t choose(const int (&classes)[3]);
  cudaError_t finish(unsigned char* m, LineTables (&out)[3], cudaStream_t s);
};

struct QTable {
  double q[HS2G_MAX_CLASSES];
};

// Device-resident source schedule of a handle, read by the x sweep of a step with a source.  The host writes
// every field: the rows, their flags and the shape field when the schedule or the shapes change, `step` (the
// row of the next step with a source) before such a step is queued, `row` (the history row of the next step)
// at the start of a run; the history kernel then advances `row` after each step.
struct DevSchedule {
  const double* q;         // [n][HS2G_MAX_CLASSES] class source values (W/m^3)
  const uint8_t* active;   // [n] 1 when row s has a non-zero value
  const double* shape;     // per-voxel multiplier of the class sources, or null when no class has a shape
  int64_t n;               // rows; steps at or beyond n have no source
  int64_t step;
  int64_t row;
  unsigned int hist_done;  // CTAs of the current history kernel that have finished (the last one advances row)
};

// Stores with an L2 evict-last policy, for a value the same warp reads back soon (a line's forward values).
__device__ __forceinline__ uint64_t l2_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void st_hint(double* p, double v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_hint(float* p, float v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(policy) : "memory");
}

// Programmatic dependent launch inside the captured step graphs: a sweep launched with the attribute may be set
// up on the SMs while the sweep before it on the stream completes (no kernel triggers early, so that happens
// only once every CTA of the previous sweep has exited, and the CTAs of the new one spread over the whole GPU as
// in an ordinary launch).  Each sweep waits here, before it touches memory the previous one reads or writes,
// until that sweep has completed and its writes are visible.  A no-op in a kernel launched without the
// attribute.
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Kernel launch with the programmatic-serialization attribute when pdl is set (an ordinary launch otherwise).
template <typename... P, typename... A>
cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl,
                          A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
}

// Record the message hs2g_last_error() returns for this thread (hs2g_api.cu); returns code.
int set_last_error(int code, const char* message);

// First error recorded by a device kernel: (code << 56) | (axis << 54) | index, 0 when none.
__device__ __forceinline__ void record_error(unsigned long long* err, int code, int axis, int64_t index) {
  unsigned long long v = ((unsigned long long)(-code) << 56) | ((unsigned long long)axis << 54) |
                         ((unsigned long long)index & ((1ull << 54) - 1));
  atomicCAS(err, 0ull, v);
}

// setup kernels (hs2g_compile.cu)
// the face conductances of the three axes (z, y, x), from the boundary classes of their faces
cudaError_t launch_faces(const Dims& d, const uint8_t* material, const uint8_t* const bclass[3], const hs2g_material* mats,
                         int nmat, const hs2g_face_form* forms, int nbnd, double* const G[3], unsigned long long* err,
                         void* table, cudaStream_t s);
size_t face_table_bytes(int nmat, int nbnd);  // of launch_faces's table; 0: it takes none
cudaError_t launch_capacity_from_classes(const Dims& d, const uint8_t* material, const hs2g_material* mats,
                                         int nmat, double* M, uint8_t* compute, unsigned long long* err,
                                         cudaStream_t s);
cudaError_t launch_validate_dense(const Dims& d, const double* Gz, const double* Gy, const double* Gx,
                                  double* M, uint8_t* compute, unsigned long long* err, cudaStream_t s);
// The face conductances a problem is factorised from: one array per axis indexed by face, or (rows[0] set) per-row
// conductances {z lo, z hi, y lo, y hi, x lo, x hi}, each (nz, ny, nx).
struct Faces {
  const double *Gz = nullptr, *Gy = nullptr, *Gx = nullptr;
  const double* rows[6] = {};
};
// The line factors into c (row pitch c.px), in FP64 from both ends; s2 and sigma are scratch, s2 holds the stage-0 row
// scale f0 afterwards.
cudaError_t launch_factor(const Dims& d, const Faces& f, const double* M, const uint8_t* compute, double* s2,
                          double* sigma, const Coeffs& c, cudaStream_t s, bool two_ended);
// What the step keeps of the factors (hs2g_compile.cu): the stencil blocks, and the x, y and z line tables where the
// lines have few classes (lines[a].cls null: c's arrays stay).  scratch: compress_scratch(d) bytes, or null: no search,
// everything in voxel order.  Waits for the stream.
struct Compressed {
  XBlocks blocks;
  LineTables lines[3];
  void *mem = nullptr, *own = nullptr;  // device memory of the tables and the distinct blocks, and of all blocks
  void release();
};
size_t compress_scratch(const Dims& d);
cudaError_t compress_coeffs(const Dims& d, const Faces& f, const uint8_t* compute, const double* f0, const Coeffs& c,
                            int precision, unsigned char* scratch, Compressed* out, cudaStream_t s);
cudaError_t launch_validate_rows(const Dims& d, const double* const rows[6], double* M, uint8_t* compute,
                                 unsigned long long* err, cudaStream_t s);

// per-voxel source shapes (hs2g_sources.cu)
cudaError_t launch_fill(double* p, int64_t n, double v, cudaStream_t s);
cudaError_t launch_zdecay_shape(int64_t n, const uint8_t* vclass, int cls, const double* zgrid, double direction,
                                double offset, double ddz, double jpm2, double length, double dt, double* shape,
                                cudaStream_t s);
int64_t point_shape_tiles(int64_t n);
cudaError_t launch_point_shape(int64_t n, const uint8_t* vclass, int cls, int64_t* tile_scratch, const double* joules,
                               int64_t count, const double* volumes, double volume, double dt, double* shape,
                               cudaStream_t s);

// step kernels (hs2g_sweep.cu)
struct StepArgs {
  Dims d;
  const double* T_in;
  double* T_out;
  double* W0;
  double* W1;
  const uint8_t* vclass;
  const double* qdense;  // may be null
  const double* qshape;  // per-voxel multiplier of the class sources (null: 1 everywhere)
  bool has_qtab;
  bool pdl;              // launch the y and z sweeps with programmatic dependent launch (captured step graphs)
  bool pdl_x;            // the same for the x sweep (not for the first kernel of a graph)
};

// raise the dynamic shared-memory limits of the sweep kernels that a problem launches, on the current device (when a
// handle is created)
cudaError_t sweeps_prepare(const Dims& d, const Coeffs& c);
cudaError_t launch_step(const StepArgs& a, const Coeffs& c, const QTable& q, cudaStream_t s);
// the same three kernels with an event recorded before each and after the last (ev[0..3])
cudaError_t launch_step_events(const StepArgs& a, const Coeffs& c, const QTable& q, cudaStream_t s,
                               cudaEvent_t ev[4]);
// One step whose class sources are row ds->step of the device schedule (no source when that row is inactive or
// past the schedule's end): the x sweep reads the row on the device.  Used for the steps with a source in the
// captured step graphs of hs2g_run; the steps without one use launch_step with no table.
cudaError_t launch_step_row(const StepArgs& a, const Coeffs& c, const DevSchedule* ds, cudaStream_t s);
// History of the step just taken into hist[ds->row][ny][nx]: layer `layer` of T (dz2 <= 0) or the insulating
// z = 0 surface estimate from layers 0 and 1 with dz2 = dz**2 (dz2 > 0); the kernel's last CTA advances
// ds->row.
cudaError_t launch_history_row(const Dims& d, const double* T, int layer, double dz2, double* hist, DevSchedule* ds,
                               cudaStream_t s, bool pdl = false);
// the reference's dz**2.0 (the C library's pow)
double surface_dz2(double dz);
// one flag per schedule row: active[s] = any of q[s][0..nclass-1] non-zero
cudaError_t launch_schedule_flags(const double* q, int64_t nrows, uint8_t* active, cudaStream_t s);
cudaError_t fp64_fma_rate(double* fma_per_s);
cudaError_t launch_copy_layer(const Dims& d, const double* T, int layer, double* dst, cudaStream_t s);
// insulating z = 0 surface temperature from layers 0 and 1 of T (an nxy-element plane each) into dst[nxy]
cudaError_t launch_surface_estimate(int64_t nxy, const double* T, double dz, double* dst, cudaStream_t s);
// one bounded mbarrier wait on a barrier that receives its arrival (arrive != 0) or none (hs2g_lines.cu)
cudaError_t wait_selftest(uint64_t limit_ns, int arrive, int* status_dev, cudaStream_t s);
// the step in pieces, for overlapping host copies with it: the x sweep over x-lines [line_begin, line_end)
// (line = k*ny + j), the whole y sweep, the z sweep over the rows of columns
// [j_begin, j_end)
cudaError_t launch_x_range(const StepArgs& a, const Coeffs& c, const QTable& q, int64_t line_begin,
                           int64_t line_end, cudaStream_t s);
cudaError_t launch_y(const StepArgs& a, const Coeffs& c, cudaStream_t s);
cudaError_t launch_z_rows(const StepArgs& a, const Coeffs& c, int64_t j_begin, int64_t j_end, cudaStream_t s);

}  // namespace hs2g
