// Fused collide-and-stream for sm_100a on the in-place AA pattern.
//
// Memory layout in HBM: one column per population i, `stride` elements long
// (the cell count rounded up to 64 elements, so every column starts on a 256 B
// boundary), cell = (x*ny + y)*nz + z with z fastest — OpenLB's order
// (src/core/blockStructure.h:65-75) without the overlap layers.  Periodic and
// non-periodic faces alike wrap per axis; at non-periodic faces the wrapped
// values only ever reach wall cells, exactly as OpenLB's unspecified padding
// values only reach its wall cells.
//
// AA pattern (one array, in place):
//   even step t: cell x reads f_i from column i at x, collides, writes f*_i to
//                column opp(i) at x.
//   odd step   : cell x reads f_i from column opp(i) at x - c_i, collides,
//                writes f*_i to column i at x + c_i.
// After an odd step the array holds the post-stream state in natural order
// (f_i(x) in column i at x); after an even step f_i(x) sits in column opp(i)
// at x - c_i.  Every cell reads and writes exactly the same q slots, so no two
// cells touch the same slot.  This is equivalent to OpenLB's collide followed
// by the periodic-shift stream (src/core/blockLattice.hh:317-339,
// src/core/platform/cpu/sisd/column.h:193-204).
//
// Full-way bounce-back (collision::Revert) writes f*_i = f_opp(i) to exactly
// the slot f_opp(i) was read from, so wall cells need no memory access at
// all; moving walls add their Nguyen-Ladd term in place.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "lbm_device.cuh"

namespace olb_b200 {

struct Geometry {
  int32_t nx, ny, nz;
  uint32_t stride;  // column length in storage elements
  int32_t paired;   // 1: 16-bit storage with cells x and x + nx/2 in one 4-byte element
  // masked lattices: a box [lo, hi) whose cells all use the bulk entry, so the
  // step kernel skips their dynamics id (empty when lo == hi)
  int32_t bulk_lo[3], bulk_hi[3];
  // FORCE per cell for the Guo-forced dynamics (3 columns of `stride` values
  // of the compute type, natural cell order), or nullptr: the entries' forces
  const void* force;
  // masked lattices: 1 when every entry of the bulk entry's collision kind has
  // the bulk entry's constants, so the step kernel takes them from the kernel
  // argument instead of loading them from the cell's table entry
  int32_t uniform;
  // flat tiles of the step kernels (tile_cells): 0 or the threads of a block,
  // with floor(n / nz) = (mulhi(n, flat_mul) + n) >> flat_shift
  int32_t flat;
  uint32_t flat_mul, flat_shift;
};

// the entry index the masked kernels give a cell of the bulk box (the table
// holds at most 256 entries): it collides with the bulk entry, the kernel
// argument, and loads nothing from the table
constexpr int kBoxCell = 256;

OLB_HD bool in_bulk_box(const Geometry& g, int x, int y, int z)
{
  return x >= g.bulk_lo[0] && x < g.bulk_hi[0] && y >= g.bulk_lo[1] && y < g.bulk_hi[1] && z >= g.bulk_lo[2] &&
         z < g.bulk_hi[2];
}

// Scalar slot of a cell within a population column.
//   natural layout: (x*ny + y)*nz + z
//   paired layout (16-bit storage, nx even): element ((x mod nx/2)*ny + y)*nz + z
//   holds cell x in its low half and cell x + nx/2 in its high half, so the
//   slot is 2*element + (x >= nx/2).  Shifts along y and z keep elements
//   aligned; only the x seam swaps the halves.
OLB_HD uint32_t cell_slot(const Geometry& g, int x, int y, int z)
{
  if (!g.paired) {
    return (uint32_t(x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  }
  const int nxh = g.nx >> 1;
  const int hi = x >= nxh;
  const uint32_t e = (uint32_t(hi ? x - nxh : x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  return 2u * e + uint32_t(hi);
}

OLB_HD int wrap(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// A copy of v the compiler cannot see through: store addresses computed from
// it are recomputed after the collision (one multiply-add each) instead of
// being kept live in registers from the load phase.
OLB_DEV uint32_t opaque(uint32_t v)
{
  uint32_t r;
  asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// per-block partial of the fused statistics reduction (FP64)
struct StatPartial {
  double sum_rho;
  double sum_usqr;
  double max_usqr;
  unsigned long long n_cells;
  unsigned long long n_nonfinite;
};

// Scratch of a reduction over several blocks, zero before the first use;
// `arrived` is zero again after each.
constexpr int kReduceBlocks = 64;
struct StatStage {
  StatPartial part[kReduceBlocks];
  unsigned arrived;
};

// a reduced statistic and the number of the reduction that wrote it (written
// last: a host that reads it from pinned memory waits for its number)
struct StatResult {
  StatPartial p;
  unsigned long long seq;
};

// Where the blocks of a kernel leave their partials.  With a stage the last
// block to finish also reduces them into `result`; without, a
// reduce_partials_kernel does.
struct StatSink {
  StatPartial* partials = nullptr;
  StatStage* stage = nullptr;
  StatResult* result = nullptr;
  unsigned long long seq = 0;
};

// ---------------------------------------------------------------------------
// launches chained on a stream (programmatic dependent launch)
//
// A step of a small lattice takes about as long as a launch: a kernel that lets
// its successor start (next_may_start, first thing) and waits for its
// predecessor's results only when it needs them (after_previous) hides the
// launch and the drain of the last blocks.  Every block of a kernel passes
// after_previous before it ends, so a finished kernel implies finished
// predecessors.  The pointer goes through the wait: no load from it can move
// ahead of it.  In a launch without the attribute both do nothing.
OLB_DEV void next_may_start() { asm volatile("griddepcontrol.launch_dependents;"); }

template <class T>
OLB_DEV T* after_previous(T* p)
{
  asm volatile("griddepcontrol.wait;" : "+l"(p) : : "memory");
  return p;
}

// ---------------------------------------------------------------------------
// storage element conversions (plain loads: the array is read and written in
// place by the same kernel, so the read-only data path is not used)

template <class S, class R> struct Store;

template <class R> struct Store<float, R> {
  template <class L, int I> OLB_DEV static R load(const float* p) { return R(*p); }
  template <class L, int I> OLB_DEV static void store(float* p, R v) { *p = float(v); }
};
template <class R> struct Store<double, R> {
  template <class L, int I> OLB_DEV static R load(const double* p) { return R(*p); }
  template <class L, int I> OLB_DEV static void store(double* p, R v) { *p = double(v); }
};
template <class R> struct Store<__half, R> {
  template <class L, int I> OLB_DEV static R load(const __half* p)
  {
    constexpr float inv = 1.f / storage_scale<L>(I);
    return R(__half2float(*p) * inv);
  }
  template <class L, int I> OLB_DEV static void store(__half* p, R v)
  {
    constexpr float s = storage_scale<L>(I);
    *p = __float2half_rn(float(v) * s);
  }
};
template <class R> struct Store<__nv_bfloat16, R> {
  template <class L, int I> OLB_DEV static R load(const __nv_bfloat16* p)
  {
    constexpr float inv = 1.f / storage_scale<L>(I);
    return R(__bfloat162float(*p) * inv);
  }
  template <class L, int I> OLB_DEV static void store(__nv_bfloat16* p, R v)
  {
    constexpr float s = storage_scale<L>(I);
    *p = __float2bfloat16_rn(float(v) * s);
  }
};

// ---------------------------------------------------------------------------
// neighbour offsets with per-axis wrap-around

struct Neighbours {
  uint32_t xo[3], yo[3], zo[3];
  OLB_DEV Neighbours(const Geometry& g, int x, int y, int z)
  {
    const uint32_t sxy = uint32_t(g.ny) * uint32_t(g.nz);
    xo[0] = uint32_t(x == 0 ? g.nx - 1 : x - 1) * sxy;
    xo[1] = uint32_t(x) * sxy;
    xo[2] = uint32_t(x == g.nx - 1 ? 0 : x + 1) * sxy;
    yo[0] = uint32_t(y == 0 ? g.ny - 1 : y - 1) * uint32_t(g.nz);
    yo[1] = uint32_t(y) * uint32_t(g.nz);
    yo[2] = uint32_t(y == g.ny - 1 ? 0 : y + 1) * uint32_t(g.nz);
    zo[0] = uint32_t(z == 0 ? g.nz - 1 : z - 1);
    zo[1] = uint32_t(z);
    zo[2] = uint32_t(z == g.nz - 1 ? 0 : z + 1);
  }
  template <int DX, int DY, int DZ>
  OLB_DEV uint32_t at() const { return xo[DX + 1] + yo[DY + 1] + zo[DZ + 1]; }
};

// ---------------------------------------------------------------------------
// block-level FP64 statistics reduction

OLB_DEV void warp_reduce(double& a, double& b, double& m, unsigned long long& n, unsigned long long& nf)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    n += __shfl_down_sync(0xffffffffu, n, o);
    nf += __shfl_down_sync(0xffffffffu, nf, o);
  }
}

// sum over the block's threads (256 or a multiple of 32), valid in thread 0
OLB_DEV StatPartial block_sum(StatPartial v)
{
  __shared__ StatPartial warp_part[32];
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nthreads = blockDim.x * blockDim.y;
  warp_reduce(v.sum_rho, v.sum_usqr, v.max_usqr, v.n_cells, v.n_nonfinite);
  const int lane = tid & 31, warp = tid >> 5;
  if (lane == 0) {
    warp_part[warp] = v;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = (nthreads + 31) >> 5;
    v = lane < nw ? warp_part[lane] : StatPartial{0, 0, 0, 0, 0};
    warp_reduce(v.sum_rho, v.sum_usqr, v.max_usqr, v.n_cells, v.n_nonfinite);
  }
  return v;
}

// the block's share of parts[begin, end): a fixed assignment to threads and a
// fixed tree (deterministic for a given block size); valid in thread 0
OLB_DEV StatPartial sum_partials(const StatPartial* parts, size_t begin, size_t end)
{
  StatPartial v{0, 0, 0, 0, 0};
  for (size_t k = begin + threadIdx.x + blockDim.x * threadIdx.y; k < end; k += blockDim.x * blockDim.y) {
    // from L2: other blocks wrote them
    v.sum_rho += __ldcg(&parts[k].sum_rho);
    v.sum_usqr += __ldcg(&parts[k].sum_usqr);
    v.max_usqr = fmax(v.max_usqr, __ldcg(&parts[k].max_usqr));
    v.n_cells += __ldcg(&parts[k].n_cells);
    v.n_nonfinite += __ldcg(&parts[k].n_nonfinite);
  }
  return block_sum(v);
}

OLB_DEV void write_result(StatResult* out, const StatPartial& p, unsigned long long seq)
{
  out->p = p;
  __threadfence_system();
  *reinterpret_cast<volatile unsigned long long*>(&out->seq) = seq;
}

// true in every thread of the block that arrives last of `blocks`; what the
// others wrote before arriving is visible to it
OLB_DEV bool last_to_arrive(unsigned* arrived, unsigned blocks)
{
  __shared__ bool last;
  if (threadIdx.x + threadIdx.y == 0) {
    __threadfence();
    last = atomicAdd(arrived, 1u) == blocks - 1;
    if (last) *arrived = 0;
    __threadfence();
  }
  __syncthreads();
  return last;
}

OLB_DEV void block_stats(double a, double b, double m, unsigned long long n, unsigned long long nf,
                         const StatSink& sink)
{
  const StatPartial v = block_sum(StatPartial{a, b, m, n, nf});
  const unsigned blocks = gridDim.x * gridDim.y * gridDim.z;
  if (threadIdx.x + threadIdx.y == 0) {
    sink.partials[blockIdx.x + size_t(gridDim.x) * (blockIdx.y + size_t(gridDim.y) * blockIdx.z)] = v;
  }
  if (sink.stage && last_to_arrive(&sink.stage->arrived, blocks)) {
    const StatPartial sum = sum_partials(sink.partials, 0, blocks);
    if (threadIdx.x + threadIdx.y == 0) write_result(sink.result, sum, sink.seq);
  }
}

// ---------------------------------------------------------------------------
// the step kernel

// Step-kernel variants: cells per thread (along y, blockDim.y rows apart) and
// the register cap (__launch_bounds__(kStepThreads, min_blocks)).  All loads of
// a thread's cells are issued before any of them is collided, so more cells
// per thread — or more resident warps — means more bytes in flight per SM, the
// quantity that bounds this HBM-streaming kernel.  Which variant is fastest
// depends on the lattice, the storage type and the mask; the library picks a
// default per lattice and can time all of them (olb_b200_autotune).  Every
// variant performs the same arithmetic on every cell, so results are
// independent of the choice.
constexpr int kStepThreads = 256;
struct StepVariant {
  int cells_per_thread;
  int min_blocks;
};
#ifdef OLB_B200_SINGLE_VARIANT
// builds that only check arithmetic compile one variant; every id maps to it
constexpr StepVariant kStepVariants[] = {{1, 3}, {1, 3}, {1, 3}, {1, 3}};
#elif defined(OLB_B200_EXACT)
// the reference-order build serves parity, not speed: both work distributions
// (one and two cells per thread), one register cap each
constexpr StepVariant kStepVariants[] = {{1, 3}, {1, 3}, {2, 3}, {2, 3}};
#else
constexpr StepVariant kStepVariants[] = {{1, 3}, {1, 4}, {2, 2}, {2, 3}};
#endif
constexpr int kNumStepVariants = 4;

// 16-bit storage in the natural layout (one cell per element) has two kernels:
// one cell per thread (variants 0 and 2), and two as the lanes of the packed
// collision (variants 1 and 3, aa_step_split_kernel).  The reference-order build
// collides one cell at a time.
#ifdef OLB_B200_EXACT
constexpr bool kSplitNatural16 = false;
#else
constexpr bool kSplitNatural16 = true;
#endif
constexpr int kSplitMinBlocks = 3;

// Variant v for a storage element of `bytes`.  16-bit storage compiles the
// one-cell-per-thread variants only (its kernels hold two cells per thread
// already; at 256^3 two elements per thread reached 0.87 of the copy bandwidth
// against 0.94 with one in D3Q19, 0.87 against 0.93 in D3Q27), so the ids of
// the others give the one-cell variant of the same rank.
constexpr StepVariant step_variant(int bytes, int v)
{
  return kStepVariants[bytes == 2 ? v & 1 : v];
}

// whether a natural 16-bit lattice runs aa_step_split_kernel in variant v
constexpr bool split_variant(int v) { return kSplitNatural16 && (v & 1) != 0; }

// running sums of the fused statistics of one thread
struct StatAcc {
  double rho = 0., usqr = 0., max = 0.;
  unsigned long long n = 0, nf = 0;
  OLB_DEV void add(double r, double u2)
  {
    if (isfinite(r) && isfinite(u2)) {
      rho += r; usqr += u2; max = fmax(max, u2); n += 1;
    } else {
      nf += 1;
    }
  }
};

// The (y, z) of this thread's CPT cells.  Two ways to cut a plane x into blocks:
//   rectangles  blockDim.x cells along z by blockDim.y * CPT rows (the launch
//               shape); lanes beyond nz and rows beyond ny idle;
//   flat        CPT runs of g.flat (the block size) consecutive cells of the plane's
//               index y*nz + z, so every lane but the plane's last few has a
//               cell, whatever nz and ny; y costs one multiply-high
//               (Granlund & Montgomery, PLDI 1994).
// Lanes without a cell get y = ny.
OLB_DEV void flat_cell(const Geometry& g, uint32_t n, int& y, int& z)
{
  const uint32_t yy = (__umulhi(n, g.flat_mul) + n) >> g.flat_shift;
  z = int(n - yy * uint32_t(g.nz));
  y = n < uint32_t(g.ny) * uint32_t(g.nz) ? int(yy) : g.ny;
}

template <int CPT>
OLB_DEV void tile_cells(const Geometry& g, int (&y)[CPT], int (&z)[CPT])
{
  if (g.flat) {
    static_for<0, CPT>([&](auto k) {
      const uint32_t n = (blockIdx.x * uint32_t(CPT) + uint32_t(k.value)) * uint32_t(g.flat) + threadIdx.x;
      flat_cell(g, n, y[k], z[k]);
    });
  } else {
    const int zz = blockIdx.x * blockDim.x + threadIdx.x;
    static_for<0, CPT>([&](auto k) {
      z[k] = zz;
      y[k] = zz < g.nz ? int(blockIdx.y * (blockDim.y * CPT) + threadIdx.y + k.value * blockDim.y) : g.ny;
      y[k] = min(y[k], g.ny);
    });
  }
}

// One tile of the step: the CPT cells (x, y[k], z[k]) of this thread (none
// where y[k] = ny).  Masked lattices pass each cell's table entry in id[k]
// (loaded ahead by aa_step_masked_kernel); unmasked lattices use `bulk` for
// every cell.
template <int Q, class S, class R, int KIND, bool ODD, bool MASKED, bool STATS, int CPT>
OLB_DEV void step_tile(S* __restrict__ pops, const Geometry& g, const DynDevice<R>* __restrict__ table,
                       const DynDevice<R>& bulk, int x, const int (&y)[CPT], const int (&z)[CPT],
                       const int (&id)[CPT], StatAcc& acc)
{
  using L = Lattice<Q>;
  using ST = Store<S, R>;
  constexpr bool kForced = KIND == K_FORCED_BGK || KIND == K_FORCED_TRT;
  R f[CPT][Q];
  R fc[CPT][3];  // the cell's FORCE when the lattice has a force field
  int kind[CPT];
  bool go[CPT];
  uint32_t n[CPT];

  // phase 1: issue all loads.  Masked lattices load every cell's populations
  // before its dynamics id has arrived (the id and the populations travel
  // together instead of one after the other); a full-way bounce-back cell
  // then stores nothing, its AA update being a no-op (see file comment).
  static_for<0, CPT>([&](auto k) {
    go[k] = y[k] < g.ny;
    kind[k] = KIND;
    n[k] = 0;
    if (go[k]) {
      n[k] = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y[k])) * uint32_t(g.nz) + uint32_t(z[k]);
      Neighbours nb(g, x, y[k], z[k]);
      static_for<0, Q>([&](auto i) {
        if constexpr (!ODD) {
          f[k][i] = ST::template load<L, i.value>(pops + size_t(i.value) * g.stride + n[k]);
        } else {
          constexpr int o = L::opp(i);
          const uint32_t src = nb.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>();
          f[k][i] = ST::template load<L, o>(pops + size_t(o) * g.stride + src);
        }
      });
      if constexpr (kForced) {
        fc[k][0] = fc[k][1] = fc[k][2] = R(0);
        if (g.force) {
          const R* __restrict__ F = static_cast<const R*>(g.force);
          fc[k][0] = __ldg(F + n[k]);
          fc[k][1] = __ldg(F + size_t(g.stride) + n[k]);
          fc[k][2] = __ldg(F + 2 * size_t(g.stride) + n[k]);
        }
      }
    }
  });
  if constexpr (MASKED) {
    static_for<0, CPT>([&](auto k) {
      if (go[k] && id[k] != kBoxCell) kind[k] = __ldg(&table[id[k]].kind);
      go[k] = go[k] && kind[k] != K_BOUNCE_BACK;
    });
  }

  // phase 2: collide and store
  static_for<0, CPT>([&](auto k) {
    if (!go[k]) return;
    R st_rho = R(0), st_usqr = R(0);
    bool counted = false;
    if (kind[k] == KIND) {
      if constexpr (MASKED) {
        // the entry's collision constants (the bulk entry's for box cells)
        DynDevice<R> q;
        if (id[k] == kBoxCell || g.uniform) {
          q.omega = bulk.omega;
          q.omega_minus = bulk.omega_minus;
          q.smago_pre = bulk.smago_pre;
          q.tau_mol = bulk.tau_mol;
          q.force[0] = bulk.force[0];
          q.force[1] = bulk.force[1];
          q.force[2] = bulk.force[2];
          q.force_relax = bulk.force_relax;
        } else {
          const DynDevice<R>* e = table + id[k];
          q.omega = __ldg(&e->omega);
          q.omega_minus = __ldg(&e->omega_minus);
          q.smago_pre = __ldg(&e->smago_pre);
          q.tau_mol = __ldg(&e->tau_mol);
          q.force[0] = __ldg(&e->force[0]);
          q.force[1] = __ldg(&e->force[1]);
          q.force[2] = __ldg(&e->force[2]);
          q.force_relax = __ldg(&e->force_relax);
        }
        if constexpr (kForced) {
          if (g.force) {
            q.force[0] = fc[k][0]; q.force[1] = fc[k][1]; q.force[2] = fc[k][2];
          }
        }
        collide_bulk<L, KIND>(f[k], q, st_rho, st_usqr);
      } else if constexpr (kForced) {
        DynDevice<R> q;
        q.omega = bulk.omega;
        q.omega_minus = bulk.omega_minus;
        q.force_relax = bulk.force_relax;
        q.force[0] = g.force ? fc[k][0] : bulk.force[0];
        q.force[1] = g.force ? fc[k][1] : bulk.force[1];
        q.force[2] = g.force ? fc[k][2] : bulk.force[2];
        collide_bulk<L, KIND>(f[k], q, st_rho, st_usqr);
      } else {
        collide_bulk<L, KIND>(f[k], bulk, st_rho, st_usqr);
      }
      counted = true;
    } else if (MASKED && kind[k] == K_BOUNCE_BACK_VELOCITY) {
      const DynDevice<R>* e = table + id[k];
      revert<L>(f[k]);
      static_for<1, Q>([&](auto i) {
        f[k][i] += __ldg(&e->wall_term[i][0]);
        f[k][i] += __ldg(&e->wall_term[i][1]);
        f[k][i] += __ldg(&e->wall_term[i][2]);
      });
      st_rho = __ldg(&e->wall_rho);
      const R wu[3] = {__ldg(&e->wall_u[0]), __ldg(&e->wall_u[1]), __ldg(&e->wall_u[2])};
      st_usqr = norm_sqr(wu);
      counted = true;
    }
    // NoDynamics and the boundary cells that carry values (their collision
    // ran in place before this kernel, boundary_collide_kernel): populations
    // pass through unchanged.
    // The store offsets are recomputed here rather than kept live through
    // the collision.
    Neighbours nb(g, int(opaque(uint32_t(x))), int(opaque(uint32_t(y[k]))), int(opaque(uint32_t(z[k]))));
    const uint32_t stride = opaque(g.stride);
    const uint32_t nk = opaque(n[k]);
    static_for<0, Q>([&](auto i) {
      if constexpr (!ODD) {
        constexpr int o = L::opp(i);
        ST::template store<L, o>(pops + size_t(o) * stride + nk, f[k][i]);
      } else {
        const uint32_t dst = nb.template at<L::c(i, 0), L::c(i, 1), L::c(i, 2)>();
        ST::template store<L, i.value>(pops + size_t(i.value) * stride + dst, f[k][i]);
      }
    });
    if constexpr (STATS) {
      if (counted) acc.add(double(st_rho), double(st_usqr));
    }
  });
}

// Unmasked lattices (every cell uses `bulk`): one tile per block, grid
// step_grid().
template <int Q, class S, class R, int KIND, bool ODD, bool STATS, int CPT, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
aa_step_kernel(S* __restrict__ pops, const Geometry g, const DynDevice<R> bulk, const StatSink sink)
{
  next_may_start();
  int y[CPT], z[CPT];
  tile_cells(g, y, z);
  const int none[CPT] = {};
  StatAcc acc;
  pops = after_previous(pops);
  step_tile<Q, S, R, KIND, ODD, false, STATS, CPT>(pops, g, nullptr, bulk, int(blockIdx.z), y, z, none, acc);
  if constexpr (STATS) {
    block_stats(acc.rho, acc.usqr, acc.max, acc.n, acc.nf, sink);
  }
}

// table entries of a tile's cells: kBoxCell for cells of the bulk box (they
// use the bulk entry, no load), -1 for cells outside the lattice (skipped)
template <int CPT>
OLB_DEV void load_tile_ids(int (&id)[CPT], const Geometry& g, const uint8_t* __restrict__ ids, int x,
                           const int (&y)[CPT], const int (&z)[CPT])
{
  static_for<0, CPT>([&](auto k) {
    id[k] = -1;
    if (y[k] < g.ny) {
      id[k] = in_bulk_box(g, x, y[k], z[k])
                ? kBoxCell
                : int(ids[(uint32_t(x) * uint32_t(g.ny) + uint32_t(y[k])) * uint32_t(g.nz) + uint32_t(z[k])]);
    }
  });
}

// Masked lattices: one tile per block, grid step_grid().  The ids of the
// thread's cells are loaded first (none for cells of the bulk box); the
// populations follow without waiting for them (step_tile).
template <int Q, class S, class R, int KIND, bool ODD, bool STATS, int CPT, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
aa_step_masked_kernel(S* __restrict__ pops, const Geometry g, const uint8_t* __restrict__ ids,
                      const DynDevice<R>* __restrict__ table, const DynDevice<R> bulk,
                      const StatSink sink)
{
  next_may_start();
  const int x = blockIdx.z;
  int y[CPT], z[CPT], id[CPT];
  tile_cells(g, y, z);
  load_tile_ids(id, g, ids, x, y, z);
  StatAcc acc;
  pops = after_previous(pops);
  step_tile<Q, S, R, KIND, ODD, true, STATS, CPT>(pops, g, table, bulk, x, y, z, id, acc);
  if constexpr (STATS) {
    block_stats(acc.rho, acc.usqr, acc.max, acc.n, acc.nf, sink);
  }
}

// ---------------------------------------------------------------------------
// the step kernel on the paired 16-bit layout
//
// Each thread updates the two cells of one 4-byte element, (x', y, z) and
// (x' + nx/2, y, z), with one aligned 32-bit load and one aligned 32-bit store
// per population — a warp moves 128 B per instruction instead of 64 B.  The
// grid's z dimension walks x' in [0, nx/2); a neighbour across the x seam is
// the element on the other side with its halves swapped, a condition that is
// uniform per block.  Cells of a pair may have different dynamics; full-way
// bounce-back cells then apply their swap in registers (it writes back what
// it read, so the result is the same as skipping them).

template <class S> struct Pair;
template <> struct Pair<__half> {
  using T = __half2;
  OLB_DEV static float2 to_float2(T v) { return __half22float2(v); }
  OLB_DEV static T from_floats(float lo, float hi) { return __floats2half2_rn(lo, hi); }
  OLB_DEV static T from_float2(float2 v) { return __float22half2_rn(v); }
};
template <> struct Pair<__nv_bfloat16> {
  using T = __nv_bfloat162;
  OLB_DEV static float2 to_float2(T v) { return __bfloat1622float2(v); }
  OLB_DEV static T from_floats(float lo, float hi) { return __floats2bfloat162_rn(lo, hi); }
  OLB_DEV static T from_float2(float2 v) { return __float22bfloat162_rn(v); }
};

// what a lane of the two-lane collision does: collide with the lattice's fluid
// kind, bounce back (full-way, collision::Revert), or pass its populations
// through (NoDynamics, and boundary cells, whose collision ran ahead of the step
// kernel), both up to an FP32 rounding of each pair's sum and difference
enum LaneMode { kLaneFluid = 0, kLaneWall = 1, kLanePass = 2 };

// the fluid collision constants of a cell for the scaled collisions (KIND the
// lattice's fluid kind): its table entry's when `own` and it has one, else the
// bulk entry's (kernel argument); a wall or pass lane gets the constants that
// make the same arithmetic a swap or the identity (see ScaledParams)
template <int KIND>
OLB_DEV ScaledParams<float> scaled_params(const DynDevice<float>* pe, bool own, const DynDevice<float>& bulk,
                                          int lane = kLaneFluid)
{
  ScaledParams<float> q;
  if (own && pe) {
    q.omega = __ldg(&pe->omega);
    q.omega_b = __ldg(&pe->omega_minus);
    q.smago_pre = __ldg(&pe->smago_pre);
    q.tau_mol = __ldg(&pe->tau_mol);
    q.force_relax = __ldg(&pe->force_relax);
    q.force[0] = __ldg(&pe->force[0]);
    q.force[1] = __ldg(&pe->force[1]);
    q.force[2] = __ldg(&pe->force[2]);
  } else {
    q.omega = bulk.omega;
    q.omega_b = bulk.omega_minus;
    q.smago_pre = bulk.smago_pre;
    q.tau_mol = bulk.tau_mol;
    q.force_relax = bulk.force_relax;
    q.force[0] = bulk.force[0];
    q.force[1] = bulk.force[1];
    q.force[2] = bulk.force[2];
  }
  if (!(KIND == K_TRT || KIND == K_FORCED_TRT)) q.omega_b = q.omega;
  q.keep = 0.5f * (1.f - q.omega);
  q.keep_minus = 0.5f * (1.f - q.omega_b);
  q.live = 1.f;
  if (lane != kLaneFluid) {
    q.omega = q.omega_b = q.force_relax = 0.f;
    q.force[0] = q.force[1] = q.force[2] = 0.f;
    q.keep = 0.5f;
    q.keep_minus = lane == kLaneWall ? -0.5f : 0.5f;
    q.live = 0.f;
  }
  return q;
}

// the constants of two cells as the lanes of one pair
OLB_DEV ScaledParams<float2> zip_params(const ScaledParams<float>& a, const ScaledParams<float>& b)
{
  ScaledParams<float2> q;
  q.omega = make_float2(a.omega, b.omega);
  q.omega_b = make_float2(a.omega_b, b.omega_b);
  q.keep = make_float2(a.keep, b.keep);
  q.keep_minus = make_float2(a.keep_minus, b.keep_minus);
  q.smago_pre = make_float2(a.smago_pre, b.smago_pre);
  q.tau_mol = make_float2(a.tau_mol, b.tau_mol);
  q.live = make_float2(a.live, b.live);
  q.force_relax = make_float2(a.force_relax, b.force_relax);
  q.force[0] = make_float2(a.force[0], b.force[0]);
  q.force[1] = make_float2(a.force[1], b.force[1]);
  q.force[2] = make_float2(a.force[2], b.force[2]);
  return q;
}

// byte permutation of a packed pair (one PRMT): 0x3210 keeps it, 0x1032 swaps
// the halves; pair_merge_lo/hi take the low/high halves of a and b
template <class T>
OLB_DEV T pair_perm(T a, T b, uint32_t sel)
{
  static_assert(sizeof(T) == 4, "packed 16-bit pair");
  uint32_t ua, ub;
  memcpy(&ua, &a, 4);
  memcpy(&ub, &b, 4);
  const uint32_t r = __byte_perm(ua, ub, sel);
  T out;
  memcpy(&out, &r, 4);
  return out;
}

struct PairNeighbours {
  uint32_t xo[3], yo[3], zo[3];
  bool swap[3];
  OLB_DEV PairNeighbours(const Geometry& g, int xp, int y, int z)
  {
    const int nxh = g.nx >> 1;
    const uint32_t sxy = uint32_t(g.ny) * uint32_t(g.nz);
    xo[0] = uint32_t(xp == 0 ? nxh - 1 : xp - 1) * sxy;
    xo[1] = uint32_t(xp) * sxy;
    xo[2] = uint32_t(xp == nxh - 1 ? 0 : xp + 1) * sxy;
    swap[0] = xp == 0;
    swap[1] = false;
    swap[2] = xp == nxh - 1;
    yo[0] = uint32_t(y == 0 ? g.ny - 1 : y - 1) * uint32_t(g.nz);
    yo[1] = uint32_t(y) * uint32_t(g.nz);
    yo[2] = uint32_t(y == g.ny - 1 ? 0 : y + 1) * uint32_t(g.nz);
    zo[0] = uint32_t(z == 0 ? g.nz - 1 : z - 1);
    zo[1] = uint32_t(z);
    zo[2] = uint32_t(z == g.nz - 1 ? 0 : z + 1);
  }
  template <int DX, int DY, int DZ>
  OLB_DEV uint32_t at() const { return xo[DX + 1] + yo[DY + 1] + zo[DZ + 1]; }
};

// collision of one cell of a pair by its runtime kind (masked lattices);
// field: the Guo-forced dynamics take the cell's FORCE from fcell
template <class L, int KIND, bool MASKED>
OLB_DEV bool collide_any(float (&f)[L::q], int kind, const DynDevice<float>* e, const DynDevice<float>& bulk,
                         const float (&fcell)[3], bool field, bool uniform, float& st_rho, float& st_usqr)
{
  constexpr bool kForced = KIND == K_FORCED_BGK || KIND == K_FORCED_TRT;
  if (kind == KIND) {
    const bool own = MASKED && e && !uniform;  // the entry's constants, not the bulk entry's
    if (own || (kForced && field)) {
      DynDevice<float> q;
      if (own) {
        q.omega = __ldg(&e->omega);
        q.omega_minus = __ldg(&e->omega_minus);
        q.smago_pre = __ldg(&e->smago_pre);
        q.tau_mol = __ldg(&e->tau_mol);
        q.force[0] = __ldg(&e->force[0]);
        q.force[1] = __ldg(&e->force[1]);
        q.force[2] = __ldg(&e->force[2]);
        q.force_relax = __ldg(&e->force_relax);
      } else {
        q.omega = bulk.omega;
        q.omega_minus = bulk.omega_minus;
        q.smago_pre = bulk.smago_pre;
        q.tau_mol = bulk.tau_mol;
        q.force[0] = bulk.force[0];
        q.force[1] = bulk.force[1];
        q.force[2] = bulk.force[2];
        q.force_relax = bulk.force_relax;
      }
      if constexpr (kForced) {
        if (field) {
          q.force[0] = fcell[0]; q.force[1] = fcell[1]; q.force[2] = fcell[2];
        }
      }
      collide_bulk<L, KIND>(f, q, st_rho, st_usqr);
    } else {
      collide_bulk<L, KIND>(f, bulk, st_rho, st_usqr);
    }
    return true;
  }
  if constexpr (MASKED) {
    if (kind == K_BOUNCE_BACK) {
      revert<L>(f);
    } else if (kind == K_BOUNCE_BACK_VELOCITY) {
      revert<L>(f);
      static_for<1, L::q>([&](auto i) {
        f[i] += __ldg(&e->wall_term[i][0]);
        f[i] += __ldg(&e->wall_term[i][1]);
        f[i] += __ldg(&e->wall_term[i][2]);
      });
      st_rho = __ldg(&e->wall_rho);
      const float wu[3] = {__ldg(&e->wall_u[0]), __ldg(&e->wall_u[1]), __ldg(&e->wall_u[2])};
      st_usqr = norm_sqr(wu);
      return true;
    }
  }
  return false;  // NoDynamics / bounce-back / boundary cells (collided ahead): no statistic here
}

// Collision of two cells held as packed 16-bit pairs (low half: cell n_lo of
// the natural order, high half: cell n_hi), in place; kind and table entry per
// cell.  count_hi: the high cell enters the statistics.  KEEP: a cell that passes
// its populations through (kLanePass) keeps their bits, an infinity or NaN among
// them with the others untouched; without, it runs as a lane and comes back
// rounded like a wall lane (see ScaledParams).
template <int Q, class S, int KIND, bool MASKED, bool STATS, bool KEEP = false>
OLB_DEV void collide_packed(typename Pair<S>::T (&raw)[Q], const Geometry& g,
                            const DynDevice<float>* __restrict__ table, const DynDevice<float>& bulk, int kind_lo,
                            int kind_hi, int id_lo, int id_hi, uint32_t n_lo, uint32_t n_hi, bool count_hi,
                            StatAcc& acc)
{
  using L = Lattice<Q>;
  using P = Pair<S>;
  using T = typename P::T;
  constexpr bool kForced = KIND == K_FORCED_BGK || KIND == K_FORCED_TRT;
  // the table entries (nullptr: the bulk entry, the kernel argument)
  const DynDevice<float>* pe_lo = MASKED && id_lo != kBoxCell ? table + id_lo : nullptr;
  const DynDevice<float>* pe_hi = MASKED && id_hi != kBoxCell ? table + id_hi : nullptr;
  const bool field = kForced && g.force != nullptr;
  // the cell's FORCE when the lattice has a force field (Guo-forced
  // dynamics; loaded here, after the populations)
  auto load_force = [&](uint32_t nn, float (&fc)[3]) {
    const float* __restrict__ F = static_cast<const float*>(g.force);
    fc[0] = __ldg(F + nn);
    fc[1] = __ldg(F + size_t(g.stride) + nn);
    fc[2] = __ldg(F + 2 * size_t(g.stride) + nn);
  };
#ifndef OLB_B200_EXACT
  if constexpr (MASKED && !kForced) {
    // A warp whose cells are all fluid with the bulk constants takes them from
    // the kernel argument, as an unmasked lattice does: no selects per lane, no
    // registers for two sets of constants (256^3 box of walls, D3Q27 BF16
    // Smagorinsky 376 -> 351 us per step, D3Q19 FP16 BGK 230 -> 228).  Not for
    // the forced collisions: the second copy of theirs spills (384x192x192 with
    // 35 % scattered walls, FP16 forced TRT: 218 -> 226 us).
    const bool plain = g.uniform && kind_lo == KIND && kind_hi == KIND;
    if (__all_sync(__activemask(), plain)) {
      collide_packed<Q, S, KIND, false, STATS>(raw, g, nullptr, bulk, KIND, KIND, 0, 0, n_lo, n_hi, count_hi, acc);
      return;
    }
  }
  // both cells go through the two-lane collision unless one is a moving wall
  // (a pair of two bounce-back walls stores nothing)
  bool both = true;
  int lane_lo = kLaneFluid, lane_hi = kLaneFluid;
  if constexpr (MASKED) {
    auto mode = [](int kind) {
      return kind == KIND ? kLaneFluid : (kind == K_BOUNCE_BACK ? kLaneWall : kLanePass);
    };
    lane_lo = mode(kind_lo);
    lane_hi = mode(kind_hi);
    // a moving wall adds its momentum terms: one cell after the other
    both = KEEP ? lane_lo != kLanePass && lane_hi != kLanePass
                : kind_lo != K_BOUNCE_BACK_VELOCITY && kind_hi != K_BOUNCE_BACK_VELOCITY;
  }
  if (both) {
    // Both cells at once, in the scaled representation g_i = s_i (f_i - w_i)
    // of the storage: lane x the low cell, lane y the high one, straight
    // from and back to the packed pairs (packed FP32 arithmetic); a wall or
    // pass lane takes the constants that make the collision a bounce-back or
    // the identity.
    float2 g2[Q];
    static_for<0, Q>([&](auto i) { g2[i] = P::to_float2(raw[i]); });
    ScaledParams<float> lo = scaled_params<KIND>(pe_lo, MASKED && !g.uniform, bulk, lane_lo);
    ScaledParams<float> hi = scaled_params<KIND>(pe_hi, MASKED && !g.uniform, bulk, lane_hi);
    if constexpr (kForced) {
      if (field) {
        if (lane_lo == kLaneFluid) load_force(n_lo, lo.force);
        if (lane_hi == kLaneFluid) load_force(n_hi, hi.force);
      }
    }
    const ScaledParams<float2> q2 = zip_params(lo, hi);
    float2 r2, u22;
    collide_scaled<L, KIND>(g2, q2, r2, u22);
    static_for<0, Q>([&](auto i) { raw[i] = P::from_float2(g2[i]); });
    if constexpr (STATS) {
      if (lane_lo == kLaneFluid) acc.add(double(r2.x), double(u22.x));
      if (lane_hi == kLaneFluid && count_hi) acc.add(double(r2.y), double(u22.y));
    }
  } else
#endif
  {
  // One cell after the other (a pair with a wall or boundary cell, and the
  // exact build).  BGK and TRT cells collide on g directly (collide_scaled);
  // any other dynamics decodes f_i = g_i / s_i, collides and re-encodes.
  // s_i of a population equals that of its opposite, so the column read or
  // written (i or opp(i)) does not change the scale.
  // the low cell's results wait in packed pairs of populations (half the
  // registers); the high cell's are packed the same way and the two are
  // merged with one byte permutation per population
  constexpr int QP = (Q + 1) / 2;
  T lo_pack[QP];
  auto cell = [&](auto half_tag, int kind, const DynDevice<float>* pe) {
    constexpr bool HI = decltype(half_tag)::value;
    float gout[Q];
    static_for<0, Q>([&](auto i) {
      const float2 fv = P::to_float2(raw[i]);
      gout[i] = HI ? fv.y : fv.x;
    });
    float r = 0.f, u2 = 0.f;
    bool counted = false, done = false;
    float fcell[3] = {0.f, 0.f, 0.f};
    if constexpr (kForced) {
      if (field && (!MASKED || kind == KIND)) load_force(HI ? n_hi : n_lo, fcell);
    }
#ifndef OLB_B200_EXACT
    if (!MASKED || kind == KIND) {
      ScaledParams<float> q = scaled_params<KIND>(pe, MASKED && !g.uniform, bulk);
      if (field) {
        q.force[0] = fcell[0]; q.force[1] = fcell[1]; q.force[2] = fcell[2];
      }
      collide_scaled<L, KIND>(gout, q, r, u2);
      counted = true;
      done = true;
    }
#endif
    if (!done) {
      static_for<0, Q>([&](auto i) {
        constexpr float inv = 1.f / storage_scale<L>(i);
        gout[i] *= inv;
      });
      counted = collide_any<L, KIND, MASKED>(gout, kind, pe, bulk, fcell, field, g.uniform != 0, r, u2);
      static_for<0, Q>([&](auto i) {
        constexpr float sc = storage_scale<L>(i);
        gout[i] *= sc;
      });
    }
    static_for<0, QP>([&](auto jj) {
      constexpr int a = 2 * jj.value;
      constexpr int b = a + 1 < Q ? a + 1 : a;
      const T packed = P::from_floats(gout[a], gout[b]);
      if constexpr (!HI) {
        lo_pack[jj] = packed;
      } else {
        raw[a] = pair_perm(lo_pack[jj], packed, 0x5410u);
        if constexpr (a + 1 < Q) {
          raw[a + 1] = pair_perm(lo_pack[jj], packed, 0x7632u);
        }
      }
    });
    if constexpr (STATS) {
      if (counted && (!HI || count_hi)) acc.add(double(r), double(u2));
    }
  };
  cell(std::integral_constant<bool, false>{}, kind_lo, pe_lo);
  cell(std::integral_constant<bool, true>{}, kind_hi, pe_hi);
  }
}

// One tile of the paired step: the CPT elements (x', y[k], z[k]) of this
// thread (none where y[k] = ny), each the two cells x' and x' + nx/2.  Masked lattices pass the
// table entries of both cells (loaded a tile ahead); unmasked ones use `bulk`.
template <int Q, class S, int KIND, bool ODD, bool MASKED, bool STATS, int CPT>
OLB_DEV void paired_tile(S* __restrict__ pops_scalar, const Geometry& g, const DynDevice<float>* __restrict__ table,
                         const DynDevice<float>& bulk, int xp, const int (&y)[CPT], const int (&z)[CPT],
                         const int (&id_lo)[CPT], const int (&id_hi)[CPT], StatAcc& acc)
{
  using L = Lattice<Q>;
  using P = Pair<S>;
  using T = typename P::T;
  T* __restrict__ pops = reinterpret_cast<T*>(pops_scalar);
  // Halves swap across the x seam only, on two planes of nx/2: one branch that
  // is uniform per block instead of a byte permutation per population (256^3
  // D3Q27 BF16 Smagorinsky 345 -> 340 us, D3Q27 BF16 TRT 292 -> 289, D3Q19 FP16
  // with walls 227 -> 224).  Not for the forced collisions, where it spills
  // (256x192x192 D3Q27 FP16 forced TRT 207 -> 220).
  constexpr bool kSeamBranch = KIND != K_FORCED_BGK && KIND != K_FORCED_TRT;
  const uint32_t pstride = g.stride >> 1;  // elements per column

  // the loaded pairs stay packed (low half = cell x', high half = x' + nx/2):
  // one 32-bit register per population for both cells
  T raw[CPT][Q];
  int kind_lo[CPT], kind_hi[CPT];
  bool go[CPT];
  uint32_t e[CPT];

  static_for<0, CPT>([&](auto k) {
    go[k] = y[k] < g.ny;
    kind_lo[k] = kind_hi[k] = KIND;
    e[k] = 0;
    if (go[k]) {
      // the pair's populations are loaded before its ids have arrived (as in
      // step_tile); a pair of two bounce-back cells then stores nothing
      e[k] = (uint32_t(xp) * uint32_t(g.ny) + uint32_t(y[k])) * uint32_t(g.nz) + uint32_t(z[k]);
      PairNeighbours nb(g, xp, y[k], z[k]);
      static_for<0, Q>([&](auto i) {
        // 32-bit element indices: the paired layout is only used while
        // q * pstride < 2^32 (olb_b200_create)
        if constexpr (!ODD) {
          raw[k][i] = pops[uint32_t(i.value) * pstride + e[k]];
        } else {
          constexpr int o = L::opp(i);
          const uint32_t src = nb.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>();
          raw[k][i] = pops[uint32_t(o) * pstride + src];
          if constexpr (!kSeamBranch && L::c(i, 0) != 0) {
            raw[k][i] = pair_perm(raw[k][i], raw[k][i], nb.swap[1 - L::c(i, 0)] ? 0x1032u : 0x3210u);
          }
        }
      });
      if constexpr (ODD && kSeamBranch) {
        if (nb.swap[0] || nb.swap[2]) {
          static_for<0, Q>([&](auto i) {
            if constexpr (L::c(i, 0) != 0) {
              raw[k][i] = pair_perm(raw[k][i], raw[k][i], nb.swap[1 - L::c(i, 0)] ? 0x1032u : 0x3210u);
            }
          });
        }
      }
    }
  });
  if constexpr (MASKED) {
    static_for<0, CPT>([&](auto k) {
      if (go[k]) {
        if (id_lo[k] != kBoxCell) kind_lo[k] = __ldg(&table[id_lo[k]].kind);
        if (id_hi[k] != kBoxCell) kind_hi[k] = __ldg(&table[id_hi[k]].kind);
        go[k] = !(kind_lo[k] == K_BOUNCE_BACK && kind_hi[k] == K_BOUNCE_BACK);
      }
    });
  }

  static_for<0, CPT>([&](auto k) {
    if (!go[k]) return;
    const uint32_t at = (uint32_t(xp) * uint32_t(g.ny) + uint32_t(y[k])) * uint32_t(g.nz) + uint32_t(z[k]);
    collide_packed<Q, S, KIND, MASKED, STATS>(raw[k], g, table, bulk, kind_lo[k], kind_hi[k], id_lo[k], id_hi[k], at,
                                              at + uint32_t(g.nx >> 1) * uint32_t(g.ny) * uint32_t(g.nz), true, acc);
    // recomputed after the collision rather than kept live through it
    PairNeighbours nb(g, int(opaque(uint32_t(xp))), int(opaque(uint32_t(y[k]))), int(opaque(uint32_t(z[k]))));
    const uint32_t ps = opaque(pstride);
    const uint32_t ek = opaque(e[k]);
    if constexpr (ODD && kSeamBranch) {
      if (nb.swap[0] || nb.swap[2]) {
        static_for<0, Q>([&](auto i) {
          if constexpr (L::c(i, 0) != 0) {
            raw[k][i] = pair_perm(raw[k][i], raw[k][i], nb.swap[1 + L::c(i, 0)] ? 0x1032u : 0x3210u);
          }
        });
      }
    }
    static_for<0, Q>([&](auto i) {
      if constexpr (!ODD) {
        constexpr int o = L::opp(i);
        pops[uint32_t(o) * ps + ek] = raw[k][i];
      } else {
        const uint32_t dst = nb.template at<L::c(i, 0), L::c(i, 1), L::c(i, 2)>();
        T v = raw[k][i];
        if constexpr (!kSeamBranch && L::c(i, 0) != 0) {
          v = pair_perm(v, v, nb.swap[1 + L::c(i, 0)] ? 0x1032u : 0x3210u);
        }
        pops[uint32_t(i.value) * ps + dst] = v;
      }
    });
  });
}

// ---------------------------------------------------------------------------
// the step kernel on the natural 16-bit layout (caller-owned buffers, odd nx)
// Bounded by memory latency: a warp's access moves 64 bytes, half of what the
// paired layout moves, so bytes in flight are short.  One cell per thread
// (f_i decoded, collided, encoded) reached 3.67 TB/s on a 191x173x150 D3Q27
// BF16 box (146 us per step) and 3.87 TB/s on 257^3 D3Q19 FP16 (330 us); two
// cells per thread, collided together as in the paired kernel, 4.39 TB/s
// (122 us) and 4.6 TB/s (280 us).  80 registers (3 blocks of 256 per SM) beat
// 64 where the cells are masked or forced (131x95x122 forced TRT: 33 us
// against 37) and are even elsewhere.
//
// Each thread updates two cells of a plane, one of each of the block's two
// runs (tile_cells), as the two lanes of the packed collision.  The cells'
// populations are separate 16-bit accesses, so nothing is asked of their
// alignment.
template <int Q, class S, int KIND, bool ODD, bool MASKED, bool STATS>
OLB_DEV void split_tile(S* __restrict__ pops, const Geometry& g, const DynDevice<float>* __restrict__ table,
                        const DynDevice<float>& bulk, int x, int (&y)[2], int (&z)[2], int (&id)[2], StatAcc& acc)
{
  using L = Lattice<Q>;
  using T = typename Pair<S>::T;
  if (y[0] >= g.ny) return;
  // a missing second cell (the plane's last run) repeats the first, unstored
  const bool two = y[1] < g.ny;
  if (!two) {
    y[1] = y[0];
    z[1] = z[0];
    id[1] = id[0];
  }
  uint32_t n[2];
  static_for<0, 2>([&](auto k) {
    n[k] = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y[k])) * uint32_t(g.nz) + uint32_t(z[k]);
  });
  T raw[Q];
  {
    const Neighbours a(g, x, y[0], z[0]), b(g, x, y[1], z[1]);
    static_for<0, Q>([&](auto i) {
      constexpr int col = ODD ? L::opp(i) : i.value;
      const S* __restrict__ p = pops + size_t(col) * g.stride;
      if constexpr (!ODD) {
        raw[i] = T(p[n[0]], p[n[1]]);
      } else {
        raw[i] = T(p[a.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>()],
                   p[b.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>()]);
      }
    });
  }
  int kind[2] = {KIND, KIND};
  bool store[2] = {true, two};
  if constexpr (MASKED) {
    static_for<0, 2>([&](auto k) {
      if (id[k] != kBoxCell) kind[k] = __ldg(&table[id[k]].kind);
      store[k] = store[k] && kind[k] != K_BOUNCE_BACK;  // a bounce-back cell's update is a no-op
    });
    if (!store[0] && !store[1]) return;
  }
  collide_packed<Q, S, KIND, MASKED, STATS, true>(raw, g, table, bulk, kind[0], kind[1], id[0], id[1], n[0], n[1], two, acc);
  const Neighbours a(g, int(opaque(uint32_t(x))), int(opaque(uint32_t(y[0]))), int(opaque(uint32_t(z[0])))),
    b(g, int(opaque(uint32_t(x))), int(opaque(uint32_t(y[1]))), int(opaque(uint32_t(z[1]))));
  const uint32_t stride = opaque(g.stride);
  const uint32_t n0 = opaque(n[0]), n1 = opaque(n[1]);
  static_for<0, Q>([&](auto i) {
    constexpr int col = ODD ? i.value : L::opp(i);
    S* __restrict__ p = pops + size_t(col) * stride;
    uint32_t to0 = n0, to1 = n1;
    if constexpr (ODD) {
      to0 = a.template at<L::c(i, 0), L::c(i, 1), L::c(i, 2)>();
      to1 = b.template at<L::c(i, 0), L::c(i, 1), L::c(i, 2)>();
    }
    if (store[0]) p[to0] = raw[i].x;
    if (store[1]) p[to1] = raw[i].y;
  });
}

// MASKED = false takes no ids or table (nullptr)
template <int Q, class S, int KIND, bool ODD, bool MASKED, bool STATS>
__global__ void __launch_bounds__(kStepThreads, kSplitMinBlocks)
aa_step_split_kernel(S* __restrict__ pops, const Geometry g, const uint8_t* __restrict__ ids,
                     const DynDevice<float>* __restrict__ table, const DynDevice<float> bulk,
                     const StatSink sink)
{
  next_may_start();
  const int x = blockIdx.z;
  int y[2], z[2], id[2] = {};
  tile_cells(g, y, z);
  if constexpr (MASKED) load_tile_ids(id, g, ids, x, y, z);
  StatAcc acc;
  pops = after_previous(pops);
  split_tile<Q, S, KIND, ODD, MASKED, STATS>(pops, g, table, bulk, x, y, z, id, acc);
  if constexpr (STATS) {
    block_stats(acc.rho, acc.usqr, acc.max, acc.n, acc.nf, sink);
  }
}

template <int Q, class S, int KIND, bool ODD, bool STATS, int CPT, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
aa_step_paired_kernel(S* __restrict__ pops, const Geometry g, const DynDevice<float> bulk,
                      const StatSink sink)
{
  next_may_start();
  int y[CPT], z[CPT];
  tile_cells(g, y, z);
  const int none[CPT] = {};
  StatAcc acc;
  pops = after_previous(pops);
  paired_tile<Q, S, KIND, ODD, false, STATS, CPT>(pops, g, nullptr, bulk, int(blockIdx.z), y, z, none, none, acc);
  if constexpr (STATS) {
    block_stats(acc.rho, acc.usqr, acc.max, acc.n, acc.nf, sink);
  }
}

// the masked paired kernel: one tile per block (aa_step_masked_kernel)
template <int Q, class S, int KIND, bool ODD, bool STATS, int CPT, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB)
aa_step_masked_paired_kernel(S* __restrict__ pops, const Geometry g, const uint8_t* __restrict__ ids,
                             const DynDevice<float>* __restrict__ table, const DynDevice<float> bulk,
                             const StatSink sink)
{
  next_may_start();
  const int xp = blockIdx.z;
  int y[CPT], z[CPT], lo[CPT], hi[CPT];
  tile_cells(g, y, z);
  load_tile_ids(lo, g, ids, xp, y, z);
  load_tile_ids(hi, g, ids, xp + (g.nx >> 1), y, z);
  StatAcc acc;
  pops = after_previous(pops);
  paired_tile<Q, S, KIND, ODD, true, STATS, CPT>(pops, g, table, bulk, xp, y, z, lo, hi, acc);
  if constexpr (STATS) {
    block_stats(acc.rho, acc.usqr, acc.max, acc.n, acc.nf, sink);
  }
}

// Deterministic second pass over the per-block partials: up to kReduceBlocks
// blocks (one block needs no stage), the last of which adds up the others.
__global__ void reduce_partials_kernel(const StatPartial* parts, size_t count, StatStage* stage, StatResult* out,
                                       unsigned long long seq);
constexpr int kReduceThreads = 256;

// ---------------------------------------------------------------------------
// logical-layout gather / scatter and moments

// Logical population i at cell (x,y,z): column i at the cell after an even
// number of steps, else column opp(i) at (x,y,z) - c_i (per-axis wrap).
template <int Q, class S, class R, int I>
OLB_DEV R logical_pop(const S* __restrict__ pops, const Geometry& g, int x, int y, int z, bool shifted)
{
  using L = Lattice<Q>;
  if (!shifted) {
    return Store<S, R>::template load<L, I>(pops + size_t(I) * g.stride + cell_slot(g, x, y, z));
  }
  constexpr int o = L::opp(I);
  const uint32_t src = cell_slot(g, wrap(x - L::c(I, 0), g.nx), wrap(y - L::c(I, 1), g.ny),
                                 wrap(z - L::c(I, 2), g.nz));
  return Store<S, R>::template load<L, o>(pops + size_t(o) * g.stride + src);
}

// The addresses of one cell's logical populations: slot<DX,DY,DZ>() is the
// scalar slot, within any column, of the cell itself (not shifted) or of its
// neighbour at (DX,DY,DZ) (shifted, per-axis wrap).
struct LogicalSlots {
  uint32_t xo[3], yo[3], zo[3];
  OLB_DEV LogicalSlots(const Geometry& g, int x, int y, int z, bool shifted)
  {
    const int s = shifted ? 1 : 0, nxh = g.nx >> 1;
    const uint32_t m = g.paired ? 2u : 1u;
    const uint32_t sy = uint32_t(g.nz) * m, sx = uint32_t(g.ny) * sy;
#pragma unroll
    for (int d = -1; d <= 1; ++d) {
      const int xx = wrap(x + d * s, g.nx);
      const bool hi = g.paired && xx >= nxh;
      xo[d + 1] = uint32_t(hi ? xx - nxh : xx) * sx + uint32_t(hi);
      yo[d + 1] = uint32_t(wrap(y + d * s, g.ny)) * sy;
      zo[d + 1] = uint32_t(wrap(z + d * s, g.nz)) * m;
    }
  }
  template <int DX, int DY, int DZ>
  OLB_DEV uint32_t at() const { return xo[DX + 1] + yo[DY + 1] + zo[DZ + 1]; }
};

// All logical populations of a cell (logical_pop of each).  The layout is
// settled once, outside the populations, so that nothing stands between the
// loads and they travel together: with logical_pop's two branches per
// population every load waited for the one before it.
template <int Q, class S, class R>
OLB_DEV void load_logical(const S* pops, const Geometry& g, int x, int y, int z, bool shifted, R (&f)[Q])
{
  using L = Lattice<Q>;
  const LogicalSlots c(g, x, y, z, shifted);
  static_for<0, Q>([&](auto i) {
    const size_t col = shifted ? size_t(L::opp(i)) * g.stride : size_t(i.value) * g.stride;
    f[i] = Store<S, R>::template load<L, i.value>(pops + col + c.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>());
  });
}

// the inverse: all logical populations of a cell written back
template <int Q, class S, class R>
OLB_DEV void store_logical(S* pops, const Geometry& g, int x, int y, int z, bool shifted, const R (&f)[Q])
{
  using L = Lattice<Q>;
  const LogicalSlots c(g, x, y, z, shifted);
  static_for<0, Q>([&](auto i) {
    const size_t col = shifted ? size_t(L::opp(i)) * g.stride : size_t(i.value) * g.stride;
    Store<S, R>::template store<L, i.value>(
      pops + col + c.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>(), f[i]);
  });
}

template <int Q, class S, class R>
__global__ void gather_logical_kernel(const S* __restrict__ pops, const Geometry g, bool shifted,
                                      R* __restrict__ out, int i_begin, int i_end)
{
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny) return;
  const uint32_t n = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  const size_t cells = size_t(g.nx) * g.ny * g.nz;
  static_for<0, Q>([&](auto i) {
    if (i.value >= i_begin && i.value < i_end) {
      out[size_t(i.value - i_begin) * cells + n] = logical_pop<Q, S, R, i.value>(pops, g, x, y, z, shifted);
    }
  });
}

// write of logical populations in the unshifted order (resets the AA parity)
template <int Q, class S, class R>
__global__ void scatter_natural_kernel(S* __restrict__ pops, const Geometry g,
                                       const R* __restrict__ in, int i_begin, int i_end)
{
  using L = Lattice<Q>;
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny) return;
  const uint32_t n = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  const size_t cells = size_t(g.nx) * g.ny * g.nz;
  const uint32_t slot = cell_slot(g, x, y, z);
  static_for<0, Q>([&](auto i) {
    if (i.value >= i_begin && i.value < i_end) {
      Store<S, R>::template store<L, i.value>(pops + size_t(i.value) * g.stride + slot,
                                              in[size_t(i.value - i_begin) * cells + n]);
    }
  });
}

// Cell::iniEquilibrium on every cell: the second-order equilibrium of the
// cell's density and velocity (equilibrium::secondOrder, src/dynamics/lbm.h:50-64,
// as the shifted value f_eq - w), written in the natural layout; rho_u holds
// rho of every cell, then u_x, u_y, u_z.
template <int Q, class S, class R>
__global__ void equilibrium_kernel(S* __restrict__ pops, const Geometry g, const R* __restrict__ rho_u)
{
  using L = Lattice<Q>;
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny) return;
  const uint32_t n = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  const size_t cells = size_t(g.nx) * g.ny * g.nz;
  const uint32_t slot = cell_slot(g, x, y, z);
  const R rho = rho_u[n];
  const R u[3] = {rho_u[cells + n], rho_u[2 * cells + n], rho_u[3 * cells + n]};
  const R usqr = norm_sqr(u);
  static_for<0, Q>([&](auto i) {
    Store<S, R>::template store<L, i.value>(pops + size_t(i.value) * g.stride + slot,
                                            feq2<L, i.value>(rho, u, usqr));
  });
}

// FORCE of cell n of a Guo-forced dynamics: the lattice's force field when it
// has one, else the entry's constant
template <class R>
OLB_DEV void cell_force(const Geometry& g, const DynDevice<R>* e, uint32_t n, R (&gg)[3])
{
  if (g.force) {
    const R* F = static_cast<const R*>(g.force);
    gg[0] = F[n];
    gg[1] = F[size_t(g.stride) + n];
    gg[2] = F[2 * size_t(g.stride) + n];
  } else {
    gg[0] = e->force[0];
    gg[1] = e->force[1];
    gg[2] = e->force[2];
  }
}

// Density and velocity of cell (x,y,z) with populations f, written to the
// outputs: as the reference's Density3D / Velocity3D report them (per-dynamics
// momenta: src/dynamics/momenta/elements.h).
template <int Q, class R>
OLB_DEV void cell_moments(const R (&f)[Q], const Geometry& g, const DynDevice<R>* __restrict__ p, int x, int y, int z,
                          uint32_t n, R* __restrict__ rho_out, R* __restrict__ u_out)
{
  using L = Lattice<Q>;
  const size_t cells = size_t(g.nx) * g.ny * g.nz;
  const int kind = p->kind;
  R rho, u[3];
  if (kind == K_BGK || kind == K_TRT || kind == K_SMAGORINSKY || kind == K_FORCED_BGK ||
      kind == K_FORCED_TRT) {
    if (kind == K_FORCED_BGK || kind == K_FORCED_TRT) {
      R gg[3];
      cell_force(g, p, n, gg);
      compute_rho_u_forced<L>(f, gg, rho, u);
    } else {
      compute_rho_u<L>(f, rho, u);
    }
  } else if (kind == K_BOUNCE_BACK) {
    rho = p->wall_rho; u[0] = u[1] = u[2] = R(0);
  } else if (kind == K_BOUNCE_BACK_VELOCITY) {
    rho = p->wall_rho; u[0] = p->wall_u[0]; u[1] = p->wall_u[1]; u[2] = p->wall_u[2];
  } else if (is_interpolated(kind) || is_local(kind)) {
    bc_rho_u<L>(f, kind, p->bc_dir, p->bc_orient, p->bc_values + 4 * size_t(bc_index(p, x, y, z)), rho, u);
  } else if (is_inner(kind)) {
    // InnerEdge/CornerDensity3D + FixedVelocityMomentumGeneric
    const R* v = p->bc_values + 4 * size_t(bc_index(p, x, y, z));
    u[0] = v[1]; u[1] = v[2]; u[2] = v[3];
    const int32_t nn[3] = {p->nrm[0], p->nrm[1], p->nrm[2]};
    rho = inner_rho<L>(f, kind, nn, u);
  } else if (is_outer(kind)) {
    // BulkDensity + FixedVelocityMomentumGeneric
    rho = compute_rho<L>(f);
    const R* v = p->bc_values + 4 * size_t(bc_index(p, x, y, z));
    u[0] = v[1]; u[1] = v[2]; u[2] = v[3];
  } else {
    rho = R(1); u[0] = u[1] = u[2] = R(0);
  }
  rho_out[n] = rho;
  u_out[n] = u[0];
  u_out[cells + n] = u[1];
  u_out[2 * cells + n] = u[2];
}

template <int Q, class S, class R>
__global__ void moments_kernel(const S* __restrict__ pops, const Geometry g, bool shifted,
                               const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                               R* __restrict__ rho_out, R* __restrict__ u_out)
{
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= g.nz || y >= g.ny) return;
  const uint32_t n = (uint32_t(x) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  const DynDevice<R>* p = table + (ids ? ids[n] : 0);
  // loaded before the cell's kind has arrived; walls and NoDynamics drop them
  R f[Q];
  load_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
  cell_moments<Q, R>(f, g, p, x, y, z, n, rho_out, u_out);
}

// The same on the paired 16-bit layout: a thread takes both cells of its
// elements, 4 bytes per population and access.  One cell per thread used half of
// every sector it fetched (512x256x256 D3Q27 BF16: 712 us,
// 607 with both).
template <int Q, class S>
__global__ void moments_paired_kernel(const S* __restrict__ pops, const Geometry g, bool shifted,
                                      const uint8_t* __restrict__ ids, const DynDevice<float>* __restrict__ table,
                                      float* __restrict__ rho_out, float* __restrict__ u_out)
{
  using L = Lattice<Q>;
  using T = typename Pair<S>::T;
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int xp = blockIdx.z;
  if (z >= g.nz || y >= g.ny) return;
  const uint32_t half = uint32_t(g.nx >> 1) * uint32_t(g.ny) * uint32_t(g.nz);
  const uint32_t n = (uint32_t(xp) * uint32_t(g.ny) + uint32_t(y)) * uint32_t(g.nz) + uint32_t(z);
  const DynDevice<float>* lo = table + (ids ? ids[n] : 0);
  const DynDevice<float>* hi = table + (ids ? ids[n + half] : 0);
  const PairNeighbours nb(g, xp, y, z);
  const T* __restrict__ elems = reinterpret_cast<const T*>(pops);
  const uint32_t pstride = g.stride >> 1;
  T raw[Q];
  static_for<0, Q>([&](auto i) {
    const uint32_t at = shifted ? nb.template at<-L::c(i, 0), -L::c(i, 1), -L::c(i, 2)>() : n;
    const T v = elems[size_t(shifted ? L::opp(i) : i.value) * pstride + at];
    raw[i] = v;
    if constexpr (L::c(i, 0) != 0) {
      raw[i] = pair_perm(v, v, shifted && nb.swap[1 - L::c(i, 0)] ? 0x1032u : 0x3210u);
    }
  });
  float f[Q];
  static_for<0, Q>([&](auto i) {
    constexpr float inv = 1.f / storage_scale<L>(i.value);
    f[i] = Pair<S>::to_float2(raw[i]).x * inv;
  });
  cell_moments<Q, float>(f, g, lo, xp, y, z, n, rho_out, u_out);
  static_for<0, Q>([&](auto i) {
    constexpr float inv = 1.f / storage_scale<L>(i.value);
    f[i] = Pair<S>::to_float2(raw[i]).y * inv;
  });
  cell_moments<Q, float>(f, g, hi, xp + (g.nx >> 1), y, z, n + half, rho_out, u_out);
}

// ---------------------------------------------------------------------------
// PostStream: PlaneFdBoundaryProcessor3D on the interpolated boundary cells
//
// src/boundary/boundaryPostProcessors3D.hh:39-92.  Each boundary cell is
// rebuilt from the post-stream state as feq(rho, u) + fneq(Pi), Pi from the
// finite-difference strain rate: one-sided second order along the normal
// (cells x - orient e and x - 2 orient e), central across it
// (fd::DirectedGradients3D, src/utilities/finiteDifference3D.h:58-200).
// Two passes: the first stores the velocity of every boundary cell (its
// momenta on the post-stream state), the second rebuilds every boundary cell;
// a boundary cell never reads another boundary cell's populations in the
// second pass, so the passes need no ordering among cells.

OLB_DEV void decode_cell(const Geometry& g, uint32_t n, int& x, int& y, int& z)
{
  const uint32_t nynz = uint32_t(g.ny) * uint32_t(g.nz);
  const uint32_t xx = n / nynz;
  const uint32_t r = n - xx * nynz;
  const uint32_t yy = r / uint32_t(g.nz);
  x = int(xx);
  y = int(yy);
  z = int(r - yy * uint32_t(g.nz));
}

// Cell::computeU through the cell's dynamics on the post-stream state: bulk
// (momenta/elements.h:466-475), forced bulk (:1480-1488), VELOCITY of moving
// walls, the stored velocity of interpolated cells, zero otherwise.  A cell
// beyond a non-periodic face is the reference's NoDynamics padding: zero.
template <int Q, class S, class R>
OLB_DEV void cell_velocity(const S* __restrict__ pops, const Geometry& g, bool shifted,
                           const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                           int periodic, int x, int y, int z, R (&u)[3])
{
  using L = Lattice<Q>;
  u[0] = u[1] = u[2] = R(0);
  int p[3] = {x, y, z};
  const int ext[3] = {g.nx, g.ny, g.nz};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (p[d] < 0 || p[d] >= ext[d]) {
      if (!((periodic >> d) & 1)) return;
      p[d] = p[d] < 0 ? p[d] + ext[d] : p[d] - ext[d];
    }
  }
  const uint32_t n = (uint32_t(p[0]) * uint32_t(g.ny) + uint32_t(p[1])) * uint32_t(g.nz) + uint32_t(p[2]);
  const DynDevice<R>* e = table + ids[n];
  const int kind = e->kind;
  if (kind == K_BGK || kind == K_TRT || kind == K_SMAGORINSKY || kind == K_FORCED_BGK || kind == K_FORCED_TRT) {
    R f[Q];
    load_logical<Q, S, R>(pops, g, p[0], p[1], p[2], shifted, f);
    R rho;
    if (kind == K_FORCED_BGK || kind == K_FORCED_TRT) {
      R gg[3];
      cell_force(g, e, n, gg);
      compute_rho_u_forced<L>(f, gg, rho, u);
    } else {
      compute_rho_u<L>(f, rho, u);
    }
  } else if (kind == K_BOUNCE_BACK_VELOCITY) {
    u[0] = e->wall_u[0]; u[1] = e->wall_u[1]; u[2] = e->wall_u[2];
  } else if (is_interpolated(kind)) {
    const R* bu = e->bc_u + 3 * size_t(bc_index(e, p[0], p[1], p[2]));
    u[0] = bu[0]; u[1] = bu[1]; u[2] = bu[2];
  } else if (kind == K_LOCAL_PRESSURE) {
    // FixedPressureMomentum::computeU: VELOCITY, the normal part from the populations
    R f[Q];
    load_logical<Q, S, R>(pops, g, p[0], p[1], p[2], shifted, f);
    R rho;
    bc_rho_u<L>(f, kind, e->bc_dir, e->bc_orient, e->bc_values + 4 * size_t(bc_index(e, p[0], p[1], p[2])), rho,
                u);
  } else if (kind == K_LOCAL_VELOCITY || is_outer(kind) || is_inner(kind)) {
    // FixedVelocityMomentumGeneric: the VELOCITY field
    const R* v = e->bc_values + 4 * size_t(bc_index(e, p[0], p[1], p[2]));
    u[0] = v[1]; u[1] = v[2]; u[2] = v[3];
  }
}

// Cell::computeRho through the cell's dynamics on the current state:
// BulkDensity (fluid, external edges and corners), velocityBMRho (flat velocity
// boundaries), FixedDensity RHO (walls, pressure boundaries), 1 for NoDynamics
// and for the reference's padding beyond a non-periodic face.
template <int Q, class S, class R>
OLB_DEV R cell_density(const S* __restrict__ pops, const Geometry& g, bool shifted,
                       const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table, int periodic,
                       int x, int y, int z)
{
  using L = Lattice<Q>;
  int p[3] = {x, y, z};
  const int ext[3] = {g.nx, g.ny, g.nz};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (p[d] < 0 || p[d] >= ext[d]) {
      if (!((periodic >> d) & 1)) return R(1);
      p[d] = p[d] < 0 ? p[d] + ext[d] : p[d] - ext[d];
    }
  }
  const uint32_t n = (uint32_t(p[0]) * uint32_t(g.ny) + uint32_t(p[1])) * uint32_t(g.nz) + uint32_t(p[2]);
  const DynDevice<R>* e = table + ids[n];
  const int kind = e->kind;
  if (kind == K_BOUNCE_BACK || kind == K_BOUNCE_BACK_VELOCITY) return e->wall_rho;
  if (kind == K_NONE) return R(1);
  R f[Q];
  load_logical<Q, S, R>(pops, g, p[0], p[1], p[2], shifted, f);
  if (is_interpolated(kind) || is_local(kind)) {
    R rho, u[3];
    bc_rho_u<L>(f, kind, e->bc_dir, e->bc_orient, e->bc_values + 4 * size_t(bc_index(e, p[0], p[1], p[2])), rho,
                u);
    return rho;
  }
  if (is_inner(kind)) {
    const R* v = e->bc_values + 4 * size_t(bc_index(e, p[0], p[1], p[2]));
    const R u[3] = {v[1], v[2], v[3]};
    const int32_t nn[3] = {e->nrm[0], e->nrm[1], e->nrm[2]};
    return inner_rho<L>(f, kind, nn, u);
  }
  return compute_rho<L>(f);
}

// pass 1: velocity of every interpolated cell (its momenta, post-stream state)
template <int Q, class S, class R>
__global__ void bc_velocity_kernel(const S* pops, const Geometry g, bool shifted,
                                   const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                                   const uint32_t* __restrict__ cells, uint32_t count)
{
  using L = Lattice<Q>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  next_may_start();
  pops = after_previous(pops);
  if (k >= count) return;
  const uint32_t n = cells[k];
  int x, y, z;
  decode_cell(g, n, x, y, z);
  const DynDevice<R>* e = table + ids[n];
  const uint32_t bi = bc_index(e, x, y, z);
  R f[Q];
  load_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
  R rho, u[3];
  bc_rho_u<L>(f, e->kind, e->bc_dir, e->bc_orient, e->bc_values + 4 * size_t(bi), rho, u);
  R* bu = e->bc_u + 3 * size_t(bi);
  bu[0] = u[0];
  bu[1] = u[1];
  bu[2] = u[2];
}

// grad[d][c], the derivative along axis d of velocity component c at (x,y,z)
// whose velocity is u: one-sided second order along the axes with
// inward[d] != 0 (cells inward[d] and 2 inward[d] away), central along the
// others (fd::DirectedGradients3D, src/utilities/finiteDifference3D.h:58-200).
// The axes and the two neighbours of each go through one copy of
// cell_velocity instead of twelve (every dynamics kind, q loads each): with
// the populations of a cell loaded together (load_logical) plane_fd_kernel
// takes 26 us on the 129 032 boundary cells of a 512x256x256 D3Q27 BF16
// channel, 80-85 with the loop alone, 90 with neither.
template <int Q, class S, class R>
OLB_DEV void velocity_gradients(const S* pops, const Geometry& g, bool shifted, const uint8_t* __restrict__ ids,
                                const DynDevice<R>* __restrict__ table, int periodic, int x, int y, int z,
                                const R (&u)[3], const int (&inward)[3], R (&grad)[3][3])
{
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    const int s = d == 0 ? inward[0] : (d == 1 ? inward[1] : inward[2]);
    R a[3], b[3];  // at s and 2 s, or at +1 and -1
#pragma unroll 1
    for (int m = 0; m < 2; ++m) {
      const int step = s != 0 ? (m + 1) * s : 1 - 2 * m;
      R v[3];
      cell_velocity<Q, S, R>(pops, g, shifted, ids, table, periodic, x + (d == 0 ? step : 0),
                             y + (d == 1 ? step : 0), z + (d == 2 ? step : 0), v);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (m == 0) a[c] = v[c]; else b[c] = v[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const R v = s != 0 ? R(s) * ((-R(3) * u[c] + R(4) * a[c] - R(1) * b[c]) / R(2)) : (a[c] - b[c]) / R(2);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (d == k) grad[k][c] = v;
      }
    }
  }
}

// pass 2: PlaneFdBoundaryProcessor3D<direction,orientation>::apply
template <int Q, class S, class R>
__global__ void plane_fd_kernel(S* __restrict__ pops, const Geometry g, bool shifted,
                                const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                                int periodic, const uint32_t* __restrict__ cells, uint32_t count)
{
  using L = Lattice<Q>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  next_may_start();
  pops = after_previous(pops);
  if (k >= count) return;
  const uint32_t n = cells[k];
  int x, y, z;
  decode_cell(g, n, x, y, z);
  const DynDevice<R>* e = table + ids[n];
  const int dir = e->bc_dir, orient = e->bc_orient;
  R f[Q];
  load_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
  R rho, u[3];
  bc_rho_u<L>(f, e->kind, dir, orient, e->bc_values + 4 * size_t(bc_index(e, x, y, z)), rho, u);
  const int inward[3] = {dir == 0 ? -orient : 0, dir == 1 ? -orient : 0, dir == 2 ? -orient : 0};
  R grad[3][3];
  velocity_gradients<Q, S, R>(pops, g, shifted, ids, table, periodic, x, y, z, u, inward, grad);
  const R s_to_pi = -rho / R(3) / e->omega;
  R pi[6];
  pi[0] = R(2) * grad[0][0] * s_to_pi;
  pi[3] = R(2) * grad[1][1] * s_to_pi;
  pi[5] = R(2) * grad[2][2] * s_to_pi;
  pi[1] = (grad[0][1] + grad[1][0]) * s_to_pi;
  pi[2] = (grad[0][2] + grad[2][0]) * s_to_pi;
  pi[4] = (grad[1][2] + grad[2][1]) * s_to_pi;
  const R usqr = norm_sqr(u);
  static_for<0, Q>([&](auto i) {
    f[i] = feq2<L, i.value>(rho, u, usqr) + from_pi_to_fneq<L, i.value>(pi);
  });
  store_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
}

// Collision of the boundary cells that carry values (interpolated, local
// velocity, external edges and corners), in place, ahead of the step kernel.
// Each cell's populations are read where the step kernel will read them
// (the current AA parity) and written back there, so the step kernel, which
// passes these cells through, streams the collided values.  Keeping the
// boundary collisions out of the step kernel leaves its register allocation
// to the bulk collision: inlined, they raised the register demand of every
// cell and the masked kernels spilled.  Statistics of the boundary cells go
// to the partials after the step kernel's blocks.
template <int Q, class S, class R, int KIND, bool STATS>
__global__ void boundary_collide_kernel(S* __restrict__ pops, const Geometry g, bool shifted,
                                        const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                                        const uint32_t* __restrict__ cells, uint32_t count,
                                        const StatSink sink)
{
  using L = Lattice<Q>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  double s_rho = 0., s_usqr = 0., s_max = 0.;
  unsigned long long s_n = 0, s_nf = 0;
  next_may_start();
  pops = after_previous(pops);
  if (k < count) {
    const uint32_t n = cells[k];
    int x, y, z;
    decode_cell(g, n, x, y, z);
    const DynDevice<R>* e = table + ids[n];
    R f[Q];
    load_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
    R st_rho = R(0), st_usqr = R(0);
    collide_boundary<L, KIND>(f, e->kind, e, x, y, z, st_rho, st_usqr);
    store_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
    if constexpr (STATS) {
      const double r = double(st_rho), u2 = double(st_usqr);
      if (isfinite(r) && isfinite(u2)) {
        s_rho = r; s_usqr = u2; s_max = u2; s_n = 1;
      } else {
        s_nf = 1;
      }
    }
  }
  if constexpr (STATS) {
    block_stats(s_rho, s_usqr, s_max, s_n, s_nf, sink);
  }
}

// OuterVelocityEdgeProcessor3D<plane,normal1,normal2>::apply (pass 3) and
// OuterVelocityCornerProcessor3D<xN,yN,zN>::apply (pass 4),
// src/boundary/boundaryPostProcessors3D.hh:164-292: the density extrapolated
// from the cells inward along the normal(s), velocity gradients one-sided
// across the boundary and central along an edge, the cell rebuilt as
// feq(rho, VELOCITY) + fneq(Pi).  The corner pass runs after the edge pass
// (priority 1 after 0): a corner's density reads the edge cells it ends.
template <int Q, class S, class R, bool CORNER>
__global__ void outer_velocity_kernel(S* __restrict__ pops, const Geometry g, bool shifted,
                                      const uint8_t* __restrict__ ids, const DynDevice<R>* __restrict__ table,
                                      int periodic, const uint32_t* __restrict__ cells, uint32_t count)
{
  using L = Lattice<Q>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  next_may_start();
  pops = after_previous(pops);
  if (k >= count) return;
  const uint32_t n = cells[k];
  int x, y, z;
  decode_cell(g, n, x, y, z);
  const DynDevice<R>* e = table + ids[n];
  const int nrm[3] = {e->nrm[0], e->nrm[1], e->nrm[2]};
  const R* v = e->bc_values + 4 * size_t(bc_index(e, x, y, z));
  const R u[3] = {v[1], v[2], v[3]};
  R rho;
  // neighbour densities: edges getNeighborRho(step1, step2), steps 1 and 2
  // along each of the two normal axes d1, d2; corners along the three axes
  const int plane = nrm[0] == 0 ? 0 : (nrm[1] == 0 ? 1 : 2);
  const int d1 = CORNER ? 0 : (plane == 2 ? 0 : plane + 1), d2 = plane == 0 ? 2 : (plane == 1 ? 0 : 1);
  constexpr int kAxes = CORNER ? 3 : 2;
  R near[3] = {R(0), R(0), R(0)}, far[3] = {R(0), R(0), R(0)};  // one and two cells inward
#pragma unroll 1
  for (int m = 0; m < 2 * kAxes; ++m) {
    const int k = m % kAxes, step = m / kAxes + 1;
    const int axis = CORNER ? k : (k == 0 ? d1 : d2);
    const int off = -(axis == 0 ? nrm[0] : (axis == 1 ? nrm[1] : nrm[2])) * step;
    const R r = cell_density<Q, S, R>(pops, g, shifted, ids, table, periodic, x + (axis == 0 ? off : 0),
                                      y + (axis == 1 ? off : 0), z + (axis == 2 ? off : 0));
#pragma unroll
    for (int j = 0; j < kAxes; ++j) {
      if (k == j) {
        if (step == 1) near[j] = r; else far[j] = r;
      }
    }
  }
  if constexpr (!CORNER) {
    rho = R(2) / R(3) * (near[1] + near[0]) - R(1) / R(6) * (far[1] + far[0]);
  } else {
    rho = R(4) / R(9) * (near[2] + near[1] + near[0]) - R(1) / R(9) * (far[2] + far[1] + far[0]);
  }
  const int inward[3] = {-nrm[0], -nrm[1], -nrm[2]};
  R grad[3][3];
  velocity_gradients<Q, S, R>(pops, g, shifted, ids, table, periodic, x, y, z, u, inward, grad);
  const R s_to_pi = -rho / R(3) / e->omega;
  R pi[6];
  pi[0] = R(2) * grad[0][0] * s_to_pi;
  pi[3] = R(2) * grad[1][1] * s_to_pi;
  pi[5] = R(2) * grad[2][2] * s_to_pi;
  pi[1] = (grad[0][1] + grad[1][0]) * s_to_pi;
  pi[2] = (grad[0][2] + grad[2][0]) * s_to_pi;
  pi[4] = (grad[1][2] + grad[2][1]) * s_to_pi;
  const R usqr = norm_sqr(u);
  R f[Q];
  static_for<0, Q>([&](auto i) { f[i] = feq2<L, i.value>(rho, u, usqr) + from_pi_to_fneq<L, i.value>(pi); });
  store_logical<Q, S, R>(pops, g, x, y, z, shifted, f);
}

// ---------------------------------------------------------------------------
// host-side launch entry points (explicitly instantiated per lattice/storage)

// Launch whose kernel may start before the stream's previous kernel has ended
// (it waits by after_previous); an ordinary launch when !chained.
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), bool chained, dim3 grid, dim3 block, cudaStream_t stream, A&&... args)
{
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, P(args)...);
}

struct StepLaunch {
  void* pops;
  Geometry g;
  const uint8_t* ids;      // device, or nullptr
  const void* table;       // device DynDevice<R>[]
  const void* bulk;        // host DynDevice<R>
  StatSink sink;           // partials: gridDim product entries (statistics only)
  bool chained = false;    // the previous work on the stream may be overlapped (launch_chained)
  int block_z, block_y;
  int variant;             // of the step kernel (running_variant)
  cudaStream_t stream;
};

template <int Q, class S, class R>
cudaError_t launch_step(const StepLaunch& a, int kind, bool odd, bool masked, bool stats);

template <int Q, class S, class R>
cudaError_t launch_gather(const void* pops, const Geometry& g, bool shifted, void* out, int i_begin,
                          int i_end, cudaStream_t stream);

template <int Q, class S, class R>
cudaError_t launch_scatter(void* pops, const Geometry& g, const void* in, int i_begin, int i_end,
                           cudaStream_t stream);

// every cell's populations from its density and velocity (rho_u: 4 columns of R)
template <int Q, class S, class R>
cudaError_t launch_equilibrium(void* pops, const Geometry& g, const void* rho_u, cudaStream_t stream);

template <int Q, class S, class R>
cudaError_t launch_moments(const void* pops, const Geometry& g, bool shifted, const uint8_t* ids,
                           const void* table, void* rho, void* u, cudaStream_t stream);

// the boundary pre-pass over `count` cells; sink.partials == nullptr: no statistics
template <int Q, class S, class R>
cudaError_t launch_boundary_collide(void* pops, const Geometry& g, bool shifted, const uint8_t* ids,
                                    const void* table, int kind, const uint32_t* cells, uint32_t count,
                                    const StatSink& sink, cudaStream_t stream);
constexpr int kBoundaryThreads = 128;

// the PostStream passes: cells[0, n_flat) are the interpolated flat cells
// (velocity pass, then PlaneFd), the next n_edge the external edge cells,
// the last n_corner the external corner cells
template <int Q, class S, class R>
cudaError_t launch_boundary(void* pops, const Geometry& g, bool shifted, const uint8_t* ids, const void* table,
                            int periodic, const uint32_t* cells, uint32_t n_flat, uint32_t n_edge,
                            uint32_t n_corner, cudaStream_t stream);

// grid of the step kernels: flat tiles, or rectangles of bz x (by * cells per thread)
inline dim3 step_grid(const Geometry& g, int bz, int by, int cells_per_thread)
{
  const unsigned planes = unsigned(g.paired ? g.nx / 2 : g.nx);
  if (g.flat) {
    const uint64_t tile = uint64_t(g.flat) * uint64_t(cells_per_thread);
    return dim3(unsigned((uint64_t(g.ny) * uint64_t(g.nz) + tile - 1) / tile), 1, planes);
  }
  const int rows = by * cells_per_thread;
  return dim3((g.nz + bz - 1) / bz, (g.ny + rows - 1) / rows, planes);
}

// Threads of a block of flat tiles, which every lattice takes unless the caller
// or the autotuner has fixed a launch shape.
//   Against rectangles: those leave lanes without cells when nz or ny is no
// multiple of theirs (0.58 of the lanes have cells at 191x173x150: 144 us
// against 125 with flat tiles for an FP32 cavity; 35 against 31 at 200x120x100
// FP16; 15.4 against 12.3 at 97x61x75), and at 256^3, where every lane is busy,
// flat tiles still gain 0.1 % to 3 % (FP32 402 us against 389: a block's loads
// are one contiguous run of every column).
//   Block size: the 16-bit kernels alternate between waiting for loads and
// bursts of arithmetic, and the warps of one block do so together; blocks of
// 64 threads (the same registers and warps per SM) mix the phases better:
// 256^3 D3Q27 BF16 Smagorinsky 389 -> 372 us (377 with 128 threads), D3Q27 BF16
// TRT 302 -> 292, D3Q19 FP16 212 -> 206, 384x192x192 FP16 forced TRT 228 -> 217.
// FP32 gains nothing from it (257^3 cavity 418 against 417 us with 128).
inline int flat_threads(int bytes) { return bytes == 2 ? 64 : kStepThreads; }

// What runs on a lattice when variant v is selected.
inline StepVariant running_variant(const Geometry& g, int bytes, int v)
{
  if (bytes == 2 && !g.paired && kSplitNatural16) {
    return split_variant(v) ? StepVariant{2, kSplitMinBlocks} : kStepVariants[0];
  }
  return step_variant(bytes, v);
}

inline dim3 step_block(const Geometry& g, int bz, int by)
{
  return g.flat ? dim3(g.flat, 1) : dim3(bz, by);
}

// the constants of floor(n / d) = (mulhi(n, mul) + n) >> shift for n < 2^31
inline void division_constants(uint32_t d, uint32_t& mul, uint32_t& shift)
{
  shift = 0;
  while ((uint64_t(1) << shift) < d) ++shift;
  mul = uint32_t(((uint64_t(1) << 32) * ((uint64_t(1) << shift) - d)) / d + 1);
}

// flat tiles of `threads` threads
inline void set_flat(Geometry& g, int threads)
{
  g.flat = threads;
  division_constants(uint32_t(g.nz), g.flat_mul, g.flat_shift);
}

// grid of the gather / moments kernels (one cell per thread)
inline dim3 cell_grid(const Geometry& g, int bz, int by)
{
  return dim3((g.nz + bz - 1) / bz, (g.ny + by - 1) / by, g.nx);
}

} // namespace olb_b200
