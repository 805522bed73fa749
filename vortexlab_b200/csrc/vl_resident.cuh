// The resident step kernel: many steps of one sim in one cooperative launch.
//
// A domain whose two population buffers stay in the L2 takes a few microseconds of memory traffic
// per step, less than the launches, the fork / join and the serial outlet sum of the two-kernel
// step cost. Here one block per SM stays on the chip for all the steps of a call and a grid-wide
// arrival counter separates them. Per step:
//
//   boundary tasks  8 to 32 boundary nodes with like links, a warp each, dealt out over the blocks: the
//                   loads of a column's nodes are a transaction each. The wall links of a task run one
//                   per lane from records whose coefficients the host has worked out (WallRec); then one
//                   lane per node takes the returning populations, collides and stores. The nodes' own
//                   populations stay in shared memory, and the part of the open-boundary rules that
//                   needs only them is worked out after the block has arrived. The outlet nodes have
//                   tasks and blocks of their own; there one warp sums the outlet velocities that the
//                   previous step left (sequentially, src/sim.rs:444-455) beside the tasks.
//   bulk            segments of 32 V cells of a row, taken by the block's other warps in turn.
//   one part        (kBlock threads of the last block) the force sums and history record of the step
//                   before the previous one, and the pressure probe of the previous step.
//
// The force terms of a task are formed after the block has arrived, per node in link order; that
// part sums them by the tree of k_links over the same chunks of kBlock nodes.
//
// Populations are read from the L2 (ld.global.cg: another block wrote them a step before). A block's
// stores are ordered before its arrival by the release; the counter is polled with relaxed loads, and a
// fence of GPU scope after the last of them, before the barrier that lets the block go on, makes the wait
// an acquire. The fence drops the L1, so what a block reads in every step (its tasks' tables, the control
// block, the chunks with force) is kept in its shared memory. us per step without the fence and with the
// tables in the L1 / with the fence / with the tables in shared memory: rig of 442 x 84 FP64 5.31 / 6.04 /
// 5.36, 1762 x 330 15.8 / 15.7 / 13.9, tank of 482 x 242 FP32 6.5 / 7.1 / 6.5, 1802 x 902 28.4 / 28.5 /
// 26.0, disk box of 700 x 450 FP64 9.4 / 10.1 / 8.5. Every value is computed by the functions of
// the two-kernel step in their order, so states, forces and records are bit-identical to it.
//
// Every wait is bounded (kWaitPolls polls); a block that gives up sets Ctl::stalled and the host's flag
// and leaves, and so do the blocks that wait for it and all blocks of later launches. The launch is
// cooperative: all blocks are on the chip at once.
#pragma once

#include "vl_device.cuh"
#include "vl_pair.cuh"

namespace vl {

constexpr unsigned kWaitPolls = 1u << 22;   // seconds
constexpr int kResidentThreads = 1024;      // 32 warps of 64 registers: enough loads in flight for the L2
constexpr int kResidentWarps = kResidentThreads / 32;
constexpr int kResidentTaskWarps = 16;      // the warps that take boundary tasks
constexpr int kResidentSumPart = 2;         // the part of the last block that sums the forces
constexpr int kResidentSmem = 160 * 1024;   // most dynamic shared memory of a block, and of one with its tables
constexpr int kResidentSmemTables = 200 * 1024;

// A wall link of a task: c1, c2 are the coefficients of its rule (link_back: 0.5 / q and 1 - 0.5 / q, or
// 2 q and 1 - 2 q), worked out in the arithmetic type; `behind` the population a[j][behind] of the near
// rule.
enum : unsigned { WALL_FAR = 0, WALL_NEAR = 1, WALL_HALF = 2 };   // q >= 1/2; q < 1/2; no node behind
struct alignas(16) WallRec {
  unsigned behind;
  unsigned slot;                // (j - 1) * 32 + lane of its node
  unsigned meta;                // type | vgroup << 2
  unsigned pad0;
  double c1, c2;
  double cu6, pad1;
};

enum : int { TASK_WALL = 0, TASK_OPEN = 1, TASK_OUTLET = 2 };   // nodes with wall links only; with open links

constexpr unsigned kOutletIndex = (1u << 28) - 1u;

struct ResidentParams {
  int steps;
  int grid;
  const int32_t* seg_first;     // [grid + 1] first row segment of each block
  const int32_t* task_first;    // [grid + 1] first task of each block
  int segs_per_row;             // segments of 32 V cells
  // Per task and lane {cell or -1; link directions j: wall 1 << j, open 1 << (j + 9), and with force or (an
  // outlet node) pressure 1 << (j + 18); first link in `links`; rank in the boundary-node list, or index in the outlet
  // list and the normal's components + 1 << 28 and << 30}.
  const int4* nodes;
  // with a cell at the grid's edge: x = 0 1 << 27, x = nx - 1 1 << 28, y = 0 1 << 29, y = ny - 1 1 << 30
  const WallRec* walls;
  const int4* tasks;            // {first wall record, end, kind, end of its nodes' records in `links`}
  const void* links;            // LinkRecDev[]: the links of the nodes with open links or force, by task and node
  const int32_t* block_outlets; // outlet tasks of each block
  int max_tasks;                // most tasks of a block
  int max_walls, max_links;     // most wall records and records of `links` of a block
  int tables;                   // the block's tasks, nodes, wall and link records are copied to its shared memory
  const int32_t* force_chunks;  // chunks that hold a node with force
  int nforce;
  volatile int* host_stalled;   // in host memory: set with Ctl::stalled
  unsigned* arrived;            // arrivals since the sim was built
  unsigned arrived0;            // arrivals before this launch
  double* node_force;           // three sets of [2 * ngroups][nbs], zero for nodes without force
  double* un;                   // two sets of the outlet nodes' normal velocities
  double* drho;                 // [3]
};

// Dynamic shared memory: the outlet velocities, then per task of the block (by lane of the node) the
// returning populations of the links by direction j - 1, for an open link the part of it that needs no
// outlet offset, and the nodes' own populations before and after the step (by its parity).
template <class R>
struct TaskScratch {
  R back[8][32];
  R open[8][32];
  R own[2][9][32];
};

// The tables' part of it: nodes, tasks, wall and link records of a block.
inline size_t resident_table_bytes(const ResidentParams& r) {
  return (size_t)r.max_tasks * 33 * sizeof(int4) + (size_t)r.max_walls * sizeof(WallRec) +
         (size_t)r.max_links * sizeof(LinkRecDev);
}
// n records of a global table to shared memory, by the block.
template <class T>
__device__ __forceinline__ const T* copy_table(uint4*& at, const T* src, int n) {
  constexpr int kWords = sizeof(T) / sizeof(uint4);
  static_assert(sizeof(T) % sizeof(uint4) == 0, "copied in 16-byte words");
  const uint4* q = reinterpret_cast<const uint4*>(src);
  for (int k = (int)threadIdx.x; k < n * kWords; k += kResidentThreads) at[k] = __ldg(q + k);
  const T* out = reinterpret_cast<const T*>(at);
  at += n * kWords;
  return out;
}

// Where a block finds its tables (kept in shared memory: pointers held over the steps would be spilled, and
// the acquire drops the spilled lines too).
struct BlockTables {
  const int4* nodes;            // of its first task
  const int4* tasks;
  const WallRec* walls;
  const LinkRecDev* links;
  int ntasks;
};

// One part of a block.
struct PartOf {
  int part;
  __device__ __forceinline__ int tid() const { return (int)threadIdx.x & (kBlock - 1); }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(1 + part), "r"(kBlock) : "memory"); }
};

__device__ __forceinline__ void grid_arrive(unsigned* counter) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}

// Waits (one thread of the block) until `target` arrivals have been counted. The polls are relaxed; the fence
// behind the last one makes it an acquire of the other blocks' releases, and the barrier after it (in the
// caller) orders the block's loads behind it.
__device__ __forceinline__ bool poll_arrived(const unsigned* counter, unsigned target) {
  for (unsigned k = 0; k < kWaitPolls; ++k) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
    if ((int)(v - target) >= 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      return true;
    }
  }
  return false;
}

// A wait ran out (one thread of each block that gives up).
__device__ __forceinline__ void mark_stalled(const StepParams& p, const ResidentParams& r) {
  *(volatile int*)&p.ctl->stalled = 1;
  *r.host_stalled = 1;
  __threadfence_system();
}

// The named barrier between a block's summing warp and its outlet tasks' warps.
__device__ __forceinline__ void outlet_sum_ready(int tasks) {
  asm volatile("bar.arrive 8, %0;" ::"r"(32 * (1 + tasks)) : "memory");
}
__device__ __forceinline__ void outlet_sum_wait(int tasks) {
  asm volatile("bar.sync 8, %0;" ::"r"(32 * (1 + tasks)) : "memory");
}

// The pull of a boundary node (pull) with its wraps from the node's flags.
template <class S>
__device__ __forceinline__ void pull_node(const S* a, unsigned ns, int nx, int ny, unsigned cell, int flags,
                                          typename Store<S>::R* f) {
  const unsigned up = (flags >> 29) & 1 ? (unsigned)((ny - 1) * nx) : (unsigned)-nx;         // row y - 1
  const unsigned dn = (flags >> 30) & 1 ? (unsigned)-((ny - 1) * nx) : (unsigned)nx;         // row y + 1
  const unsigned xm = (flags >> 27) & 1 ? (unsigned)(nx - 1) : (unsigned)-1;
  const unsigned xp = (flags >> 28) & 1 ? (unsigned)(1 - nx) : 1u;
  f[0] = Store<S>::ld_cg(a + cell, 0);
  f[1] = Store<S>::ld_cg(a + 1u * ns + (cell + xm), 1);
  f[2] = Store<S>::ld_cg(a + 2u * ns + (cell + up), 2);
  f[3] = Store<S>::ld_cg(a + 3u * ns + (cell + xp), 3);
  f[4] = Store<S>::ld_cg(a + 4u * ns + (cell + dn), 4);
  f[5] = Store<S>::ld_cg(a + 5u * ns + (cell + up + xm), 5);
  f[6] = Store<S>::ld_cg(a + 6u * ns + (cell + up + xp), 6);
  f[7] = Store<S>::ld_cg(a + 7u * ns + (cell + dn + xp), 7);
  f[8] = Store<S>::ld_cg(a + 8u * ns + (cell + dn + xm), 8);
}

// Normal velocity of an outlet node from its populations as stored (outlet_offset).
__device__ __forceinline__ double outlet_velocity(const double* f, const StepParams& p, int nx, int ny) {
  double rho, jx, jy;
  moments(f, rho, jx, jy);
  const double ux = jx / rho - 0.5 * p.gx, uy = jy / rho - 0.5 * p.gy;
  return (double)nx * ux + (double)ny * uy;
}

// What a task's open links return, as far as it follows from the nodes' own populations (link_back): of
// a radiating link everything, of a pressure link the factor 1 + cu^2 / 2 - 1.5 u^2 and the link's density.
template <class S>
__device__ __forceinline__ void open_prepare(const StepParams& p, const LinkRecDev* links, const int4& nd, int kind,
                                             int parity, TaskScratch<typename Store<S>::R>& t) {
  using R = typename Store<S>::R;
  const int lane = (int)(threadIdx.x & 31u);
  if (nd.x < 0 || !((nd.y >> 9) & 0x1ff)) return;
  R own[9];
#pragma unroll
  for (int d = 0; d < 9; ++d) own[d] = t.own[parity][d][lane];
  R rho, jx, jy;
  moments(own, rho, jx, jy);
  const R ux = jx / rho - R(0.5) * (R)p.gx, uy = jy / rho - R(0.5) * (R)p.gy;
  const unsigned all = ((unsigned)nd.y | ((unsigned)nd.y >> 9)) & 0x1ffu;
#pragma unroll
  for (int j = 1; j < 9; ++j) {
    if (!((nd.y >> (j + 9)) & 1)) continue;
    const R cu = R(3.0) * ((R)cx_of(j) * ux + (R)cy_of(j) * uy);
    R g = R(1.0) + R(0.5) * cu * cu - R(1.5) * (ux * ux + uy * uy);
    const int4 w = *(reinterpret_cast<const int4*>(links + nd.z + __popc(all & ((1u << j) - 1u))) + 2);
    const R lrho = (R)__hiloint2double(w.y, w.x);
    if (kind == TASK_OUTLET && ((nd.y >> (j + 18)) & 1)) {
      t.back[j - 1][lane] = lrho;
    } else {
      const int flags = (int)(((unsigned)w.w >> 8) & 0xffu);
      const R nxv = (R)((int)((flags >> 2) & 3) - 1), nyv = (R)((int)((flags >> 4) & 3) - 1);
      const R rho_w = lrho + (nxv * ux + nyv * uy) / (R)p.sqrt_cs2;
      g = -own[j] + R(2.0) * (R)w_of(j) * rho_w * g;
    }
    t.open[j - 1][lane] = g;
  }
}

// One task of a warp: its boundary nodes updated. walls: the records, by td's indices; vs: the step's wall
// speeds; parity: the step's; outlets: the outlet tasks of the block that wait for *s_drho (an outlet task;
// 0: no target); un_new: the outlet velocities after the step.
template <class S, int CK>
__device__ __forceinline__ void boundary_task(const StepParams& p, const int4& nd, const int4& td,
                                              const WallRec* walls, const S* a, S* b, const double* vs, int parity,
                                              int outlets, const double* s_drho, double* un_new,
                                              TaskScratch<typename Store<S>::R>& t) {
  using R = typename Store<S>::R;
  const int lane = (int)(threadIdx.x & 31u);
  const unsigned cell = (unsigned)nd.x;
  R f[9];
  if (nd.x >= 0) pull_node(a, p.ns, p.nx, p.ny, cell, nd.y, f);
  const R* own = &t.own[parity][0][0];
  constexpr int U = 3;                                          // links of a lane in flight
  for (int base = td.x + lane; base < td.y; base += U * 32) {
    R bval[U];
    unsigned slot[U], meta[U];
#pragma unroll
    for (int m = 0; m < U; ++m) {
      const int l = base + m * 32;
      if (l < td.y) {
        const uint4 w = *reinterpret_cast<const uint4*>(walls + l);
        slot[m] = w.y;
        meta[m] = w.z;
        if ((w.z & 3u) == WALL_NEAR) bval[m] = Store<S>::ld_cg(a + w.x, (int)(w.y / 32) + 1);
      }
    }
#pragma unroll
    for (int m = 0; m < U; ++m) {
      const int l = base + m * 32;
      if (l < td.y) {
        const double2 cc = *(reinterpret_cast<const double2*>(walls + l) + 1);
        const R corr = (R)walls[l].cu6 * (R)vs[(meta[m] >> 2) & 3u];
        const unsigned type = meta[m] & 3u;
        const int j = (int)(slot[m] / 32) + 1, node = (int)(slot[m] & 31u);
        const R out = own[j * 32 + node];
        const R x3 = type == WALL_NEAR ? bval[m] : own[opp_of(j) * 32 + node];
        R back = type == WALL_NEAR ? out : out - corr;
        if (type != WALL_HALF) back = (R)cc.x * back + (R)cc.y * x3;
        if (type == WALL_NEAR) back = back - corr;
        t.back[j - 1][node] = back;
      }
    }
  }
  double drho = 0.0;
  __syncwarp();
  if (outlets > 0) {
    outlet_sum_wait(outlets);
    drho = *s_drho;
  }
  if (nd.x < 0) return;
  if (td.z != TASK_WALL) {
#pragma unroll
    for (int j = 1; j < 9; ++j) {
      if ((nd.y >> (j + 9)) & 1) {
        R back = t.open[j - 1][lane];
        if (td.z == TASK_OUTLET && ((nd.y >> (j + 18)) & 1)) {
          const R rho_w = t.back[j - 1][lane] + (R)drho;        // (open_prepare left the link's density here)
          back = -own[j * 32 + lane] + R(2.0) * (R)w_of(j) * rho_w * back;
        }
        f[opp_of(j)] = back;
      }
    }
  }
#pragma unroll
  for (int j = 1; j < 9; ++j)
    if ((nd.y >> j) & 1) f[opp_of(j)] = t.back[j - 1][lane];
  collide_s<S>(f, CK, (R)p.op, (R)p.om, (R)p.gx, (R)p.gy);
#pragma unroll
  for (int i = 0; i < 9; ++i) Store<S>::st(b + (unsigned)i * p.ns + cell, i, f[i]);
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i] = Store<S>::rt(i, f[i]);
  if (td.z == TASK_OUTLET) {
    double fd[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) fd[i] = (double)f[i];
    const unsigned w = (unsigned)nd.w;
    __stcg(un_new + (w & kOutletIndex), outlet_velocity(fd, p, (int)((w >> 28) & 3u) - 1, (int)(w >> 30) - 1));
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) t.own[parity ^ 1][i][lane] = f[i];
}

// The force terms of a task's nodes, per node in link order (after boundary_task).
template <class S>
__device__ __forceinline__ void task_force(const StepParams& p, const LinkRecDev* links, const int4& nd,
                                           const double* vs, int parity, double* node_force, const TaskScratch<typename Store<S>::R>& t) {
  using R = typename Store<S>::R;
  const int lane = (int)(threadIdx.x & 31u);
  const unsigned fm = ((unsigned)nd.y >> 18) & 0x1ffu;
  if (nd.x < 0 || !fm) return;
  const unsigned all = ((unsigned)nd.y | ((unsigned)nd.y >> 9)) & 0x1ffu;
  double acc[2 * kMaxGroups];
#pragma unroll
  for (int k = 0; k < 2 * kMaxGroups; ++k) acc[k] = 0.0;
  for (int j = 1; j < 9; ++j) {
    if (!((fm >> j) & 1u)) continue;
    const int4* rec = reinterpret_cast<const int4*>(links + nd.z + __popc(all & ((1u << j) - 1u)));
    const LinkView L = link_view(rec[0], rec[1], rec[2]);
    double tx, ty;
    force_terms(L, (double)t.own[parity][j][lane], (double)t.back[j - 1][lane], (double)(R)vs[L.vgroup], tx, ty);
#pragma unroll
    for (int g = 0; g < kMaxGroups; ++g) {
      if (g == L.fgroup) {
        acc[2 * g] += tx;
        acc[2 * g + 1] += ty;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 2 * kMaxGroups; ++k)
    if (k < 2 * p.ngroups) __stcg(node_force + (size_t)k * p.nbs + nd.w, acc[k]);
}

// Force sums and history record of step t by one part: per chunk with force the tree of
// block_force_partial (a warp per chunk: kBlock / 32 groups of 32 nodes, then the groups in order), then
// the tree of sum_partials by one warp per component (at most kBlock chunks). s_part[component][chunk] is
// zero for the other chunks.
template <class S>
__device__ __forceinline__ void resident_epilogue(const StepParams& p, const ResidentParams& r, unsigned long long t,
                                                  int slot, bool final_step, double (*s_part)[kBlock], double* s_force,
                                                  const int* s_chunks, const Ctl* k0, const PartOf& me) {
  Ctl* c = p.ctl;                                               // (read in the copy k0, but for `nonfinite`)
  const int tid = me.tid(), lane = tid & 31, warp = tid >> 5;
  const int ncomp = 2 * p.ngroups;
  const double* nf = r.node_force + (size_t)slot * ncomp * p.nbs;
  for (int q = warp; q < r.nforce * ncomp; q += kBlock / 32) {
    const int ch = s_chunks[q / ncomp], k = q % ncomp;
    double v[kBlock / 32];
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) {
      const int g = ch * kBlock + w * 32 + lane;
      v[w] = g < p.nb ? __ldcg(nf + (size_t)k * p.nbs + g) : 0.0;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int w = 0; w < kBlock / 32; ++w) v[w] += __shfl_down_sync(0xffffffffu, v[w], off);
    }
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) sum += v[w];
    if (lane == 0) s_part[k][ch] = sum;
  }
  me.sync();
  if (warp < ncomp) {
    double v[kBlock / 32];
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) v[w] = s_part[warp][w * 32 + lane];
#pragma unroll
    for (int h = kBlock / 64; h > 0; h >>= 1) {
#pragma unroll
      for (int w = 0; w < h; ++w) v[w] += v[w + h];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], off);
    if (lane == 0) s_force[warp] = v[0];
  }
  me.sync();
  if (tid == 0) {
    const int has_target = k0->sched_on ? k0->absorbing : k0->has_target;
    const double drho = p.np > 0 && has_target ? __ldcg(r.drho + slot) : 0.0;
    bool finite = true;
    for (int k = 0; k < ncomp; ++k) finite = finite && isfinite(s_force[k]);
    if (!finite && !c->nonfinite) {
      c->nonfinite = 1;
      c->nonfinite_t = t;
    }
    if (k0->rec_cap && t >= k0->rec_start && t - k0->rec_start < k0->rec_cap) {
      double* h = k0->hist + (size_t)(t - k0->rec_start) * kRec;
      for (int k = 0; k < 2 * kMaxGroups; ++k) h[k] = k < ncomp ? s_force[k] : 0.0;
      h[8] = drho;
      if (!k0->dp_on) h[9] = 0.0;                               // else the probe, one step before this
    }
    if (final_step) {
      for (int k = 0; k < 2 * kMaxGroups; ++k) c->force[k] = k < ncomp ? s_force[k] : 0.0;
      c->drho = drho;
      if (k0->sched_on) {
        const Controls k = read_controls(k0, t);
        c->vscale[1] = k.vs[1];
        c->vscale[2] = k.vs[2];
        c->target = k.target;
        c->has_target = k.has_target;
      }
      c->t = t + 1;
    }
  }
  me.sync();
}

template <class S, int V, int CK>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident(const __grid_constant__ StepParams p,
                                                                  const __grid_constant__ ResidentParams r, S* buf0,
                                                                  S* buf1) {
  using R = typename Store<S>::R;
  __shared__ double s_part[2 * kMaxGroups][kBlock];             // the last part's chunk sums
  __shared__ double s_force[2 * kMaxGroups];
  __shared__ double s_vs[2][4];                                 // by parity of the step
  __shared__ double s_target[2];
  __shared__ unsigned long long s_t;
  __shared__ int s_next[2];                                     // next segment of the block, by parity
  __shared__ int s_go;
  __shared__ double s_drho;
  __shared__ int s_chunks[kBlock];                              // the last part's chunks with force
  __shared__ Ctl s_ctl;                                         // the control block at the start
  __shared__ BlockTables s_tab;
  extern __shared__ double s_dyn[];
  const int bid = (int)blockIdx.x, lane = (int)(threadIdx.x & 31u), warp = (int)threadIdx.x >> 5;
  Ctl* c = p.ctl;
  // An earlier launch gave up (one thread reads the flag: the block leaves as one).
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)&c->stalled)) return;
  const unsigned long long t0 = c->t;
  const int seg0 = __ldg(r.seg_first + bid), seg1 = __ldg(r.seg_first + bid + 1);
  const int task0 = __ldg(r.task_first + bid), task1 = __ldg(r.task_first + bid + 1);
  const PartOf me{(int)threadIdx.x / kBlock};
  const bool last = bid == r.grid - 1 && me.part == kResidentSumPart;
  const int has_target = c->sched_on ? c->absorbing : c->has_target;
  double* s_un = s_dyn;                                         // the summing warp's outlet velocities
  TaskScratch<R>* scratch = (TaskScratch<R>*)(s_dyn + (p.np + 1) / 2 * 2);
  const int outlets = has_target ? __ldg(r.block_outlets + bid) : 0;
  // The block's tasks, their nodes, wall and link records: copied to shared memory where they fit (the acquire
  // of every step drops the L1, and a task would begin with a chain of L2 loads).
  {
    const int4 *nodes = r.nodes + (size_t)task0 * 32, *tds = r.tasks + task0;
    const WallRec* walls = r.walls;
    const LinkRecDev* links = (const LinkRecDev*)r.links;
    if (r.tables && task1 > task0) {
      const int w0 = __ldg(&tds[0].x), w1 = __ldg(&r.tasks[task1 - 1].y);
      const int l0 = task0 > 0 ? __ldg(&tds[-1].w) : 0, l1 = __ldg(&r.tasks[task1 - 1].w);
      uint4* at = (uint4*)(scratch + r.max_tasks);
      nodes = copy_table(at, nodes, (task1 - task0) * 32);
      tds = copy_table(at, tds, task1 - task0);
      walls = copy_table(at, walls + w0, w1 - w0) - w0;         // (indexed as the whole tables are)
      links = copy_table(at, links + l0, l1 - l0) - l0;
    }
    if (threadIdx.x == 0) s_tab = {nodes, tds, walls, links, task1 - task0};
  }
  const size_t force_set = (size_t)2 * p.ngroups * p.nbs;

  static_assert(sizeof(Ctl) % 8 == 0, "copied in 8-byte words");
  for (int k = (int)threadIdx.x; k < (int)(sizeof(Ctl) / 8); k += kResidentThreads)
    ((unsigned long long*)&s_ctl)[k] = ((const unsigned long long*)c)[k];
  if (last)
    for (int k = me.tid(); k < r.nforce; k += kBlock) s_chunks[k] = __ldg(r.force_chunks + k);

  // controls of step s into shared memory (one thread)
  auto controls = [&](int s, const Ctl* c) {
    const Controls k = read_controls(c, t0 + (unsigned long long)s);
#pragma unroll
    for (int g = 0; g < 4; ++g) s_vs[s & 1][g] = k.vs[g];
    s_target[s & 1] = k.target;
    s_t = t0 + (unsigned long long)s;
    s_next[s & 1] = seg0;
  };

  if (threadIdx.x == 0) controls(0, c);
  for (int k = (int)threadIdx.x; k < 2 * kMaxGroups * kBlock; k += kResidentThreads) (&s_part[0][0])[k] = 0.0;
  // Outlet velocities of the start state, in the shared memory of every block that sums them: no grid-wide
  // wait is needed before the first step, and no two blocks write a word.
  for (int k = (int)threadIdx.x; outlets > 0 && k < p.np; k += kResidentThreads) {
    const int idx = __ldg(p.pnode_idx + k);
    double f[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = (double)Store<S>::ld_cg(buf0 + (size_t)i * p.ns + idx, i);
    s_un[k] = outlet_velocity(f, p, p.pnode_n[2 * k], p.pnode_n[2 * k + 1]);
  }
  // The nodes' own populations in the start state.
  if (warp < kResidentTaskWarps) {
    for (int task = task0 + warp; task < task1; task += kResidentTaskWarps) {
      const int4 nd = __ldg(r.nodes + (size_t)task * 32 + lane);
      TaskScratch<R>& t = scratch[task - task0];
      if (nd.x >= 0) {
#pragma unroll
        for (int d = 0; d < 9; ++d) t.own[0][d][lane] = Store<S>::ld_cg(buf0 + (unsigned)d * p.ns + (unsigned)nd.x, d);
      }
      open_prepare<S>(p, (const LinkRecDev*)r.links, nd, __ldg(r.tasks + task).z, 0, t);
    }
  }
  __syncthreads();

  unsigned target = r.arrived0;
  int slot = 0;                                                 // step s: slot s % 3
  for (int s = 0; s < r.steps; ++s) {
    const S* a = (s & 1) ? buf1 : buf0;
    S* b = (s & 1) ? buf0 : buf1;
    const int slot2 = slot == 2 ? 0 : slot + 1;                 // (s - 2) % 3

    if (last) {
      if (s > 0) record_probe<S>(p, a, (long long)(t0 + s) - 1, &s_ctl, me);
      if (s > 1) resident_epilogue<S>(p, r, t0 + s - 2, slot2, false, s_part, s_force, s_chunks, &s_ctl, me);
    } else if (warp < kResidentTaskWarps) {
      for (int task = warp; task < s_tab.ntasks; task += kResidentTaskWarps) {
        const int4 nd = s_tab.nodes[task * 32 + lane], td = s_tab.tasks[task];
        boundary_task<S, CK>(p, nd, td, s_tab.walls, a, b, s_vs[s & 1], s & 1, td.z == TASK_OUTLET ? outlets : 0, &s_drho,
                             r.un + ((s & 1) ^ 1) * p.np, scratch[task]);
        __syncwarp();
      }
    } else if (outlets > 0 && warp == kResidentWarps - 1) {
      const double* un = r.un + (s & 1) * p.np;
      for (int base = 0; s > 0 && base < p.np; base += 16 * 32) {   // 16 loads of a lane in flight
        double v[16];
#pragma unroll
        for (int m = 0; m < 16; ++m)
          if (base + m * 32 + lane < p.np) v[m] = __ldcg(un + base + m * 32 + lane);
#pragma unroll
        for (int m = 0; m < 16; ++m)
          if (base + m * 32 + lane < p.np) s_un[base + m * 32 + lane] = v[m];
      }
      __syncwarp();
      const double drho = (serial_sum(s_un, p.np) / (double)p.np - s_target[s & 1]) / p.sqrt_cs2;
      if (lane == 0) {
        s_drho = drho;
        if (bid == 0) __stcg(r.drho + slot, drho);              // (block 0 has outlet tasks if any block has)
      }
      __syncwarp();
      outlet_sum_ready(outlets);
    }

    while (true) {
      int sg = 0;
      if (lane == 0) sg = atomicAdd(&s_next[s & 1], 1);
      sg = __shfl_sync(0xffffffffu, sg, 0);
      if (sg >= seg1) break;
      const int y = sg / r.segs_per_row;
      const int xw = (sg - y * r.segs_per_row) * (32 * V);
      if constexpr (V > 1) {
        PairTask q;
        q.nx = p.nx;
        q.ny = p.ny;
        q.y = y;
        q.xw = xw;
        q.ns = p.ns;
        q.flag = p.flag;
        q.ck = CK;
        q.op = (float)p.op;
        q.om = (float)p.om;
        q.bad = &c->nonfinite;
        q.bad_t = &c->nonfinite_t;
        q.t_now = &s_t;
        group_update<S, V, 0, 1>(q, a, b);
      } else {
        const int x = xw + lane;
        if (x < p.nx) {
          const unsigned idx = (unsigned)(y * p.nx + x);
          const uint8_t fl = __ldg(p.flag + idx);
          R f[9];
          pull<S, 1>(a, p.ns, p.nx, p.ny, x, y, f);
          if (fl == 0) {
            collide_s<S>(f, CK, (R)p.op, (R)p.om, (R)p.gx, (R)p.gy);
            if (Saturates<S>::value && !density_plausible(f)) mark_diverged(&c->nonfinite, &c->nonfinite_t, &s_t);
#pragma unroll
            for (int i = 0; i < 9; ++i) Store<S>::st(b + (unsigned)i * p.ns + idx, i, f[i]);
          }
        }
      }
    }

    grid_arrive(r.arrived);
    target += (unsigned)r.grid;
    // After the arrival (the block has synchronised: the step's controls and counter are free).
    if (warp < kResidentTaskWarps) {
      for (int task = warp; task < s_tab.ntasks; task += kResidentTaskWarps) {
        const int4 nd = s_tab.nodes[task * 32 + lane];
        const int kind = s_tab.tasks[task].z;
        TaskScratch<R>& t = scratch[task];
        if (kind == TASK_OUTLET || kind == TASK_OPEN) open_prepare<S>(p, s_tab.links, nd, kind, (s & 1) ^ 1, t);
        if (kind != TASK_OUTLET) task_force<S>(p, s_tab.links, nd, s_vs[s & 1], s & 1, r.node_force + slot * force_set, t);
      }
    }
    if (threadIdx.x == kResidentThreads - 32) controls(s + 1, &s_ctl);
    if (threadIdx.x == kResidentThreads - 64) s_go = poll_arrived(r.arrived, target);
    __syncthreads();
    if (!s_go) {
      if (threadIdx.x == 0) mark_stalled(p, r);
      return;
    }
    slot = slot2;
  }
  // The force terms of the last step are complete after one more arrival.
  grid_arrive(r.arrived);
  target += (unsigned)r.grid;
  if (bid != r.grid - 1) return;
  if (threadIdx.x == 0) s_go = poll_arrived(r.arrived, target);
  __syncthreads();
  if (!s_go && threadIdx.x == 0) mark_stalled(p, r);
  if (!s_go || !last) return;
  record_probe<S>(p, (r.steps & 1) ? buf1 : buf0, (long long)(t0 + r.steps) - 1, &s_ctl, me);
  if (r.steps > 1)
    resident_epilogue<S>(p, r, t0 + r.steps - 2, slot == 2 ? 0 : slot + 1, false, s_part, s_force, s_chunks, &s_ctl, me);
  resident_epilogue<S>(p, r, t0 + r.steps - 1, slot == 0 ? 2 : slot - 1, true, s_part, s_force, s_chunks, &s_ctl, me);
}

}  // namespace vl
