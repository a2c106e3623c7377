// rg_team.cuh - what the persistent step kernels (rg_nsc.cu, rg_verlet.cu)
// share: teams of co-resident blocks, their bounded barriers, scans and phase
// clocks, and the neighbour-list rebuild of one system by its team.
#pragma once
#include "rg_nsc_dev.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// Teams and team barriers.
// ---------------------------------------------------------------------------
struct Team {
  int b0, nb;
  unsigned int* bar;      // 4 barrier words, then the residual ring
  int* err;
  long long spin_limit;   // polls per barrier wait before ERR_TIMEOUT
  unsigned int absent;    // test hook: blocks the barriers wait for in vain
  __device__ int rank() const { return (int)blockIdx.x - b0; }
  __device__ int tid() const { return rank() * (int)blockDim.x + (int)threadIdx.x; }
  __device__ int size() const { return nb * (int)blockDim.x; }
  // residuals of the split solve's chunks: three buffers of kChunk, zero at
  // the start of a launch
  __device__ double* ring() const { return reinterpret_cast<double*>(bar + 4); }
};

// Barrier of the whole team.  The arrivals are counted, never reset: barrier k
// of a launch is over when the count reaches (k + 1) times the blocks, so a
// block needs one atomic and then only reads (the sense-reversing grid_sync
// also reads the generation and the error word first, each a round trip to
// L2).  The count starts at zero (memset before the launch) and every block
// keeps k in shared memory (team_barriers_reset at kernel start).  Bounded
// like grid_sync.  Measured
// with 148 blocks, waits for slower blocks included: 3.0 -> 1.9 us.
static __shared__ unsigned team_barrier_k;
__device__ inline void team_barriers_reset() {
  if (threadIdx.x == 0) team_barrier_k = 0;
  __syncthreads();
}
__device__ inline bool team_sync(const Team& T) {
  __syncthreads();
  const unsigned nb = (unsigned)T.nb + T.absent;
  if (nb <= 1) return !(*(volatile int*)T.err & ERR_TIMEOUT);
  int ok = 1;
  if (threadIdx.x == 0) {
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> count(*T.bar);
    const unsigned target = (++team_barrier_k) * nb;  // modulo 2^32, as the count
    count.fetch_add(1u, cuda::memory_order_release);
    long long it = 0;
    while ((int)(count.load(cuda::memory_order_acquire) - target) < 0) {
      ++it;
      if ((it & 63) == 0 && (*(volatile int*)T.err & ERR_TIMEOUT)) { ok = 0; break; }
      if (it > T.spin_limit) {
        atomicOr(T.err, ERR_TIMEOUT);
        ok = 0;
        break;
      }
      if (it > 256) __nanosleep(32);
    }
  }
  return __syncthreads_and(ok) != 0;
}
// Barrier among the first nsub blocks of the team (the others must not call it).
__device__ inline bool team_sync_sub(const Team& T, int nsub) {
  GridBar g{T.bar + 2, T.bar + 3, T.err, T.spin_limit, T.absent};
  return grid_sync(g, (unsigned)nsub);
}

__device__ inline double block_reduce_max(double v, double* sm) {
  v = warp_max(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
  if (threadIdx.x < 32) r = warp_max(r);
  return r;  // valid in thread 0
}
__device__ inline int block_reduce_sum_i(int v, int* sm) {
  v = warp_sum_i(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  int r = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0;
  if (threadIdx.x < 32) r = warp_sum_i(r);
  return r;  // valid in thread 0
}

// Phase timers (team rank 0, thread 0; %globaltimer in ns) when enabled.
// ---------------------------------------------------------------------------
__device__ inline unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
struct PhaseClock {
  Ctl* ctl;
  bool on;
  unsigned long long t;
  __device__ PhaseClock(Ctl* c, bool enabled) : ctl(c), on(enabled), t(enabled ? gtimer() : 0) {}
  __device__ void mark(int k) {
    if (!on) return;
    unsigned long long u = gtimer();
    ctl->phase_ns[k] += (long long)(u - t);
    t = u;
  }
};

// Dynamic shared memory of the persistent kernels: the list-build tiles while
// a rebuild runs (NSC: the small-solve arrays at other times).
extern __shared__ __align__(16) unsigned char team_dyn_smem[];
// list-build candidate queues, after the tiles
constexpr int kBuildQ = 4096;
constexpr size_t kBuildQOff = (sizeof(BuildSmem) + 15) & ~(size_t)15;

struct SmemNsc {
  double red_d[32];
  int red_i[32];
  int scan_w[32];
  int pre[32];
  int coff[kMaxColors + 1];
  int bcast;
};

// Every block computes Σ blk[0..rank) and Σ blk[0..nb).
__device__ inline void block_prefix(const int* blk, int nb, int rank, int& prefix, int& total, SmemNsc& sm) {
  int a = 0, b = 0;
  for (int r = threadIdx.x; r < nb; r += blockDim.x) {
    int v = *(volatile const int*)&blk[r];
    b += v;
    if (r < rank) a += v;
  }
  int pa = warp_sum_i(a), pb = warp_sum_i(b);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    sm.pre[threadIdx.x >> 5] = pa;
    sm.red_i[threadIdx.x >> 5] = pb;
  }
  __syncthreads();
  int x = 0, y = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    x += sm.pre[w];
    y += sm.red_i[w];
  }
  prefix = x;
  total = y;
  __syncthreads();
}

// Exclusive scan of in[0..m) into out[0..m], out[m] = total (team, blocked).
__device__ inline bool team_excl_scan(const Team& T, const int* in, int* out, int m, int* blk, SmemNsc& sm) {
  const int rank = T.rank();
  const int seg = (m + T.nb - 1) / T.nb;
  const int lo = rank * seg < m ? rank * seg : m;
  const int hi = lo + seg < m ? lo + seg : m;
  int s = 0;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) s += in[i];
  int bsum = block_reduce_sum_i(s, sm.red_i);
  if (threadIdx.x == 0) blk[rank] = bsum;
  if (!team_sync(T)) return false;
  int prefix, total;
  block_prefix(blk, T.nb, rank, prefix, total, sm);
  int run = prefix;
  for (int base = lo; base < hi; base += blockDim.x) {
    int i = base + threadIdx.x;
    int v = i < hi ? in[i] : 0;
    int tot;
    int ex = block_excl_scan(v, sm.scan_w, tot);
    if (i < hi) out[i] = run + ex;
    run += tot;
  }
  if (rank == 0 && threadIdx.x == 0) out[m] = total;
  return team_sync(T);
}

// ---------------------------------------------------------------------------
// Detection inside the persistent kernel.
// ---------------------------------------------------------------------------
// Rods in the 27 cells about cell c, a row of three at a time (the wrap along x
// left out: an estimate).
static __device__ inline int cells_around(const GridDev& g, const Box& box, const int* cell_start, int c) {
  const int cx = c % g.n[0], cy = (c / g.n[0]) % g.n[1], cz = c / (g.n[0] * g.n[1]);
  const int x0 = max(cx - 1, 0), x1 = min(cx + 2, g.n[0]);
  int sum = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int y = cy + dy, z = cz + dz;
      if (box.pbc) {
        y = (y + g.n[1]) % g.n[1];
        z = (z + g.n[2]) % g.n[2];
      } else if (y < 0 || z < 0 || y >= g.n[1] || z >= g.n[2]) {
        continue;
      }
      const int row = (z * g.n[1] + y) * g.n[0];
      sum += cell_start[row + x1] - cell_start[row + x0];
    }
  return sum;
}

// The pairs of a team's cells, each block its share; those without rods are
// passed over a word of cells at a time (one after the other, 0.5 us each).
static __device__ RG_BUILD_INLINE void build_cells(const Team& T, const NscView& V, const GridDev& g,
                                                   const double* invL, SmemNsc& sm, int& overflow) {
  const int rank = T.rank(), lane = threadIdx.x & 31, nwarp = (int)(blockDim.x >> 5);
  for (int first = rank; first < g.ncells; first += (int)blockDim.x * T.nb) {
    const int c = first + (int)threadIdx.x * T.nb;
    const unsigned any = __ballot_sync(0xffffffffu, c < g.ncells && V.cell_start[c + 1] > V.cell_start[c]);
    if (lane == 0) sm.pre[threadIdx.x >> 5] = (int)any;
    __syncthreads();
    for (int w = 0; w < nwarp; ++w)
      for (unsigned m = (unsigned)sm.pre[w]; m; m &= m - 1)
        build_cell_pairs(V.seg, g, V.box, invL, V.cell_start, V.cell_rods, V.margin, V.skin, V.nbr_cnt, V.nbr, V.maxnb,
                         first + (32 * w + __ffs((int)m) - 1) * T.nb, *reinterpret_cast<BuildSmem*>(team_dyn_smem),
                         reinterpret_cast<unsigned*>(team_dyn_smem + kBuildQOff),
                         reinterpret_cast<unsigned*>(team_dyn_smem + kBuildQOff) + kBuildQ, kBuildQ, overflow);
    __syncthreads();
  }
}

// Cell lists and the candidates within margin + skin of every rod (unordered).
static __device__ bool build_lists(const Team& T, const NscView& V, SmemNsc& sm, int& overflow) {
  const int n = V.st.n;
  const int tid = T.tid(), TS = T.size(), rank = T.rank();
  if (!V.box.pbc) {
    if (rank == 0 && threadIdx.x < 3) {
      V.bounds[threadIdx.x] = ~0ull;
      V.bounds[3 + threadIdx.x] = 0ull;
    }
    if (!team_sync(T)) return false;
    for (int i = tid; i < n; i += TS) {
      Seg s = V.seg[i];
      atomicMin(&V.bounds[0], ord_key(s.cx)); atomicMax(&V.bounds[3], ord_key(s.cx));
      atomicMin(&V.bounds[1], ord_key(s.cy)); atomicMax(&V.bounds[4], ord_key(s.cy));
      atomicMin(&V.bounds[2], ord_key(s.cz)); atomicMax(&V.bounds[5], ord_key(s.cz));
    }
    if (!team_sync(T)) return false;
    if (rank == 0 && threadIdx.x == 0) open_grid(V.bounds, V.bounds + 3, V.cut_center, 64, V.grid);
    if (!team_sync(T)) return false;
  }
  GridDev g;
  {
    const volatile GridDev* vg = V.grid;
    for (int k = 0; k < 3; ++k) {
      g.lo[k] = vg->lo[k];
      g.cell[k] = vg->cell[k];
      g.n[k] = vg->n[k];
    }
    g.ncells = vg->ncells;
  }
  for (int c = tid; c <= g.ncells; c += TS) {
    V.cell_cnt[c] = 0;
    V.cell_fill[c] = 0;
  }
  for (int i = tid; i < n; i += TS) V.nbr_cnt[i] = 0;
  if (rank == 0 && threadIdx.x < 2) V.bounds[threadIdx.x] = 0ull;  // (an open box's grid has been made from them)
  if (!team_sync(T)) return false;
  for (int i = tid; i < n; i += TS) {
    Seg s = V.seg[i];
    int cx = cell_coord(s.cx, g.lo[0], g.cell[0], g.n[0], V.box.pbc);
    int cy = cell_coord(s.cy, g.lo[1], g.cell[1], g.n[1], V.box.pbc);
    int cz = cell_coord(s.cz, g.lo[2], g.cell[2], g.n[2], V.box.pbc);
    int c = (cz * g.n[1] + cy) * g.n[0] + cx;
    V.cell_of[i] = c;
    atomicAdd(&V.cell_cnt[c], 1);
  }
  if (!team_sync(T)) return false;
  if (!team_excl_scan(T, V.cell_cnt, V.cell_start, g.ncells, V.blk, sm)) return false;
  // (and how crowded the cells are: the other rods in a rod's cell and in its
  // neighbourhood, over every rod of a small system, every 16th of a large one)
  const int step = n > 16384 ? 16 : 1;
  int own = 0, near = 0;
  for (int i = tid; i < n; i += TS) {
    int c = V.cell_of[i];
    const int first = V.cell_start[c];
    V.cell_rods[first + atomicAdd(&V.cell_fill[c], 1)] = i;
    if (i % step) continue;
    own += min(V.cell_start[c + 1] - first - 1, 4095);
    near += min(cells_around(g, V.box, V.cell_start, c) - 1, 4095);
  }
  own = block_reduce_sum_i(own, sm.red_i);
  near = block_reduce_sum_i(near, sm.red_i);
  if (threadIdx.x == 0) {
    atomicAdd(&V.bounds[0], (unsigned long long)own);
    atomicAdd(&V.bounds[1], (unsigned long long)near);
  }
  if (!team_sync(T)) return false;
  const int seen = (n + step - 1) / step;
  const double K = (double)*(volatile unsigned long long*)&V.bounds[1] / seen;
  const double shared = 1.0 + (double)*(volatile unsigned long long*)&V.bounds[0] / seen;
  double invL[3] = {1.0, 1.0, 1.0};
  for (int k = 0; k < 3; ++k)
    if (V.box.L[k] > 0.0) invL[k] = 1.0 / V.box.L[k];
  // One thread per home rod, or the block splits the pairs of one home cell at
  // a time.  A thread alone with its rod's K candidates is a serial chain,
  // 12 + 2.1 K us (several turns of the threads overlap by a quarter); a cell
  // that holds rods costs its block some 12 us of barriers and staging, more
  // when its pairs fill several rounds, and there are a little over n / shared
  // of them.
  // Measured, whole builds by rod and by cell, us (some 40 of them the cells
  // themselves), uniform boxes with rho rods a cell (K = 27 rho): 1000 rods on 8
  // blocks, rho 0.03 54 and 2132 (32768 cells), 1 115 and 818, 4 242 and 351, 8
  // 552 and 144; 20000 on 148, rho 1 137 and 1168, 4 288 and 460, 8 506 and 237;
  // 20000 on 40, rho 8 502 and 774, 16 945 and 662; a million on 148, rho 1 1384
  // and 49811, 8 5154 and 11045, 16 8723 and 7469.  60 rods in a tube on one
  // block (few neighbours a rod, and those along one axis): 26 and 133.
  const double t_rod = (12.0 + 2.1 * K) * fmax(1.0, 0.75 * n / TS);
  const double t_cell = (13.5 + 4e-5 * K * K) * n / (shared * T.nb);
  if (t_rod < t_cell) {
    for (int i = tid; i < n; i += TS)
      build_rod_list(i, V.seg, g, V.box, invL, V.cell_of, V.cell_start, V.cell_rods, V.margin, V.skin,
                     V.nbr_cnt, V.nbr, V.maxnb, overflow);
  } else {
    build_cells(T, V, g, invL, sm, overflow);
  }
  return team_sync(T);
}

static __device__ __noinline__ bool rebuild_phase(const Team& T, const NscView& V, SmemNsc& sm) {
  Ctl* ctl = V.ctl;
  const int n = V.st.n;
  const int tid = T.tid(), TS = T.size(), rank = T.rank();
  unsigned long long t_start = (ctl->prof_phases && rank == 0 && threadIdx.x == 0) ? gtimer() : 0;
  int overflow = 0;
  if (V.all_pairs) list_all_pairs(n, tid >> 5, TS >> 5, V.nbr_cnt, V.nbr, V.maxnb, overflow);
  else if (!build_lists(T, V, sm, overflow)) return false;
  for (int i = tid; i < n; i += TS) {
    if (!V.all_pairs) sort_list(V.nbr, V.nbr_cnt, V.maxnb, i, overflow);
    Seg s = V.seg[i];
    V.ref[i] = s.cx; V.ref[n + i] = s.cy; V.ref[2 * n + i] = s.cz;
    V.ref[3 * n + i] = s.ux; V.ref[4 * n + i] = s.uy; V.ref[5 * n + i] = s.uz;
  }
  if (overflow) atomicOr(&ctl->err, ERR_NBR_CAP);
  if (!team_sync(T)) return false;
  if (*(volatile int*)&ctl->err) return false;
  if (rank == 0 && threadIdx.x == 0) {
    ctl->rebuild = 0;
    ctl->rebuilds += 1;
    if (t_start) ctl->phase_ns[9] += (long long)(gtimer() - t_start);
  }
  return true;
}

}  // namespace rg
