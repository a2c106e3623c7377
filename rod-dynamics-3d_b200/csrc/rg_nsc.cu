// rg_nsc.cu - the non-smooth-contact (PSOR) step as one persistent kernel.
//
// NscContactSolver (src/physics/nsc_contact.cpp):
//   detectAndBuildManifolds :239-321, buildTangentBasis :78-85,
//   computeDiag :106-117, solveVelocities :325-655 (warm start :344-380,
//   sweeps :385-552, residual :546-551, cache :646-654),
//   projectPositions :659-880 (multi-body path :698-879);
// step order of App::physicsStep (src/app/main.cpp:4383-4528).
//
// Execution model.  A "team" of co-resident blocks (cooperative launch) runs
// every phase of one system's step - free flight, detection, colouring,
// manifold rows, PSOR sweeps, position update, projection, wrap - for
// nsteps steps in ONE launch.  Phases are separated by a bounded team
// barrier instead of kernel boundaries.  Independent systems run as separate
// teams of one launch (batching).
//
// Gauss-Seidel is graph-coloured: Jones-Plassmann first-fit colouring of the
// contacts (no two contacts of a colour share a dynamic body), computed with
// per-body atomic maxima of contact priorities and per-body colour masks
// instead of adjacency lists.  A sweep visits colours in order and the
// contacts of a colour in parallel; this is sequential Gauss-Seidel over the
// colour-major permutation of the (a,b)-sorted contacts, bit for bit.  Rows
// live in colour-major slots so each colour is a contiguous, coalesced range;
// the per-sweep residual max is a warp-shuffle reduction plus one atomic per
// block, and the exit test runs on the device.
#include <cstring>

#include "rg_team.cuh"

namespace rg {

#ifndef RG_NARROW_LANES
#define RG_NARROW_LANES 2  // lanes per rod in the narrow phase over the lists
#endif

GridDev* detector_grid(rg_system* s);
unsigned long long* detector_bounds(rg_system* s);
MlpDev mlp_dev(rg_system* s);

constexpr int kChunk = 32;  // most sweeps of a chunk of the split solve
static_assert(kTeamBarBytes >= 16 + sizeof(double) * 3 * kChunk, "barrier words and residual ring of a team");

struct SmallSmem;
// The small-solve arrays, by their symbol: a function that takes them as a
// reference would reach them through generic loads and stores.
__device__ __forceinline__ SmallSmem& small_smem() { return *reinterpret_cast<SmallSmem*>(team_dyn_smem); }

// Contacts at the current segment records (V.seg current, ctl->maxdisp
// accumulated by the caller, all blocks past a team barrier).  Returns the
// contact count, or -1 on error.
// Two-level lists: the near list holds the list entries within the contact
// reach (r_a + r_b + margin) plus near_skin, rebuilt from the lists when a
// rod has moved near_skin/2 since its build (or the lists were rebuilt).  A
// pair outside it was at least near_skin beyond contact at the build, and
// each rod has since moved less than near_skin/2 (|dx| + h|du| bounds every
// point of a segment), so it cannot touch: the contact set found from the
// near list is the exact one.  Contacts come out in near-list order, which
// is (a, b) order.
__device__ __noinline__ int detect_near(const Team& T, const NscView& V, double delta, SmemNsc& sm,
                                        bool lists_rebuilt, bool position_level) {
  Ctl* ctl = V.ctl;
  const int n = V.st.n;
  const int rank = T.rank();
  const int mode = V.all_pairs ? 2 : 1;
  double invL[3] = {1.0, 1.0, 1.0};
  for (int k = 0; k < 3; ++k)
    if (V.box.L[k] > 0.0) invL[k] = 1.0 / V.box.L[k];
  const bool rebuild_near = lists_rebuilt || !*(volatile int*)&ctl->near_valid ||
                            *(volatile double*)&ctl->near_disp >= 0.5 * V.near_skin * (1.0 - 1e-9);
  int prefix, total;
  if (rebuild_near) {
    const int seg = (n + T.nb - 1) / T.nb;
    const int lo = rank * seg < n ? rank * seg : n;
    const int hi = lo + seg < n ? lo + seg : n;
    constexpr int G = RG_NARROW_LANES;
    int mine = 0;
    for (int base = lo; base < hi; base += blockDim.x / G) {
      const int i = base + threadIdx.x / G;
      const bool valid = i < hi;
      const int c = near_count_lanes<G>(i, valid, V.seg, V.st.inv_mass, V.box, invL, mode, V.margin + V.near_skin,
                                        V.nbr_cnt, V.nbr, V.maxnb, V.words, V.mask);
      if (valid && (threadIdx.x & (G - 1)) == 0) {
        V.hit_cnt[i] = c;
        mine += c;
      }
    }
    const int bsum = block_reduce_sum_i(mine, sm.red_i);
    if (threadIdx.x == 0) V.blk[rank] = bsum;
    if (!team_sync(T)) return -1;
    if (rank == 0 && threadIdx.x == 0) {
      ctl->near_disp = 0.0;  // every block has read it
      ctl->near_rebuilds += 1;
    }
    block_prefix(V.blk, T.nb, rank, prefix, total, sm);
    int run = prefix;
    for (int base = lo; base < hi; base += blockDim.x) {
      const int i = base + threadIdx.x;
      const int c = i < hi ? V.hit_cnt[i] : 0;
      int tot;
      const int ex = block_excl_scan(c, sm.scan_w, tot);
      if (i < hi) {
        if (c) near_write_rod(i, run + ex, V.nbr_cnt, V.nbr, V.maxnb, V.words, V.mask, V.near);
        const Seg s = V.seg[i];
        V.ref2[i] = s.cx; V.ref2[n + i] = s.cy; V.ref2[2 * n + i] = s.cz;
        V.ref2[3 * n + i] = s.ux; V.ref2[4 * n + i] = s.uy; V.ref2[5 * n + i] = s.uz;
      }
      run += tot;
    }
    if (rank == 0 && threadIdx.x == 0) {
      ctl->near_n = total;
      ctl->near_valid = 1;
    }
    if (!team_sync(T)) return -1;
  }
  // exact narrow phase over the near list: each block a 64-aligned range
  const int P = *(volatile int*)&ctl->near_n;
  const int segp = (((P + T.nb - 1) / T.nb) + 63) & ~63;
  const int plo = rank * segp < P ? rank * segp : P;
  const int phi = plo + segp < P ? plo + segp : P;
  unsigned long long* bits = V.mask;  // one bit per near pair
  const double* im = V.st.inv_mass;
  // the block's words (none for an empty range: plo is then P, whose word
  // may belong to the block before)
  const int wlo = plo >> 6, whi = plo < phi ? (phi + 63) >> 6 : wlo;
  // The velocity-level detection follows the previous step's position-level
  // one over the same near list; only the position projection and the
  // periodic wrap moved rods in between.  A pair of two unmoved rods has
  // bit-identical segments, so its hit bit carries over; the other pairs
  // are tested again.
  const bool carry = !position_level && !rebuild_near && V.moved && *(volatile int*)&ctl->det_valid;
  if (carry) {
    constexpr int U = 4;  // pairs per thread and round: independent loads in flight
    for (int p0 = plo + threadIdx.x; p0 < phi; p0 += U * blockDim.x) {
      int2 pr[U];
      bool mv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int p = p0 + u * blockDim.x;
        pr[u] = p < phi ? V.near[p] : make_int2(0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) mv[u] = p0 + u * (int)blockDim.x < phi && (V.moved[pr[u].x] | V.moved[pr[u].y]);
#pragma unroll 1
      for (int u = 0; u < U; ++u) {
        if (!mv[u]) continue;
        const int p = p0 + u * blockDim.x;
        const bool was = (__ldcg(&bits[p >> 6]) >> (p & 63)) & 1ull;
        bool hit = false;
        if (im[pr[u].x] > 0.0 || im[pr[u].y] > 0.0) {
          const Seg A = V.seg[pr[u].x], B = V.seg[pr[u].y];
          if (!seg_far(A, B, prefilter_offset(A, B, V.box, invL, mode), A.r + B.r + delta)) {
            const Narrow nr = narrow_pair(A, B, V.box);
            hit = contact_test(nr.d2, A.r + B.r, delta);
          }
        }
        if (hit != was) atomicXor(&bits[p >> 6], 1ull << (p & 63));
      }
    }
  } else {
    for (int w = wlo + threadIdx.x; w < whi; w += blockDim.x) bits[w] = 0ull;
    __syncthreads();
    for (int p = plo + threadIdx.x; p < phi; p += blockDim.x) {
      const int2 pr = V.near[p];
      if (!(im[pr.x] > 0.0) && !(im[pr.y] > 0.0)) continue;
      const Seg A = V.seg[pr.x], B = V.seg[pr.y];
      if (seg_far(A, B, prefilter_offset(A, B, V.box, invL, mode), A.r + B.r + delta)) continue;
      const Narrow nr = narrow_pair(A, B, V.box);
      if (contact_test(nr.d2, A.r + B.r, delta)) atomicOr(&bits[p >> 6], 1ull << (p & 63));
    }
  }
  __syncthreads();
  int mine = 0;
  for (int w = wlo + threadIdx.x; w < whi; w += blockDim.x) mine += __popcll(__ldcg(&bits[w]));
  const int bsum = block_reduce_sum_i(mine, sm.red_i);
  if (threadIdx.x == 0) V.blk[rank] = bsum;
  if (!team_sync(T)) return -1;
  // every block has read maxdisp.  After a position-level pass it stays:
  // the next free flight refreshes only the rods moved since, and the
  // unmoved rods' bounds are the ones it holds (unless the lists were just
  // rebuilt, when every bound restarts at zero).
  if (rank == 0 && threadIdx.x == 0 && (!position_level || lists_rebuilt)) ctl->maxdisp = 0.0;
  block_prefix(V.blk, T.nb, rank, prefix, total, sm);
  if (total > V.ccap) {
    if (rank == 0 && threadIdx.x == 0) atomicOr(&ctl->err, ERR_CONTACT_CAP);
    return -1;
  }
  // contacts in pair order: one word (64 pairs) per thread, scanned by
  // population count, places each hit's pair in its slot; then one thread
  // per slot runs the exact narrow phase (a word may hold several hits,
  // which one thread would otherwise evaluate one after the other)
  int run = prefix;
  for (int wb = wlo; wb < whi; wb += blockDim.x) {
    const int w = wb + threadIdx.x;
    const unsigned long long m = w < whi ? __ldcg(&bits[w]) : 0ull;
    int tot;
    int slot = run + block_excl_scan(__popcll(m), sm.scan_w, tot);
    for (unsigned long long r = m; r; r &= r - 1) {
      const int2 pr = V.near[(w << 6) + __ffsll((long long)r) - 1];
      V.con.a[slot] = pr.x;
      V.con.b[slot] = pr.y;
      ++slot;
    }
    run += tot;
  }
  __syncthreads();
  for (int c = prefix + (int)threadIdx.x; c < run; c += blockDim.x) {
    const int a = V.con.a[c], b = V.con.b[c];
    const Seg A = V.seg[a], B = V.seg[b];
    const Narrow nr = narrow_pair(A, B, V.box);
    write_contact(V.con, c, a, b, A.r + B.r, nr);
  }
  if (rank == 0 && threadIdx.x == 0) {
    ctl->contacts = total;
    ctl->det_valid = position_level ? 1 : 0;
  }
  if (!team_sync(T)) return -1;
  return total;
}

__device__ __noinline__ int detect_phase(const Team& T, const NscView& V, double delta, SmemNsc& sm,
                                         bool position_level) {
  Ctl* ctl = V.ctl;
  const int n = V.st.n;
  const int rank = T.rank();
  const bool need = *(volatile int*)&ctl->rebuild ||
                    (!V.all_pairs && *(volatile double*)&ctl->maxdisp >= 0.5 * V.skin * (1.0 - 1e-9));
  if (need && !rebuild_phase(T, V, sm)) return -1;
  if (V.near) return detect_near(T, V, delta, sm, need, position_level);
  const int seg = (n + T.nb - 1) / T.nb;
  const int lo = rank * seg < n ? rank * seg : n;
  const int hi = lo + seg < n ? lo + seg : n;
  constexpr int G = RG_NARROW_LANES;  // lanes per rod
  int mine = 0;
  for (int base = lo; base < hi; base += blockDim.x / G) {
    int i = base + threadIdx.x / G;
    bool valid = i < hi;
    int c = narrow_count_lanes<G>(i, valid, V.seg, V.st.inv_mass, V.box, delta, V.nbr_cnt, V.nbr, V.maxnb,
                                  V.words, V.mask, V.all_pairs ? 2 : 1);
    if (valid && (threadIdx.x & (G - 1)) == 0) {
      V.hit_cnt[i] = c;
      mine += c;
    }
  }
  int run = block_reduce_sum_i(mine, sm.red_i);
  if (threadIdx.x == 0) V.blk[rank] = run;
  if (!team_sync(T)) return -1;
  // every block has read maxdisp (kept after a position-level pass, as above)
  if (rank == 0 && threadIdx.x == 0 && (!position_level || need)) ctl->maxdisp = 0.0;
  int prefix, total;
  block_prefix(V.blk, T.nb, rank, prefix, total, sm);
  if (total > V.ccap) {
    if (rank == 0 && threadIdx.x == 0) atomicOr(&ctl->err, ERR_CONTACT_CAP);
    return -1;
  }
  run = prefix;
  for (int base = lo; base < hi; base += blockDim.x) {
    int i = base + threadIdx.x;
    int c = i < hi ? V.hit_cnt[i] : 0;
    int tot;
    int ex = block_excl_scan(c, sm.scan_w, tot);
    if (c) narrow_write_rod(i, run + ex, V.seg, V.box, V.nbr_cnt, V.nbr, V.maxnb, V.words, V.mask, V.con);
    run += tot;
  }
  if (rank == 0 && threadIdx.x == 0) ctl->contacts = total;
  if (!team_sync(T)) return -1;
  return total;
}

// ---------------------------------------------------------------------------
// Colouring: Jones-Plassmann first fit with per-body priority maxima.
// ---------------------------------------------------------------------------
__device__ __noinline__ bool color_phase(const Team& T, const NscView& V, int C, SmemNsc& sm) {
  Ctl* ctl = V.ctl;
  const int n = V.st.n;
  const int tid = T.tid(), TS = T.size(), rank = T.rank();
  const double* im = V.st.inv_mass;
  for (int c = tid; c < C; c += TS) {
    int x[2] = {V.con.a[c], V.con.b[c]};
    for (int k = 0; k < 2; ++k) {
      if (!(im[x[k]] > 0.0)) continue;
      V.pmax[x[k]] = 0;
      V.pmax[n + x[k]] = 0;
      V.cmask[x[k]] = 0;
      V.owner[x[k]] = 0x7fffffff;
    }
    V.color[c] = -1;
  }
  if (rank == 0) {
    for (int k = threadIdx.x; k <= kMaxColors; k += blockDim.x) {
      V.color_cnt[k] = 0;
      V.cursor[k] = 0;
    }
    for (int r = threadIdx.x; r < kMaxRounds; r += blockDim.x) V.remaining[r] = 0;
    if (threadIdx.x == 0) ctl->colors = 0;
  }
  if (!team_sync(T)) return false;
  int round = 0;
  for (; round < kMaxRounds; ++round) {
    unsigned long long* pm = V.pmax + (size_t)(round & 1) * n;
    unsigned long long* pn = V.pmax + (size_t)((round + 1) & 1) * n;
    for (int c = tid; c < C; c += TS) {
      if (V.color[c] >= 0) continue;
      int x[2] = {V.con.a[c], V.con.b[c]};
      unsigned long long p = jp_priority((unsigned)c);
      for (int k = 0; k < 2; ++k) {
        if (!(im[x[k]] > 0.0)) continue;
        atomicMax(&pm[x[k]], p);
        if (round == 0) atomicMin(&V.owner[x[k]], c);
      }
    }
    if (!team_sync(T)) return false;
    int rem = 0, maxc = 0;
    for (int c = tid; c < C; c += TS) {
      if (V.color[c] >= 0) continue;
      int x[2] = {V.con.a[c], V.con.b[c]};
      unsigned long long p = jp_priority((unsigned)c);
      bool win = true;
      unsigned long long used = 0;
      for (int k = 0; k < 2; ++k) {
        if (!(im[x[k]] > 0.0)) continue;
        if (*(volatile unsigned long long*)&pm[x[k]] != p) win = false;
        used |= *(volatile unsigned long long*)&V.cmask[x[k]];
        pn[x[k]] = 0;
      }
      if (win) {
        int col = __ffsll((long long)~used) - 1;
        if (used == ~0ull) {
          atomicOr(&ctl->err, ERR_COLOR);
          col = kMaxColors - 1;
        }
        V.color[c] = col;
        for (int k = 0; k < 2; ++k)
          if (im[x[k]] > 0.0) atomicOr(&V.cmask[x[k]], 1ull << col);
        atomicAdd(&V.color_cnt[col], 1);
        maxc = col + 1 > maxc ? col + 1 : maxc;
      } else {
        ++rem;
      }
    }
    int br = block_reduce_sum_i(rem, sm.red_i);
    if (threadIdx.x == 0 && br) atomicAdd(&V.remaining[round], br);
    if (maxc) atomicMax(&ctl->colors, maxc);
    if (!team_sync(T)) return false;
    if (*(volatile int*)&V.remaining[round] == 0) break;
  }
  if (round >= kMaxRounds) {
    if (rank == 0 && threadIdx.x == 0) atomicOr(&ctl->err, ERR_COLOR);
    return false;
  }
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int k = 0; k <= kMaxColors; ++k) {
      sm.coff[k] = acc;
      if (k < kMaxColors) acc += *(volatile int*)&V.color_cnt[k];
    }
  }
  __syncthreads();
  if (rank == 0)
    for (int k = threadIdx.x; k <= kMaxColors; k += blockDim.x) V.color_off[k] = sm.coff[k];
  for (int c = tid; c < C; c += TS) {
    int k = V.color[c];
    V.order[sm.coff[k] + atomicAdd(&V.cursor[k], 1)] = c;
  }
  return team_sync(T);
}

// ---------------------------------------------------------------------------
// PSOR sweeps.
// ---------------------------------------------------------------------------
__device__ inline int active_blocks(const int* coff, int ncol, int bs, int nb) {
  int m = 0;
  for (int k = 0; k < ncol; ++k) {
    int c = coff[k + 1] - coff[k];
    m = c > m ? c : m;
  }
  int need = (m + bs - 1) / bs;
  if (need < 1) need = 1;
  return need < nb ? need : nb;
}

__device__ __noinline__ bool psor_phase(const Team& T, const NscView& V, int C, SmemNsc& sm) {
  Ctl* ctl = V.ctl;
  const int K = *(volatile int*)&ctl->colors;
  const int rank = T.rank();
  const rg_config& cfg = V.cfg;
  if (C > 0) {
    const int na = active_blocks(V.color_off, K, blockDim.x, T.nb);
    if (rank < na) {
      const int tid = rank * blockDim.x + threadIdx.x, stride = na * blockDim.x;
      RowIO R{V.row, V.lam, V.ccap};
      Vel Vv{V.st.v, V.st.w};
      const double omega = cfg.nsc_omega, cfm = cfg.nsc_cfm, mu = cfg.nsc_mu;
      const int iters = cfg.nsc_velocity_iters;
      const int* coff = V.color_off;
      for (int i = tid; i < iters; i += stride) ctl->res_sweep[i] = 0.0;
      if (cfg.nsc_warm_start != RG_WARM_NONE) {
        for (int k = 0; k < K; ++k) {
          for (int p = coff[k] + tid; p < coff[k + 1]; p += stride) {
            int c = V.order[p];
            warm_apply(R, Vv, p, V.con.a[c], V.con.b[c]);
          }
          if (!team_sync_sub(T, na)) return false;
        }
      } else if (!team_sync_sub(T, na)) {
        return false;
      }
      double res = 0.0;
      int sweeps = 0;
      for (int it = 0; it < iters; ++it) {
        double loc = 0.0;
        for (int k = 0; k < K; ++k) {
          for (int p = coff[k] + tid; p < coff[k + 1]; p += stride) {
            int c = V.order[p];
            loc = fmax(loc, psor_row(R, Vv, p, V.con.a[c], V.con.b[c], omega, cfm, mu));
          }
          if (k + 1 < K && !team_sync_sub(T, na)) return false;
        }
        double bm = block_reduce_max(loc, sm.red_d);
        if (threadIdx.x == 0) atomic_max_nonneg(&ctl->res_sweep[it], bm);
        if (!team_sync_sub(T, na)) return false;
        res = *(volatile double*)&ctl->res_sweep[it];
        sweeps = it + 1;
        if (res < cfg.nsc_tol) break;
      }
      if (tid == 0) {
        ctl->residual = res;
        ctl->sweeps_last = sweeps;
        ctl->sweeps_sum += sweeps;
        ctl->row_sweeps += (long long)C * sweeps;
        ctl->contact_steps += C;
        if (res >= cfg.nsc_tol) ctl->not_conv += 1;
        if (res > ctl->max_residual) ctl->max_residual = res;
      }
    }
  } else if (rank == 0 && threadIdx.x == 0) {
    ctl->residual = 0.0;
    ctl->sweeps_last = 0;
  }
  return team_sync(T);
}

// ---------------------------------------------------------------------------
// Position projection (rows from the pass-0 detection, then narrow phase on
// the cached pairs in later passes).  Runs on the na active blocks.
// ---------------------------------------------------------------------------
__device__ __noinline__ bool project_rows(const NscView& V, int C, int K, int na, int rank, const Team& T, SmemNsc& sm) {
  Ctl* ctl = V.ctl;
  const rg_config& cfg = V.cfg;
  const State& st = V.st;
  const int n = st.n;
  const int tid = rank * blockDim.x + threadIdx.x, stride = na * blockDim.x;
  const double omega = cfg.nsc_omega, cfm = cfg.nsc_cfm, slop = cfg.nsc_slop;
  const int* coff = V.color_off;
  const size_t ccap = (size_t)V.ccap;
  double* PR = V.prow;
  Vec3A DX{V.dx, V.dx + n, V.dx + 2 * n}, DT{V.dx + 3 * n, V.dx + 4 * n, V.dx + 5 * n};
  double* slots = ctl->res_sweep;
  const int piters = cfg.nsc_position_psor_iters;
  for (int outer = 0; outer < cfg.nsc_position_iters; ++outer) {
    for (int i = tid; i < piters + 1; i += stride) slots[i] = 0.0;
    if (!team_sync_sub(T, na)) return false;
    int cnt = 0;
    for (int p = tid; p < C; p += stride) {
      const int c = V.order[p];
      const int a = V.con.a[c], b = V.con.b[c];
      d3 xa = st.x.ld(a), xb = st.x.ld(b);
      d3 nv, ra, rb;
      double phi;
      if (outer == 0) {
        phi = V.con.comp(12)[c] - V.con.comp(13)[c];
        nv = mk3(V.con.comp(6)[c], V.con.comp(7)[c], V.con.comp(8)[c]);
        d3 pa{V.con.comp(0)[c], V.con.comp(1)[c], V.con.comp(2)[c]};
        d3 pb{V.con.comp(3)[c], V.con.comp(4)[c], V.con.comp(5)[c]};
        d3 sh{V.con.comp(9)[c], V.con.comp(10)[c], V.con.comp(11)[c]};
        ra = pa - xa;
        rb = pb - (xb + sh);
      } else {
        Seg A = make_seg(st, a), B = make_seg(st, b);
        Narrow nr = narrow_pair(A, B, V.box);
        d3 diff = nr.pb - nr.pa;
        double dist = len(diff);
        phi = dist - V.con.comp(13)[c];
        nv = dist > 1e-10 ? diff / dist : mk3(1, 0, 0);
        ra = nr.pa - xa;
        rb = nr.pb - (xb + nr.sh);
      }
      int act = phi < -slop ? 1 : 0;
      V.pactive[p] = act;
      if (act) {
        ++cnt;
        PR[P_N * ccap + p] = nv.x; PR[(P_N + 1) * ccap + p] = nv.y; PR[(P_N + 2) * ccap + p] = nv.z;
        PR[P_RA * ccap + p] = ra.x; PR[(P_RA + 1) * ccap + p] = ra.y; PR[(P_RA + 2) * ccap + p] = ra.z;
        PR[P_RB * ccap + p] = rb.x; PR[(P_RB + 1) * ccap + p] = rb.y; PR[(P_RB + 2) * ccap + p] = rb.z;
        PR[P_PHI * ccap + p] = phi + slop;
        PR[P_G * ccap + p] = diag_of(st, a, b, ra, rb, nv, cfm);
        PR[P_L * ccap + p] = 0.0;
      }
      DX.st(a, mk3(0, 0, 0)); DT.st(a, mk3(0, 0, 0));
      DX.st(b, mk3(0, 0, 0)); DT.st(b, mk3(0, 0, 0));
    }
    int bc = block_reduce_sum_i(cnt, sm.red_i);
    if (threadIdx.x == 0 && bc)
      atomicAdd(reinterpret_cast<unsigned long long*>(&slots[piters]), (unsigned long long)bc);
    if (!team_sync_sub(T, na)) return false;
    if (*(volatile unsigned long long*)&slots[piters] == 0ull) return true;  // nothing penetrates
    for (int it = 0; it < piters; ++it) {
      double loc = 0.0;
      for (int k = 0; k < K; ++k) {
        for (int p = coff[k] + tid; p < coff[k + 1]; p += stride) {
          if (!V.pactive[p]) continue;
          const int c = V.order[p];
          const int a = V.con.a[c], b = V.con.b[c];
          d3 nv{PR[P_N * ccap + p], PR[(P_N + 1) * ccap + p], PR[(P_N + 2) * ccap + p]};
          d3 ra{PR[P_RA * ccap + p], PR[(P_RA + 1) * ccap + p], PR[(P_RA + 2) * ccap + p]};
          d3 rb{PR[P_RB * ccap + p], PR[(P_RB + 1) * ccap + p], PR[(P_RB + 2) * ccap + p]};
          double l = PR[P_L * ccap + p];
          double corr = dot(nv, ((DX.ld(b) + cross(DT.ld(b), rb)) - DX.ld(a)) - cross(DT.ld(a), ra));
          double r = corr + PR[P_PHI * ccap + p] + cfm * l;
          double d = -(omega / PR[P_G * ccap + p]) * r;
          double nl = smax(0.0, l + d);
          double dl = nl - l;
          if (dl != 0.0) {
            PR[P_L * ccap + p] = nl;
            d3 rAxn = cross(ra, nv);
            DX.st(a, DX.ld(a) - nv * (dl * st.inv_mass[a]));
            DT.st(a, DT.ld(a) - iinv_apply(st, a, rAxn) * dl);
            d3 rBxn = cross(rb, nv);
            DX.st(b, DX.ld(b) + nv * (dl * st.inv_mass[b]));
            DT.st(b, DT.ld(b) + iinv_apply(st, b, rBxn) * dl);
          }
          loc = fmax(loc, fabs(dl));
        }
        if (k + 1 < K && !team_sync_sub(T, na)) return false;
      }
      double bm = block_reduce_max(loc, sm.red_d);
      if (threadIdx.x == 0) atomic_max_nonneg(&slots[it], bm);
      if (!team_sync_sub(T, na)) return false;
      if (*(volatile double*)&slots[it] < 1e-8) break;
    }
    // apply: each body once, by the lowest-index contact touching it
    for (int p = tid; p < C; p += stride) {
      const int c = V.order[p];
      for (int side = 0; side < 2; ++side) {
        int bd = side ? V.con.b[c] : V.con.a[c];
        if (st.inv_mass[bd] <= 0.0 || V.owner[bd] != c) continue;
        if (V.moved) V.moved[bd] = 1;
        st.x.st(bd, st.x.ld(bd) + DX.ld(bd));
        d3 th = DT.ld(bd);
        double ang = len(th);
        if (ang > 1e-8) {
          d3 ax = th / ang;
          st.q.st(bd, qnormalize(qmul(angle_axis(ang, ax), st.q.ld(bd))));
        }
      }
    }
    if (!team_sync_sub(T, na)) return false;
  }
  return true;
}

__device__ __noinline__ bool project_phase(const Team& T, const NscView& V, int C, SmemNsc& sm) {
  const int rank = T.rank();
  const int K = *(volatile int*)&V.ctl->colors;
  if (C > 0 && V.cfg.nsc_position_stabilization) {
    const int na = active_blocks(V.color_off, K, blockDim.x, T.nb);
    if (rank < na && !project_rows(V, C, K, na, rank, T, sm)) return false;
  }
  return team_sync(T);
}


// ---------------------------------------------------------------------------
// Contact sets of up to kSmallC contacts: solved on chip, island by island.
//
// Every block of the team colours the whole contact graph in its own shared
// memory (no barrier, the same colours everywhere) and finds its connected
// components.  Components share no dynamic body, so Gauss-Seidel on one never
// reads what another writes: block r takes the r-th share of them and keeps
// their body velocities in shared memory.  The sweeps stop when the largest
// change of any contact falls below the tolerance, so the blocks run a chunk
// of sweeps, keep the state after each, publish the chunk's residuals, and
// after one team barrier all put back the state of the sweep at which the
// whole set stopped: the same sweeps as one sequential solver makes, bit for
// bit.  A component that a sweep left unchanged stays unchanged and is not
// swept again.
//
// A contact is owned by two adjacent lanes, one per body: a lane holds its
// side of the manifold row, updates its body, and gets the three numbers it
// needs of the other side by shuffle.  That halves the chain of dependent
// FP64 operations, and the row of one contact per lane pair stays in
// registers; up to 16 contacts need a single warp and no block barrier.
//
// Sets of at most kPairs contacts stay on the team's first block (solo): a
// chunk's barrier and its surplus sweeps cost more there than the split saves.
//
// Bound: latency of a row update (about 1,200 cycles: some 50 dependent FP64
// operations, two square roots, three exchanges) times colours times sweeps.
// Measured per sweep: N = 20,000, 200 contacts 10 -> 2.9 us (one block; rows
// in shared memory and one lane per contact before), N = 50,000, 450 contacts
// 23 -> 2.4 us (rows and velocities in global memory before); whole steps
// 274 -> 180 us and 2,020 -> 385 us.  Above kSmallC contacts the shared
// memory for velocities ends and the team path takes over.
// ---------------------------------------------------------------------------
#ifndef RG_NSC_BLOCK
#define RG_NSC_BLOCK (2 * kTile)
#endif
constexpr int kBlock = RG_NSC_BLOCK;     // threads per block of the persistent step
constexpr int kPairs = kBlock / 2;       // lane pairs of a block
constexpr int kSmallC = 4 * kPairs;      // contacts of the on-chip solve
constexpr int kSmallB = 2 * kSmallC;     // body slots
constexpr int kHash = 2 * kSmallB;       // body -> slot table (power of two)
constexpr int kSplit = 512;              // most blocks the components are split over
constexpr int kVel = 6 * kSmallB;        // doubles of the velocity space
static_assert((kHash & (kHash - 1)) == 0 && kSmallB <= 65536, "hash table and 16-bit slots");

struct SmallSmem {
  // v, w (or dx, dθ) per local body slot, 6 doubles each, then the states
  // after the sweeps of a chunk.  Before the velocities are loaded the space
  // serves the colouring and the split (SmallScratch), then the warm-cache
  // keys, then the network's third layer.
  alignas(16) double vel[kVel];
  // the network's W1, W4 and small parameters; before that the degrees
  alignas(16) unsigned char stage[(kStageSmallBytes + 15) / 16 * 16];
  alignas(16) __nv_bfloat16 wh[kStageWh];  // the network's second layer
  double locs[kChunk * 32];          // residuals of a chunk's sweeps, per lane or warp
  double res[kChunk];                // residuals of the chunk over the team
  int body[kSmallB];                 // body of a local slot
  unsigned char dyn[kSmallB];        // 1: dynamic body
  // this block's contacts in colour-major slots: contact, colour, body slots
  unsigned short order[kSmallC], pa[kSmallC], pb[kSmallC];
  unsigned short comp[kSmallC];      // component of the slot's contact (split solves)
  unsigned char pcol[kSmallC];
  unsigned char cached[kSmallC];     // 1: the slot's contact is in the warm cache
  int cnt[kMaxColors + 1], coff[kMaxColors + 1], cur[kMaxColors + 1];
  int nloc, ncol, nbody;
  int scan_w[32];
  int mtile[kSmallC / 16];           // 16-contact tiles that need the network
};
struct SmallScratch {  // whole contact set: slots of all bodies, colours
  union {
    unsigned long long pmax[2 * kSmallB];
    struct {  // after the colouring
      int lab[kSmallC], blab[kSmallB], irank[kSmallC], hist[kSplit], bl[kSmallB];
    };
  };
  unsigned long long cmask[kSmallB];
  int hkey[kHash];
  unsigned short hslot[kHash];
  int body[kSmallB];
  unsigned char dyn[kSmallB];
  unsigned short la[kSmallC], lb[kSmallC], color[kSmallC];  // by contact
};
static_assert(sizeof(SmallScratch) <= sizeof(double) * kVel, "colouring scratch");
static_assert(sizeof(SmallSmem::stage) >= sizeof(int) * kSmallB, "degrees");
static_assert(sizeof(__nv_bfloat16) * kStageWh <= sizeof(double) * kVel, "third network layer");
static_assert(sizeof(SmallSmem) >= kBuildQOff + 2 * sizeof(unsigned) * kBuildQ,
              "list-build tiles and queues share the small-solve memory");

// True when contact c has an entry in the warm cache of the previous step
// (W entries): the learned start by default serves only the others.
__device__ inline bool warm_cached(const NscView& V, int c, int W) {
  if (W <= 0) return false;
  const unsigned long long k = ((unsigned long long)(unsigned)V.con.a[c] << 32) | (unsigned)V.con.b[c];
  const int q = lower_bound_key(V.wkey, W, k);
  return q < W && V.wkey[q] == k;
}

// Slots for the bodies of contacts 0..C-1 (C <= kSmallC), through a hash
// table of body numbers in shared memory.
__device__ __noinline__ void small_map(const NscView& V, int C) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x;
  SmallScratch& X = *reinterpret_cast<SmallScratch*>(S.vel);
  const int size = C <= 64 ? 256 : (C <= kPairs ? 4 * kPairs : kHash);  // at least 4 C, a power of two
  if (t == 0) S.nloc = 0;
  for (int k = t; k < size; k += blockDim.x) X.hkey[k] = -1;
  __syncthreads();
  for (int e = t; e < 2 * C; e += blockDim.x) {
    const int c = e >> 1;
    const int x = (e & 1) ? V.con.b[c] : V.con.a[c];
    unsigned pos = ((unsigned)x * 0x9E3779B1u) >> 7;
    for (;;) {  // at most 2 C of the entries are ever taken
      pos &= size - 1;
      const int old = atomicCAS(&X.hkey[pos], -1, x);
      if (old == -1) {
        const int idx = atomicAdd(&S.nloc, 1);
        X.hslot[pos] = (unsigned short)idx;
        X.body[idx] = x;
        X.dyn[idx] = V.st.inv_mass[x] > 0.0 ? 1 : 0;
      }
      if (old == -1 || old == x) break;
      ++pos;
    }
    if (e & 1) X.lb[c] = (unsigned short)pos;
    else X.la[c] = (unsigned short)pos;
  }
  __syncthreads();
  for (int c = t; c < C; c += blockDim.x) {
    X.la[c] = X.hslot[X.la[c]];
    X.lb[c] = X.hslot[X.lb[c]];
  }
  __syncthreads();
}

// Jones-Plassmann first fit on the slots: X.color per contact.  Returns the
// colour count or -1.
__device__ __noinline__ int small_color(const NscView& V, int C, bool lead) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x;
  SmallScratch& X = *reinterpret_cast<SmallScratch*>(S.vel);
  constexpr unsigned short kNone = 0xffff;
  if (S.nloc == 2 * C) {  // no body twice: one colour
    for (int c = t; c < C; c += blockDim.x) X.color[c] = 0;
    if (t == 0) S.ncol = C > 0;
    if (t == 0 && lead) V.ctl->colors = C > 0;
    __syncthreads();
    return C > 0;
  }
  for (int s = t; s < S.nloc; s += blockDim.x) {
    X.pmax[s] = 0; X.pmax[kSmallB + s] = 0; X.cmask[s] = 0;
  }
  for (int c = t; c < C; c += blockDim.x) X.color[c] = kNone;
  if (t == 0) S.ncol = 0;
  __syncthreads();
  int round = 0;
  for (; round < kMaxRounds; ++round) {
    unsigned long long* pm = X.pmax + (round & 1) * kSmallB;
    unsigned long long* pn = X.pmax + ((round + 1) & 1) * kSmallB;
    for (int c = t; c < C; c += blockDim.x) {
      if (X.color[c] != kNone) continue;
      const unsigned long long p = jp_priority((unsigned)c);
      if (X.dyn[X.la[c]]) atomicMax(&pm[X.la[c]], p);
      if (X.dyn[X.lb[c]]) atomicMax(&pm[X.lb[c]], p);
    }
    __syncthreads();
    int rem = 0;
    for (int c = t; c < C; c += blockDim.x) {
      if (X.color[c] != kNone) continue;
      const unsigned long long p = jp_priority((unsigned)c);
      const int sl[2] = {X.la[c], X.lb[c]};
      bool win = true;
      unsigned long long used = 0;
      for (int k = 0; k < 2; ++k) {
        if (!X.dyn[sl[k]]) continue;
        if (pm[sl[k]] != p) win = false;
        // two winners of a round never share a dynamic body, so a mask that
        // changes in this round is only read by losers
        used |= *(volatile unsigned long long*)&X.cmask[sl[k]];
        pn[sl[k]] = 0;
      }
      if (win) {
        int col = __ffsll((long long)~used) - 1;
        if (used == ~0ull) {
          atomicOr(&V.ctl->err, ERR_COLOR);
          col = kMaxColors - 1;
        }
        X.color[c] = (unsigned short)col;
        for (int k = 0; k < 2; ++k)
          if (X.dyn[sl[k]]) atomicOr(&X.cmask[sl[k]], 1ull << col);
        atomicMax(&S.ncol, col + 1);
      } else {
        rem = 1;
      }
    }
    if (!__syncthreads_or(rem)) break;
  }
  if (round >= kMaxRounds) {
    if (t == 0) atomicOr(&V.ctl->err, ERR_COLOR);
    return -1;
  }
  const int ncol = S.ncol;
  if (t == 0 && lead) V.ctl->colors = ncol;
  __syncthreads();  // every thread has its copy before ncol is used again
  return ncol;
}

// This block's share of a contact set: its contacts in colour-major slots
// 0..count-1 of the on-chip arrays, and slots [base, base + count) of the
// global row, impulse and feature arrays; most: the largest share.
struct Share {
  int count, base, most, colors;
};
// A team's blocks get the connected components in the order of their lowest
// contacts.
__device__ __noinline__ Share small_split(const Team& T, int C, int ncol) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x, rank = T.rank();
  SmallScratch& X = *reinterpret_cast<SmallScratch*>(S.vel);
  const bool split = T.nb > 1;
  const int nbu = T.nb < kSplit ? T.nb : kSplit;
  if (!split && ncol <= 1) {  // one block, one colour: the contacts as they are
    for (int s = t; s < S.nloc; s += blockDim.x) {
      S.body[s] = X.body[s];
      S.dyn[s] = X.dyn[s];
    }
    for (int c = t; c < C; c += blockDim.x) {
      S.order[c] = (unsigned short)c;
      S.pcol[c] = 0;
      S.pa[c] = X.la[c];
      S.pb[c] = X.lb[c];
      S.comp[c] = 0;
    }
    if (t == 0) {
      S.nbody = S.nloc;
      S.coff[0] = 0;
      S.cnt[0] = C;
    }
    __syncthreads();
    return Share{C, 0, C, ncol};
  }
  for (int k = t; k <= kMaxColors; k += blockDim.x) { S.cnt[k] = 0; S.cur[k] = 0; }
  if (t == 0) { S.nbody = 0; S.ncol = 0; }
  __syncthreads();  // (also: the colouring's maxima are done with)
  if (split) {
    for (int c = t; c < C; c += blockDim.x) X.lab[c] = c;
    for (int s = t; s < S.nloc; s += blockDim.x) X.blab[s] = 0x7fffffff;
    for (int r = t; r < kSplit; r += blockDim.x) X.hist[r] = 0;
    // labels fall to the lowest contact of the component
    int changed = 1;
    while (__syncthreads_or(changed)) {
      for (int c = t; c < C; c += blockDim.x) {
        const int l = X.lab[c];
        if (X.dyn[X.la[c]]) atomicMin(&X.blab[X.la[c]], l);
        if (X.dyn[X.lb[c]]) atomicMin(&X.blab[X.lb[c]], l);
      }
      __syncthreads();
      changed = 0;
      for (int c = t; c < C; c += blockDim.x) {
        const int l = X.lab[c];
        int m = l;
        if (X.dyn[X.la[c]]) m = min(m, X.blab[X.la[c]]);
        if (X.dyn[X.lb[c]]) m = min(m, X.blab[X.lb[c]]);
        m = min(m, *(volatile int*)&X.lab[m]);
        if (m < l) {
          *(volatile int*)&X.lab[c] = m;
          changed = 1;
        }
      }
    }
    // component numbers
    int total = 0;
    for (int base = 0; base < C; base += blockDim.x) {
      const int c = base + t;
      const int root = c < C && X.lab[c] == c;
      int tot;
      const int ex = block_excl_scan(root, S.scan_w, tot);
      if (root) X.irank[c] = total + ex;
      total += tot;
    }
    __syncthreads();
    for (int c = t; c < C; c += blockDim.x) {
      const int blk = X.irank[X.lab[c]] * nbu / total;
      X.blab[c] = blk;  // (the labels of the bodies are done with; C <= kSmallB)
      atomicAdd(&X.hist[blk], 1);
    }
  }
  for (int s = t; s < S.nloc; s += blockDim.x) X.bl[s] = -1;
  __syncthreads();
  // colours and bodies of the own contacts
  int maxc = 0;
  for (int c = t; c < C; c += blockDim.x) {
    if (split && X.blab[c] != rank) continue;
    atomicAdd(&S.cnt[X.color[c]], 1);
    maxc = max(maxc, X.color[c] + 1);
    for (int k = 0; k < 2; ++k) {
      const int s = k ? X.lb[c] : X.la[c];
      if (atomicCAS(&X.bl[s], -1, -2) == -1) {
        const int idx = atomicAdd(&S.nbody, 1);
        S.body[idx] = X.body[s];
        S.dyn[idx] = X.dyn[s];
        X.bl[s] = idx;
      }
    }
  }
  if (maxc) atomicMax(&S.ncol, maxc);
  int low = 0, most = 0;
  if (split)
    for (int r = t; r < nbu; r += blockDim.x) {
      if (r < rank) low += X.hist[r];
      most = max(most, X.hist[r]);
    }
  low = warp_sum_i(low);
  most = (int)__reduce_max_sync(0xffffffffu, (unsigned)most);
  if ((t & 31) == 0) {
    S.scan_w[t >> 5] = low;
    S.mtile[t >> 5] = most;
  }
  __syncthreads();
  Share sh{0, 0, split ? 0 : C, S.ncol};
  if (split)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      sh.base += S.scan_w[w];
      sh.most = max(sh.most, S.mtile[w]);
    }
  for (int k = 0; k < S.ncol; ++k) sh.count += S.cnt[k];
  if (t == 0) {
    int acc = 0;
    for (int k = 0; k < S.ncol; ++k) {
      S.coff[k] = acc;
      acc += S.cnt[k];
    }
  }
  __syncthreads();
  for (int c = t; c < C; c += blockDim.x) {
    if (split && X.blab[c] != rank) continue;
    const int k = X.color[c];
    const int p = S.coff[k] + atomicAdd(&S.cur[k], 1);
    S.order[p] = (unsigned short)c;
    S.pcol[p] = (unsigned char)k;
    S.pa[p] = (unsigned short)X.bl[X.la[c]];
    S.pb[p] = (unsigned short)X.bl[X.lb[c]];
    S.comp[p] = split ? (unsigned short)X.lab[c] : 0;
  }
  __syncthreads();
  return sh;
}

// One side of a manifold row: directions, this side's arm, inertia-applied
// arms and inverse mass, omega / g per direction, bias terms, impulses.
struct HalfRow {
  d3 n, t1, t2, r, In, It1, It2;
  double im, gn, gt1, gt2, bn, brest;
  double ln, l1, l2;
};

__device__ inline d3 shfl_pair(unsigned mask, d3 a) {
  return {__shfl_xor_sync(mask, a.x, 1), __shfl_xor_sync(mask, a.y, 1), __shfl_xor_sync(mask, a.z, 1)};
}

// build_row of contact c for one side (lane pairs of whole warps call it);
// with feat, side 0 writes the learned start's features 0-6 of slot p.
// Returns bit 0: impact, bit 1: in the warm cache (or a wall row).
__device__ __noinline__ int build_half(const NscView& V, int c, int side, int W, const unsigned long long* keys,
                                       HalfRow& h, float* feat, int p, double& phi_out, double& vnp_out) {
  const State& st = V.st;
  const Contacts& con = V.con;
  const rg_config& cfg = V.cfg;
  const unsigned all = 0xffffffffu;
  const double beta = cfg.nsc_position_stabilization ? cfg.nsc_beta * 0.01 : cfg.nsc_beta;
  const int a = con.a[c], b = con.b[c];
  const int bd = side ? b : a;
  const bool wall = a == b, live = !(wall && side);
  const d3 n{con.comp(6)[c], con.comp(7)[c], con.comp(8)[c]};
  const double phi = con.comp(12)[c] - con.comp(13)[c];
  const int pk = side ? 3 : 0;
  const d3 pt{con.comp(pk)[c], con.comp(pk + 1)[c], con.comp(pk + 2)[c]};
  const d3 x = st.x.ld(bd), v = st.v.ld(bd), w = st.w.ld(bd), Iinv = st.Iinv.ld(bd);
  const dq q = st.q.ld(bd);
  const double im = live ? st.inv_mass[bd] : 0.0, rest = st.rest[bd];
  const d3 sh{con.comp(9)[c], con.comp(10)[c], con.comp(11)[c]};
  const d3 ref = fabs(n.x) < 0.9 ? mk3(1, 0, 0) : mk3(0, 1, 0);
  const d3 cr = cross(n, ref);
  const d3 t1 = cr / len(cr);
  const d3 t2 = cross(n, t1);
  d3 r = side ? pt - (x + sh) : pt - x;
  if (!live) r = mk3(0, 0, 0);
  // iinv_apply of the three arms (the columns of the rotation once)
  d3 c0, c1, c2;
  rot_cols(q, c0, c1, c2);
  auto iinv = [&](d3 m) {
    if (im <= 0.0) return mk3(0, 0, 0);
    const double b0 = dot(c0, m) * Iinv.x, b1 = dot(c1, m) * Iinv.y, b2 = dot(c2, m) * Iinv.z;
    return c0 * b0 + c1 * b1 + c2 * b2;
  };
  const d3 rn = cross(r, n), rt1 = cross(r, t1), rt2 = cross(r, t2);
  h.n = n; h.t1 = t1; h.t2 = t2; h.r = r; h.im = im;
  h.In = iinv(rn); h.It1 = iinv(rt1); h.It2 = iinv(rt2);
  // diag_of: both sides' terms in the order 1/ma + 1/mb + A + B + cfm
  const double imo = __shfl_xor_sync(all, im, 1);
  const double ima = side ? imo : im, imb = side ? im : imo;
  auto diag = [&](double mine) {
    const double other = __shfl_xor_sync(all, mine, 1);
    const double A = side ? other : mine, B = side ? mine : other;
    const double g = ima + imb + A + B + cfg.nsc_cfm;
    return cfg.nsc_omega / smax(g, 1e-12);
  };
  h.gn = diag(dot(rn, h.In));
  h.gt1 = diag(dot(rt1, h.It1));
  h.gt2 = diag(dot(rt2, h.It2));
  d3 u = v + cross(w, r);
  if (!live) u = mk3(0, 0, 0);
  const d3 uo = shfl_pair(all, u);
  const d3 uA = side ? uo : u, uB = side ? u : uo;
  const d3 vrel = wall ? -uA : uB - uA;
  const double vnp = dot(n, vrel);
  const double ro = __shfl_xor_sync(all, rest, 1);
  const double e = wall ? rest : (side ? smin(ro, rest) : smin(rest, ro));
  h.bn = phi < 0.0 ? beta * phi / cfg.dt : 0.0;
  h.brest = vnp < 0.0 ? e * vnp : 0.0;
  int cached = wall ? 2 : 0;  // walls start cold and are left alone by the learned start
  h.ln = h.l1 = h.l2 = 0.0;
  if (!wall && cfg.nsc_warm_start != RG_WARM_NONE && W > 0) {
    const unsigned long long k = ((unsigned long long)(unsigned)a << 32) | (unsigned)b;
    const int f = lower_bound_key(keys, W, k);
    if (f < W && keys[f] == k) {
      cached = 2;
      h.ln = smax(0.0, V.wlam[f]);
      h.l1 = V.wlam[V.wcap + f];
      h.l2 = V.wlam[2 * V.wcap + f];
    }
  }
  if (feat && side == 0) {
    const size_t fld = (size_t)V.ccap;
    feat[p] = (float)phi;
    feat[fld + p] = (float)vnp;
    feat[2 * fld + p] = (float)dot(t1, vrel);
    feat[3 * fld + p] = (float)dot(t2, vrel);
    feat[4 * fld + p] = (float)h.ln;
    feat[5 * fld + p] = (float)h.l1;
    feat[6 * fld + p] = (float)h.l2;
  }
  phi_out = phi;
  vnp_out = vnp;
  return (vnp < -1e-6 ? 1 : 0) | cached;
}

// Half rows of slots beyond the registers: the global row arrays (RowIO).
__device__ inline void half_store(const RowIO& R, int p, int side, const HalfRow& h) {
  if (side == 0) {
    R.w3(R_N, p, h.n); R.w3(R_T1, p, h.t1); R.w3(R_T2, p, h.t2);
    R.r(R_GN, p) = h.gn; R.r(R_GT1, p) = h.gt1; R.r(R_GT2, p) = h.gt2;
    R.r(R_BN, p) = h.bn; R.r(R_BREST, p) = h.brest;
    R.lam[p] = h.ln; R.lam[R.ccap + p] = h.l1; R.lam[2 * (size_t)R.ccap + p] = h.l2;
  }
  R.w3(side ? R_RB : R_RA, p, h.r);
  R.w3(side ? R_IBN : R_IAN, p, h.In);
  R.w3(side ? R_IBT1 : R_IAT1, p, h.It1);
  R.w3(side ? R_IBT2 : R_IAT2, p, h.It2);
  R.r(side ? R_IMB : R_IMA, p) = h.im;
}
__device__ inline void half_load(const RowIO& R, int p, int side, HalfRow& h) {
  h.n = R.r3(R_N, p); h.t1 = R.r3(R_T1, p); h.t2 = R.r3(R_T2, p);
  h.gn = R.r(R_GN, p); h.gt1 = R.r(R_GT1, p); h.gt2 = R.r(R_GT2, p);
  h.bn = R.r(R_BN, p); h.brest = R.r(R_BREST, p);
  h.ln = R.lam[p]; h.l1 = R.lam[R.ccap + p]; h.l2 = R.lam[2 * (size_t)R.ccap + p];
  h.r = R.r3(side ? R_RB : R_RA, p);
  h.In = R.r3(side ? R_IBN : R_IAN, p);
  h.It1 = R.r3(side ? R_IBT1 : R_IAT1, p);
  h.It2 = R.r3(side ? R_IBT2 : R_IAT2, p);
  h.im = R.r(side ? R_IMB : R_IMA, p);
}

// The six numbers of a body slot (three 16-byte words).
__device__ inline void slot_ld(const double* vs, d3& v, d3& w) {
  const double2 p = *reinterpret_cast<const double2*>(vs), q = *reinterpret_cast<const double2*>(vs + 2),
                r = *reinterpret_cast<const double2*>(vs + 4);
  v = mk3(p.x, p.y, q.x);
  w = mk3(q.y, r.x, r.y);
}
__device__ inline void slot_st(double* vs, d3 v, d3 w) {
  *reinterpret_cast<double2*>(vs) = make_double2(v.x, v.y);
  *reinterpret_cast<double2*>(vs + 2) = make_double2(v.z, w.x);
  *reinterpret_cast<double2*>(vs + 4) = make_double2(w.y, w.z);
}

// Warm-start impulses of one side (warm_apply).
__device__ inline void warm_half(const HalfRow& h, double* vs, int side) {
  d3 v, w;
  slot_ld(vs, v, w);
  auto imp = [&](d3 d, d3 I, double l) {
    if (l == 0.0) return;
    const d3 dv = d * (l * h.im), dw = I * l;
    v = side ? v + dv : v - dv;
    w = side ? w + dw : w - dw;
  };
  imp(h.n, h.In, h.ln);
  imp(h.t1, h.It1, h.l1);
  imp(h.t2, h.It2, h.l2);
  slot_st(vs, v, w);
}

// sqrt(max(0, a)), without the square root's special-value path for the
// a <= 0 of contacts at or inside their friction limit's end.
__device__ inline double cone_limit(double a) { return a > 0.0 ? sqrt(a) : 0.0; }

// One Gauss-Seidel row update by a lane pair (psor_row); act: the lanes of
// the warp that call it.  Both lanes form the same relative velocity and
// impulses; each updates its own body.  Straight-line: an impulse change of
// zero adds zero instead of branching around the update (a branch per
// direction and the reconvergence after it took a fifth of the 1,450 cycles
// of the branching form; 1,160 now, two square roots among them).  Returns
// |dλn| + |dλt1| + |dλt2|.
__device__ __forceinline__ double psor_half(HalfRow& h, double* vs, int side, bool wall, unsigned act, double cfm,
                                            double mu) {
  const bool live = !(wall && side);  // a wall takes no impulse and stays at rest
  d3 v{0, 0, 0}, w{0, 0, 0};
  if (live) slot_ld(vs, v, w);
  const d3 u = v + cross(w, h.r);
  const d3 uo = shfl_pair(act, u);
  const d3 uA = side ? uo : u, uB = side ? u : uo;
  d3 vrel = wall ? -uA : uB - uA;
  // impulse change d along dir: this side's velocities, and the change of
  // the relative velocity it makes (side A's first, then side B's)
  auto kick = [&](d3 dir, d3 I, double d, bool last) {
    const d3 dv = dir * (d * h.im), dw = I * d;
    v = side ? v + dv : v - dv;
    w = side ? w + dw : w - dw;
    if (last) return;
    const d3 X = dv + cross(dw, h.r);
    const d3 Xo = shfl_pair(act, X);
    vrel = vrel + (side ? Xo : X);
    vrel = vrel + (side ? X : Xo);
  };
  const double wn = dot(h.n, vrel) + h.bn + h.brest + cfm * h.ln;
  const double ln = smax(0.0, h.ln + -h.gn * wn);
  const double dn = ln - h.ln;
  kick(h.n, h.In, dn, false);
  const double mf = mu * ln;
  const double lim1 = cone_limit(mf * mf - h.l2 * h.l2);
  const double w1 = dot(h.t1, vrel) + cfm * h.l1;
  const double l1 = smin(smax(h.l1 + -h.gt1 * w1, -lim1), lim1);
  const double d1 = l1 - h.l1;
  kick(h.t1, h.It1, d1, false);
  const double lim2 = cone_limit(mf * mf - l1 * l1);
  const double w2 = dot(h.t2, vrel) + cfm * h.l2;
  const double l2 = smin(smax(h.l2 + -h.gt2 * w2, -lim2), lim2);
  const double d2 = l2 - h.l2;
  kick(h.t2, h.It2, d2, true);
  if (live) slot_st(vs, v, w);
  h.ln = ln; h.l1 = l1; h.l2 = l2;
  return fabs(dn) + fabs(d1) + fabs(d2);
}

// ---- sweeps of a block's share ----------------------------------------------
// Up to n sweeps; with stop >= 0 the block alone decides and leaves after the
// first sweep whose every change is below `stop`.  S.locs gets each sweep's
// residuals (per lane of the one warp, else per warp).  Returns the sweeps
// made; fewer than n with stop < 0 only when the last one changed nothing
// (so further ones would not either).  The state after sweep i < keep goes to
// S.vel[snap + i stride]: 6 nbody velocities, then the impulses per slot.
struct Sweep {
  int colors, n;
  double stop;
  int keep, snap, stride;
};
template <bool ONE>
__device__ __forceinline__ void sweep_sync() {
  if (ONE) __syncwarp();
  else __syncthreads();
}
// ONE: at most 16 contacts, the first warp only and no block barrier.
template <bool ONE, class Row, class Update>
__device__ __forceinline__ int sweep_share(const Sweep w, int C, Row& h, Update update) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x, pair = t >> 1, side = t & 1;
  if (ONE && t >= 32) return 0;
  const int col = pair < C ? (int)S.pcol[pair] : -1;
  const int q0 = pair < C ? pair : 0;
  const bool wall = S.pa[q0] == S.pb[q0];
  double* vs = &S.vel[6 * (side ? S.pb[q0] : S.pa[q0])];
  const int nv = 6 * S.nbody;
  // One warp: a component that a sweep left unchanged stays so and its lanes
  // rest; a colour without other contacts costs nothing (in the sweeps of a
  // set that will not converge, most components are done early: a step of
  // 50000 rods 358 -> 346 us, of a set with more such sweeps 403 -> 384).
  const unsigned same = ONE ? __match_any_sync(0xffffffffu, pair < C ? (int)S.comp[pair] : -1) : 0u;
  bool rest = false;
  int i = 0;
  while (i < w.n) {
    double loc = 0.0;
    for (int k = 0; k < w.colors; ++k) {
      const bool mine = col == k && !rest;
      const unsigned act = __ballot_sync(0xffffffffu, mine);
      if (ONE && act == 0u) continue;
      if (mine) loc = update(h, vs, side, wall, act);
      if (k + 1 < w.colors) sweep_sync<ONE>();
    }
    double* ls = &S.locs[(i & (kChunk - 1)) * 32];
    if (ONE) {
      ls[t] = loc;
    } else {
      const double m = warp_max(loc);
      if ((t & 31) == 0) ls[t >> 5] = m;
    }
    ++i;
    if (ONE) {
      __syncwarp();  // (the votes below order nothing)
      rest = (__ballot_sync(0xffffffffu, loc != 0.0) & same) == 0u;
    }
    // one vote: goes on while a change reaches the limit (or, in a chunk,
    // while anything changes)
    const int more = w.stop >= 0.0 ? loc >= w.stop : loc != 0.0;
    if (!(ONE ? __any_sync(0xffffffffu, more) : __syncthreads_or(more))) break;
    if (i <= w.keep) {  // state after sweep i - 1
      double* sn = &S.vel[w.snap + (i - 1) * w.stride];
      for (int k = t; k < nv; k += ONE ? 32 : blockDim.x) sn[k] = S.vel[k];
      if (pair < C && side == 0) h.keep(sn + nv, pair);
      sweep_sync<ONE>();
    }
  }
  return i;
}
// The same over more contacts than lane pairs: rows from the global arrays.
template <class Row, class Update>
__device__ __forceinline__ int sweep_rows(const Sweep w, int C, const RowIO R, Update update) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x, pair = t >> 1, side = t & 1;
  int i = 0;
  while (i < w.n) {
    double loc = 0.0;
    for (int k = 0; k < w.colors; ++k) {
      for (int p0 = S.coff[k] & ~(kPairs - 1); p0 < S.coff[k] + S.cnt[k]; p0 += kPairs) {
        const int p = p0 + pair;
        const bool mine = p >= S.coff[k] && p < S.coff[k] + S.cnt[k];
        const unsigned act = __ballot_sync(0xffffffffu, mine);
        if (!mine) continue;
        Row g;
        g.load(R, p, side);
        const int sa = S.pa[p], sb = S.pb[p];
        loc = fmax(loc, update(g, &S.vel[6 * (size_t)(side ? sb : sa)], side, sa == sb, act));
        __syncwarp(act);  // both lanes have read the impulses
        if (side == 0) g.put(R, p);
      }
      if (k + 1 < w.colors) __syncthreads();
    }
    const double m = warp_max(loc);
    if ((t & 31) == 0) S.locs[(i & (kChunk - 1)) * 32 + (t >> 5)] = m;
    ++i;
    const int more = w.stop >= 0.0 ? loc >= w.stop : loc != 0.0;
    if (!__syncthreads_or(more)) break;
  }
  return i;
}

// Sweeps until the residual over the whole team is below tol, or max_it.
// run(w) makes sweeps, back(state) puts a kept state's impulses (nl a slot)
// back.  Returns false on a team error; res and sweeps as a single solver's.
template <class Run, class Back>
__device__ __forceinline__ bool sweep_until(const Team& T, const Share& sh, int nl, int max_it, double tol, int first,
                                            unsigned& chunk, Run run, Back back, double& res, int& sweeps) {
  SmallSmem& S = small_smem();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarp = (int)(blockDim.x >> 5);
  const int width = sh.count <= 16 ? 32 : nwarp;
  auto residual = [&](int i) {  // of sweep i, by every warp that calls it
    return warp_max(lane < width ? S.locs[(i & (kChunk - 1)) * 32 + lane] : 0.0);
  };
  res = 0.0;
  sweeps = 0;
  if (T.nb == 1) {
    const int made = sh.count ? run(Sweep{sh.colors, max_it, tol, 0, 0, 0}) : 0;
    if (t == 0) S.nloc = made;  // (the one-warp form returns 0 in the other warps)
    __syncthreads();
    sweeps = S.nloc;
    if (sweeps) res = residual(sweeps - 1);
    __syncthreads();
    return true;
  }
  if (max_it <= 0) return team_sync(T);  // every block has read what the others now write
  const int nv = 6 * S.nbody, stride = nv + nl * sh.count;
  // states that fit the velocity space of every block (two bodies a contact
  // at most); none where the impulses live in the global arrays
  const int room = sh.most > kPairs ? 0 : (kVel - 12 * sh.most) / ((12 + nl) * sh.most);
  int size = first;
  bool still = sh.count == 0;
  while (sweeps < max_it) {
    const int n = min(min(size, room + 1), max_it - sweeps);
    size = kChunk;
    int made = 0;
    if (!still) {
      made = run(Sweep{sh.colors, n, -1.0, n - 1, nv, stride});
      if (t == 0) S.nloc = made;
      __syncthreads();
      made = S.nloc;
    }
    // publish; the buffer after this one is cleared for the next chunk (every
    // block has read its last use: it arrived at the barrier after that)
    double* ring = T.ring() + (chunk % 3) * kChunk;
    for (int i = warp; i < made; i += nwarp) {
      const double v = residual(i);
      if (lane == 0 && v > 0.0) atomic_max_nonneg(&ring[i], v);
    }
    if (T.rank() == 0 && t < kChunk) T.ring()[((chunk + 1) % 3) * kChunk + t] = 0.0;
    ++chunk;
    if (!team_sync(T)) return false;
    if (t < n) S.res[t] = __ldcg(&ring[t]);
    __syncthreads();
    int m = 0;
    while (m < n && !(S.res[m] < tol)) ++m;
    const bool done = m < n;
    if (!done) m = n - 1;
    res = S.res[m];
    sweeps += m + 1;
    if (!still && m < made - 1) {  // back to the state after sweep m
      const double* sn = &S.vel[nv + m * stride];
      for (int k = t; k < nv; k += blockDim.x) S.vel[k] = sn[k];
      back(sn + nv);
    }
    // a share that a sweep left unchanged is done
    if (!done && made < n) still = true;
    __syncthreads();
    if (done) break;
  }
  return true;
}

// The impulse part of a velocity row, and its place in the global arrays.
struct VelRow : HalfRow {
  __device__ void keep(double* o, int p) const { o[3 * p] = ln; o[3 * p + 1] = l1; o[3 * p + 2] = l2; }
  __device__ void back(const double* o, int p) { ln = o[3 * p]; l1 = o[3 * p + 1]; l2 = o[3 * p + 2]; }
  __device__ void load(const RowIO& R, int p, int side) { half_load(R, p, side, *this); }
  __device__ void put(const RowIO& R, int p) const {
    R.lam[p] = ln; R.lam[R.ccap + p] = l1; R.lam[2 * (size_t)R.ccap + p] = l2;
  }
};
template <bool ONE>
__device__ __noinline__ int vel_sweep(const Sweep w, int C, VelRow& row, double cfm, double mu) {
  VelRow h = row;
  const int made = sweep_share<ONE>(w, C, h, [&](VelRow& r, double* vs, int side, bool wall, unsigned act) {
    return psor_half(r, vs, side, wall, act, cfm, mu);
  });
  row.ln = h.ln; row.l1 = h.l1; row.l2 = h.l2;
  return made;
}
__device__ __noinline__ int vel_sweep_rows(const Sweep w, int C, const RowIO R, double cfm, double mu) {
  return sweep_rows<VelRow>(w, C, R, [&](VelRow& r, double* vs, int side, bool wall, unsigned act) {
    return psor_half(r, vs, side, wall, act, cfm, mu);
  });
}

// Contact sets that the team's first block solves alone: those that fit its
// registers (a chunk's barrier costs more than the sweeps it saves), and
// recorded ones, whose records keep one block's slot order.
__device__ inline bool solo(int C, bool recording) { return C <= kPairs || recording; }

// Colouring, manifold rows, PSOR and the warm cache for C <= kSmallC.
__device__ __noinline__ bool small_solve(const Team& team, const NscView& V, int C, int Cp, unsigned& chunk,
                                         PhaseClock& pc) {
  SmallSmem& S = small_smem();
  if (solo(C, V.rec_cap > 0) && team.rank() != 0) return true;
  Team T = team;
  if (solo(C, V.rec_cap > 0)) T.nb = 1;
  Ctl* ctl = V.ctl;
  const rg_config& cfg = V.cfg;
  const int t = threadIdx.x, pair = t >> 1, side = t & 1;
  if (C == 0) {
    if (t == 0) {
      *V.wn = 0;
      ctl->colors = 0;
      ctl->vel_contacts = 0;
      ctl->residual = 0.0;
      ctl->sweeps_last = 0;
    }
    return true;
  }
  // the learned start's gate is known now: its first hidden layer travels to
  // shared memory while the colouring and the rows are built
  const bool mlp_gate = V.use_mlp && (*(volatile int*)V.wn == 0 ||
                                      *(volatile int*)&ctl->sweeps_last > V.mlp_min_sweeps);
  const int W = *(volatile int*)V.wn;
  const int rec_base = V.rec_cap > 0 ? *(volatile int*)&ctl->rec_n : 0;
  if (mlp_gate) stage_bf16(S.wh, kWhLd, V.mlp.w2, kMlpH, kMlpH);
  small_map(V, C);
  pc.mark(10);
  const int K = small_color(V, C, T.rank() == 0);
  if (K < 0) {
    if (mlp_gate) stage_wait();
    return false;
  }
  const Share sh = small_split(T, C, K);
  const int Cl = sh.count;
  pc.mark(2);
  // ---- manifold rows: slot j kPairs + pair of a lane pair, j = 0, 1, .. ----
  const unsigned long long* keys = V.wkey;
  if (cfg.nsc_warm_start != RG_WARM_NONE && W <= kVel && Cl > 0) {
    unsigned long long* ks = reinterpret_cast<unsigned long long*>(S.vel);
    for (int k = t; k < W; k += blockDim.x) ks[k] = V.wkey[k];
    keys = ks;
  }
  int* deg = reinterpret_cast<int*>(S.stage);
  if (V.feat_on)
    for (int s = t; s < S.nbody; s += blockDim.x) deg[s] = 0;
  __syncthreads();
  const size_t cc = (size_t)V.ccap;
  const RowIO R{V.row + sh.base, V.lam + sh.base, V.ccap};  // this block's slots
  float* feat = V.feat + sh.base;
  const int nt = (Cl + kPairs - 1) / kPairs;
  VelRow row = {};
  int coll = 0;
#pragma unroll 1
  for (int j = 0; j < nt; ++j) {
    const int p = j * kPairs + pair;
    if (j * kPairs + (t >> 5) * 16 >= Cl) continue;  // no contact in this warp
    const bool valid = p < Cl;
    const int c = S.order[valid ? p : Cl - 1];
    double phi, vnp;
    const int br = build_half(V, c, side, W, keys, row, V.feat_on && valid ? feat : nullptr, p, phi, vnp);
    if (!valid) continue;
    if (nt > 1) half_store(R, p, side, row);
    if (side == 0) {
      coll += br & 1;
      S.cached[p] = (unsigned char)(br >> 1);
    }
    if (c < Cp) {  // wall rows (after the pairs) have no graph degree and no export
      const int sl = side ? S.pb[p] : S.pa[p];
      if (V.feat_on && S.dyn[sl]) atomicAdd(&deg[sl], 1);
      if (V.xrow) {  // contact-network export, warm-cache order
        const size_t wc = (size_t)V.wcap;
        double* xr = V.xrow + c;
        const int k0 = side ? 6 : 3;
        xr[k0 * wc] = row.r.x; xr[(k0 + 1) * wc] = row.r.y; xr[(k0 + 2) * wc] = row.r.z;
        if (side == 0) {
          xr[0] = row.n.x; xr[wc] = row.n.y; xr[2 * wc] = row.n.z;
          xr[9 * wc] = phi; xr[10 * wc] = vnp;
        }
      }
    }
  }
  coll = warp_sum_i(coll);
  if ((t & 31) == 0 && coll) atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->collisions), (unsigned long long)coll);
  __syncthreads();
  if (V.feat_on) {
    for (int p = t; p < Cl; p += blockDim.x) {
      const int sa = S.pa[p], sb = S.pb[p];
      feat[7 * cc + p] = (float)((S.dyn[sa] ? deg[sa] - 1 : 0) + (S.dyn[sb] ? deg[sb] - 1 : 0));
    }
    if (mlp_gate) {
      // the contacts the learned start is for (every contact, or those new
      // since the last step); the network runs only on tiles that hold one
      for (int k = t; k < kSmallC / 16; k += blockDim.x) S.mtile[k] = 0;
      __syncthreads();
      unsigned want = 0;
      for (int j = 0; j < nt; ++j) {
        const int p = j * kPairs + pair;
        if (p < Cl && S.order[p] < Cp && (V.mlp_all || !S.cached[p])) want |= 1u << j;  // never a wall row
        if ((want >> j) & 1u) S.mtile[p >> 4] = 1;
      }
      if (__syncthreads_or((int)want)) {
        // one warp per 16 contacts on the tensor cores, then the cone.  The
        // weights come from shared memory: W1, W4 and the small parameters
        // in stage, W2 in wh, W3 in the space of the velocities.
        const MlpStage ms = mlp_stage_at(S.stage);
        __nv_bfloat16* w3s = reinterpret_cast<__nv_bfloat16*>(S.vel);
        float* pred = V.pred + sh.base;
        stage_small(ms, V.mlp);  // W2 is already on its way (start of the solve)
        stage_bf16(w3s, kWhLd, V.mlp.w3, kMlpH, kMlpH);
        stage_wait();
        __syncthreads();
        const MlpSmall q = ms.small();
        const int lane = t & 31;
        for (int tile = t >> 5; tile * 16 < Cl; tile += blockDim.x >> 5) {
          if (!S.mtile[tile]) continue;
          unsigned a[8][4];
          mlp_layer1(ms.w1, kW1Ld, q, feat, V.ccap, tile * 16, Cl, lane, a);
          hidden_layer(a, S.wh, kWhLd, q.b2, lane);
          hidden_layer(a, w3s, kWhLd, q.b3, lane);
          mlp_layer4(a, ms.w4, kWhLd, q, pred, V.ccap, tile * 16, Cl, lane);
        }
        __syncthreads();
        for (int j = 0; j < nt; ++j) {
          if (!((want >> j) & 1u)) continue;
          const int p = j * kPairs + pair;
          if (nt == 1) mlp_apply(row.ln, row.l1, row.l2, pred, V.ccap, p, cfg.nsc_mu);
          else if (side == 0) mlp_apply(R.lam[p], R.lam[cc + p], R.lam[2 * cc + p], pred, V.ccap, p, cfg.nsc_mu);
        }
      }
    }
  }
  if (mlp_gate) stage_wait();  // no copy outlives the solve
  // body velocities on chip (the keys and the third layer are done with)
  __syncthreads();
  for (int s = t; s < S.nbody; s += blockDim.x) {
    const int x = S.body[s];
    slot_st(&S.vel[6 * s], V.st.v.ld(x), V.st.w.ld(x));
  }
  __syncthreads();
  pc.mark(3);
  // ---- PSOR ----
  const double cfm = cfg.nsc_cfm, mu = cfg.nsc_mu, tol = cfg.nsc_tol;
  if (cfg.nsc_warm_start != RG_WARM_NONE) {
    for (int k = 0; k < sh.colors; ++k) {
      for (int j = 0; j < nt; ++j) {
        const int p = j * kPairs + pair;
        if (p >= Cl || S.pcol[p] != k || (S.pa[p] == S.pb[p] && side)) continue;
        double* vs = &S.vel[6 * (size_t)(side ? S.pb[p] : S.pa[p])];
        if (nt == 1) {
          warm_half(row, vs, side);
        } else {
          VelRow g;
          g.load(R, p, side);
          warm_half(g, vs, side);
        }
      }
      __syncthreads();
    }
  }
  double res = 0.0;
  int sweeps = 0;
  const bool ok = sweep_until(
      T, sh, 3, cfg.nsc_velocity_iters, tol, 8, chunk,
      [&](const Sweep& w) {
        if (nt > 1) return vel_sweep_rows(w, Cl, R, cfm, mu);
        return Cl <= 16 ? vel_sweep<true>(w, Cl, row, cfm, mu) : vel_sweep<false>(w, Cl, row, cfm, mu);
      },
      [&](const double* o) {
        if (pair < Cl) row.back(o, pair);
      },
      res, sweeps);
  if (!ok) return false;
  pc.mark(4);
  // velocities back; warm cache and impulse sums (contact order)
  for (int s = t; s < S.nbody; s += blockDim.x) {
    if (!S.dyn[s]) continue;
    const int x = S.body[s];
    d3 v, w;
    slot_ld(&S.vel[6 * s], v, w);
    V.st.v.st(x, v);
    V.st.w.st(x, w);
  }
  double jn = 0, jt = 0;
  for (int j = 0; j < nt && side == 0; ++j) {
    const int p = j * kPairs + pair;
    if (p >= Cl) break;
    const int c = S.order[p];
    const bool reg = nt == 1;
    const double l0 = reg ? row.ln : R.lam[p], l1 = reg ? row.l1 : R.lam[cc + p], l2 = reg ? row.l2 : R.lam[2 * cc + p];
    if (c < Cp) {  // wall rows start cold every step: they stay out of the cache
      V.wkey[c] = ((unsigned long long)(unsigned)V.con.a[c] << 32) | (unsigned)V.con.b[c];
      V.wlam[c] = l0;
      V.wlam[V.wcap + c] = l1;
      V.wlam[2 * V.wcap + c] = l2;
      reinterpret_cast<int*>(V.wlam + 3 * (size_t)V.wcap)[c] = S.pcol[p];
    }
    if (V.rec_cap > 0 && rec_base + p < V.rec_cap) {
      // record (features, converged impulses) in slot order
      const size_t r = (size_t)(rec_base + p);
      for (int k = 0; k < kMlpIn; ++k) V.rec_x[r * kMlpIn + k] = feat[(size_t)k * cc + p];
      V.rec_y[r * kMlpOut] = (float)l0;
      V.rec_y[r * kMlpOut + 1] = (float)l1;
      V.rec_y[r * kMlpOut + 2] = (float)l2;
    }
    jn += fabs(l0);  // profile-CSV sums of main.cpp:3339-3343
    jt += fabs(l1) + fabs(l2);
  }
  jn = warp_sum(jn);
  jt = warp_sum(jt);
  if ((t & 31) == 0 && (jn != 0.0 || jt != 0.0)) {
    atomicAdd(&ctl->jn_sum, jn);
    atomicAdd(&ctl->jt_sum, jt);
  }
  __syncthreads();
  if (t == 0 && T.rank() == 0) {
    if (V.rec_cap > 0 && C > 0) ctl->rec_n = rec_base + C;
    *V.wn = Cp;
    ctl->vel_contacts = C;
    ctl->residual = res;
    ctl->sweeps_last = sweeps;
    if (C > 0) {
      ctl->sweeps_sum += sweeps;
      ctl->row_sweeps += (long long)C * sweeps;
      ctl->contact_steps += C;
      if (res >= cfg.nsc_tol) ctl->not_conv += 1;
      if (res > ctl->max_residual) ctl->max_residual = res;
    }
  }
  return true;
}

// One side of a projection row: normal, arm, inertia-applied arm, inverse
// mass, phi + slop, omega / g and the accumulated correction.
struct HalfPos {
  d3 n, r, In;
  double im, phi, og, l;
};
// What a lane keeps of its body and contact over the projection passes.
struct PosSide {
  d3 Iinv;
  double im, h, rsum;
};
// The row of a contact for one side at its body's position x, q (lane pairs
// of whole warps call it): the geometry the detection computes, from the
// pair's own positions.  Returns 1 when the contact penetrates.
__device__ __noinline__ int build_half_pos(const NscView& V, const d3 x, const dq q, const PosSide& b, int side,
                                           HalfPos& h) {
  const rg_config& cfg = V.cfg;
  const unsigned all = 0xffffffffu;
  const d3 u = axis_y(q);
  const d3 xo = shfl_pair(all, x), uo = shfl_pair(all, u);
  const double ho = __shfl_xor_sync(all, b.h, 1), imo = __shfl_xor_sync(all, b.im, 1);
  const d3 xa = side ? xo : x, ua = side ? uo : u, xb = side ? x : xo, ub = side ? u : uo;
  const Seg A{xa.x, xa.y, xa.z, side ? ho : b.h, ua.x, ua.y, ua.z, 0.0};
  const Seg B{xb.x, xb.y, xb.z, side ? b.h : ho, ub.x, ub.y, ub.z, 0.0};
  const Narrow nr = narrow_pair(A, B, V.box);
  const d3 diff = nr.pb - nr.pa;
  const double dist = len(diff);
  const double phi = dist - b.rsum;
  const int act = phi < -cfg.nsc_slop ? 1 : 0;
  if (!__any_sync(all, act)) return 0;
  const d3 nv = dist > 1e-10 ? diff / dist : mk3(1, 0, 0);
  const d3 r = side ? nr.pb - (xb + nr.sh) : nr.pa - xa;
  const d3 rn = cross(r, nv);
  h.n = nv; h.r = r;
  h.im = b.im;
  h.In = b.im <= 0.0 ? mk3(0, 0, 0) : rot_diag_apply(q, b.Iinv, rn);
  const double mine = dot(rn, h.In), other = __shfl_xor_sync(all, mine, 1);
  const double g = (side ? imo : h.im) + (side ? h.im : imo) + (side ? other : mine) + (side ? mine : other) + cfg.nsc_cfm;
  h.og = cfg.nsc_omega / smax(g, 1e-12);
  h.phi = phi + cfg.nsc_slop;
  h.l = 0.0;
  return act;
}
__device__ inline void half_pos_store(const RowIO& R, int p, int side, const HalfPos& h) {
  if (side == 0) {
    R.w3(R_N, p, h.n);
    R.r(R_PHI, p) = h.phi;
    R.r(R_GN, p) = h.og;
    R.lam[p] = h.l;
  }
  R.w3(side ? R_RB : R_RA, p, h.r);
  R.w3(side ? R_IBN : R_IAN, p, h.In);
  R.r(side ? R_IMB : R_IMA, p) = h.im;
}
__device__ inline void half_pos_load(const RowIO& R, int p, int side, HalfPos& h) {
  h.n = R.r3(R_N, p);
  h.phi = R.r(R_PHI, p);
  h.og = R.r(R_GN, p);
  h.l = R.lam[p];
  h.r = R.r3(side ? R_RB : R_RA, p);
  h.In = R.r3(side ? R_IBN : R_IAN, p);
  h.im = R.r(side ? R_IMB : R_IMA, p);
}
// One projection row update by a lane pair; vs: dx, dθ of this side's slot.
// Returns |dλ|.
__device__ __forceinline__ double pos_half(HalfPos& h, double* vs, int side, unsigned act, int penetrates, double cfm) {
  d3 dx, dt;
  slot_ld(vs, dx, dt);
  const d3 cr = cross(dt, h.r);
  // n . (((dx_b + dθ_b x r_b) - dx_a) - dθ_a x r_a)
  const d3 mine = side ? dx + cr : dx;
  const d3 other = shfl_pair(act, mine), cro = shfl_pair(act, cr);
  const d3 rel = side ? (mine - other) - cro : (other - mine) - cr;
  if (!penetrates) return 0.0;
  const double r = dot(h.n, rel) + h.phi + cfm * h.l;
  const double nl = smax(0.0, h.l + -h.og * r);
  const double dl = nl - h.l;
  if (dl != 0.0) {
    h.l = nl;
    const d3 ddx = h.n * (dl * h.im), ddt = h.In * dl;
    slot_st(vs, side ? dx + ddx : dx - ddx, side ? dt + ddt : dt - ddt);
  }
  return fabs(dl);
}

struct PosRow : HalfPos {
  int act;  // 1: the contact penetrates
  __device__ void keep(double* o, int p) const { o[p] = l; }
  __device__ void load(const RowIO& R, int p, int side) {
    half_pos_load(R, p, side, *this);
    act = og != 0.0;
  }
  __device__ void put(const RowIO& R, int p) const { R.lam[p] = l; }
};
template <bool ONE>
__device__ __noinline__ int pos_sweep(const Sweep w, int C, PosRow& row, double cfm) {
  PosRow h = row;
  const int made = sweep_share<ONE>(w, C, h, [&](PosRow& r, double* vs, int side, bool, unsigned act) {
    return pos_half(r, vs, side, act, r.act, cfm);
  });
  row.l = h.l;
  return made;
}
__device__ __noinline__ int pos_sweep_rows(const Sweep w, int C, const RowIO R, double cfm) {
  return sweep_rows<PosRow>(w, C, R, [&](PosRow& r, double* vs, int side, bool, unsigned act) {
    return pos_half(r, vs, side, act, r.act, cfm);
  });
}

// Position projection for C <= kSmallC (nsc_contact.cpp:698-879), split as
// the velocity solve.
__device__ __noinline__ bool small_project(const Team& team, const NscView& V, int C, unsigned& chunk) {
  SmallSmem& S = small_smem();
  if (solo(C, false) && team.rank() != 0) return true;
  Team T = team;
  if (solo(C, false)) T.nb = 1;
  const rg_config& cfg = V.cfg;
  const State& st = V.st;
  const int t = threadIdx.x, pair = t >> 1, side = t & 1;
  if (C == 0) return true;
  small_map(V, C);
  const int K = small_color(V, C, T.rank() == 0);
  if (K < 0) return false;
  const Share sh = small_split(T, C, K);
  const int Cl = sh.count;
  const double cfm = cfg.nsc_cfm;
  const RowIO R{V.row + sh.base, V.lam + sh.base, V.ccap};
  const int nt = (Cl + kPairs - 1) / kPairs;
  // Positions over the passes: in shared memory (the network's space) when
  // the share has one contact per lane pair, else in the state arrays.
  double* pos = reinterpret_cast<double*>(S.wh);
  static_assert(sizeof(S.wh) >= sizeof(double) * 7 * 2 * kPairs, "positions of a one-tier share");
  const bool chip = nt <= 1;
  auto side_of = [&](int p) {
    const int c = S.order[p], bd = S.body[side ? S.pb[p] : S.pa[p]];
    return PosSide{st.Iinv.ld(bd), st.inv_mass[bd], st.h[bd], V.con.comp(13)[c]};
  };
  PosSide mine = {};
  const int own = pair < Cl ? pair : Cl - 1;  // (unused lanes follow the last contact)
  if (Cl > 0 && chip) {
    mine = side_of(own);
    for (int s = t; s < S.nbody; s += blockDim.x) {
      const int x = S.body[s];
      const d3 p = st.x.ld(x);
      const dq q = st.q.ld(x);
      double* o = pos + 7 * s;
      o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = q.w; o[4] = q.x; o[5] = q.y; o[6] = q.z;
    }
  }
  bool moved = false;
  __syncthreads();
  for (int outer = 0; outer < cfg.nsc_position_iters; ++outer) {
    int any = 0;
    PosRow row = {};
#pragma unroll 1
    for (int j = 0; j < nt; ++j) {
      if (j * kPairs + (t >> 5) * 16 >= Cl) continue;  // no contact in this warp
      const int p = j * kPairs + pair;
      const bool valid = p < Cl;
      if (chip) {
        const double* o = pos + 7 * (side ? S.pb[own] : S.pa[own]);
        row.act = build_half_pos(V, mk3(o[0], o[1], o[2]), dq{o[3], o[4], o[5], o[6]}, mine, side, row);
      } else {
        const int pc = valid ? p : Cl - 1, bd = S.body[side ? S.pb[pc] : S.pa[pc]];
        const PosSide b = side_of(pc);
        row.act = build_half_pos(V, st.x.ld(bd), st.q.ld(bd), b, side, row);
      }
      if (!valid) continue;
      any |= row.act;
      if (!row.act) row.og = 0.0;
      if (nt > 1) half_pos_store(R, p, side, row);
    }
    for (int s = t; s < 6 * S.nbody; s += blockDim.x) S.vel[s] = 0.0;
    any = __syncthreads_or(any);
    if (T.nb == 1 && !any) break;  // nothing penetrates
    Share act = sh;
    if (!any) act.count = 0;  // nothing of this share moves, now or in a later pass
    double res;
    int its = 0;
    // a team's blocks learn whether anything penetrates from the first
    // sweep's residual: it is above zero exactly when something does.  Most
    // passes stop after one or two sweeps.
    const bool ok = sweep_until(
        T, act, 1, cfg.nsc_position_psor_iters, 1e-8, 2, chunk,
        [&](const Sweep& w) {
          if (nt > 1) return pos_sweep_rows(w, Cl, R, cfm);
          return Cl <= 16 ? pos_sweep<true>(w, Cl, row, cfm) : pos_sweep<false>(w, Cl, row, cfm);
        },
        [&](const double* o) {
          if (pair < Cl) row.l = o[pair];
        },
        res, its);
    if (!ok) return false;
    if (any) {
      moved = true;
      for (int s = t; s < S.nbody; s += blockDim.x) {
        if (!S.dyn[s]) continue;
        const int x = S.body[s];
        double* o = pos + 7 * s;
        d3 dx, th;
        slot_ld(&S.vel[6 * s], dx, th);
        d3 p = chip ? mk3(o[0], o[1], o[2]) : st.x.ld(x);
        dq q = chip ? dq{o[3], o[4], o[5], o[6]} : st.q.ld(x);
        p = p + dx;
        const double ang = len(th);
        if (ang > 1e-8) {
          const d3 ax = th / ang;
          q = qnormalize(qmul(angle_axis(ang, ax), q));
        }
        if (chip) {
          o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = q.w; o[4] = q.x; o[5] = q.y; o[6] = q.z;
        } else {
          st.x.st(x, p);
          st.q.st(x, q);
        }
      }
    }
    __syncthreads();
    if (T.nb > 1 && its == 1 && res == 0.0) break;  // nothing penetrated anywhere
  }
  if (moved)
    for (int s = t; s < S.nbody; s += blockDim.x) {
      if (!S.dyn[s]) continue;
      const int x = S.body[s];
      if (V.moved) V.moved[x] = 1;
      if (!chip) continue;
      const double* o = pos + 7 * s;
      st.x.st(x, mk3(o[0], o[1], o[2]));
      st.q.st(x, dq{o[3], o[4], o[5], o[6]});
    }
  return true;
}

// ---------------------------------------------------------------------------
// Cylinder walls of the velocity solve: for every dynamic capsule, contacts
// where its surface passes the tube wall at the two end points or the centre
// of its axis (collideCapsuleInsideCylinder, collision.cpp:197-241), in body
// order then sample order, appended after the Cp pair contacts as rows with
// b == a (main.cpp:4431-4447).  The team's first block lists them (block
// scan per round of rods); returns the total contact count.
// ---------------------------------------------------------------------------
__device__ inline int wall_hits(const NscView& V, int i, d3 ax, double R, d3* pt, d3* nrm, double* pen) {
  const State& st = V.st;
  if (!(st.inv_mass[i] > 0.0)) return 0;
  const double h = st.h[i], r = st.r[i];
  const d3 x = st.x.ld(i);
  d3 u = axis_y(st.q.ld(i));
  u = u / len(u);
  const d3 smp[3] = {x - u * h, x, x + u * h};
  int k = 0;
  for (int j = 0; j < 3; ++j) {
    const d3 p = smp[j];
    const d3 pp = p - ax * dot(p, ax);
    const double d = len(pp);
    const double pe = d + r - R;
    if (pe <= 0.0) continue;
    d3 nv;
    if (d > 1e-8) {
      nv = pp / d;
    } else {
      const d3 cr = cross(ax, fabs(ax.x) < 0.9 ? mk3(1, 0, 0) : mk3(0, 1, 0));
      nv = cr / len(cr);
    }
    if (pt) {
      pt[k] = p + nv * (R - d);
      nrm[k] = nv;
      pen[k] = pe;
    }
    ++k;
  }
  return k;
}

__device__ __noinline__ int wall_phase(const Team& T, const NscView& V, int Cp, SmemNsc& sm) {
  Ctl* ctl = V.ctl;
  const int n = V.st.n;
  const rg_config& cfg = V.cfg;
  if (T.rank() == 0) {
    d3 ax{cfg.cylinder_axis[0], cfg.cylinder_axis[1], cfg.cylinder_axis[2]};
    ax = ax / len(ax);
    const double R = cfg.cylinder_radius;
    int run = Cp;
    for (int base = 0; base < n; base += blockDim.x) {
      const int i = base + threadIdx.x;
      d3 pt[3], nv[3];
      double pe[3];
      const int k = i < n ? wall_hits(V, i, ax, R, pt, nv, pe) : 0;
      int tot;
      const int ex = block_excl_scan(k, sm.scan_w, tot);
      for (int j = 0; j < k; ++j) {
        const int c = run + ex + j;
        if (c >= V.ccap) break;
        V.con.a[c] = i;
        V.con.b[c] = i;
        V.con.type[c] = 3;  // wall
        V.con.comp(0)[c] = pt[j].x; V.con.comp(1)[c] = pt[j].y; V.con.comp(2)[c] = pt[j].z;
        V.con.comp(3)[c] = pt[j].x; V.con.comp(4)[c] = pt[j].y; V.con.comp(5)[c] = pt[j].z;
        V.con.comp(6)[c] = nv[j].x; V.con.comp(7)[c] = nv[j].y; V.con.comp(8)[c] = nv[j].z;
        V.con.comp(9)[c] = 0.0; V.con.comp(10)[c] = 0.0; V.con.comp(11)[c] = 0.0;
        V.con.comp(12)[c] = -pe[j];  // phi = comp12 - comp13 = -penetration
        V.con.comp(13)[c] = 0.0;
      }
      run += tot;
    }
    if (threadIdx.x == 0) {
      if (run > V.ccap) atomicOr(&ctl->err, ERR_CONTACT_CAP);
      ctl->contacts = run;
    }
  }
  if (!team_sync(T)) return -1;
  const int C = *(volatile int*)&ctl->contacts;
  return C > V.ccap ? -1 : C;
}

// ---------------------------------------------------------------------------
// One NSC step of one system by one team.
// ---------------------------------------------------------------------------
__device__ bool nsc_step(const Team& T, const NscView& V, SmemNsc& sm, unsigned& chunk, bool first) {
  SmallSmem& S = small_smem();
  Ctl* ctl = V.ctl;
  const State& st = V.st;
  const rg_config& cfg = V.cfg;
  const int n = st.n;
  const int tid = T.tid(), TS = T.size(), rank = T.rank();
  if (*(volatile int*)&ctl->err) return false;
  PhaseClock pc(ctl, rank == 0 && threadIdx.x == 0 && ctl->prof_phases);
  if (rank == 0 && threadIdx.x == 0) {
    ctl->collisions = 0;
    ctl->jn_sum = 0;
    ctl->jt_sum = 0;
  }
  // 1) free flight (main.cpp:4397-4408) + segment records + displacement
  {
    const d3 g{cfg.gravity[0], cfg.gravity[1], cfg.gravity[2]};
    double dmax = 0.0, dnear = 0.0;
    const double* ref2 = V.near ? V.ref2 : nullptr;
    double invL[3] = {1.0, 1.0, 1.0};
    for (int k = 0; k < 3; ++k)
      if (V.box.L[k] > 0.0) invL[k] = 1.0 / V.box.L[k];
    const StateBase SB{st.sbase, st.pbase, n};
    const double dt = cfg.dt;
    const double* ref = V.ref;
    Seg* seg = V.seg;
    const Box box = V.box;
    // Only the position update, the projection and the wrap move rods, and
    // the last two flag what they move: other rods keep the segment record
    // and displacement bounds of the position update (still folded into
    // ctl->maxdisp / near_disp), and need their velocities only.  The first
    // step of a launch refreshes every rod (the state may have been set
    // from the host).
    const unsigned char* moved = first ? nullptr : V.moved;
    for (int i = tid; i < n; i += TS) {
      if (moved && !moved[i]) free_flight_velocity(SB, i, g, dt);
      else free_flight_fused(SB, i, g, dt, ref, ref2, box, invL, seg, dmax, dnear);
    }
    double bm = block_reduce_max(dmax, sm.red_d);
    if (threadIdx.x == 0) atomic_max_nonneg(&ctl->maxdisp, bm);
    if (V.near) {
      double bn = block_reduce_max(dnear, sm.red_d);
      if (threadIdx.x == 0) atomic_max_nonneg(&ctl->near_disp, bn);
    }
    if (!team_sync(T)) return false;
  }
  pc.mark(0);
  // 2) detection (pairs, then cylinder walls), colouring, manifold rows
  const int Cp = detect_phase(T, V, 0.0, sm, false);
  if (Cp < 0) return false;
  const int C = cfg.cylinder_enabled ? wall_phase(T, V, Cp, sm) : Cp;
  if (C < 0) return false;
  pc.mark(1);
  const bool small = C <= kSmallC;
  if (small) {
    // colouring, rows, PSOR and warm cache on chip
    // (serial time of the batch's cost model: what one block does alone)
    const bool alone = solo(C, V.rec_cap > 0) && rank == 0 && threadIdx.x == 0;
    const unsigned long long ts = alone ? gtimer() : 0ull;
    if (!small_solve(T, V, C, Cp, chunk, pc)) return false;
    if (alone) ctl->serial_ns += (long long)(gtimer() - ts);
    pc.mark(10);
    if (!team_sync(T)) return false;
    pc.mark(11);
  } else {
  if (!color_phase(T, V, C, sm)) return false;
  pc.mark(2);
  {
    RowIO R{V.row, V.lam, V.ccap};
    const int W = *(volatile int*)V.wn;
    const double* im = st.inv_mass;
    int* deg = V.owner;  // free between colouring and the next colouring
    if (V.feat_on) {
      for (int c = tid; c < C; c += TS) {
        deg[V.con.a[c]] = 0;
        deg[V.con.b[c]] = 0;
      }
      if (!team_sync(T)) return false;
    }
    int coll = 0;
    for (int p = tid; p < C; p += TS) {
      const int c = V.order[p];
      coll += build_row(st, V.con, cfg, c, p, R, V.wkey, V.wlam, W, V.wcap, V.feat_on ? V.feat : nullptr, V.ccap) & 1;
      if (V.feat_on && c < Cp) {  // wall rows have no graph degree
        if (im[V.con.a[c]] > 0.0) atomicAdd(&deg[V.con.a[c]], 1);
        if (im[V.con.b[c]] > 0.0) atomicAdd(&deg[V.con.b[c]], 1);
      }
    }
    int bcoll = block_reduce_sum_i(coll, sm.red_i);
    if (threadIdx.x == 0 && bcoll)
      atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->collisions), (unsigned long long)bcoll);
    if (!team_sync(T)) return false;
    if (V.feat_on) {
      for (int p = tid; p < C; p += TS) {
        const int c = V.order[p], a = V.con.a[c], b = V.con.b[c];
        V.feat[7 * (size_t)V.ccap + p] = (float)((im[a] > 0.0 ? deg[a] - 1 : 0) + (im[b] > 0.0 ? deg[b] - 1 : 0));
      }
      if (V.use_mlp && (W == 0 || *(volatile int*)&ctl->sweeps_last > V.mlp_min_sweeps)) {
        // each warp of the team evaluates tiles of 16 slots on the tensor
        // cores; its own lanes then apply the tile's predictions.  Every
        // block stages the whole network in its (here unused) small-solve
        // shared memory: W1, W4 and the small parameters in stage, W2 in wh,
        // W3 in the space of the velocities.
        const MlpStage ms = mlp_stage_at(S.stage);
        __nv_bfloat16* w3s = reinterpret_cast<__nv_bfloat16*>(S.vel);
        stage_small(ms, V.mlp);
        stage_bf16(S.wh, kWhLd, V.mlp.w2, kMlpH, kMlpH);
        stage_bf16(w3s, kWhLd, V.mlp.w3, kMlpH, kMlpH);
        stage_wait();
        __syncthreads();
        if (!team_sync(T)) return false;
        const MlpSmall q = ms.small();
        const int lane = threadIdx.x & 31, gw = tid >> 5, nw = TS >> 5;
        for (int row0 = gw * 16; row0 < C; row0 += nw * 16) {
          const int p = row0 + (lane & 15);
          const bool want = lane < 16 && p < C && V.order[p] < Cp &&  // never a wall row
                            (V.mlp_all || !warm_cached(V, V.order[p], W));
          if (!__ballot_sync(0xffffffffu, want)) continue;  // no row of this tile needs the network
          unsigned a[8][4];
          mlp_layer1(ms.w1, kW1Ld, q, V.feat, V.ccap, row0, C, lane, a);
          hidden_layer(a, S.wh, kWhLd, q.b2, lane);
          hidden_layer(a, w3s, kWhLd, q.b3, lane);
          mlp_layer4(a, ms.w4, kWhLd, q, V.pred, V.ccap, row0, C, lane);
          __syncwarp();
          if (want)
            mlp_apply(R.lam[p], R.lam[R.ccap + p], R.lam[2 * (size_t)R.ccap + p], V.pred, V.ccap, p, cfg.nsc_mu);
          __syncwarp();
        }
      }
      if (!team_sync(T)) return false;
    }
  }
  pc.mark(3);
  // 3) PSOR
  if (!psor_phase(T, V, C, sm)) return false;
  pc.mark(4);
  }
  // 4) warm cache and impulse sums (large path); position update + segments
  {
    RowIO R{V.row, V.lam, V.ccap};
    double jn = 0, jt = 0;
    for (int p = tid; !small && p < C; p += TS) {
      int c = V.order[p];
      double l0 = R.lam[p], l1 = R.lam[R.ccap + p], l2 = R.lam[2 * R.ccap + p];
      if (c < Cp) {  // wall rows start cold every step: they stay out of the cache
        V.wkey[c] = ((unsigned long long)(unsigned)V.con.a[c] << 32) | (unsigned)V.con.b[c];
        V.wlam[c] = l0;
        V.wlam[V.wcap + c] = l1;
        V.wlam[2 * V.wcap + c] = l2;
        reinterpret_cast<int*>(V.wlam + 3 * (size_t)V.wcap)[c] = V.color[c];
        if (V.xrow) export_row(V.xrow, V.wcap, c, R, p);
      }
      jn += fabs(l0);  // profile-CSV sums of main.cpp:3339-3343
      jt += fabs(l1) + fabs(l2);
    }
    jn = warp_sum(jn);
    jt = warp_sum(jt);
    if ((threadIdx.x & 31) == 0 && (jn != 0.0 || jt != 0.0)) {
      atomicAdd(&ctl->jn_sum, jn);
      atomicAdd(&ctl->jt_sum, jt);
    }
    if (tid == 0 && !small) {
      *V.wn = Cp;
      ctl->vel_contacts = C;
    }
    int rec_base = 0;
    if (V.rec_cap > 0 && !small && C > 0) {
      // records (features, converged impulses) in slot order
      rec_base = *(volatile int*)&ctl->rec_n;
      for (int p = tid; p < C && rec_base + p < V.rec_cap; p += TS) {
        const size_t r = (size_t)(rec_base + p);
        for (int k = 0; k < kMlpIn; ++k) V.rec_x[r * kMlpIn + k] = V.feat[(size_t)k * V.ccap + p];
        for (int k = 0; k < kMlpOut; ++k) V.rec_y[r * kMlpOut + k] = (float)R.lam[(size_t)k * R.ccap + p];
      }
    }
    int bad = 0;
    double dmax = 0.0, dnear = 0.0;
    const double* ref2 = V.near ? V.ref2 : nullptr;
    double invL[3] = {1.0, 1.0, 1.0};
    for (int k = 0; k < 3; ++k)
      if (V.box.L[k] > 0.0) invL[k] = 1.0 / V.box.L[k];
    {
      const StateBase SB{st.sbase, st.pbase, n};
      const double dt = cfg.dt, w_max = cfg.w_max;
      const double ld = 1.0 - cfg.lin_damp * dt, ad = 1.0 - cfg.ang_damp * dt;
      const double* ref = V.ref;
      Seg* seg = V.seg;
      unsigned char* moved = V.moved;
      const bool spin = cfg.cylinder_enabled != 0;
      const Box box = V.box;
      for (int i = tid; i < n; i += TS)
        bad |= position_update_fused(SB, i, dt, ld, ad, w_max, ref, ref2, box, invL, seg, dmax, dnear, moved,
                                     spin);
    }
    if (bad) atomicOr(&ctl->err, ERR_NONFINITE);
    double bm = block_reduce_max(dmax, sm.red_d);
    if (threadIdx.x == 0) atomic_max_nonneg(&ctl->maxdisp, bm);
    if (V.near) {
      double bn = block_reduce_max(dnear, sm.red_d);
      if (threadIdx.x == 0) atomic_max_nonneg(&ctl->near_disp, bn);
    }
    if (!team_sync(T)) return false;
    // every block has read rec_n before the barrier
    if (V.rec_cap > 0 && !small && C > 0 && tid == 0) ctl->rec_n = rec_base + C;
  }
  pc.mark(5);
  // 5) position projection (nsc_contact.cpp:659-880)
  if (cfg.nsc_position_stabilization) {
    int C2 = detect_phase(T, V, 0.0, sm, true);
    if (C2 < 0) return false;
    pc.mark(6);
    if (C2 <= kSmallC) {
      const bool alone = solo(C2, false) && rank == 0 && threadIdx.x == 0;
      const unsigned long long ts = alone ? gtimer() : 0ull;
      if (!small_project(T, V, C2, chunk)) return false;
      if (alone) ctl->serial_ns += (long long)(gtimer() - ts);
      if (!team_sync(T)) return false;
    } else {
      if (!color_phase(T, V, C2, sm)) return false;
      pc.mark(7);
      if (!project_phase(T, V, C2, sm)) return false;
    }
    pc.mark(8);
  }
  // 6) PBC wrap + clear forces (main.cpp:4508-4527); the next step touches
  // rod i from this same thread, so no barrier is needed here.
  {
    const StateBase SB{st.sbase, st.pbase, n};
    const Box box = V.box;
    unsigned char* moved = V.moved;
    for (int i = tid; i < n; i += TS) wrap_clear_body(SB, box, i, moved);
  }
  return true;
}

// Each block finds its team (teams are sorted by b0), then runs nsteps steps
// of the team's systems, one system after the other within a step.  A
// system whose step failed (error bits set) returns at once from its later
// steps; the others carry on.
#ifndef RG_NSC_MIN_BLOCKS
#define RG_NSC_MIN_BLOCKS 1
#endif
__global__ void __launch_bounds__(kBlock, RG_NSC_MIN_BLOCKS) k_nsc_run(const NscView* views, const TeamDesc* teams, int nteams,
                                                   const int* members, int nsteps) {
  __shared__ SmemNsc sm;
  int lo = 0, hi = nteams;  // last team with b0 <= blockIdx.x
  while (hi - lo > 1) {
    int m = (lo + hi) >> 1;
    if (teams[m].b0 <= (int)blockIdx.x) lo = m;
    else hi = m;
  }
  const TeamDesc td = teams[lo];
  if ((int)blockIdx.x < td.b0 || (int)blockIdx.x >= td.b0 + td.nb) return;
  team_barriers_reset();
  const bool team_timer = td.t_ns && threadIdx.x == 0 && (int)blockIdx.x == td.b0;
  const unsigned long long t_start = team_timer ? gtimer() : 0ull;
  // The view is read in every phase, right after a barrier whose acquire has
  // emptied the L1 cache: from shared memory a field costs 30 cycles instead
  // of an L2 round trip in front of the load that needs it.
  __shared__ __align__(16) unsigned char view_words[sizeof(NscView)];
  const NscView& V = *reinterpret_cast<const NscView*>(view_words);
  unsigned chunk = 0;  // chunks of the split solve so far (all blocks of a team count alike)
  for (int s = 0; s < nsteps; ++s) {
    bool any = false;
    for (int m = td.first; m < td.first + td.count; ++m) {
      if (s == 0 || td.count > 1) {
        static_assert(sizeof(NscView) % 8 == 0, "copied in 8-byte words");
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&views[members ? members[m] : m]);
        __syncthreads();  // the member before is done with its view
        for (int k = threadIdx.x; k < (int)(sizeof(NscView) / 8); k += blockDim.x)
          reinterpret_cast<unsigned long long*>(view_words)[k] = src[k];
        __syncthreads();
      }
      Team T{td.b0, td.nb, td.bar, &V.ctl->err,
             V.cfg.spin_limit > 0 ? (long long)V.cfg.spin_limit : kSpinLimit,
             V.cfg.test_absent_blocks > 0 ? (unsigned)V.cfg.test_absent_blocks : 0u};
      const bool timer = threadIdx.x == 0 && (int)blockIdx.x == td.b0;
      const unsigned long long t0 = timer ? gtimer() : 0ull;
      any |= nsc_step(T, V, sm, chunk, s == 0);
      if (timer) V.ctl->member_ns += (long long)(gtimer() - t0);  // one writer per system
    }
    if (!any) break;
  }
  if (team_timer) *td.t_ns = (long long)(gtimer() - t_start);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
NscView make_view(rg_system* s) {
  NscView V;
  std::memset(&V, 0, sizeof(V));
  V.st = s->st;
  V.box = s->box;
  V.cfg = s->cfg;
  V.ctl = s->d_ctl;
  const Detector& d = s->det;
  V.seg = d.seg; V.nbr_cnt = d.nbr_cnt; V.nbr = d.nbr; V.maxnb = d.maxnb; V.ref = d.ref;
  V.words = d.mask_words; V.mask = d.hit_mask; V.hit_cnt = d.hit_cnt;
  V.cell_of = d.cell_of; V.cell_cnt = d.cell_cnt; V.cell_start = d.cell_start;
  V.cell_fill = d.cell_fill; V.cell_rods = d.cell_rods;
  V.grid = detector_grid(s);
  V.bounds = detector_bounds(s);
  V.skin = d.skin; V.margin = d.margin; V.cut_center = d.cut_center; V.all_pairs = d.all_pairs ? 1 : 0;
  V.con = s->con;
  const Nsc& N = s->nsc;
  V.row = N.row; V.lam = N.lam; V.color = N.color; V.order = N.order;
  V.color_cnt = N.color_cnt; V.color_off = N.color_off; V.cursor = N.cursor; V.remaining = N.remaining;
  V.pmax = N.pmax; V.cmask = N.cmask; V.owner = N.owner;
  V.wkey = N.wkey; V.wlam = N.wlam; V.wn = N.wn; V.wcap = N.wcap;
  V.xrow = s->export_on ? N.xrow : nullptr;
  V.dx = N.dx; V.prow = N.prow; V.pactive = N.pactive;
  V.ccap = s->ccap;
  V.blk = N.blk;
  V.near = d.near;
  V.ref2 = d.ref2;
  V.moved = d.moved;
  V.near_skin = d.near_skin;
  V.feat = s->d_feat;
  V.pred = s->d_pred;
  V.use_mlp = (s->cfg.nsc_warm_start == RG_WARM_MLP && s->mlp_ready) ? 1 : 0;
  V.mlp_all = s->cfg.nsc_mlp_scope == 1 ? 1 : 0;
  V.mlp_min_sweeps = s->cfg.nsc_mlp_min_sweeps;
  V.rec_cap = s->recording ? s->rec_cap : 0;
  V.rec_x = s->d_rec_x;
  V.rec_y = s->d_rec_y;
  V.feat_on = (V.use_mlp || V.rec_cap > 0) ? 1 : 0;
  if (V.use_mlp) V.mlp = mlp_dev(s);
  return V;
}

int nsc_team_blocks(const rg_system* s) {
  int nb = s->team_blocks;  // explicit team size (tests, sweeps)
  if (nb <= 0) nb = (s->n + 127) / 128;  // about one block per 128 rods, up to every SM
  if (nb < 1) nb = 1;
  if (nb > s->coop_blocks) nb = s->coop_blocks;
  return nb;
}

static void launch_coop(const void* fn, int grid, int block, void** args, cudaStream_t st,
                        size_t smem = 0) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RGL cudaLaunchKernelExC(&cfg, fn, args);
}

// nsteps NSC steps of one system as one persistent cooperative launch.
void nsc_run_launch(rg_system* s, int nsteps) {
  NscView V = make_view(s);
  const int nb = nsc_team_blocks(s);
  TeamDesc td{0, nb, 0, 1, s->nsc.bar};
  cudaMemcpyAsync(s->nsc.view_dev, &V, sizeof(NscView), cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->nsc.team_dev, &td, sizeof(TeamDesc), cudaMemcpyHostToDevice, s->stream);
  cudaMemsetAsync(s->nsc.bar, 0, kTeamBarBytes, s->stream);
  const NscView* views = reinterpret_cast<const NscView*>(s->nsc.view_dev);
  const TeamDesc* teams = reinterpret_cast<const TeamDesc*>(s->nsc.team_dev);
  int nteams = 1;
  const int* members = nullptr;
  void* args[] = {&views, &teams, &nteams, &members, &nsteps};
  ProfScope p(s, ST_OTHER);
  launch_coop((const void*)k_nsc_run, nb, kBlock, args, s->stream, sizeof(SmallSmem));
  s->contacts_fresh = Fresh::kNo;
}

cudaError_t nsc_allow_smem() {
  return cudaFuncSetAttribute((const void*)k_nsc_run, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(SmallSmem));
}

// nsteps steps of many systems as one persistent cooperative launch: teams
// (device array, sorted by b0) cover blocks [0, grid); team k runs the
// systems members[first_k .. first_k + count_k) of views.
void nsc_batch_launch(const NscView* views, const TeamDesc* teams, int nteams, const int* members, int grid,
                      int nsteps, cudaStream_t st) {
  void* args[] = {&views, &teams, &nteams, &members, &nsteps};
  launch_coop((const void*)k_nsc_run, grid, kBlock, args, st, sizeof(SmallSmem));
}

// Co-resident blocks of the persistent kernel per SM of the current device
// (its registers and shared memory decide; the cooperative launch needs them
// all resident).
int nsc_blocks_per_sm() {
  int k = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_nsc_run, kBlock, sizeof(SmallSmem)) != cudaSuccess || k < 1) {
    cudaGetLastError();
    k = 1;
  }
  return k;
}
size_t nsc_view_bytes() { return sizeof(NscView); }
size_t nsc_team_bytes() { return sizeof(TeamDesc); }

}  // namespace rg
