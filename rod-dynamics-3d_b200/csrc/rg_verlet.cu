// rg_verlet.cu - the velocity-Verlet step (soft and Hertz-Mindlin models) as
// one persistent kernel.
//
// The same step as the multi-kernel form (rg_api.cu verlet_step; App::
// physicsStep, src/app/main.cpp:4529-4810): forces at t, half kick and drift,
// detection, forces at t + dt, second half kick - the same expressions in the
// same order, so states, contacts and histories are bit-identical.  A team of
// co-resident blocks runs all steps of a call in one cooperative launch, with
// five bounded team barriers a step where the multi-kernel form has 25
// dependent kernels.  Teams of one launch are independent systems (batches).
//
// What makes five barriers enough:
//  * a contact's force is computed by the thread that writes the contact, in
//    the pass after the hit counts are known; the forces at the next step's
//    start reuse those contacts in place;
//  * a body's contacts are found without a sorted incidence table: those where
//    it is the first body are a run of the (a, b)-sorted list,
//    those where it is the second hang off it in a linked list, walked in
//    ascending order; together the contact order of the reference's sums;
//  * the history entry of a persisting contact is found through the previous
//    contact list (same first body, a handful of candidates) and rewritten in
//    place; the sorted table is merged only in evaluations that add a pair,
//    and entries past their retention are only passed over until the call
//    ends (or the table fills up), when they are removed.
//
// Bound: instruction and L2 latency of the five phases plus the barriers (1 to
// 2 us each) up to some 50,000 rods, then the two passes over the body state.
// Measured, multi-kernel form (one captured graph a step) -> this one, us per
// step: 1,000 rods 80 -> 33, 5,000 (soft) 104 -> 38, 20,000 103 -> 41, 100,000
// 130 -> 61, 400,000 279 -> 163, 1,000,000 441 -> 299 (5,000 contacts) and 641
// -> 360 (80,000 contacts).  It is the faster one at every size, so the
// multi-kernel form only serves the stage timers and contact queries.
#include <cstring>
#include <vector>

// Functions of their own here: inlined into the list rebuild, the registers
// that they take from its callers made every step 1 % slower (the PSOR kernel:
// the other way round).
#define RG_BUILD_INLINE __noinline__
#include "rg_team.cuh"
#include "rg_verlet_dev.cuh"

namespace rg {

constexpr int kVBlock = 2 * kTile;  // threads per block
constexpr int kIns = 512;           // inserted pairs sorted on chip

// Where one team stands in its system's call (the same in every block).
struct VerletRun {
  int H, cur;      // history entries (dead ones included), current table
  int C, cb;       // contacts, current contact list
  long long fr;    // evaluation counter
  bool idx_ok;     // hidx[cb] names the contacts' table entries
  int lo, hi;      // this block's rods
  HmConst hm;
};
struct VerletSmem {
  SmemNsc s;
  unsigned long long key[kIns], sorted[kIns];
};

__device__ inline bool v_is_hm(const VerletView& W) { return W.v.cfg.model == RG_MODEL_HERTZ_MINDLIN; }

// Entry of the current table, or -1.
__device__ inline int v_find(const VerletView& W, const VerletRun& r, int a, int b) {
  const unsigned long long k = pkey(a, b);
  const int p = lower_bound_u64(W.hkey[r.cur], r.H, k);
  return (p < r.H && W.hkey[r.cur][p] == k) ? p : -1;
}

// Geometry of a contact.
struct VContact {
  d3 pa, pb, n, sh;
  double dist, surf;
};
// Force of contact c of bodies in `in`, with table entry f (-1: none) whose
// value and frame are `old`, `frame`; updates the entry, or lists the pair
// for insertion.  energy: the contact's potential energy is wanted (of a call
// only the last evaluation's sum is kept).
__device__ inline void v_eval(const VerletView& W, const VerletRun& r, int c, const PairIn& in, const VContact& g, int f,
                              d3 old, long long frame, bool energy) {
  const int hc = W.hcap, cc = W.v.ccap;
  const bool hm = v_is_hm(W);
  // an entry past its retention was dropped by the evaluation before this one
  if (f < 0 || (hm && r.fr - frame > 5)) old = mk3(0, 0, 0);
  const PairForce p = hm ? hm_pair(in, W.v.cfg, r.hm, g.pa, g.pb, g.n, g.sh, g.dist, g.surf, old, energy)
                         : soft_pair(in, W.v.cfg, g.pa, g.pb, g.n, g.sh, g.dist, g.surf, old, energy);
  store_addends(W.cf, cc, c, p);
  if (energy) W.cf[12 * (size_t)cc + c] = p.pe;
  int added = 0;
  if (p.touch) {
    if (f >= 0) {
      double* hv = W.hval[r.cur];
      hv[f] = p.hist.x; hv[hc + f] = p.hist.y; hv[2 * (size_t)hc + f] = p.hist.z;
      W.hframe[r.cur][f] = r.fr;
    } else {
      W.newval[c] = p.hist.x; W.newval[cc + c] = p.hist.y; W.newval[2 * (size_t)cc + c] = p.hist.z;
      W.ins[atomicAdd(&W.v.ctl->ins_n[r.fr & 1], 1)] = c;
      added = 1;
    }
  }
  W.touched[c] = added;
  W.hidx[r.cb][c] = f;
}
__device__ inline d3 v_old(const VerletView& W, const VerletRun& r, int f, long long& frame) {
  if (f < 0) return mk3(0, 0, 0);
  const double* hv = W.hval[r.cur];
  const int hc = W.hcap;
  frame = W.hframe[r.cur][f];
  return mk3(hv[f], hv[hc + f], hv[2 * (size_t)hc + f]);
}
// Evaluation r.fr of a contact already in place (every load before the first
// store: the loads then overlap).
__device__ inline void v_eval_again(const VerletView& W, const VerletRun& r, int c) {
  const Contacts& con = W.v.con;
  const int f = W.hidx[r.cb][c], a = con.a[c], b = con.b[c];
  const VContact g{{con.comp(0)[c], con.comp(1)[c], con.comp(2)[c]}, {con.comp(3)[c], con.comp(4)[c], con.comp(5)[c]},
                   {con.comp(6)[c], con.comp(7)[c], con.comp(8)[c]}, {con.comp(9)[c], con.comp(10)[c], con.comp(11)[c]},
                   con.comp(12)[c], con.comp(13)[c]};
  const PairIn in = load_pair(W.v.st, a, b);
  long long frame = 0;
  const d3 old = v_old(W, r, f, frame);
  v_eval(W, r, c, in, g, f, old, frame, false);
}

// Removes the entries past their retention (Hertz-Mindlin) after evaluation
// r.fr; keeps the contacts' indices.
__device__ __noinline__ bool v_purge(const Team& T, const VerletView& W, VerletRun& r, SmemNsc& sm) {
  if (!v_is_hm(W) || r.H == 0) return true;
  const int tid = T.tid(), TS = T.size(), hc = W.hcap, src = r.cur, dst = 1 - r.cur;
  for (int e = tid; e < r.H; e += TS) W.kept[e] = r.fr - W.hframe[src][e] <= 4 ? 1 : 0;
  if (!team_sync(T)) return false;
  if (!team_excl_scan(T, W.kept, W.kept_off, r.H, W.v.blk, sm)) return false;
  const int K = W.kept_off[r.H];
  if (K == r.H) return true;
  for (int e = tid; e < r.H; e += TS) {
    if (!W.kept[e]) continue;
    const int p = W.kept_off[e];
    W.hkey[dst][p] = W.hkey[src][e];
    for (int k = 0; k < 3; ++k) W.hval[dst][(size_t)k * hc + p] = W.hval[src][(size_t)k * hc + e];
    W.hframe[dst][p] = W.hframe[src][e];
  }
  for (int c = tid; c < r.C; c += TS) {
    const int f = W.hidx[r.cb][c];
    if (f >= 0) W.hidx[r.cb][c] = W.kept[f] ? W.kept_off[f] : -1;
  }
  if (!team_sync(T)) return false;
  r.cur = dst;
  r.H = K;
  return true;
}

// Merges the pairs that evaluation r.fr added into the sorted table (every
// block past a barrier since); the next evaluation is behind another barrier.
__device__ __noinline__ bool v_insert(const Team& T, const VerletView& W, VerletRun& r, VerletSmem& S, int added) {
  const NscView& V = W.v;
  const int t = threadIdx.x, hc = W.hcap, cc = V.ccap;
  if (r.H + added > hc - hc / 4 && !v_purge(T, W, r, S.s)) return false;
  if (r.H + added > hc) {
    if (T.rank() == 0 && t == 0) atomicOr(&V.ctl->err, ERR_HIST_CAP);
    return false;
  }
  const int src = r.cur, dst = 1 - r.cur;
  const unsigned long long* ok = W.hkey[src];
  const bool chip = added <= kIns;
  if (chip) {  // every block sorts the added keys by counting
    for (int i = t; i < added; i += blockDim.x) {
      const int c = W.ins[i];
      S.key[i] = pkey(V.con.a[c], V.con.b[c]);
    }
    __syncthreads();
    for (int i = t; i < added; i += blockDim.x) {
      int rank = 0;
      for (int j = 0; j < added; ++j) rank += S.key[j] < S.key[i];
      S.sorted[rank] = S.key[i];
    }
    __syncthreads();
  } else if (!team_excl_scan(T, W.touched, W.touched_off, r.C, V.blk, S.s)) {
    return false;
  }
  // each block an equal range (a table of a few hundred entries would
  // otherwise be moved by the first block alone)
  const int he = (r.H + T.nb - 1) / T.nb, ce = (r.C + T.nb - 1) / T.nb, rank = T.rank();
  for (int e = rank * he + t; e < min((rank + 1) * he, r.H); e += blockDim.x) {
    const unsigned long long k = ok[e];
    int before;
    if (chip) {
      before = lower_bound_u64(S.sorted, added, k);
    } else {
      int lo = 0, hi = r.C;  // contacts are sorted by key
      while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (pkey(V.con.a[m], V.con.b[m]) < k) lo = m + 1;
        else hi = m;
      }
      before = W.touched_off[lo];
    }
    const int p = e + before;
    W.hkey[dst][p] = k;
    for (int j = 0; j < 3; ++j) W.hval[dst][(size_t)j * hc + p] = W.hval[src][(size_t)j * hc + e];
    W.hframe[dst][p] = W.hframe[src][e];
  }
  for (int c = rank * ce + t; c < min((rank + 1) * ce, r.C); c += blockDim.x) {
    const int f = W.hidx[r.cb][c];
    const bool in = W.touched[c];
    if (!in && f < 0) continue;
    const unsigned long long k = pkey(V.con.a[c], V.con.b[c]);
    const int before = chip ? lower_bound_u64(S.sorted, added, k) : W.touched_off[c];
    const int p = before + (in ? lower_bound_u64(ok, r.H, k) : f);
    W.hidx[r.cb][c] = p;
    if (!in) continue;
    W.hkey[dst][p] = k;
    for (int j = 0; j < 3; ++j) W.hval[dst][(size_t)j * hc + p] = W.newval[(size_t)j * cc + c];
    W.hframe[dst][p] = r.fr;
  }
  __syncthreads();  // the on-chip keys are free again
  r.cur = dst;
  r.H += added;
  return true;
}

// Sorts the list of contacts whose head is at *at: turned over (a warp's
// contacts then mostly ascend, having been pushed in lane order), then pairs of
// ascending runs merged until one is left.
__device__ __noinline__ void v_sort_list(int* next, int* at) {
  int head = *at;
  int rev = -1;
  while (head >= 0) {
    const int k = next[head];
    next[head] = rev;
    rev = head;
    head = k;
  }
  head = rev;
  auto run_end = [&](int p, int& rest) {  // last of the run at p; what follows it
    while ((rest = next[p]) > p) p = rest;
    return p;
  };
  for (;;) {
    int p = head, tail = -1, runs = 0;
    auto append = [&](int k) {
      if (tail < 0) head = k;
      else next[tail] = k;
      tail = k;
    };
    while (p >= 0) {
      int q, rest;
      const int pe = run_end(p, q);
      next[pe] = -1;
      ++runs;
      if (q < 0) {
        append(p);
        break;
      }
      const int qe = run_end(q, rest);
      next[qe] = -1;
      while (p >= 0 && q >= 0) {
        const int k = min(p, q);
        append(k);  // (k's own link is read before the next append sets it)
        if (k == p) p = next[p];
        else q = next[q];
      }
      append(p >= 0 ? p : q);
      tail = p >= 0 ? pe : qe;
      p = rest;
    }
    if (runs <= 1) break;
  }
  *at = head;
}

// Sums of body i's contact addends in contact order.  A walk of the list of the
// contacts that it is second body of, for each of them, suits the usual two or
// three; a longer list (a large body under many small ones) has to be sorted:
// false where it is not, and the caller sorts it and comes again, once a
// detection.  A rod under 1000 others, some 6000 contacts in all: 23 -> 1.1 ms
// a step.  (The call stays outside the callers' loops: inside, its registers
// slowed all steps by 1 to 2 %.)
constexpr int kShortList = 8;
__device__ inline bool v_body_sum(const VerletView& W, const VerletRun& r, int i, d3& f, d3& t) {
  const size_t cc = (size_t)W.v.ccap;
  const int* next = W.next;
  const int h0 = W.head[i];
  auto add = [&](const double* g) {
    f.x = f.x + g[0]; f.y = f.y + g[cc]; f.z = f.z + g[2 * cc];
    t.x = t.x + g[3 * cc]; t.y = t.y + g[4 * cc]; t.z = t.z + g[5 * cc];
  };
  const double* fb = W.cf + 6 * cc;
  // second body of: each walk of the list finds the contact after `last`
  for (int last = -1, more = h0 >= 0 ? 2 : 0; more > 1;) {
    int c = 0x7fffffff;
    more = 0;
    for (int k = h0; k >= 0; k = next[k])
      if (k > last) {
        ++more;
        if (k < c) c = k;
      }
    if (more > kShortList) {
      int p = -1;
      for (int k = h0; k >= 0; p = k, k = next[k]) {
        if (k < p) return false;
        add(fb + k);
      }
      break;
    }
    add(fb + c);
    last = c;
  }
  const int2* pk = W.pk[r.cb];
  const int c0 = W.first[r.cb][i];
  for (int c = c0; c >= 0 && c < r.C && pk[c].x == i; ++c) add(W.cf + c);  // first body of
  return true;
}

// Rod i's records on their way to L2: a thread's next rod, while the present
// one is worked on.  With thousands of rods a block the state is streamed from
// memory each phase, and 16 warps (128 registers a thread) do not cover its
// latency: a million rods 350 -> 332 us a step, 325 with the next pairs'
// segments in the detection too; up to 20000 rods (one turn a thread) the
// same.  Loading the next values into registers spilled: 365.
__device__ inline void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ inline void v_prefetch(const VerletView& W, const VerletRun& r, int i, bool drift, const DriftOut& o) {
  const State& st = W.v.st;
  const int n = st.n;
  prefetch_l2(W.head + i);
  prefetch_l2(W.first[r.cb] + i);
  prefetch_l2(st.inv_mass + i);
  prefetch_l2(st.mass + i);
  auto p3 = [&](const auto& a) { prefetch_l2(a.x + i); prefetch_l2(a.y + i); prefetch_l2(a.z + i); };
  p3(st.v); p3(st.w); p3(st.I);
  prefetch_l2(st.q.w + i); p3(st.q);
  if (!drift) return;
  p3(st.x);
  prefetch_l2(st.h + i);
  prefetch_l2(st.r + i);
  for (int k = 0; k < 6; ++k) {
    if (o.ref) prefetch_l2(o.ref + (size_t)k * n + i);
    if (o.ref2) prefetch_l2(o.ref2 + (size_t)k * n + i);
  }
}

// The largest displacement bounds of the block's rods.
__device__ inline void v_publish_disp(const NscView& V, double m, double m2, SmemNsc& sm) {
  m = block_reduce_max(m, sm.red_d);
  m2 = block_reduce_max(m2, sm.red_d);
  if (threadIdx.x == 0) {
    atomic_max_nonneg(&V.ctl->maxdisp, m);
    atomic_max_nonneg(&V.ctl->near_disp, m2);
  }
}

// The flat pair list: near lists from the lists where they are due (else the
// lists themselves), then all rods' entries as (i, j) pairs in order.
__device__ __noinline__ bool v_flatten(const Team& T, const VerletView& W, const VerletRun& r, VerletSmem& S, bool due) {
  const NscView& V = W.v;
  Ctl* ctl = V.ctl;
  const int n = V.st.n, rank = T.rank(), t = threadIdx.x;
  const double* im = V.st.inv_mass;
  const bool near = W.near_cnt != nullptr;
  int mine = 0;
  for (int i = r.lo + t; i < r.hi; i += blockDim.x) {
    const int cnt = V.nbr_cnt[i];
    int m = cnt;
    if (near && due) {
      const Seg A = V.seg[i];
      const bool a_static = !(im[i] > 0.0);
      const int* list = V.nbr + (size_t)i * V.maxnb;
      int* out = W.near_nbr + (size_t)i * V.maxnb;
      m = 0;
      for (int k = 0; k < cnt; ++k) {
        const int j = list[k];
        if (a_static && !(im[j] > 0.0)) continue;
        const Seg B = V.seg[j];
        const d3 xa{A.cx, A.cy, A.cz}, xb{B.cx, B.cy, B.cz};
        if (seg_far(A, B, (xb - xa) + min_image_shift(V.box, xa, xb), A.r + B.r + W.extra)) continue;
        out[m++] = j;
      }
      W.near_cnt[i] = m;
      V.ref2[i] = A.cx; V.ref2[n + i] = A.cy; V.ref2[2 * n + i] = A.cz;
      V.ref2[3 * n + i] = A.ux; V.ref2[4 * n + i] = A.uy; V.ref2[5 * n + i] = A.uz;
    } else if (near) {
      m = W.near_cnt[i];
    }
    mine += m;
  }
  const int bsum = block_reduce_sum_i(mine, S.s.red_i);
  if (t == 0) V.blk[rank] = bsum;
  if (!team_sync(T)) return false;
  int prefix, total;
  block_prefix(V.blk, T.nb, rank, prefix, total, S.s);
  if (total > W.flat_cap) {
    if (rank == 0 && t == 0) atomicOr(&ctl->err, ERR_FLAT_CAP);
    return false;
  }
  const int* cnts = near ? W.near_cnt : V.nbr_cnt;
  const int* lists = near ? W.near_nbr : V.nbr;
  int run = prefix;
  for (int base = r.lo; base < r.hi; base += blockDim.x) {
    const int i = base + t;
    const int m = i < r.hi ? cnts[i] : 0;
    int tot;
    const int o = run + block_excl_scan(m, S.s.scan_w, tot);
    const int* list = lists + (size_t)i * V.maxnb;
    for (int k = 0; k < m; ++k) W.flat[o + k] = make_int2(i, list[k]);
    run += tot;
  }
  if (rank == 0 && t == 0) {  // every block has read them
    ctl->near_n = total;
    ctl->flat_valid = 1;
    if (near && due) {
      ctl->near_valid = 1;
      ctl->near_disp = 0.0;
      ctl->near_rebuilds += 1;
    }
  }
  return team_sync(T);
}

// Detection at the current segment records (every block past a barrier since
// they and the displacement bounds were written), and evaluation r.fr on the
// contacts found.  One thread tests one pair of the flat list (a thread per
// rod over its near list left most lanes idle: a rod has 0.2 to 0.6 entries,
// a warp's busiest one three or four).
__device__ __noinline__ bool v_detect_eval(const Team& T, const VerletView& W, VerletRun& r, VerletSmem& S,
                                           bool energy) {
  const NscView& V = W.v;
  Ctl* ctl = V.ctl;
  const int rank = T.rank(), t = threadIdx.x;
  const bool need = *(volatile int*)&ctl->rebuild ||
                    (!V.all_pairs && *(volatile double*)&ctl->maxdisp >= 0.5 * V.skin * (1.0 - 1e-9));
  const bool due = need || (W.near_cnt && (!*(volatile int*)&ctl->near_valid ||
                                           *(volatile double*)&ctl->near_disp >= 0.5 * V.near_skin * (1.0 - 1e-9)));
  const bool flat = due || !*(volatile int*)&ctl->flat_valid;
  if (need && !rebuild_phase(T, V, S.s)) return false;
  if (flat && !v_flatten(T, W, r, S, due)) return false;
  // test: each block a 32-aligned range of pairs, one bit per pair
  const int P = *(volatile int*)&ctl->near_n;
  const int per = (((P + T.nb - 1) / T.nb) + 31) & ~31;
  const int plo = min(rank * per, P), phi = min(plo + per, P);
  unsigned* bits = reinterpret_cast<unsigned*>(V.mask);
  const double* im = V.st.inv_mass;
  int mine = 0;
  const int ahead = blockDim.x;  // a thread's next pair, its segments on their way to L2
  int2 pr{0, 0}, next{0, 0};
  if (plo + t < phi) pr = W.flat[plo + t];
  if (plo + t + ahead < phi) next = W.flat[plo + t + ahead];
  for (int p0 = plo; p0 < phi; p0 += blockDim.x) {
    const int p = p0 + t;
    bool hit = false;
    int2 after{0, 0};
    if (p + ahead < phi) {
      prefetch_l2(V.seg + next.x);
      prefetch_l2(V.seg + next.y);
      if (p + 2 * ahead < phi) after = W.flat[p + 2 * ahead];
    }
    if (p < phi) {
      if (im[pr.x] > 0.0 || im[pr.y] > 0.0) {
        const Seg A = V.seg[pr.x], B = V.seg[pr.y];
        const Narrow nr = narrow_pair(A, B, V.box);
        hit = contact_test(nr.d2, A.r + B.r, W.delta);
      }
    }
    const unsigned word = __ballot_sync(0xffffffffu, hit);
    if ((t & 31) == 0 && p < phi) {
      bits[p >> 5] = word;
      mine += __popc(word);
    }
    pr = next;
    next = after;
  }
  const int bsum = block_reduce_sum_i(mine, S.s.red_i);
  if (t == 0) V.blk[rank] = bsum;
  if (!team_sync(T)) return false;
  if (rank == 0 && t == 0) ctl->maxdisp = 0.0;
  int prefix, total;
  block_prefix(V.blk, T.nb, rank, prefix, total, S.s);
  if (total > V.ccap) {
    if (rank == 0 && t == 0) atomicOr(&ctl->err, ERR_CONTACT_CAP);
    return false;
  }
  // contacts in pair order: the hits' pairs to their slots first, then one
  // thread per slot
  const int ob = r.cb, cb = 1 - r.cb, oc = r.C;  // the contact lists before and now
  int run = prefix;
  const int wlo = plo >> 5, whi = plo < phi ? (phi + 31) >> 5 : wlo;
  for (int base = wlo; base < whi; base += blockDim.x) {
    const int w = base + t;
    const unsigned word = w < whi ? bits[w] : 0u;  // (this block wrote it)
    int tot;
    int o = run + block_excl_scan(__popc(word), S.s.scan_w, tot);
    for (unsigned m = word; m; m &= m - 1) W.pk[cb][o++] = W.flat[(w << 5) + __ffs((int)m) - 1];
    run += tot;
  }
  if (rank == 0 && t == 0) {
    ctl->contacts = total;
    ctl->contact_steps += total;
  }
  r.C = total;
  r.cb = cb;
  __syncthreads();
  for (int c = prefix + t; c < run; c += blockDim.x) {
    // every load that needs no result comes before the first store
    const int2 pr = W.pk[cb][c];
    const int a = pr.x, b = pr.y;
    // the first contact of a: the slot before belongs to another rod (of a
    // block's first slot the block before may hold more of the same run: the
    // lowest slot wins below)
    const bool head_of_a = c > prefix ? W.pk[cb][c - 1].x != a : true;
    const Seg A = V.seg[a], B = V.seg[b];
    const PairIn in = load_pair(V.st, a, b);
    int f = -1;
    bool known = false;
    if (r.idx_ok) {  // among a's first contacts before (of a longer run: by search)
      const int k0 = W.first[ob][a], lim = min(oc, k0 + 8);
      for (int k = k0; k >= 0 && k < lim; ++k) {
        const int2 q = W.pk[ob][k];
        if (q.x != a) break;
        if (q.y == b) {
          f = W.hidx[ob][k];
          known = true;
        }
      }
    }
    if (!known && r.H > 0) f = v_find(W, r, a, b);
    long long frame = 0;
    const d3 old = v_old(W, r, f, frame);
    const Narrow nr = narrow_pair(A, B, V.box);
    const double dist = sqrt(nr.d2);
    const d3 diff = nr.pb - nr.pa;
    const VContact g{nr.pa, nr.pb, dist > 1e-10 ? diff / dist : mk3(1, 0, 0), nr.sh, dist, A.r + B.r};
    W.next[c] = atomicExch(&W.head[b], c);
    if (head_of_a) atomicMin(reinterpret_cast<unsigned*>(&W.first[cb][a]), (unsigned)c);
    write_contact(V.con, c, a, b, g.surf, nr);
    v_eval(W, r, c, in, g, f, old, frame, energy);
  }
  r.idx_ok = true;
  return true;
}

// Potential energy in the order of the multi-kernel form's one 1024-thread
// block (k_pe_sum), by the first block.
__device__ inline void v_energy(const VerletView& W, int C, SmemNsc& sm) {
  const double* pe = W.cf + 12 * (size_t)W.v.ccap;
  const int t = threadIdx.x, warp = t >> 5;
  for (int h = 0; h < 1024; h += blockDim.x) {
    double v = 0;
    for (int c = h + t; c < C; c += 1024) v += pe[c];
    v = warp_sum(v);
    if ((t & 31) == 0) sm.red_d[(h >> 5) + warp] = v;
  }
  __syncthreads();
  if (t < 32) {
    const double u = warp_sum(sm.red_d[t]);
    if (t == 0) W.v.ctl->pe = u;
  }
  __syncthreads();
}

// nsteps steps of one system by its team (0: one force evaluation).
__device__ __noinline__ bool v_run(const Team& T, const VerletView& W, int nsteps, VerletSmem& S) {
  const NscView& V = W.v;
  const State& st = V.st;
  const rg_config& cfg = V.cfg;
  Ctl* ctl = V.ctl;
  const int n = st.n, rank = T.rank(), t = threadIdx.x;
  const int seg = (n + T.nb - 1) / T.nb;
  VerletRun r;
  r.lo = min(rank * seg, n);
  r.hi = min(r.lo + seg, n);
  r.H = ctl->hist_n;
  r.cur = W.hcur;
  r.cb = W.cb;
  r.C = ctl->contacts;
  r.fr = ctl->frame;
  r.idx_ok = W.fresh != 0;
  r.hm = hm_const(cfg);
  const bool wall = !v_is_hm(W) && cfg.cylinder_enabled;
  const d3 ax = wall ? soft_wall_axis(cfg) : mk3(0, 0, 0);
  const double el = exp(-cfg.lin_damp * cfg.dt), ea = exp(-cfg.ang_damp * cfg.dt);
  double invL[3] = {1.0, 1.0, 1.0};
  for (int k = 0; k < 3; ++k)
    if (V.box.L[k] > 0.0) invL[k] = 1.0 / V.box.L[k];
  const DriftOut out{V.seg, V.all_pairs ? nullptr : V.ref, W.near_cnt ? V.ref2 : nullptr, V.skin};
  if (!W.fresh) {  // segment records and displacement bounds of the first detection
    double m = 0.0, m2 = 0.0;
    for (int i = r.lo + t; i < r.hi; i += blockDim.x) {
      const Seg s = make_seg(st, i);
      V.seg[i] = s;
      W.head[i] = -1;
      W.first[1 - r.cb][i] = -1;
      if (out.ref) m = fmax(m, seg_disp(s, out.ref, n, i, V.box));
      if (out.ref2) m2 = fmax(m2, seg_disp(s, out.ref2, n, i, V.box));
    }
    v_publish_disp(V, m, m2, S.s);
  }
  // (every block has read the control words before the first one changes any)
  if (!team_sync(T)) return false;
  if (nsteps == 0) {  // one force evaluation at the current state, kept in f and tau
    ++r.fr;
    if (!v_detect_eval(T, W, r, S, true)) return false;
    if (!team_sync(T)) return false;
    const int added = *(volatile int*)&ctl->ins_n[r.fr & 1];
    for (int i = r.lo + t; i < r.hi;) {
      bool sort = false;
      for (; i < r.hi; i += blockDim.x) {
        d3 f{0, 0, 0}, tq{0, 0, 0};
        sort = !v_body_sum(W, r, i, f, tq);
        if (sort) break;
        if (wall && st.inv_mass[i] > 0.0) soft_wall_apply(cfg, ax, st.r[i], st.x.ld(i), st.v.ld(i), f);
        st.f.st(i, f);
        st.tau.st(i, tq);
      }
      if (sort) v_sort_list(W.next, W.head + i);
    }
    if (rank == 0) v_energy(W, r.C, S.s);
    if (added && !v_insert(T, W, r, S, added)) return false;
    if (!team_sync(T)) return false;
  }
  for (int step = 0; step < nsteps; ++step) {
    const bool last = step == nsteps - 1;
    // forces at t: with the first detection, or on the contacts in place
    ++r.fr;
    if (step == 0 && !W.fresh) {
      if (!v_detect_eval(T, W, r, S, false)) return false;
    } else {
      const int per = (r.C + T.nb - 1) / T.nb, c1 = min((rank + 1) * per, r.C);
      for (int c = rank * per + t; c < c1; c += blockDim.x) v_eval_again(W, r, c);
      if (rank == 0 && t == 0) ctl->contact_steps += r.C;
    }
    if (!team_sync(T)) return false;
    // half kick and drift
    {
      const int added = *(volatile int*)&ctl->ins_n[r.fr & 1];
      if (rank == 0 && t == 0) ctl->ins_n[(r.fr + 1) & 1] = 0;
      double m = 0.0, m2 = 0.0;
      for (int i = r.lo + t; i < r.hi;) {
        bool sort = false;
        for (; i < r.hi; i += blockDim.x) {
          if (i + (int)blockDim.x < r.hi) v_prefetch(W, r, i + blockDim.x, true, out);
          d3 f{0, 0, 0}, tq{0, 0, 0};
          if (st.inv_mass[i] > 0.0) sort = !v_body_sum(W, r, i, f, tq);
          if (sort) break;
          W.head[i] = -1;  // for the detection that follows
          W.first[1 - r.cb][i] = -1;
          drift_rod(st, V.box, cfg, ax, wall, i, f, tq, out, invL, m, m2);
        }
        if (sort) v_sort_list(W.next, W.head + i);
      }
      if (out.ref || out.ref2) v_publish_disp(V, m, m2, S.s);
      if (added && !v_insert(T, W, r, S, added)) return false;
    }
    if (!team_sync(T)) return false;
    // forces at t + dt
    ++r.fr;
    if (!v_detect_eval(T, W, r, S, last)) return false;
    if (!team_sync(T)) return false;
    // second half kick
    {
      const int added = *(volatile int*)&ctl->ins_n[r.fr & 1];
      if (rank == 0 && t == 0) ctl->ins_n[(r.fr + 1) & 1] = 0;
      int bad = 0;
      for (int i = r.lo + t; i < r.hi;) {
        bool sort = false;
        for (; i < r.hi; i += blockDim.x) {
          if (i + (int)blockDim.x < r.hi) v_prefetch(W, r, i + blockDim.x, false, out);
          d3 f{0, 0, 0}, tq{0, 0, 0};
          sort = !v_body_sum(W, r, i, f, tq);
          if (sort) break;
          bad |= kick_rod(st, cfg, ax, wall, i, f, tq, el, ea);
          if (last) {  // the forces that the call's last kick used
            st.f.st(i, f);
            st.tau.st(i, tq);
          }
        }
        if (sort) v_sort_list(W.next, W.head + i);
      }
      if (bad) atomicOr(&ctl->err, ERR_NONFINITE);
      if (last && rank == 0) v_energy(W, r.C, S.s);
      if (added && !v_insert(T, W, r, S, added)) return false;
    }
    if (!team_sync(T)) return false;
    if (*(volatile int*)&ctl->err) return false;
  }
  // the table in the buffer it was found in, without entries past retention
  if (!v_purge(T, W, r, S.s)) return false;
  if (r.cur != W.hcur) {
    const int hc = W.hcap, src = r.cur, dst = W.hcur;
    for (int e = T.tid(); e < r.H; e += T.size()) {
      W.hkey[dst][e] = W.hkey[src][e];
      for (int k = 0; k < 3; ++k) W.hval[dst][(size_t)k * hc + e] = W.hval[src][(size_t)k * hc + e];
      W.hframe[dst][e] = W.hframe[src][e];
    }
  }
  if (rank == 0 && t == 0) {
    ctl->hist_n = r.H;
    ctl->frame = r.fr;
  }
  return true;
}

// A team's systems one after the other, each through all steps.
__global__ void __launch_bounds__(kVBlock, 1) k_verlet_run(const VerletView* views, const TeamDesc* teams, int nteams,
                                                           const int* members, int nsteps) {
  __shared__ VerletSmem S;
  __shared__ __align__(16) unsigned char view_words[sizeof(VerletView)];
  int lo = 0, hi = nteams;  // last team with b0 <= blockIdx.x
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (teams[m].b0 <= (int)blockIdx.x) lo = m;
    else hi = m;
  }
  const TeamDesc td = teams[lo];
  if ((int)blockIdx.x < td.b0 || (int)blockIdx.x >= td.b0 + td.nb) return;
  team_barriers_reset();
  static_assert(sizeof(VerletView) % 8 == 0, "copied in 8-byte words");
  for (int m = td.first; m < td.first + td.count; ++m) {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&views[members ? members[m] : m]);
    __syncthreads();  // the system before is done with its view
    for (int k = threadIdx.x; k < (int)(sizeof(VerletView) / 8); k += blockDim.x)
      reinterpret_cast<unsigned long long*>(view_words)[k] = src[k];
    __syncthreads();
    const VerletView& W = *reinterpret_cast<const VerletView*>(view_words);
    const Team T{td.b0, td.nb, td.bar, &W.v.ctl->err,
                 W.v.cfg.spin_limit > 0 ? (long long)W.v.cfg.spin_limit : kSpinLimit,
                 W.v.cfg.test_absent_blocks > 0 ? (unsigned)W.v.cfg.test_absent_blocks : 0u};
    if (*(volatile int*)&W.v.ctl->err == 0) v_run(T, W, nsteps, S);
  }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
constexpr size_t kVSmem = kBuildQOff + 2 * sizeof(unsigned) * kBuildQ;

VerletView make_verlet_view(rg_system* s) {
  VerletView W;
  std::memset(&W, 0, sizeof(W));
  W.v = make_view(s);
  const Detector& d = s->det;
  W.near_cnt = d.near_cnt;
  W.near_nbr = d.near_nbr;
  W.extra = d.margin + d.near_skin;
  W.delta = s->cfg.model == RG_MODEL_HERTZ_MINDLIN ? 0.0 : s->cfg.soft_delta;
  W.cf = s->d_cf;
  const History& H = s->hist;
  for (int k = 0; k < 2; ++k) {
    W.hkey[k] = H.key[k];
    W.hval[k] = H.val[k];
    W.hframe[k] = H.frame[k];
    W.first[k] = s->vteam.first[k];
    W.pk[k] = s->vteam.pk[k];
    W.hidx[k] = s->vteam.hidx[k];
  }
  W.hcap = H.cap;
  W.hcur = H.cur;
  W.touched = H.touched;
  W.touched_off = H.touched_off;
  W.kept = H.kept;
  W.kept_off = H.kept_off;
  W.newval = H.newval;
  W.head = s->vteam.head;
  W.next = s->vteam.next;
  W.ins = s->vteam.ins;
  W.flat = s->vteam.flat;
  W.flat_cap = s->vteam.flat_cap;
  W.fresh = s->contacts_fresh == Fresh::kTeam ? 1 : 0;
  W.cb = s->vteam.cb;
  return W;
}

// Bookkeeping of a launch of nsteps steps: the contacts it leaves when it ends
// without an error.  Until then (a barrier that timed out, a launch that never
// ran) they are not to be relied on: the lists hold whatever the kernel had
// reached, and indices read from them could lie outside the tables.
void verlet_launched(rg_system* s, int nsteps) {
  const int detections = nsteps + (s->contacts_fresh == Fresh::kTeam ? 0 : 1);
  s->vteam.cb_after = (s->vteam.cb + detections) & 1;
  s->fresh_after = Fresh::kTeam;
  s->contacts_fresh = Fresh::kNo;
}

bool verlet_team_fits(const rg_system* s) {
  const int m = s->cfg.model;
  return (m == RG_MODEL_HARMONIC || m == RG_MODEL_HERTZ_MINDLIN) && !s->prof_on && s->vteam.head;
}

cudaError_t verlet_allow_smem() {
  return cudaFuncSetAttribute((const void*)k_verlet_run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVSmem);
}

void verlet_launch(const VerletView* views, const TeamDesc* teams, int nteams, const int* members, int grid, int nsteps,
                   cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kVBlock);
  cfg.dynamicSmemBytes = kVSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&views, &teams, &nteams, &members, &nsteps};
  RGL cudaLaunchKernelExC(&cfg, (const void*)k_verlet_run, args);
}

void verlet_run_launch(rg_system* s, int nsteps) {
  // (a force evaluation alone crosses few barriers, so a new state's list
  // build decides: four times the blocks; 1000 rods, first pass 435 -> 300 us,
  // later ones the same)
  const int per = nsteps > 0 ? kVerletRodsPerBlock : kVerletRodsPerBlock / 4;
  int nb = s->team_blocks > 0 ? s->team_blocks : (s->n + per - 1) / per;
  if (nb > s->sm_count) nb = s->sm_count;
  const VerletView W = make_verlet_view(s);
  const TeamDesc td{0, nb, 0, 1, s->nsc.bar, nullptr};
  cudaMemcpyAsync(s->vteam.view_dev, &W, sizeof(W), cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->nsc.team_dev, &td, sizeof(td), cudaMemcpyHostToDevice, s->stream);
  cudaMemsetAsync(s->nsc.bar, 0, kTeamBarBytes, s->stream);
  verlet_launch(static_cast<const VerletView*>(s->vteam.view_dev), static_cast<const TeamDesc*>(s->nsc.team_dev), 1,
                nullptr, nb, nsteps, s->stream);
  verlet_launched(s, nsteps);
}

// One allocation behind the arrays (each a multiple of 16 bytes); the flat
// list belongs to the detector's lists.
cudaError_t VerletTeam::alloc(int n, int ccap) {
  const size_t rods = ((size_t)n + 3) / 4 * 4, cons = ((size_t)ccap + 3) / 4 * 4;
  const size_t view = (sizeof(VerletView) + 15) / 16 * 16;
  const cudaError_t e = cudaMalloc(&view_dev, view + sizeof(int) * (3 * rods + 8 * cons));
  if (e) return e;
  int* p = reinterpret_cast<int*>(static_cast<char*>(view_dev) + view);
  for (int k = 0; k < 2; ++k) {
    pk[k] = reinterpret_cast<int2*>(p);
    hidx[k] = p + 2 * cons;
    first[k] = p + 3 * cons;
    p += 3 * cons + rods;
  }
  next = p;
  ins = p + cons;
  head = p + 2 * cons;
  return cudaSuccess;
}
void VerletTeam::free_() {
  cudaFree(view_dev);
  int2* const f = flat;
  const int fc = flat_cap;
  *this = VerletTeam();
  flat = f;
  flat_cap = fc;
}

}  // namespace rg
