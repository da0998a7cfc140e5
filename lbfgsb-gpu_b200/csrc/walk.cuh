// walk.cuh -- the breakpoint walk of the generalized Cauchy point (the part of
// culbfgsb/lbfgsbcpu.cpp:725-816 after the first breakpoint test).
//
// The reference keeps the breakpoints in a heap (hpsolb, 1175-1233) and pops them one at
// a time.  Here, only when the scan found that the first breakpoint is passed, the
// breakpoints (t_i, i) are listed (same arithmetic as the scan, so the same t_i) and walked
// in chunks of the smallest remaining keys (96-bit key: the bits of t, then i):
//   select   a radix select over the list, 8 bits a level, that stops as soon as the
//            buckets below the boundary hold a large enough chunk (usually after one or
//            two levels), and the extraction of that chunk;
//   walk     the chunk is sorted in shared memory (bitonic), each candidate's row of W,
//            M*wbp and wbp'M wbp are formed in parallel, and one thread walks the chunk in
//            key order with the reference's recurrence for f', f'', c and p.
// Two forms: k_walk_coop (single-instance solves) lists, selects, sorts and prepares with the
// whole grid, a cooperative launch with a bounded grid barrier, and walks in CTA 0 as a
// pipeline of warps; walk_pass (batched solves: kb_walk, one CTA per instance, after
// kb_walk_gather) does everything in one CTA as described above.  Breakpoints with equal t are
// passed in increasing variable index (the heap's order among exact ties is an artefact of its
// layout).
#pragma once

#include "common.cuh"
#include "passes.cuh"
#include "small.cuh"
#include "state.cuh"

namespace lbfgsb_b200 {

// Appends the breakpoints of the CTA's share of the variables to (wl_t, wl_i).
template <typename R, typename H, typename S>
__device__ __forceinline__ void gather_breakpoints(const Ctx<R, H, S>& c, CtaPos cp, int nthreads,
                                                   const R* __restrict__ x, const R* __restrict__ g) {
  const int n = c.n;
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)cp.rank * nthreads; base < n;
       base += (long long)cp.count * nthreads) {
    const long long i = base + threadIdx.x;
    bool has_bp = false;
    R t = 0;
    if (i < n) classify(x[i], g[i], c.l[i], c.u[i], c.nbd[i], has_bp, t);
    const uint32_t mask = __ballot_sync(0xffffffffu, has_bp);
    if (mask == 0) continue;
    unsigned int start = 0;
    if (lane == 0) start = atomicAdd(c.wl_n, (unsigned int)__popc(mask));
    start = __shfl_sync(0xffffffffu, start, 0);
    if (has_bp) {
      const unsigned int pos = start + __popc(mask & ((1u << lane) - 1u));
      c.wl_t[pos] = (double)t;
      c.wl_i[pos] = (int)i;
    }
  }
}

template <typename R, typename H, typename S>
__device__ __forceinline__ void walk_gather_pass(const Ctx<R, H, S>& c, CtaPos cp,
                                                 const R* __restrict__ x, const R* __restrict__ g) {
  if (c.rounds) {
    const DevState<S>* st = c.st;
    if (!st->rp_sub || st->gcp_state != GCP_WALK || st->internal_fail != 0) return;
    x = c.X[st->xr[0]];
    g = c.G[st->gr[0]];
  }
  gather_breakpoints<R, H, S>(c, cp, kThreads, x, g);
}
template <typename R, typename H, typename S>
__global__ void __launch_bounds__(kThreads) k_walk_gather(Ctx<R, H, S> c, const R* __restrict__ x,
                                                          const R* __restrict__ g) {
  walk_gather_pass<R, H, S>(c, cta_here(), x, g);
}

constexpr int kWalkThreads = 512;
constexpr int kChunk = kWalkChunk;
constexpr int kChunkMin = kChunk / 4;  // the smallest chunk the select may stop at
constexpr int kBatch = 64;    // candidates prepared in parallel per walking step

struct Key96 {
  unsigned long long hi;  // bits of t (t >= 0, so the bits order like the values)
  unsigned int lo;        // variable index
};
__device__ __forceinline__ bool key_less(const Key96& a, const Key96& b) {
  return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo);
}
__device__ __forceinline__ Key96 make_key(double t, int i) {
  return Key96{(unsigned long long)__double_as_longlong(t), (unsigned int)i};
}
__device__ __forceinline__ int key_digit(const Key96& k, int level) {
  return level < 8 ? (int)((k.hi >> (56 - 8 * level)) & 255ull) : (int)((k.lo >> (24 - 8 * (level - 8))) & 255u);
}
// true when the first `level` digits of k equal those of p
__device__ __forceinline__ bool key_prefix_eq(const Key96& k, const Key96& p, int level) {
  if (level == 0) return true;
  if (level <= 8) {
    const int sh = 64 - 8 * level;
    return (sh == 0) ? k.hi == p.hi : (k.hi >> sh) == (p.hi >> sh);
  }
  if (k.hi != p.hi) return false;
  const int sh = 32 - 8 * (level - 8);
  return (sh == 0) ? k.lo == p.lo : (k.lo >> sh) == (p.lo >> sh);
}
__device__ __forceinline__ void key_set_digit(Key96& k, int level, int d) {
  if (level < 8) {
    const int sh = 56 - 8 * level;
    k.hi = (k.hi & ~(255ull << sh)) | ((unsigned long long)d << sh);
  } else {
    const int sh = 24 - 8 * (level - 8);
    k.lo = (k.lo & ~(255u << sh)) | ((unsigned int)d << sh);
  }
}
// the key just below k (k > 0)
__device__ __forceinline__ Key96 key_prev(Key96 k) {
  if (k.lo > 0) return Key96{k.hi, k.lo - 1};
  return Key96{k.hi - 1, ~0u};
}

// One level of the radix select, from the level's histogram (the same in every thread that
// runs it): the boundary digit d, the keys below it, and whether the select may stop here
// with the chunk "every candidate below bucket d" (at least chunk_min keys in all).  taken:
// keys already below the prefix from earlier levels; kk: keys still wanted.
__device__ __forceinline__ void select_level(const unsigned int* hist, long long taken,
                                             long long kk, long long chunk_min, int& d,
                                             long long& cum, bool& stop) {
  cum = 0;
  d = 255;
  for (int b = 0; b < 256; b++) {
    if (cum + hist[b] >= kk) {
      d = b;
      break;
    }
    cum += hist[b];
  }
  stop = taken + cum >= chunk_min;
}

// Thread 0's running walk (lbfgsbcpu.cpp:725-809) across chunks.
template <typename S>
struct WalkCarry {
  S f1, f2, f2org, dtm, tsum, tj;
  int nleft, nint;
  bool all_fixed;
};

template <typename S>
struct WalkSmem {
  unsigned long long k_hi[kChunk];
  unsigned int k_lo[kChunk];
  unsigned int hist[256];
  int count, done, info;
  Key96 prefix, last;
  long long kk, taken;
  S wbp[kBatch][2 * kMaxM + 1];
  S v[kBatch][2 * kMaxM + 1];
  S wmw[kBatch], dibp[kBatch], zibp[kBatch];
  S work[kBatch][kMaxM + 1];
};

// Bitonic sort of the cnt keys in sm.k_hi / k_lo by (hi, lo), padded with maximal keys
// (all threads of the CTA).
template <typename S>
__device__ void sort_chunk(WalkSmem<S>& sm, int cnt) {
  for (int e = cnt + threadIdx.x; e < kChunk; e += blockDim.x) {
    sm.k_hi[e] = ~0ull;
    sm.k_lo[e] = ~0u;
  }
  __syncthreads();
  for (int size = 2; size <= kChunk; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int e = threadIdx.x; e < kChunk; e += blockDim.x) {
        const int p = e ^ stride;
        if (p > e) {
          const bool up = (e & size) == 0;
          const Key96 a{sm.k_hi[e], sm.k_lo[e]}, b{sm.k_hi[p], sm.k_lo[p]};
          if (key_less(b, a) == up) {
            sm.k_hi[e] = b.hi;
            sm.k_lo[e] = b.lo;
            sm.k_hi[p] = a.hi;
            sm.k_lo[p] = a.lo;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Walk the cnt sorted keys of sm (all threads of the CTA) with the reference's recurrence
// (lbfgsbcpu.cpp:725-809).  prep(q, k) fills sm.dibp[q], sm.zibp[q] and sm.wbp[q][1..2col]
// for key k of the chunk (run by thread q of a batch); pass(k, dibp) records that the walk
// passed key k (thread 0).  Sets sm.done: 1 the walk ended, 2 a step of M*wbp failed (the
// driver resets the memory).
template <typename S, typename Prep, typename Pass>
__device__ void walk_sorted(DevState<S>* st, WalkSmem<S>& sm, int cnt, WalkCarry<S>& w,
                            Prep&& prep, Pass&& pass) {
  const int n = st->n, col = st->col, col2 = 2 * col, nbreak = st->nbreak, bnded = st->bnded;
  const S theta = st->theta;
  for (int b0 = 0; b0 < cnt; b0 += kBatch) {
    const int nb = (cnt - b0) < kBatch ? (cnt - b0) : kBatch;
    if (threadIdx.x < nb) {
      prep((int)threadIdx.x, b0 + (int)threadIdx.x);
      const S* wbp = sm.wbp[threadIdx.x];
      if (col > 0) {
        int info = 0;
        sbmv(st->sy, st->wt, col, wbp, sm.v[threadIdx.x], &info, sm.work[threadIdx.x]);
        if (info != 0) atomicExch(&sm.info, info);
        sm.wmw[threadIdx.x] = sdot(&wbp[1], 1, &sm.v[threadIdx.x][1], 1, col2);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (sm.info != 0) {
        st->internal_fail = sm.info;
        sm.done = 2;
      }
      #pragma unroll 1
      for (int q = 0; q < nb && sm.done == 0; q++) {
        const int k = b0 + q;
        const S tk = (S)__longlong_as_double((long long)sm.k_hi[k]);
        const S tj0 = w.tj;
        w.tj = tk;
        const S dt = w.tj - tj0;
        if (w.dtm < dt) {
          sm.done = 1;
          break;
        }
        w.tsum = w.tsum + dt;
        w.nleft = w.nleft - 1;
        const S dibp = sm.dibp[q];
        pass(k, dibp);
        if (w.nleft == 0 && nbreak == n) {
          w.dtm = dt;
          #pragma unroll 1
          for (int j = 1; j <= col2; j++) st->c[j] += w.dtm * st->p[j];
          w.all_fixed = true;
          sm.done = 1;
          break;
        }
        w.nint = w.nint + 1;
        const S dibp2 = dibp * dibp;
        w.f1 = w.f1 + dt * w.f2 + dibp2 - theta * dibp * sm.zibp[q];
        w.f2 = w.f2 - theta * dibp2;
        if (col > 0) {
          #pragma unroll 1
          for (int j = 1; j <= col2; j++) st->c[j] += dt * st->p[j];
          const S wmc = sdot(&st->c[1], 1, &sm.v[q][1], 1, col2);
          const S wmp = sdot(&st->p[1], 1, &sm.v[q][1], 1, col2);
          const S wmw = sm.wmw[q];
          #pragma unroll 1
          for (int j = 1; j <= col2; j++) st->p[j] += (-dibp) * sm.wbp[q][j];
          w.f1 = w.f1 + dibp * wmc;
          w.f2 = w.f2 + (S)2.0 * dibp * wmp - dibp2 * wmw;
        }
        w.f2 = smax((S)(5e-16 * (double)w.f2org), w.f2);
        if (w.nleft > 0) {
          w.dtm = -w.f1 / w.f2;
          continue;
        }
        if (bnded) {
          w.f1 = 0;
          w.f2 = 0;
          w.dtm = 0;
        } else {
          w.dtm = -w.f1 / w.f2;
        }
        sm.done = 1;
        break;
      }
    }
    __syncthreads();
    if (sm.done) break;
  }
}

// Sort the cnt keys in sm.k_hi / k_lo and walk them, reading each candidate's x, g, bounds
// and history row from the solve's arrays (all threads of the CTA).
template <typename R, typename H, typename S>
__device__ void walk_chunk(const Ctx<R, H, S>& c, const R* __restrict__ x, const R* __restrict__ g,
                           const H* const (&Y)[kMaxM], const H* const (&Sl)[kMaxM], WalkSmem<S>& sm,
                           int cnt, WalkCarry<S>& w) {
  DevState<S>* st = c.st;
  const int col = st->col;
  const S theta = st->theta;
  sort_chunk(sm, cnt);
  walk_sorted(st, sm, cnt, w,
      [&](int q, int k) {
        const int i = (int)sm.k_lo[k];
        const R xi = x[i], gi = g[i];
        const R dibp = -gi;
        const R zibp = (dibp > R(0)) ? rsub(c.u[i], xi) : rsub(c.l[i], xi);
        sm.dibp[q] = (S)dibp;
        sm.zibp[q] = (S)zibp;
        S* wbp = sm.wbp[q];
        #pragma unroll 1
        for (int j = 0; j < col; j++) {
          wbp[1 + j] = (S)HistTraits<H>::load(Y[j] + i);
          wbp[1 + col + j] = theta * (S)HistTraits<H>::load(Sl[j] + i);
        }
      },
      [&](int k, S dibp) {
        c.code[(int)sm.k_lo[k]] = (int8_t)(dibp > S(0) ? IW_WALK_UPP : IW_WALK_LOW);
      });
}

// The walk's start from the state and its end into it (thread 0).
template <typename S>
__device__ __forceinline__ WalkCarry<S> walk_start(const DevState<S>* st) {
  WalkCarry<S> w;
  w.f1 = st->f1;
  w.f2 = st->f2;
  w.f2org = st->f2org;
  w.dtm = st->dtm;
  w.tsum = st->tsum;
  w.tj = st->tj;
  w.nleft = st->nleft;
  w.nint = st->nint;
  w.all_fixed = false;
  return w;
}
template <typename S>
__device__ __forceinline__ void walk_end(DevState<S>* st, WalkCarry<S>& w, S* work) {
  const int col = st->col, col2 = 2 * col;
  if (!w.all_fixed) {
    if (w.dtm <= S(0)) w.dtm = 0;
    w.tsum = w.tsum + w.dtm;
    #pragma unroll 1
    for (int j = 1; j <= col2; j++) st->c[j] += w.dtm * st->p[j];
  }
  st->f1 = w.f1;
  st->f2 = w.f2;
  st->dtm = w.dtm;
  st->tsum = w.tsum;
  st->tj = w.tj;
  st->nleft = w.nleft;
  st->nint = w.nint;
  if (col > 0) {
    int info = 0;
    sbmv(st->sy, st->wt, col, st->c, st->mc, &info, work);
    if (info != 0) {
      st->internal_fail = -8;
      return;
    }
  }
  st->gcp_state = GCP_DONE;
}

// The whole walk in one CTA (batched solves: one CTA per instance, after kb_walk_gather).
template <typename R, typename H, typename S>
__device__ __forceinline__ void walk_pass(const Ctx<R, H, S>& c, const R* __restrict__ x,
                                          const R* __restrict__ g) {
  DevState<S>* st = c.st;
  if (c.rounds) {
    if (!st->rp_sub || st->internal_fail != 0) return;
    x = c.X[st->xr[0]];
    g = c.G[st->gr[0]];
  }
  if (st->gcp_state != GCP_WALK) return;
  const long long L = *c.wl_n;
  const H *Y[kMaxM], *Sl[kMaxM];
  ring_ptrs(st, c.wy, c.ld, Y);
  ring_ptrs(st, c.ws, c.ld, Sl);
  __shared__ WalkSmem<S> sm;
  WalkCarry<S> w{};
  if (threadIdx.x == 0) {
    w = walk_start(st);
    sm.done = 0;
    sm.last = Key96{0ull, 0u};
    sm.info = 0;
  }
  __syncthreads();
  bool first_round = true;
  long long consumed = 0;
  while (true) {
    // ---- select the next chunk: the smallest keys greater than sm.last ----
    const long long remaining = L - consumed;
    Key96 thr;
    thr.hi = ~0ull;
    thr.lo = ~0u;
    if (remaining > kChunk) {
      if (threadIdx.x == 0) {
        sm.prefix = Key96{0ull, 0u};
        sm.kk = kChunk;
        sm.taken = 0;
        sm.done = 0;
      }
      __syncthreads();
      for (int level = 0; level < 12; level++) {
        for (int b = threadIdx.x; b < 256; b += blockDim.x) sm.hist[b] = 0;
        __syncthreads();
        const Key96 pre = sm.prefix, last = sm.last;
        for (long long e = threadIdx.x; e < L; e += blockDim.x) {
          const Key96 k = make_key(c.wl_t[e], c.wl_i[e]);
          if (!first_round && !key_less(last, k)) continue;
          if (!key_prefix_eq(k, pre, level)) continue;
          atomicAdd(&sm.hist[key_digit(k, level)], 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          int d;
          long long cum;
          bool stop;
          select_level(sm.hist, sm.taken, sm.kk, kChunkMin, d, cum, stop);
          Key96 p = sm.prefix;
          key_set_digit(p, level, d);
          if (stop) {
            // every candidate below bucket d: the prefix with digit d and zeros after it
            sm.prefix = key_prev(p);
            sm.done = 1;  // used here as "select finished early"
          } else {
            sm.prefix = p;
            sm.kk = sm.kk - cum;
            sm.taken = sm.taken + cum;
          }
        }
        __syncthreads();
        if (sm.done) break;
      }
      thr = sm.prefix;
      __syncthreads();
      if (threadIdx.x == 0) sm.done = 0;
    }
    // ---- extract keys in (sm.last, thr] into shared memory ----
    if (threadIdx.x == 0) sm.count = 0;
    __syncthreads();
    {
      const Key96 last = sm.last;
      for (long long e = threadIdx.x; e < L; e += blockDim.x) {
        const Key96 k = make_key(c.wl_t[e], c.wl_i[e]);
        if (!first_round && !key_less(last, k)) continue;
        if (key_less(thr, k)) continue;
        const int pos = atomicAdd(&sm.count, 1);
        if (pos < kChunk) {
          sm.k_hi[pos] = k.hi;
          sm.k_lo[pos] = k.lo;
        }
      }
    }
    __syncthreads();
    const int cnt = sm.count < kChunk ? sm.count : kChunk;
    walk_chunk<R, H, S>(c, x, g, Y, Sl, sm, cnt, w);
    consumed += cnt;
    if (sm.done || consumed >= L || cnt == 0) break;
    if (threadIdx.x == 0) sm.last = Key96{sm.k_hi[cnt - 1], sm.k_lo[cnt - 1]};
    first_round = false;
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  if (sm.done == 2) return;  // a failed M*wbp: the driver resets the memory
  walk_end(st, w, sm.work[0]);
}

// ---- the cooperative walk of single-instance solves ------------------------------------

// Bounded grid barrier of a cooperative launch: every CTA adds one arrival to *bar and
// waits until all of this barrier's arrivals are in (target counts up by gridDim.x per
// barrier; *bar is zero at launch).  Returns false in every CTA whose wait gave up.
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int& target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(bar, 1u);
    long long k = 0;
    while (*(volatile unsigned int*)bar < target && k < 4 * kWaitPolls) k++;
    s_ok = k < 4 * kWaitPolls ? 1 : 0;
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}

// The cooperative walk takes the breakpoints in chunks of up to kWalkRows keys.  For each
// chunk the whole grid selects it (histograms in global memory, the same digit decided
// redundantly by every CTA), sorts it (pieces of kPiece keys, one CTA each; a key's rank is
// its position in its piece plus its lower bounds in the others) and prepares each key's
// record: its row times its step, M*wbp and wbp'M wbp.  CTA 0 then walks the records.
//
// The walk is the reference's recurrence with its operations unchanged, cut into the chains
// that depend on one another, each run by its own warp over sub-batches of kSub keys one
// sub-batch behind the warp that feeds it:
//   scan    p += (-dibp) wbp and c += dt p need no f' or f'': one lane per component, one
//           dependent addition a key;
//   dots    wbp'M c and wbp'M p, one thread per key, and the terms of f' and f'';
//   f''     three dependent additions a key on one thread;
//   f'      four dependent additions a key on one thread (the walk's rate: the reference's
//           order of these additions is kept), and the sum of dt on another;
//   test    dtm = -f'/f'' against the next breakpoint's distance, one lane per key.
// The keys after the one where the walk ends are worked on in vain (at most five sub-batches).
//
// What bounds it: f', four dependent additions of 8.3 cycles each, 33-40 cycles a key; with the
// chunk's selection, sort and preparation (40-60 us for 8192 keys) a key takes 35 ns.  One
// thread walking key by key, with 64 rows of M*wbp prepared at a time by 64 threads, took
// 0.46-0.52 us a key (n = 512^2, a solve with 426,000 keys in six walks: 190.7 -> 14.6 ms); f'
// and f'' on one thread, and f' with its loads waited for, took 74-84 cycles a key (23.2 ms).
constexpr int kWalkRows = 8192;       // breakpoints of a chunk at most
constexpr int kWalkFirst = 1024;      // of the first chunk (most walks are short); then doubled
constexpr int kPiece = kWalkThreads;  // keys sorted together
constexpr int kMaxPieces = kWalkRows / kPiece;
constexpr int kSub = 128;             // keys of a pipeline step
constexpr int kRow = 2 * kMaxM;

// The records of a chunk, after the WalkScratch header (walk_scratch_bytes in all).
template <typename S>
struct WalkRecords {
  unsigned long long *raw_hi, *hi;  // keys as extracted (then sorted by piece), keys in order
  S *e, *v;                         // rows of kRow: (-dibp) wbp, M wbp
  S *dibp, *zibp, *wmw;
  unsigned int *raw_lo, *lo;
};
__host__ __device__ inline int walk_rows(int n) {
  return n < kWalkRows ? (n + kPiece - 1) / kPiece * kPiece : kWalkRows;
}
template <typename S>
__host__ __device__ inline size_t walk_scratch_bytes(int n) {
  return (sizeof(WalkScratch) + 255) / 256 * 256 +
         (size_t)walk_rows(n) * (2 * 8 + 2 * 4 + (2 * kRow + 3) * sizeof(S));
}
template <typename S>
__device__ __forceinline__ WalkRecords<S> walk_records(WalkScratch* ws, int n) {
  const size_t rows = (size_t)walk_rows(n);
  WalkRecords<S> r;
  r.raw_hi = reinterpret_cast<unsigned long long*>(reinterpret_cast<unsigned char*>(ws) +
                                                   (sizeof(WalkScratch) + 255) / 256 * 256);
  r.hi = r.raw_hi + rows;
  r.e = reinterpret_cast<S*>(r.hi + rows);
  r.v = r.e + rows * kRow;
  r.dibp = r.v + rows * kRow;
  r.zibp = r.dibp + rows;
  r.wmw = r.zibp + rows;
  r.raw_lo = reinterpret_cast<unsigned int*>(r.wmw + rows);
  r.lo = r.raw_lo + rows;
  return r;
}

// Dynamic shared memory of k_walk_coop.
template <typename S>
struct WalkCoop {
  unsigned long long k_hi[kPiece];
  unsigned int k_lo[kPiece];
  unsigned int hist[256];
  S sy[kMaxM * kMaxM], wt[kMaxM * kMaxM];
  int slot[kMaxM];  // the ring's physical slots, oldest pair first
  int rank[kBatch];
  S wbp[kBatch][kRow + 1], bv[kBatch][kRow + 1], work[kBatch][kMaxM + 1];
  union {
    struct {
      // CTA 0's pipeline; buffers are indexed by sub-batch modulo their count
      S e[2][kSub][kRow];
      S p[2][kSub][kRow + 1], c[2][kSub][kRow + 1];  // p before, c after each key
      S dt[8][kSub];
      alignas(16) S a[4][kSub][4];                               // the terms of f' (the first becomes dt f'')
      alignas(16) S b[2][kSub][4];                               // the terms of f''
      alignas(16) S f1s[2][kSub], f2s[4][kSub], ts[2][kSub];     // after each key
      S ckp[kWalkRows / kSub][kRow], ckc[kWalkRows / kSub][kRow];  // p, c before each sub-batch
    };
    struct {  // every CTA: the chunk's keys while they are ranked
      unsigned long long all_hi[kWalkRows];
      unsigned int all_lo[kWalkRows];
    };
  };
  S f1, f2, dtm, tsum, tj;                       // before the next key to be tested
  int nleft, nint, all_fixed, done, passed, info;
};

// Sorts the kPiece keys held one per thread (a bitonic network; partners within a warp by
// shuffles, farther ones through shared memory).
template <typename S>
__device__ Key96 sort_piece(WalkCoop<S>& sm, Key96 k) {
  const int e = (int)threadIdx.x;
#pragma unroll 1
  for (int size = 2; size <= kPiece; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      Key96 o;
      if (stride >= 32) {
        sm.k_hi[e] = k.hi;
        sm.k_lo[e] = k.lo;
        __syncthreads();
        o = Key96{sm.k_hi[e ^ stride], sm.k_lo[e ^ stride]};
        __syncthreads();
      } else {
        o.hi = __shfl_xor_sync(0xffffffffu, k.hi, stride);
        o.lo = __shfl_xor_sync(0xffffffffu, k.lo, stride);
      }
      // the lower of the pair keeps the smaller key where the run ascends
      const bool want_small = ((e & stride) == 0) == ((e & size) == 0);
      if (key_less(o, k) == want_small) k = o;
    }
  }
  return k;
}

// The pieces (each sorted, in shared memory) below key k of piece `own`: the lower bounds of k in
// the pieces first, first + kRankLanes, ... of the chunk's cnt keys.
constexpr int kRankLanes = 4;  // threads that share a key's pieces
__device__ __forceinline__ int rank_part(const unsigned long long* all_hi, const unsigned int* all_lo,
                                         const Key96& k, int own, int first, int cnt) {
  constexpr int kMine = kMaxPieces / kRankLanes;
  int lb[kMine];
#pragma unroll
  for (int u = 0; u < kMine; u++) lb[u] = 0;
#pragma unroll 1
  for (int step = kPiece; step > 0; step >>= 1) {
#pragma unroll
    for (int u = 0; u < kMine; u++) {
      const int pc = first + u * kRankLanes, base = pc * kPiece, at = lb[u] + step;
      if (pc != own && at <= kPiece && base + at <= cnt &&
          key_less(Key96{all_hi[base + at - 1], all_lo[base + at - 1]}, k))
        lb[u] = at;
    }
  }
  int r = 0;
#pragma unroll
  for (int u = 0; u < kMine; u++) r += lb[u];
  return r;
}

// sdot of two rows of col2 values, a in registers.
template <typename S>
__device__ __forceinline__ S row_dot(const S* b, const S (&a)[kRow], int col2) {
  S r = 0;
#pragma unroll
  for (int g = 0; g < kRow; g += 4) {
    if (g + 4 <= col2) {
      r += b[g] * a[g] + b[g + 1] * a[g + 1] + b[g + 2] * a[g + 2] + b[g + 3] * a[g + 3];
    } else if (g + 2 <= col2) {
      r += b[g] * a[g];
      r += b[g + 1] * a[g + 1];
    }
  }
  return r;
}

// Four values in one (float) or two (double) shared-memory loads, and back.
__device__ __forceinline__ void lds4(uint32_t at, double (&v)[4]) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(at) : "memory");
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "r"(at + 16) : "memory");
}
__device__ __forceinline__ void lds4(uint32_t at, float (&v)[4]) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t at, const double (&v)[4]) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(v[0]), "d"(v[1]) : "memory");
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(at + 16), "d"(v[2]), "d"(v[3]) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t at, const float (&v)[4]) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}

// One thread runs a chain over nk keys, a row of four terms each: step(row) returns the chain's
// value after the key, stored to out.  Groups of four keys, the next group's rows loaded while
// one group is added (two register sets, so that no addition waits for a load).
template <typename S, typename Step>
__device__ __forceinline__ void walk_chain(const S (*rows)[4], S* out, int nk, Step&& step) {
  constexpr int U = 4;
  const uint32_t in = smem_addr(rows), o = smem_addr(out);
  constexpr uint32_t kB = 4 * sizeof(S);
  S va[U][4], vb[U][4];
  auto load = [&](S (&v)[U][4], int q) {
#pragma unroll
    for (int u = 0; u < U; u++) lds4(in + (uint32_t)(q + u) * kB, v[u]);
  };
  auto run = [&](const S (&v)[U][4], int q) {
    S r[U];
#pragma unroll
    for (int u = 0; u < U; u++) r[u] = step(v[u]);
    sts4(o + (uint32_t)q * (uint32_t)sizeof(S), r);
  };
  // (rows past nk, of a buffer of kSub, are loaded and not used)
  int q = 0;
  load(va, 0);
#pragma unroll 1
  for (; q + 2 * U <= nk; q += 2 * U) {
    load(vb, q + U);
    run(va, q);
    load(va, q + 2 * U < kSub ? q + 2 * U : 0);
    run(vb, q + U);
  }
  for (; q < nk; q++) out[q] = step(rows[q]);
}

// f'' after each of nk keys: f2 - b[0] + b[1] - b[2] (lbfgsbcpu.cpp:789, 800-803; the last two
// terms with a history only), no lower than floor2 when kLimit.
template <bool kHist, bool kLimit, typename S>
__device__ __forceinline__ void walk_f2(const S (*b)[4], S* out, int nk, S f2, S floor2) {
  walk_chain(b, out, nk, [&](const S* v) {
    f2 = f2 - v[0];
    if constexpr (kHist) f2 = f2 + v[1] - v[2];
    if constexpr (kLimit) f2 = smax(floor2, f2);
    return f2;
  });
}

// f' after each of nk keys: f1 + a[0] + a[1] - a[2] + a[3] (788, 801; the last with a history
// only).
template <bool kHist, typename S>
__device__ __forceinline__ void walk_f1(const S (*a)[4], S* out, int nk, S f1) {
  walk_chain(a, out, nk, [&](const S* v) {
    f1 = f1 + v[0] + v[1] - v[2];
    if constexpr (kHist) f1 = f1 + v[3];
    return f1;
  });
}

// CTA 0: walks the cnt records in order (all threads).  sm.f1 .. sm.nint carry the walk from
// chunk to chunk; st->p and st->c hold p and c.  Sets sm.done when the walk has ended.
template <typename R, typename H, typename S>
__device__ void walk_records_in_order(const Ctx<R, H, S>& c, const WalkRecords<S>& rec, int cnt,
                                      WalkCoop<S>& sm) {
  DevState<S>* st = c.st;
  const int col2 = 2 * st->col, nbreak = st->nbreak, bnded = st->bnded, n = st->n;
  const S theta = st->theta, floor2 = (S)(5e-16 * (double)st->f2org);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsub = (cnt + kSub - 1) / kSub;
  auto t_of = [&](int k) { return (S)__longlong_as_double((long long)__ldcg(&rec.hi[k])); };
  // sub-batch b into shared memory, by nt threads; every load is issued before the first store
  auto stage = [&](int b, int tid, auto nt) {
    constexpr int NT = decltype(nt)::value, kTrips = (kSub * kRow + NT - 1) / NT;
    const int base = b * kSub, nk = cnt - base < kSub ? cnt - base : kSub;
    S v[kTrips];
    if (col2 > 0) {
#pragma unroll
      for (int w = 0; w < kTrips; w++) {
        const int q = tid + w * NT;
        v[w] = q < nk * kRow ? __ldcg(&rec.e[(size_t)base * kRow + q]) : S(0);
      }
    }
    for (int q = tid; q < nk; q += NT) {
      const int k = base + q;
      sm.dt[b & 7][q] = t_of(k) - (k > 0 ? t_of(k - 1) : sm.tj);
    }
    if (col2 > 0) {
#pragma unroll
      for (int w = 0; w < kTrips; w++) {
        const int q = tid + w * NT;
        if (q < nk * kRow) (&sm.e[b & 1][0][0])[q] = v[w];
      }
    }
  };
  S pj = 0, cj = 0;  // warp 0: component `lane` of p and c
  if (warp == 0 && lane < col2) {
    pj = st->p[lane + 1];
    cj = st->c[lane + 1];
  }
  if (threadIdx.x == 0) sm.passed = cnt;
  stage(0, (int)threadIdx.x, std::integral_constant<int, kWalkThreads>{});
  __syncthreads();
  // The test's warp ends the loop through the step's barrier itself: every thread gets the same
  // answer for the same step, however late it leaves the barrier (a flag in shared memory, read
  // after the barrier, would be written by the next step's test before a late warp has read it).
  bool stopped = false;
  for (int s = 0; s < nsub + 4; s++) {
    bool stop_here = false;
    if (warp == kWalkThreads / 32 - 1) {
      if (lane == 0 && s >= 3 && s - 3 < nsub) {
        // the sum of dt, at the pace of f'
        const int b = s - 3, nk = cnt - b * kSub < kSub ? cnt - b * kSub : kSub;
        const S* dt = sm.dt[b & 7];
        S ts = b > 0 ? sm.ts[(b - 1) & 1][kSub - 1] : sm.tsum;
#pragma unroll 8
        for (int q = 0; q < nk; q++) {
          ts = ts + dt[q];
          sm.ts[b & 1][q] = ts;
        }
      }
    } else if (warp >= 8) {
      if (s + 1 < nsub) stage(s + 1, (int)threadIdx.x - 256, std::integral_constant<int, kWalkThreads - 256 - 32>{});
    } else if (warp == 0) {
      if (s < nsub && col2 > 0 && lane < kRow) {
        const int b = s & 1, nk = cnt - s * kSub < kSub ? cnt - s * kSub : kSub;
        const S* dt = sm.dt[s & 7];
        sm.ckp[s][lane] = pj;
        sm.ckc[s][lane] = cj;
        constexpr int U = 4;
        S da[U], ea[U], db[U], eb[U];
        auto load = [&](S (&d)[U], S (&e)[U], int q) {
#pragma unroll
          for (int u = 0; u < U; u++) {
            d[u] = dt[q + u];
            e[u] = sm.e[b][q + u][lane];
          }
        };
        auto run = [&](const S (&d)[U], const S (&e)[U], int q) {
#pragma unroll
          for (int u = 0; u < U; u++) {
            sm.p[b][q + u][lane] = pj;
            cj += d[u] * pj;
            sm.c[b][q + u][lane] = cj;
            pj += e[u];
          }
        };
        int q = 0;
        load(da, ea, 0);
#pragma unroll 1
        for (; q + 2 * U <= nk; q += 2 * U) {
          load(db, eb, q + U);
          run(da, ea, q);
          load(da, ea, q + 2 * U < kSub ? q + 2 * U : 0);
          run(db, eb, q + U);
        }
        for (; q < nk; q++) {
          sm.p[b][q][lane] = pj;
          cj += dt[q] * pj;
          sm.c[b][q][lane] = cj;
          pj += sm.e[b][q][lane];
        }
      }
    } else if (warp >= 4) {
      const int b = s - 1, q = (int)threadIdx.x - 128;
      if (b >= 0 && b < nsub && b * kSub + q < cnt) {
        const int k = b * kSub + q, o = b & 1, oa = b & 3;
        const S dibp = __ldcg(&rec.dibp[k]), zibp = __ldcg(&rec.zibp[k]);
        const S dibp2 = dibp * dibp;
        sm.a[oa][q][1] = dibp2;
        sm.a[oa][q][2] = theta * dibp * zibp;
        sm.b[o][q][0] = theta * dibp2;
        if (col2 > 0) {
          S v[kRow];
#pragma unroll
          for (int j = 0; j < kRow; j++) v[j] = j < col2 ? __ldcg(&rec.v[(size_t)k * kRow + j]) : S(0);
          const S wmw = __ldcg(&rec.wmw[k]);
          const S wmc = row_dot(sm.c[o][q], v, col2), wmp = row_dot(sm.p[o][q], v, col2);
          sm.a[oa][q][3] = dibp * wmc;
          sm.b[o][q][1] = (S)2.0 * dibp * wmp;
          sm.b[o][q][2] = dibp2 * wmw;
        }
      }
    } else if (warp == 1) {
      const int b = s - 2;
      if (b >= 0 && b < nsub) {
        const int nk = cnt - b * kSub < kSub ? cnt - b * kSub : kSub;
        S* f2s = sm.f2s[b & 3];
        const S f2 = b > 0 ? sm.f2s[(b - 1) & 3][kSub - 1] : sm.f2;
        if (lane == 0) {
          if (col2 > 0)
            walk_f2<true, false>(sm.b[b & 1], f2s, nk, f2, floor2);
          else
            walk_f2<false, false>(sm.b[b & 1], f2s, nk, f2, floor2);
        }
        __syncwarp();
        // the lower limit of f'' hardly ever acts: the sub-batch is summed without it, and
        // once more with it when it would have acted
        bool low = false;
        for (int q = lane; q < nk; q += 32) low = low || floor2 > f2s[q];
        if (__any_sync(0xffffffffu, low) && lane == 0) {
          if (col2 > 0)
            walk_f2<true, true>(sm.b[b & 1], f2s, nk, f2, floor2);
          else
            walk_f2<false, true>(sm.b[b & 1], f2s, nk, f2, floor2);
        }
      }
    } else if (warp == 2) {
      const int b = s - 3;
      if (b >= 0 && b < nsub) {
        const int nk = cnt - b * kSub < kSub ? cnt - b * kSub : kSub;
        const S* dt = sm.dt[b & 7];
        const S* f2s = sm.f2s[b & 3];
        const S f2 = b > 0 ? sm.f2s[(b - 1) & 3][kSub - 1] : sm.f2;  // before the sub-batch
        for (int q = lane; q < nk; q += 32) sm.a[b & 3][q][0] = dt[q] * (q > 0 ? f2s[q - 1] : f2);
        __syncwarp();
        if (lane == 0) {
          const S f1 = b > 0 ? sm.f1s[(b - 1) & 1][kSub - 1] : sm.f1;
          if (col2 > 0)
            walk_f1<true>(sm.a[b & 3], sm.f1s[b & 1], nk, f1);
          else
            walk_f1<false>(sm.a[b & 3], sm.f1s[b & 1], nk, f1);
        }
      }
    } else {  // warp 3
      const int b = s - 4;
      if (b >= 0) {
        const int o = b & 1, base = b * kSub, nk = cnt - base < kSub ? cnt - base : kSub;
        const S* dt = sm.dt[b & 7];
        const S* f2s = sm.f2s[b & 3];
        int hit = -1;
        for (int r = 0; r < nk && hit < 0; r += 32) {
          const int q = r + lane;
          bool ends = false;
          if (q < nk) {
            const S dtm = q == 0 ? sm.dtm : -sm.f1s[o][q - 1] / f2s[q - 1];
            ends = dtm < dt[q];
          }
          const unsigned bal = __ballot_sync(0xffffffffu, ends);
          if (bal) hit = r + __ffs(bal) - 1;
        }
        __syncwarp();
        if (lane == 0) {
          const int q = hit >= 0 ? hit : nk;  // the sub-batch's keys passed
          const bool last = hit < 0 && sm.nleft - (base + nk) == 0;
          sm.tj = t_of(hit >= 0 ? base + hit : base + nk - 1);
          // every variable has reached its bound: the last key moves c and sum dt only
          const bool fixed = last && nbreak == n;
          const int f = fixed ? q - 1 : q;
          if (q > 0) sm.tsum = sm.ts[o][q - 1];
          if (f > 0) {
            sm.f1 = sm.f1s[o][f - 1];
            sm.f2 = f2s[f - 1];
            sm.dtm = -sm.f1 / sm.f2;
          }
          if (fixed) {
            sm.dtm = dt[q - 1];
            sm.all_fixed = 1;
          } else if (last && bnded) {
            sm.f1 = 0;
            sm.f2 = 0;
            sm.dtm = 0;
          }
          if (hit >= 0) {
            stop_here = true;
            sm.passed = base + hit;
          }
          if (hit >= 0 || last) sm.done = 1;
        }
      }
    }
    if (__syncthreads_or(stop_here)) {
      stopped = true;
      break;
    }
  }
  const int passed = sm.passed;
  if (warp == 0 && lane < col2) {
    if (stopped || sm.all_fixed) {
      // p and c where the walk ended, from the start of that sub-batch
      const int b = stopped ? passed / kSub : (cnt - 1) / kSub;
      pj = sm.ckp[b][lane];
      cj = sm.ckc[b][lane];
      for (int k = b * kSub; k < passed; k++) {
        cj += sm.dt[b & 7][k - b * kSub] * pj;
        if (!(sm.all_fixed && k == cnt - 1)) pj += __ldcg(&rec.e[(size_t)k * kRow + lane]);
      }
    }
    st->p[lane + 1] = pj;
    st->c[lane + 1] = cj;
  }
  for (int k = threadIdx.x; k < passed; k += blockDim.x)
    c.code[(int)__ldcg(&rec.lo[k])] =
        (int8_t)(__ldcg(&rec.dibp[k]) > S(0) ? IW_WALK_UPP : IW_WALK_LOW);
  __syncthreads();
  if (threadIdx.x == 0) {
    sm.nleft -= passed;
    sm.nint += passed - sm.all_fixed;
  }
}

// Lists the breakpoints with the whole grid and walks them chunk by chunk.  wsc->bar and
// *wl_n are zero at launch.
template <typename R, typename H, typename S>
__global__ void __launch_bounds__(kWalkThreads, 1) k_walk_coop(Ctx<R, H, S> c, const R* __restrict__ x,
                                                            const R* __restrict__ g) {
  DevState<S>* st = c.st;
  if (c.rounds) {
    if (!st->rp_sub || st->internal_fail != 0) return;
    x = c.X[st->xr[0]];
    g = c.G[st->gr[0]];
  }
  if (st->gcp_state != GCP_WALK) return;
  extern __shared__ __align__(128) unsigned char dyn[];
  WalkCoop<S>& sm = *reinterpret_cast<WalkCoop<S>*>(dyn);
  WalkScratch* ws = c.wsc;
  const int col = st->col, col2 = 2 * col;
  const S theta = st->theta;
  for (int k = threadIdx.x; k < kMaxM * kMaxM; k += blockDim.x) {
    sm.sy[k] = st->sy[k];
    sm.wt[k] = st->wt[k];
  }
  if (threadIdx.x == 0) {
    // a zero on the factor's diagonal fails every M*wbp (the driver resets the memory)
    sm.info = 0;
    for (int j = 0; j < col; j++) sm.slot[j] = st->phys[(st->head - 1 + j) % st->m + 1];
    for (int j = col; j >= 1; j--)
      if (LB_AT(st->wt, kMaxM, j, j) == S(0)) sm.info = j;
  }
  __syncthreads();
  const bool lead = blockIdx.x == 0;
  unsigned int target = 0;
  if (sm.info != 0) {
    // the other CTAs may still read internal_fail at the top: written after the barrier
    if (!grid_barrier(&ws->bar, target)) {
      if (threadIdx.x == 0) atomicExch(&st->device_error, 1);
      return;
    }
    if (lead && threadIdx.x == 0) st->internal_fail = sm.info;
    return;
  }
  auto fail = [&]() {
    if (threadIdx.x == 0) atomicExch(&st->device_error, 1);
  };
  const WalkRecords<S> rec = walk_records<S>(ws, c.n);
  if (lead) {
    for (int b = threadIdx.x; b < 256; b += blockDim.x) ws->hist[0][b] = 0;
    if (threadIdx.x == 0) {
      ws->chunk_n = 0;
      const WalkCarry<S> w = walk_start(st);
      sm.f1 = w.f1;
      sm.f2 = w.f2;
      sm.dtm = w.dtm;
      sm.tsum = w.tsum;
      sm.tj = w.tj;
      sm.nleft = w.nleft;
      sm.nint = w.nint;
      sm.all_fixed = 0;
      sm.done = 0;
    }
  }
  gather_breakpoints<R, H, S>(c, cta_here(), blockDim.x, x, g);
  if (!grid_barrier(&ws->bar, target)) return fail();
  const long long L = (long long)*(volatile unsigned int*)c.wl_n;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long e0 = (long long)blockIdx.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  bool first_round = true;
  Key96 last{0ull, 0u};
  long long consumed = 0;
  int want = kWalkFirst < walk_rows(c.n) ? kWalkFirst : walk_rows(c.n);
  int hb = 0;  // the histogram buffer of the next level (rotating over three)
  while (true) {
    const long long remaining = L - consumed;
    Key96 thr{~0ull, ~0u};
    if (remaining > want) {
      Key96 prefix{0ull, 0u};
      long long kk = want, taken = 0;
      for (int level = 0; level < 12; level++) {
        unsigned int* h = ws->hist[hb];
        // the buffer after this one was last read two levels ago, before the previous
        // barrier: clear it for the next level
        if (lead)
          for (int b = threadIdx.x; b < 256; b += blockDim.x) ws->hist[(hb + 1) % 3][b] = 0;
        for (int b = threadIdx.x; b < 256; b += blockDim.x) sm.hist[b] = 0;
        __syncthreads();
        for (long long e = e0 + threadIdx.x; e < L; e += stride) {
          const Key96 k = make_key(c.wl_t[e], c.wl_i[e]);
          if (!first_round && !key_less(last, k)) continue;
          if (!key_prefix_eq(k, prefix, level)) continue;
          atomicAdd(&sm.hist[key_digit(k, level)], 1u);
        }
        __syncthreads();
        for (int b = threadIdx.x; b < 256; b += blockDim.x)
          if (sm.hist[b]) atomicAdd(&h[b], sm.hist[b]);
        if (!grid_barrier(&ws->bar, target)) return fail();
        for (int b = threadIdx.x; b < 256; b += blockDim.x) sm.hist[b] = __ldcg(&h[b]);
        __syncthreads();
        hb = (hb + 1) % 3;
        int d;
        long long cum;
        bool stop;
        select_level(sm.hist, taken, kk, want / 4, d, cum, stop);
        __syncthreads();  // every thread has read the histogram before the next level clears it
        key_set_digit(prefix, level, d);
        if (stop) {
          prefix = key_prev(prefix);
          break;
        }
        kk -= cum;
        taken += cum;
      }
      thr = prefix;
    }
    // extract the chunk: keys in (last, thr]
    for (long long e1 = e0; e1 < L; e1 += stride) {
      const long long e = e1 + threadIdx.x;
      Key96 k{0ull, 0u};
      bool take = false;
      if (e < L) {
        k = make_key(c.wl_t[e], c.wl_i[e]);
        take = (first_round || key_less(last, k)) && !key_less(thr, k);
      }
      const unsigned mask = __ballot_sync(0xffffffffu, take);
      if (mask == 0) continue;
      unsigned int start = 0;
      if (lane == 0) start = atomicAdd(&ws->chunk_n, (unsigned int)__popc(mask));
      start = __shfl_sync(0xffffffffu, start, 0);
      const unsigned int pos = start + __popc(mask & ((1u << lane) - 1u));
      if (take && pos < (unsigned int)walk_rows(c.n)) {
        rec.raw_hi[pos] = k.hi;
        rec.raw_lo[pos] = k.lo;
      }
    }
    if (!grid_barrier(&ws->bar, target)) return fail();
    const unsigned int n_sel = __ldcg(&ws->chunk_n);
    const int cnt = n_sel < (unsigned int)want ? (int)n_sel : want;
    if (cnt == 0) break;
    // sort the pieces
    for (int pc = blockIdx.x; pc * kPiece < cnt; pc += gridDim.x) {
      const int q = pc * kPiece + (int)threadIdx.x;
      Key96 k{~0ull, ~0u};
      if (q < cnt) k = Key96{__ldcg(&rec.raw_hi[q]), __ldcg(&rec.raw_lo[q])};
      k = sort_piece(sm, k);
      if (q < cnt) {
        rec.raw_hi[q] = k.hi;
        rec.raw_lo[q] = k.lo;
      }
    }
    if (!grid_barrier(&ws->bar, target)) return fail();
    if (lead && threadIdx.x == 0) ws->chunk_n = 0;
    // rank every key and prepare its record there, the keys spread over the CTAs; every CTA
    // searches a copy of the pieces in its shared memory (searching them in L2, all CTAs
    // probing the same lines, took 34 us a chunk)
#pragma unroll 4
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
      sm.all_hi[q] = __ldcg(&rec.raw_hi[q]);
      sm.all_lo[q] = __ldcg(&rec.raw_lo[q]);
    }
    __syncthreads();
    for (int q0 = 0; q0 < cnt; q0 += kBatch * (int)gridDim.x) {
      if (threadIdx.x < kBatch * kRankLanes) {
        const int qr = q0 + (int)(threadIdx.x / kRankLanes) * (int)gridDim.x + (int)blockIdx.x;
        int r = 0;
        if (qr < cnt)
          r = rank_part(sm.all_hi, sm.all_lo, Key96{sm.all_hi[qr], sm.all_lo[qr]}, qr / kPiece,
                        (int)(threadIdx.x % kRankLanes), cnt);
#pragma unroll
        for (int o = 1; o < kRankLanes; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (threadIdx.x % kRankLanes == 0) sm.rank[threadIdx.x / kRankLanes] = r + qr % kPiece;
      }
      __syncthreads();
      const int q = q0 + (int)threadIdx.x * (int)gridDim.x + (int)blockIdx.x;
      if (threadIdx.x < kBatch && q < cnt) {
        const Key96 k{sm.all_hi[q], sm.all_lo[q]};
        const int i = (int)k.lo;
        S* wbp = sm.wbp[threadIdx.x];
        S* v = sm.bv[threadIdx.x];
        const R xi = x[i], gi = g[i];
#pragma unroll 4
        for (int j = 0; j < col; j++) {
          const size_t at = (size_t)sm.slot[j] * (size_t)c.ld + i;
          wbp[1 + j] = (S)HistTraits<H>::load(c.wy + at);
          wbp[1 + col + j] = theta * (S)HistTraits<H>::load(c.ws + at);
        }
        const int r = sm.rank[threadIdx.x];
        const R dibp = -gi;
        const R zibp = (dibp > R(0)) ? rsub(c.u[i], xi) : rsub(c.l[i], xi);
        rec.hi[r] = k.hi;
        rec.lo[r] = k.lo;
        rec.dibp[r] = (S)dibp;
        rec.zibp[r] = (S)zibp;
        if (col > 0) {
          int info = 0;
          sbmv(sm.sy, sm.wt, col, wbp, v, &info, sm.work[threadIdx.x]);
          rec.wmw[r] = sdot(&wbp[1], 1, &v[1], 1, col2);
          for (int j = 0; j < col2; j++) {
            rec.e[(size_t)r * kRow + j] = (-(S)dibp) * wbp[1 + j];
            rec.v[(size_t)r * kRow + j] = v[1 + j];
          }
        }
      }
      __syncthreads();  // the ranks are rewritten
    }
    if (!grid_barrier(&ws->bar, target)) return fail();
    if (lead) {
      walk_records_in_order<R, H, S>(c, rec, cnt, sm);
      if (threadIdx.x == 0) {
        ws->done = sm.done;
        ws->last_hi = __ldcg(&rec.hi[cnt - 1]);
        ws->last_lo = __ldcg(&rec.lo[cnt - 1]);
      }
    }
    if (!grid_barrier(&ws->bar, target)) return fail();
    const int done = *(volatile int*)&ws->done;
    consumed += cnt;
    if (done || consumed >= L) break;
    last = Key96{*(volatile unsigned long long*)&ws->last_hi, *(volatile unsigned int*)&ws->last_lo};
    first_round = false;
    want = 2 * want < walk_rows(c.n) ? 2 * want : walk_rows(c.n);
  }
  // the walk's end into the state (walk_end), M c by the first warp
  if (!lead || threadIdx.x >= 32) return;
  if (!sm.all_fixed) {
    if (lane == 0) {
      if (sm.dtm <= S(0)) sm.dtm = 0;
      sm.tsum = sm.tsum + sm.dtm;
    }
    __syncwarp();
    if (lane < col2) st->c[lane + 1] += sm.dtm * st->p[lane + 1];
  }
  if (lane == 0) {
    st->f1 = sm.f1;
    st->f2 = sm.f2;
    st->dtm = sm.dtm;
    st->tsum = sm.tsum;
    st->tj = sm.tj;
    st->nleft = sm.nleft;
    st->nint = sm.nint;
  }
  if (lane < col2) sm.wbp[0][lane + 1] = st->c[lane + 1];
  __syncwarp();
  if (col > 0) {
    const int info = wbmv(sm.sy, sm.wt, col, sm.wbp[0], sm.bv[0], sm.work[0], lane);
    if (info != 0) {
      if (lane == 0) st->internal_fail = -8;
      return;
    }
    if (lane < col2) st->mc[lane + 1] = sm.bv[0][lane + 1];
  }
  if (lane == 0) st->gcp_state = GCP_DONE;
}

}  // namespace lbfgsb_b200
