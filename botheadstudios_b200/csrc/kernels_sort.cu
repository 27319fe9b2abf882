// Stable LSD radix sort of (64-bit key, 32-bit value) pairs, with the Morton keys of the state computed on the way when
// the tree asks: one launch up to kOneLaunchMax keys, a chain of launches above.
//
// One launch, 10-bit digits. The chain (reduce, scan and scatter kernels for each 8-bit digit, 12 launches for a 30-bit
// code) costs its launches below a million keys: keys, sort and permutation of the state took 77 µs at 10,240 particles,
// 84 at 65,536 and 93 at 262,144, and take 34, 51 and 67 this way. Here the blocks draw tickets in order; a ticket is one tile (1,024 or 2,048 keys) of one phase. Phase 0 counts the digits of every
// pass (and writes the Morton keys), phase q + 1 moves the tiles of pass q: ranks within the tile (by warps),
// the digit counts of the tiles before it by looking back over their published counts, then a scatter through shared
// memory. A phase waits until the previous one is complete. Tickets are drawn in order, so whatever a tile waits for is
// held by a block that already runs: the launch needs no co-residency and any number of blocks. Ten-bit digits make
// three passes of a 30-bit code; a digit's counters are 16-bit in shared memory.
// Every wait is bounded: after Dev::sort_polls polls the block raises kFlagSortTimeout and goes on (the scatter checks its
// bounds), so a fault in the protocol shows as a flag and not as a hang. What comes out is then no permutation, and the
// control block says so (SortEnd): the callers do without it.
#include "sph_kernels.cuh"

namespace sphb {

constexpr int SO_THREADS = 512;
constexpr int SO_WARPS = SO_THREADS / 32;
constexpr int SO_LOOK = 8;    // predecessors read at a time

// Keys to a thread. A tile is worked on by one SM, whose shared memory and stores bound it (8,192 keys take 12 µs a
// pass), so small sorts take small tiles on many SMs; a tile's look-back reads the counts of every tile before it, so
// larger sorts take larger ones. Above 148 tiles of 2,048 the look-backs of a whole wave of tiles cost more than the
// chain's launches: at 1,048,576 keys 203 µs against the chain's 167, at 4,194,304 717 against 506.
constexpr int kSmallTiles = 64 * 2 * SO_THREADS;
constexpr int kOneLaunchMax = 148 * 4 * SO_THREADS;

// ---- the chain's workspace: [256][tiles] digit counts, 256 digit totals, behind the tile words of the one launch. The
// two forms share nothing: the one launch takes any word with its tag for a published count, and tags, like counts, are
// small numbers.
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 2048 keys per tile
constexpr int RS_WARPS = RS_THREADS / 32;

constexpr int kMaxTiles = kOneLaunchMax / (4 * SO_THREADS);
static_assert(kMaxTiles >= kSmallTiles / (2 * SO_THREADS), "no sort of one launch has more tiles");
constexpr size_t kChainAt = kSortCtlBytes + kMaxTiles * kSortTileBytes;

size_t sort_work_bytes(int n) {
  const size_t m = n < 1 ? 1 : n;
  if (m > kOneLaunchMax) return kChainAt + 256 * sizeof(unsigned) * ((m + RS_TILE - 1) / RS_TILE + 1);
  const size_t small = m < kSmallTiles ? m : kSmallTiles;
  const size_t t2 = (small + 2 * SO_THREADS - 1) / (2 * SO_THREADS), t4 = (m + 4 * SO_THREADS - 1) / (4 * SO_THREADS);
  return kSortCtlBytes + (t2 > t4 ? t2 : t4) * kSortTileBytes;
}
static_assert(SO_BINS * 8 == kSortTileBytes, "a tile publishes one word for each digit");

template <int ITEMS>
struct SortSmem {
  unsigned long long keys[SO_THREADS * ITEMS];
  unsigned vals[SO_THREADS * ITEMS];
  unsigned short wcnt[SO_WARPS][SO_BINS];  // digit counts of each warp, then their prefix over the warps
  unsigned hist[SO_PASSES * SO_BINS];      // phase 0: the tile's digit counts
  unsigned bstart[SO_BINS];                // where a digit starts inside the tile
  unsigned gbin[SO_BINS];                  // where it goes
  unsigned long long warp[33];
  unsigned ticket;
  unsigned finished;  // (not `ticket`: a warp may still be reading the ticket that ended its loop)
};

__device__ __forceinline__ unsigned long long scan_u64(unsigned long long v, unsigned long long* s_warp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(SPH_FULL_MASK, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[w] = incl;
  __syncthreads();
  if (w == 0) {
    const unsigned long long x = lane < SO_WARPS ? s_warp[lane] : 0ull;
    unsigned long long xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(SPH_FULL_MASK, xi, o);
      if (lane >= o) xi += t;
    }
    s_warp[lane] = xi - x;
  }
  __syncthreads();
  return s_warp[w] + incl - v;
}

// Lanes whose digit equals this lane's (and that hold a key: `in`). A ballot for each bit: match_any takes a time
// that grows with the number of distinct digits in the warp (12 µs of a 16 µs pass over 8,192 keys on one SM).
template <int BITS>
__device__ __forceinline__ unsigned same_digit(unsigned d, bool in) {
  unsigned peers = __ballot_sync(SPH_FULL_MASK, in);
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const bool one = (d >> b) & 1u;
    const unsigned bal = __ballot_sync(SPH_FULL_MASK, one);
    peers &= one ? bal : ~bal;
  }
  return peers;
}

// Polls *p (written by other blocks) until it reaches `want`.
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned want, unsigned limit) {
  for (unsigned k = 0; k < limit; ++k) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v >= want) return true;
  }
  return false;
}

// Counts of digits 2t and 2t + 1 in the tiles before `tile`. The published words are tag << 32 | state << 30 | count,
// state 1 the tile's own count, 2 the count up to and including the tile; SO_LOOK tiles' words are read at a time.
__device__ __forceinline__ uint2 look_back(const unsigned long long* status, int tile, int t, unsigned tag, unsigned limit,
                                           bool& ok) {
  uint2 before = make_uint2(0u, 0u);
  int ja = tile - 1, jb = tile - 1;
  for (unsigned polls = 0; ja >= 0 || jb >= 0;) {
    unsigned long long a[SO_LOOK], b[SO_LOOK];
#pragma unroll
    for (int k = 0; k < SO_LOOK; ++k) {
      a[k] = ja - k >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(status + (size_t)(ja - k) * SO_BINS + 2 * t) : 0ull;
      b[k] = jb - k >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(status + (size_t)(jb - k) * SO_BINS + 2 * t + 1) : 0ull;
    }
    const int a0 = ja, b0 = jb;
#pragma unroll
    for (int k = 0; k < SO_LOOK; ++k) {
      if (ja >= 0 && ja == a0 - k && (unsigned)(a[k] >> 32) == tag) {  // an unpublished word ends the batch
        before.x += (unsigned)a[k] & 0x3fffffffu;
        ja = ((unsigned)a[k] >> 30) == 2u ? -1 : ja - 1;
      }
      if (jb >= 0 && jb == b0 - k && (unsigned)(b[k] >> 32) == tag) {
        before.y += (unsigned)b[k] & 0x3fffffffu;
        jb = ((unsigned)b[k] >> 30) == 2u ? -1 : jb - 1;
      }
    }
    if (ja == a0 && jb == b0 && ++polls > limit) {
      ok = false;
      break;
    }
  }
  return before;
}

template <bool MORTON, int SO_ITEMS>
__global__ void __launch_bounds__(SO_THREADS, 2) k_radix_sort(
    int n, int T, int passes, unsigned long long* keys0, unsigned long long* keys1, unsigned* vals0, unsigned* vals1,
    SortCtl* ctl, unsigned long long* status, unsigned polls, unsigned* flags, const float4* __restrict__ pos,
    const unsigned* __restrict__ id, const unsigned* __restrict__ seg, const Seg* __restrict__ segs) {
  extern __shared__ __align__(16) unsigned char so_raw[];
  SortSmem<SO_ITEMS>& S = *reinterpret_cast<SortSmem<SO_ITEMS>*>(so_raw);
  constexpr int SO_TILE = SO_THREADS * SO_ITEMS;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const unsigned epoch = ctl->end.epoch;
  const auto timed_out = [&] {
    atomicOr(flags, kFlagSortTimeout);
    atomicExch(&ctl->end.failed, epoch + 1u);
  };
  const unsigned total = (unsigned)(T * (passes + 1));
  unsigned next = 0;  // thread 0: the ticket after this one, drawn while this one is worked on
  if (tid == 0) next = atomicAdd(&ctl->ticket, 1u);
  for (;;) {
    if (tid == 0) S.ticket = next;
    __syncthreads();
    const unsigned ticket = S.ticket;
    if (ticket >= total) break;
    if (tid == 0) next = atomicAdd(&ctl->ticket, 1u);
    const int phase = (int)(ticket / (unsigned)T), tile = (int)(ticket % (unsigned)T);
    const int base = tile * SO_TILE;
    if (phase == 0) {
      unsigned* h = S.hist;
      for (int k = tid; k < passes * SO_BINS; k += SO_THREADS) h[k] = 0u;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < SO_ITEMS; ++k) {
        const int i = base + k * SO_THREADS + tid;
        if (i < n) {
          unsigned long long key;
          if (MORTON) {
            const unsigned sg = seg[i];
            const unsigned* bb = segs[sg].bbox;
            float lo[3], ext[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
              lo[a] = key_float(bb[a]);
              ext[a] = fmaxf(fsub(key_float(bb[3 + a]), lo[a]), 1.0e-30f);
            }
            key = ((unsigned long long)sg << 30) | morton_code(pos[i], lo, ext);
            const unsigned o = id[i];  // a permutation of [0, n): equal keys end up in original-index order
            keys0[o] = key;
            vals0[o] = (unsigned)i;
          } else {
            key = keys0[i];
          }
          for (int q = 0; q < passes; ++q) atomicAdd(&h[q * SO_BINS + ((unsigned)(key >> (SO_BITS * q)) & (SO_BINS - 1))], 1u);
        }
      }
      __syncthreads();
      for (int k = tid; k < passes * SO_BINS; k += SO_THREADS)
        if (h[k]) atomicAdd(&ctl->hist[0][0] + k, h[k]);
    } else {
      const int q = phase - 1, shift = SO_BITS * q;
      const unsigned long long* kin = q & 1 ? keys1 : keys0;
      const unsigned* vin = q & 1 ? vals1 : vals0;
      unsigned long long* kout = q & 1 ? keys0 : keys1;
      unsigned* vout = q & 1 ? vals0 : vals1;
      for (int k = tid; k < SO_WARPS * SO_BINS / 2; k += SO_THREADS) reinterpret_cast<unsigned*>(&S.wcnt[0][0])[k] = 0u;
      if (tid == 0 && !wait_count(&ctl->done[phase - 1], (unsigned)T, polls)) timed_out();
      __syncthreads();
      unsigned long long key[SO_ITEMS];
      unsigned val[SO_ITEMS], rank[SO_ITEMS];
#pragma unroll
      for (int k = 0; k < SO_ITEMS; ++k) {
        const int i = base + (w * SO_ITEMS + k) * 32 + lane;
        key[k] = i < n ? __ldcg(kin + i) : 0ull;
        val[k] = i < n ? __ldcg(vin + i) : 0u;
      }
      const unsigned long long hist2 = __ldcg(reinterpret_cast<const unsigned long long*>(ctl->hist[q]) + tid);
#pragma unroll
      for (int k = 0; k < SO_ITEMS; ++k) {
        const bool in = base + (w * SO_ITEMS + k) * 32 + lane < n;
        const unsigned d = (unsigned)(key[k] >> shift) & (SO_BINS - 1);
        const unsigned peers = same_digit<SO_BITS>(d, in);
        const int leader = in ? __ffs(peers) - 1 : lane;
        unsigned old = 0;
        if (lane == leader && in) {
          old = S.wcnt[w][d];
          S.wcnt[w][d] = (unsigned short)(old + __popc(peers));
        }
        old = __shfl_sync(SPH_FULL_MASK, old, leader);
        rank[k] = old + __popc(peers & lt_mask);
        __syncwarp();
      }
      __syncthreads();
      // thread t: digits 2t and 2t + 1, the two halves of a word of the 16-bit counters
      unsigned run = 0;
#pragma unroll
      for (int k = 0; k < SO_WARPS; ++k) {
        unsigned* c = reinterpret_cast<unsigned*>(&S.wcnt[k][0]) + tid;
        const unsigned v = *c;
        *c = run;
        run += v;  // no carry: a tile holds fewer than 2^16 keys
      }
      const unsigned c0 = run & 0xffffu, c1 = run >> 16;
      const unsigned tag = epoch * 8u + (unsigned)q + 1u;
      const unsigned long long word = (unsigned long long)tag << 32;
      volatile unsigned long long* mine = status + (size_t)tile * SO_BINS + 2 * tid;
      const unsigned state = tile == 0 ? 2u << 30 : 1u << 30;
      mine[0] = word | state | c0;
      mine[1] = word | state | c1;
      // one scan for the digits' places in the whole output (high half) and in the tile (low half)
      const unsigned h0 = (unsigned)hist2, h1 = (unsigned)(hist2 >> 32);
      const unsigned long long ex = scan_u64(((unsigned long long)(h0 + h1) << 32) | (c0 + c1), S.warp);
      bool ok = true;
      const uint2 before = look_back(status, tile, tid, tag, polls, ok);
      if (!ok) timed_out();
      if (tile > 0) {
        mine[0] = word | (2u << 30) | (before.x + c0);
        mine[1] = word | (2u << 30) | (before.y + c1);
      }
      const unsigned g = (unsigned)(ex >> 32), l = (unsigned)ex;
      S.bstart[2 * tid] = l;
      S.bstart[2 * tid + 1] = l + c0;
      S.gbin[2 * tid] = g + before.x;
      S.gbin[2 * tid + 1] = g + h0 + before.y;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < SO_ITEMS; ++k) {
        if (base + (w * SO_ITEMS + k) * 32 + lane < n) {
          const unsigned d = (unsigned)(key[k] >> shift) & (SO_BINS - 1);
          const unsigned at = S.bstart[d] + S.wcnt[w][d] + rank[k];
          S.keys[at] = key[k];
          S.vals[at] = val[k];
        }
      }
      __syncthreads();
      const int cnt = min(SO_TILE, n - base);
      for (int i = tid; i < cnt; i += SO_THREADS) {
        const unsigned long long k = S.keys[i];
        const unsigned d = (unsigned)(k >> shift) & (SO_BINS - 1);
        const unsigned to = S.gbin[d] + (unsigned)i - S.bstart[d];
        if (to < (unsigned)n) {
          kout[to] = k;
          vout[to] = S.vals[i];
        }
      }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(&ctl->done[phase]) : "memory");
  }
  // the last block to run out of tickets leaves the control block ready for the next sort
  if (tid == 0) S.finished = atomicAdd(&ctl->finished, 1u);
  __syncthreads();
  if (S.finished == gridDim.x - 1) {
    for (int k = tid; k < SO_PASSES * SO_BINS; k += SO_THREADS) (&ctl->hist[0][0])[k] = 0u;
    if (tid <= SO_PASSES) ctl->done[tid] = 0u;
    if (tid == 0) {
      ctl->ticket = 0u;
      ctl->finished = 0u;
      ctl->end.epoch = epoch + 1u;
    }
  }
}

template <bool MORTON, int ITEMS>
static int radix_sort(int n, int bits, unsigned long long* const keys[2], unsigned* const vals[2], void* work,
                      unsigned polls, unsigned* flags, const State* st, const Seg* segs, cudaStream_t s) {
  static SmemLimit attr;
  smem_limit(k_radix_sort<MORTON, ITEMS>, (int)sizeof(SortSmem<ITEMS>), attr);
  const int tile = SO_THREADS * ITEMS, T = (n + tile - 1) / tile, passes = (bits + SO_BITS - 1) / SO_BITS;
  const int grid = T < 2 * 148 ? T : 2 * 148;
  SortCtl* ctl = static_cast<SortCtl*>(work);
  unsigned long long* status = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(work) + kSortCtlBytes);
  k_radix_sort<MORTON, ITEMS><<<grid, SO_THREADS, sizeof(SortSmem<ITEMS>), s>>>(
      n, T, passes, keys[0], keys[1], vals[0], vals[1], ctl, status, polls, flags, st ? st->pos_h : nullptr,
      st ? st->id : nullptr, st ? st->seg : nullptr, segs);
  return passes & 1;
}

template <bool MORTON>
static int one_launch(int n, int bits, unsigned long long* const keys[2], unsigned* const vals[2], void* work,
                      unsigned polls, unsigned* flags, const State* st, const Seg* segs, cudaStream_t s) {
  if (n <= kSmallTiles) return radix_sort<MORTON, 2>(n, bits, keys, vals, work, polls, flags, st, segs, s);
  return radix_sort<MORTON, 4>(n, bits, keys, vals, work, polls, flags, st, segs, s);
}

// ---------------------------------------------------------------------------------------------------
// The chain: 8-bit digits, reduce-then-scan (no inter-block waits): upsweep histograms per tile, per-digit scans over
// tiles, stable downsweep (ranks by warps, staged through shared memory).
// ---------------------------------------------------------------------------------------------------
__global__ void k_keys(const float4* __restrict__ pos, const unsigned* __restrict__ id,
                       const unsigned* __restrict__ seg, int n, const Seg* __restrict__ segs,
                       unsigned long long* __restrict__ keys, unsigned* __restrict__ vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned sg = seg[i];
  const unsigned* bb = segs[sg].bbox;
  float lo[3], ext[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = key_float(bb[k]);
    ext[k] = fmaxf(fsub(key_float(bb[3 + k]), lo[k]), 1.0e-30f);
  }
  const unsigned code = morton_code(pos[i], lo, ext);
  const unsigned o = id[i];  // a permutation of [0, n)
  keys[o] = ((unsigned long long)sg << 30) | code;
  vals[o] = (unsigned)i;
}

__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const unsigned long long* __restrict__ keys, int n,
                                                           int shift, unsigned* __restrict__ hist, int T) {
  __shared__ unsigned h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int base = blockIdx.x * RS_TILE;
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const int idx = base + it * RS_THREADS + threadIdx.x;
    if (idx < n) atomicAdd(&h[(unsigned)(keys[idx] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[threadIdx.x * T + blockIdx.x] = h[threadIdx.x];
}

// One block per digit: exclusive scan of hist[d][0..T) in place; tot[d] = sum.
__global__ void __launch_bounds__(1024) k_rs_scan(unsigned* __restrict__ hist, unsigned* __restrict__ tot, int T) {
  __shared__ unsigned s_warp[33];
  unsigned* h = hist + (size_t)blockIdx.x * T;
  const int per = (T + blockDim.x - 1) / blockDim.x;
  const int b0 = threadIdx.x * per;
  unsigned sum = 0;
  for (int i = 0; i < per; ++i)
    if (b0 + i < T) sum += h[b0 + i];
  unsigned total;
  unsigned run = block_exclusive_scan(sum, s_warp, total);
  for (int i = 0; i < per; ++i)
    if (b0 + i < T) {
      const unsigned v = h[b0 + i];
      h[b0 + i] = run;
      run += v;
    }
  if (threadIdx.x == 0) tot[blockIdx.x] = total;
}

__global__ void __launch_bounds__(RS_THREADS) k_rs_downsweep(const unsigned long long* __restrict__ kin,
                                                             const unsigned* __restrict__ vin,
                                                             unsigned long long* __restrict__ kout,
                                                             unsigned* __restrict__ vout, int n, int shift,
                                                             const unsigned* __restrict__ hist,
                                                             const unsigned* __restrict__ tot, int T) {
  __shared__ unsigned long long s_keys[RS_TILE];
  __shared__ unsigned s_vals[RS_TILE];
  __shared__ unsigned s_wcnt[RS_WARPS][256];
  __shared__ unsigned s_gbin[256];     // global output start of digit d for this tile
  __shared__ unsigned s_bstart[256];   // start of digit d inside the tile
  __shared__ unsigned s_warp[33];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int base = blockIdx.x * RS_TILE;

  // global digit starts: exclusive scan of the digit totals + this tile's prefix
  unsigned total;
  const unsigned dstart = block_exclusive_scan(tot[tid], s_warp, total);
  s_gbin[tid] = dstart + hist[tid * T + blockIdx.x];
#pragma unroll
  for (int k = 0; k < RS_WARPS; ++k) s_wcnt[k][tid] = 0;
  __syncthreads();

  unsigned long long key[RS_ITEMS];
  unsigned val[RS_ITEMS], dig[RS_ITEMS], loc[RS_ITEMS];
  const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const int idx = base + (w * RS_ITEMS + it) * 32 + lane;
    const bool ok = idx < n;
    key[it] = ok ? kin[idx] : 0ull;
    val[it] = ok ? vin[idx] : 0u;
    const unsigned d = (unsigned)(key[it] >> shift) & 255u;
    dig[it] = ok ? d : 256u;
    const unsigned peers = same_digit<8>(d, ok);
    const int leader = ok ? __ffs(peers) - 1 : lane;
    unsigned old = 0;
    if (lane == leader && ok) {
      old = s_wcnt[w][d];
      s_wcnt[w][d] = old + __popc(peers);
    }
    old = __shfl_sync(SPH_FULL_MASK, old, leader);
    loc[it] = old + __popc(peers & lt_mask);
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive prefix over warps, then over digits within the tile
  {
    unsigned run = 0;
#pragma unroll
    for (int k = 0; k < RS_WARPS; ++k) {
      const unsigned c = s_wcnt[k][tid];
      s_wcnt[k][tid] = run;
      run += c;
    }
    unsigned t2;
    s_bstart[tid] = block_exclusive_scan(run, s_warp, t2);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    if (dig[it] < 256u) {
      const unsigned p = s_bstart[dig[it]] + s_wcnt[w][dig[it]] + loc[it];
      s_keys[p] = key[it];
      s_vals[p] = val[it];
    }
  }
  __syncthreads();
  const int cnt = min(RS_TILE, n - base);
  for (int i = tid; i < cnt; i += RS_THREADS) {
    const unsigned long long k = s_keys[i];
    const unsigned d = (unsigned)(k >> shift) & 255u;
    const unsigned g = s_gbin[d] + (unsigned)i - s_bstart[d];
    kout[g] = k;
    vout[g] = s_vals[i];
  }
}

// Sorts keys[0]; returns the kernels launched, `src` the buffer with the result.
static int chain_sort(unsigned long long* const keys[2], unsigned* const vals[2], int n, int bits, void* work, int& src,
                      cudaStream_t s) {
  const int T = (n + RS_TILE - 1) / RS_TILE;
  unsigned* hist = reinterpret_cast<unsigned*>(static_cast<unsigned char*>(work) + kChainAt);
  unsigned* tot = hist + 256 * (size_t)T;
  src = 0;
  int launches = 0;
  for (int shift = 0; shift < bits; shift += 8) {
    k_rs_upsweep<<<T, RS_THREADS, 0, s>>>(keys[src], n, shift, hist, T);
    k_rs_scan<<<256, 1024, 0, s>>>(hist, tot, T);
    k_rs_downsweep<<<T, RS_THREADS, 0, s>>>(keys[src], vals[src], keys[src ^ 1], vals[src ^ 1], n, shift, hist, tot, T);
    src ^= 1;
    launches += 3;
  }
  return launches;
}

int launch_radix_sort(unsigned long long* const keys[2], unsigned* const vals[2], int n, int bits, void* work,
                      unsigned polls, unsigned* flags, int& src, cudaStream_t s) {
  src = 0;
  if (n <= 1) return 0;
  if (n > kOneLaunchMax) return chain_sort(keys, vals, n, bits, work, src, s);
  src = one_launch<false>(n, bits, keys, vals, work, polls, flags, nullptr, nullptr, s);
  return 1;
}

int launch_morton_sort(const Dev& d, int& src, const SortEnd*& end, cudaStream_t s) {
  end = nullptr;  // the chain waits for nothing
  const State& in = d.st[d.cur];
  if (d.n > kOneLaunchMax) {
    k_keys<<<(d.n + 255) / 256, 256, 0, s>>>(in.pos_h, in.id, in.seg, d.n, d.segs, d.keys[0], d.vals[0]);
    return 1 + chain_sort(d.keys, d.vals, d.n, 30 + d.segbits, d.sort_work, src, s);
  }
  end = &static_cast<SortCtl*>(d.sort_work)->end;
  src = one_launch<true>(d.n, 30 + d.segbits, d.keys, d.vals, d.sort_work, d.sort_polls, &d.P->flags, &in, d.segs, s);
  return 1;
}

}  // namespace sphb
