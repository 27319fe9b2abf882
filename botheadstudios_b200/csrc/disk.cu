// Disk measurement and the Moon candidate of one impact, on the device.
//
// The reference measures a finished impact on the host in two places: the impact-run tool
// (tools/impact-run/src/main.rs:732-878, `measure` + `moon_candidate`) and the engine's HUD statistics
// (crates/engine/src/gpu_sph.rs:399-469, `disk_stats_json` + accretion.rs:73-160 `find_clumps`). Both:
//   1. mass, centre of mass and bulk velocity of the impact;
//   2. the remnant radius: the smallest radius about the centre of mass enclosing 85 % of the mass (radius
//      sort + running sum);
//   3. each particle's two-body orbit about the remnant: escaping, remnant (periapsis inside it) or disk;
//   4. friends-of-friends over the disk particles with a linking length of twice the mean smoothing length
//      (the tool: an O(k²) pair loop; the engine: a cell grid), union-find;
//   5. per clump of two or more: mass, centre of mass and velocity, volume, internal kinetic energy and the
//      pairwise self-potential (O(s²)); bound when KE + PE < 0; outside the fluid Roche limit
//      2.44 R (ρ_remnant / ρ_clump)^(1/3); the Moon candidate is the heaviest bound clump outside it.
//
// Here every step is a kernel over the impact's particle range of the state (already contiguous per impact):
// deterministic two-pass f64 reductions; the 85 % crossing is a selection over the exact f64 bit patterns of the
// radii, its running masses summed as integers; classification writes per-block partials and an order-preserving
// compaction of the disk; the friends-of-friends search sorts the disk by a lexicographic cell key (cell edge just above the linking
// length, so every linked pair lies in the 3 × 3 column of z-runs around a particle), and one warp per
// particle scans its partners and unites linked pairs with a lock-free union-find (a root is hooked under a
// node of lower rank with atomicCAS, path halving; ranks fall along every path, so every walk ends); clumps are
// contiguous after a radix sort by root; one block per clump sums its moments; the self-potential is split
// into 128 × 128 tile pairs of the clump's pair triangle, each summed in f64 by one block, then reduced per
// clump in a fixed order. The per-particle arithmetic that decides a classification (radii, periapsis, pair
// distances) is written with explicitly rounded operations in the reference's order; the sums differ from
// the reference's sequential ones only in association. Two host reads size the work: the disk count and the
// number of self-potential tile pairs.
#include <cstdint>
#include <cstring>

#include "sph_kernels.cuh"

namespace sphb {

struct RadiusSelect;

struct DiskWork {
  int cap = 0;
  void* base = nullptr;
  unsigned long long* keys[2] = {nullptr, nullptr};
  unsigned* vals[2] = {nullptr, nullptr};
  void* sort_work = nullptr;
  double* part = nullptr;   // [kDmBlocks][kDmVals] block partials
  RadiusSelect* sel = nullptr;  // the mass-fraction crossing's counters
  double* scal = nullptr;   // [S_COUNT]
  unsigned* cnt = nullptr;  // [C_COUNT]
  unsigned* bcnt = nullptr; // [kDmBlocks] disk particles per block, then their output offsets
  unsigned char* cat = nullptr;  // [cap] category of each particle
  float4* pm = nullptr;                  // [cap] x, y, z, mass of the points whose radii are sorted
  float4* dpos[2] = {nullptr, nullptr};  // disk particles: x, y, z, h
  float4* dvel[2] = {nullptr, nullptr};  // vx, vy, vz, mass
  float2* drp[2] = {nullptr, nullptr};   // rho, prov bits
  unsigned* parent = nullptr;  // [cap] union-find forest over the cell-sorted disk
  unsigned* gcnt = nullptr;    // [cap] members per root
  uint4* clump = nullptr;      // [cap/2+1] first member, members, root, units
  unsigned long long* uoff = nullptr;  // [cap/2+2] first self-potential unit of each clump
  double* cstat = nullptr;     // [cap/2+1][8] mass, com xyz, volume, target mass, internal KE, Σ m m / r
  double* upe = nullptr;       // [upe_cap] unit sums Σ m_a m_b / r (grown on demand)
  unsigned long long upe_cap = 0;
  double* out = nullptr;       // [16]
  double* bb = nullptr;        // [16] body bulk: centre, radius, new centre, new mass, new radius + mass, mass
  double* place = nullptr;     // [kMaxPlacements][12] offset, vel, spin, centre of each source body
};

namespace {

// The 48-byte exchange record (SphParticle, gpu_sph.rs:28).
struct P48x {
  float px, py, pz, h, vx, vy, vz, u, mass;
  unsigned mat;
  float rho;
  unsigned prov;
};
static_assert(sizeof(P48x) == 48, "48-byte particle");

constexpr int kDmThreads = 256;
constexpr int kDmBlocks = 592;  // 4 × 148 SMs; block b reduces the b-th contiguous chunk of the impact
constexpr int kDmVals = 8;
constexpr int kPeRows = 128;    // particles per self-potential row
constexpr int kSelBits = 12, kSelBins = 1 << kSelBits;  // digits of the crossing's selection
constexpr int kSelBrute = 256;  // candidates that one block ranks directly, in about 15 µs (1,000: 285)
// (beside their number) the candidates need not agree in any bit of the radius; they agree in all
constexpr unsigned kSelWhole = 1u << 31, kSelEqual = 1u << 30;
constexpr int kCellBits = 21;  // of a cell coordinate, at most
constexpr int kUnionTries = 1 << 16;
constexpr unsigned long long kMaxUnits = 1ull << 28;  // self-potential tile pairs (2 GB of partial sums)
constexpr double kPiD = 3.14159265358979323846;
constexpr unsigned kMaxPlacements = 256;

enum { S_M = 0, S_COM = 1, S_VCOM = 4, S_RREM = 7, S_MREM = 8, S_LINK = 9, S_RHOREM = 10, S_CAT = 11, S_COUNT = 24 };
enum { C_NDISK = 0, C_NCLUMP = 1, C_SEL = 2, C_ERR = 3, C_UNITS64 = 4, C_MINH = 6, C_CELLBITS = 7, C_MANY = 8, C_COUNT = 9 };
// (u64 in 4-5; the disk's extent before its cell bits in 7; candidates that the crossing's selection left in 8)
// body-bulk slots: the current centre and radius, the latest selection's centre and mass, its crossing radius
// and running mass, the mass of every particle of the body
enum { BB_C = 0, BB_R = 3, BB_CN = 4, BB_MN = 7, BB_RN = 8, BB_M = 10 };

// Sum kDmVals doubles over the block in a fixed order (warp trees, then warps in order). Thread 0 gets them.
__device__ __forceinline__ void block_sum(double* v, double (*s)[kDmVals]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < kDmVals; ++k) {
    const double x = warp_sum(v[k]);
    if (lane == 0) s[w][k] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < kDmVals; ++k) {
      double a = 0.0;
      for (int j = 0; j < nw; ++j) a += s[j][k];
      v[k] = a;
    }
  }
  __syncthreads();
}

// Sum of nb partials of value k over a warp, fixed order.
__device__ __forceinline__ double warp_sum_column(const double* part, int nb, int k) {
  double a = 0.0;
  for (int b = (int)(threadIdx.x & 31); b < nb; b += 32) a += part[b * kDmVals + k];
  return warp_sum(a);
}

__device__ __forceinline__ double dsq3(double x, double y, double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// The particle's position as the 48-byte exchange record holds it (f32 of the f64 master).
__device__ __forceinline__ float3 pos_f32(const State& st, unsigned t) {
  return make_float3((float)st.x[t], (float)st.y[t], (float)st.z[t]);
}

}  // namespace

// The selection's counters: zero before each use.
struct RadiusSelect {
  unsigned long long hist[2][kSelBins];  // weight in each bin of the first and of the second digit
  unsigned long long base[2];            // the weight before the crossing bin of each
  unsigned bin[2];                       // those bins
  unsigned done[3];                      // blocks that finished each pass
  unsigned count;                        // candidates listed
  unsigned amax;                         // the largest |coordinate| of the points (float bits)
  unsigned pi;                           // of many candidates: the leading bits of the crossing one's index
  unsigned long long pk;                 // ... and of its radius
  unsigned long long kmax, kinv;         // the candidates' largest radius, and the complement of their smallest
};

namespace {

// ---- 1. mass, centre of mass, bulk velocity ----------------------------------------------------------
__global__ void __launch_bounds__(kDmThreads) k_dm_moments(State st, unsigned off, unsigned m, unsigned chunk,
                                                           double* __restrict__ part, float4* __restrict__ pm,
                                                           RadiusSelect* __restrict__ sel) {
  __shared__ double s[kDmThreads / 32][kDmVals];
  double a[kDmVals] = {0, 0, 0, 0, 0, 0, 0, 0};
  float amax = 0.0f;
  const unsigned b0 = blockIdx.x * chunk, b1 = min(m, b0 + chunk);
  for (unsigned i = b0 + threadIdx.x; i < b1; i += kDmThreads) {
    const unsigned t = off + i;
    const float3 p = pos_f32(st, t);
    const float4 v = st.vel_u[t];
    const double mm = st.mass[t];
    pm[i] = make_float4(p.x, p.y, p.z, st.mass[t]);  // positions and masses for the remnant radius
    amax = fmaxf(amax, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
    a[0] += mm;
    a[1] += (double)p.x * mm;  // f32 × f32 products are exact in f64
    a[2] += (double)p.y * mm;
    a[3] += (double)p.z * mm;
    a[4] += (double)v.x * mm;
    a[5] += (double)v.y * mm;
    a[6] += (double)v.z * mm;
    a[7] += (double)st.pos_h[t].w;
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) atomicMax(&sel->amax, __float_as_uint(amax));
  block_sum(a, s);
  if (threadIdx.x == 0)
    for (int k = 0; k < kDmVals; ++k) part[blockIdx.x * kDmVals + k] = a[k];
}

__global__ void k_dm_moments_final(const double* __restrict__ part, int nb, double* __restrict__ scal) {
  __shared__ double t[kDmVals];
  const int w = threadIdx.x >> 5;
  const double v = warp_sum_column(part, nb, w);
  if ((threadIdx.x & 31) == 0) t[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    const double M = t[0];
    scal[S_M] = M;
    for (int k = 0; k < 3; ++k) {
      scal[S_COM + k] = t[1 + k] / M;
      scal[S_VCOM + k] = t[4 + k] / M;
    }
    scal[S_CAT + 7] = t[7];  // Σ h over every particle (the engine's linking length)
  }
}

// ---- 2. radii about a centre, the mass-fraction crossing --------------------------------------------------
// Shared by the remnant radius (85 % of an impact's mass) and the bulk radius of a body (98 %): the point whose running
// mass, in radius order about the centre (equal radii in index order), first reaches frac of the total. pm holds the
// points' f32 positions and masses; the radius is the exact f64 distance from the centre.
//
// A selection, not a sort: a first pass sums the weights in 4,096 bins of the radius's leading bits (64 bins an octave,
// down from a bound on the radii), a second one in the 4,096 bins of its next 12 bits inside the bin where the running
// weight crosses, a third lists the points of the crossing bin there, some ten of a million, and one block ranks those.
// Points on a lattice or a shell can leave many at one radius, or at radii that agree to 2^-18: above kSelBrute candidates
// the host, which reads the counters anyway, selects among them by further digits (launch_radius_digits).
// Weights are integers, so the sums do not depend on their order and equal masses sum exactly. Bound by three readings of the points; a radix sort of the 64-bit radii, the masses
// gathered in its order and two prefixes took 226 µs at 1,024,845 points, the three passes take 50.
__device__ __forceinline__ unsigned long long radius_bits(float4 p, const double* __restrict__ centre) {
  const double dx = __dsub_rn((double)p.x, centre[0]), dy = __dsub_rn((double)p.y, centre[1]),
               dz = __dsub_rn((double)p.z, centre[2]);
  return (unsigned long long)__double_as_longlong(__dsqrt_rn(dsq3(dx, dy, dz)));  // r >= 0: ordered like the value
}
// A point's weight: its mass in units of a power of two that puts the total between 2^61 and 2^62, so masses above
// 2^-38 of the total are whole. Without mass (or with one that is no number) every point weighs one: the first crosses.
__device__ __forceinline__ double sel_scale(double total) {
  return total > 0.0 && total < 1e300 ? __longlong_as_double((2107ll - (__double_as_longlong(total) >> 52)) << 52) : 0.0;
}
__device__ __forceinline__ unsigned long long sel_weight(float m, double scale) {
  return scale > 0.0 ? __double2ull_rn((double)m * scale) : 1ull;
}
__device__ __forceinline__ unsigned long long sel_target(double frac, double total, double scale) {
  const unsigned long long t = scale > 0.0 ? __double2ull_ru(__dmul_rn(frac, total) * scale) : 1ull;
  return t > 0ull ? t : 1ull;
}
// First digit: the leading bits below those of `bound`, larger radii first; the last bin takes everything below.
__device__ __forceinline__ unsigned sel_bin(unsigned long long key, unsigned long long bound) {
  const unsigned long long hi = bound >> 46, k = key >> 46;
  const unsigned long long d = hi > k ? hi - k : 0ull;
  return d < (unsigned long long)(kSelBins - 1) ? (unsigned)d : (unsigned)(kSelBins - 1);
}

// The bin of h (shared memory; in order of radius: from the last one down when `down`) where a running weight that starts
// at `base` reaches the target, or the sum if that falls short; base becomes the weight before that bin. The whole block.
__device__ unsigned sel_cross(const unsigned long long* h, bool down, unsigned long long& base, unsigned long long target) {
  __shared__ unsigned long long s_sum[kDmThreads / 32], s_base;
  __shared__ unsigned s_bin;
  constexpr int PER = kSelBins / kDmThreads;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned long long sum = 0ull;
#pragma unroll
  for (int k = 0; k < PER; ++k) {  // (each lane starts elsewhere in its run: no bank conflicts)
    const int i = t * PER + ((k + t) & (PER - 1));
    sum += h[down ? kSelBins - 1 - i : i];
  }
  unsigned long long incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(SPH_FULL_MASK, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_sum[w] = incl;
  __syncthreads();
  unsigned long long before = base + incl - sum, total = base;
#pragma unroll
  for (int k = 0; k < kDmThreads / 32; ++k) {
    if (k < w) before += s_sum[k];
    total += s_sum[k];
  }
  target = target < total ? target : total;
  if (before < target && before + sum >= target) {  // one thread
    int i = t * PER;
    for (;; ++i) {  // ends within the run: its sum reaches the target
      const unsigned long long v = h[down ? kSelBins - 1 - i : i];
      if (before + v >= target || i == t * PER + PER - 1) break;
      before += v;
    }
    s_bin = (unsigned)(down ? kSelBins - 1 - i : i);
    s_base = before;
  }
  __syncthreads();
  base = s_base;
  const unsigned bin = s_bin;
  __syncthreads();
  return bin;
}

// The crossing point among the n listed ones, n <= kSelBrute, ranked by (radius, index) by one block: its radius to out[0],
// the running mass there to out[1].
__device__ void sel_rank(unsigned long long* h, const float4* __restrict__ pm, unsigned n, double scale,
                         unsigned long long target, unsigned long long base, const unsigned long long* list_key,
                         const unsigned* list_idx, double* __restrict__ out) {
  const unsigned t = threadIdx.x;
  unsigned long long *s_key = h, *s_w = h + kSelBrute;
  unsigned* s_idx = reinterpret_cast<unsigned*>(h + 2 * kSelBrute);
  for (unsigned i = t; i < n; i += kDmThreads) {
    s_key[i] = __ldcg(list_key + i);
    s_idx[i] = __ldcg(list_idx + i);
    s_w[i] = sel_weight(pm[s_idx[i]].w, scale);
  }
  __syncthreads();
  for (unsigned i = t; i < n; i += kDmThreads) {
    const unsigned long long key = s_key[i], w = s_w[i];
    unsigned long long before = base, total = base;
    for (unsigned k = 0; k < n; ++k) {
      if (s_key[k] < key || (s_key[k] == key && s_idx[k] < s_idx[i])) before += s_w[k];
      total += s_w[k];
    }
    const unsigned long long goal = target < total ? target : total;
    if (before < goal && before + w >= goal) {  // one candidate
      out[0] = __longlong_as_double((long long)key);
      out[1] = scale > 0.0 ? (double)(before + w) / scale : 0.0;
    }
  }
}

// h[bin] += w; the lanes at it with the first lane's bin add together (of equal radii all of them: otherwise a turn for each
// lane, or, in shared memory, a loop for each).
__device__ __forceinline__ void sel_add(unsigned long long* h, unsigned bin, unsigned long long w) {
  const unsigned at = __activemask();
  const int first = __ffs(at) - 1;
  const bool same = bin == __shfl_sync(at, bin, first);
  const unsigned group = __ballot_sync(at, same);
  if (!same || group == 1u << (threadIdx.x & 31)) {
    atomicAdd(&h[bin], w);
    return;
  }
  const unsigned lo = __reduce_add_sync(group, (unsigned)w & 0xffffu), mid = __reduce_add_sync(group, (unsigned)(w >> 16) & 0xffffffu),
                 hi = __reduce_add_sync(group, (unsigned)(w >> 40));  // (32 values of 24 bits: no carry is lost)
  if ((int)(threadIdx.x & 31) == first) atomicAdd(&h[bin], (unsigned long long)lo + ((unsigned long long)mid << 16) + ((unsigned long long)hi << 40));
}

// Pass 0: weights by the first digit; the radii are kept for the other passes. Pass 1: by the second digit inside the
// crossing bin. Pass 2: the points of the crossing bin of both digits into the list. The last block of a pass to finish
// finds the pass's crossing bin (at the start of the next pass, in every block, that took 10 µs a pass), or ranks the list.
template <int PASS>
__global__ void __launch_bounds__(kDmThreads) k_dm_select_radius(const float4* __restrict__ pm, unsigned m, unsigned chunk,
                                                                 const double* __restrict__ centre,
                                                                 const double* __restrict__ total_mass, double frac,
                                                                 unsigned long long* __restrict__ keys,
                                                                 RadiusSelect* sel, unsigned long long* list_key,
                                                                 unsigned* list_idx, double* __restrict__ out,
                                                                 unsigned* __restrict__ cnt) {
  __shared__ unsigned long long h[kSelBins];
  unsigned* h32 = reinterpret_cast<unsigned*>(h);  // pass 0: low words, then high words (64-bit shared adds are loops: 25.4 µs, this 23.6)
  __shared__ int s_last;
  const double M = *total_mass, scale = sel_scale(M);
  // the centre is a mean of the points, so no radius is above 2 sqrt(3) times their largest coordinate
  const unsigned long long bound = (unsigned long long)__double_as_longlong(4.0 * (double)__uint_as_float(sel->amax));
  const unsigned long long target = sel_target(frac, M, scale);
  const unsigned a = PASS > 0 ? sel->bin[0] : 0u, b = PASS > 1 ? sel->bin[1] : 0u;
  const bool whole = a == (unsigned)(kSelBins - 1);  // the bin of everything far below the bound has no second digit
  if (PASS == 0) {
    for (int k = threadIdx.x; k < kSelBins; k += kDmThreads) h[k] = 0ull;
    __syncthreads();
  }
  const unsigned b0 = blockIdx.x * chunk, b1 = min(m, b0 + chunk);
  unsigned long long kmax = 0ull, kinv = 0ull;
#pragma unroll 4
  for (unsigned i = b0 + threadIdx.x; i < b1; i += kDmThreads) {
    if (PASS == 0) {
      const float4 p = pm[i];
      const unsigned long long key = radius_bits(p, centre);
      keys[i] = key;
      const unsigned d = sel_bin(key, bound);
      const unsigned long long wt = sel_weight(p.w, scale);
      const unsigned lo = (unsigned)wt;
      const unsigned carry = atomicAdd(&h32[d], lo) > ~lo ? 1u : 0u;
      const unsigned up = (unsigned)(wt >> 32) + carry;
      if (up) atomicAdd(&h32[kSelBins + d], up);
    } else {
      const unsigned long long key = keys[i];
      if (sel_bin(key, bound) == a) {
        const unsigned e = whole ? 0u : (unsigned)(key >> 34) & (kSelBins - 1);
        if (PASS == 1) {
          sel_add(sel->hist[1], e, sel_weight(pm[i].w, scale));  // (few points: no block's share of its own)
        } else if (e == b) {
          kmax = max(kmax, key);
          kinv = max(kinv, ~key);
          const unsigned at = atomicAdd(&sel->count, 1u);
          list_key[at] = key;
          list_idx[at] = i;
        }
      }
    }
  }
  if (PASS == 2 && __any_sync(SPH_FULL_MASK, kinv != 0ull)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      kmax = max(kmax, __shfl_xor_sync(SPH_FULL_MASK, kmax, o));
      kinv = max(kinv, __shfl_xor_sync(SPH_FULL_MASK, kinv, o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&sel->kmax, kmax);
      atomicMax(&sel->kinv, kinv);
    }
  }
  if (PASS == 0) {
    __syncthreads();
    for (int k = threadIdx.x; k < kSelBins; k += kDmThreads)
      if (h32[k] | h32[kSelBins + k])
        atomicAdd(&sel->hist[0][k], (unsigned long long)h32[kSelBins + k] << 32 | h32[k]);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&sel->done[PASS], 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (PASS < 2) {
    for (int k = threadIdx.x; k < kSelBins; k += kDmThreads) h[k] = __ldcg(&sel->hist[PASS][k]);
    __syncthreads();
    unsigned long long base = PASS == 0 ? 0ull : sel->base[0];
    const unsigned bin = sel_cross(h, PASS == 0, base, target);
    if (threadIdx.x == 0) {
      sel->bin[PASS] = bin;
      sel->base[PASS] = base;
    }
  } else {
    const unsigned n = __ldcg(&sel->count);
    const bool many = n > (unsigned)kSelBrute;
    if (threadIdx.x == 0) {
      const unsigned long long k = __ldcg(&sel->kmax);
      const unsigned how = k == ~__ldcg(&sel->kinv) ? kSelEqual : whole || a == 0u ? kSelWhole : 0u;  // (bin 0: no numbers)
      cnt[C_MANY] = many ? n | how : 0u;
      sel->pk = how == kSelEqual ? k : k >> 34 << 34;
    }
    if (!many) {
      sel_rank(h, pm, n, scale, target, sel->base[1], list_key, list_idx, out);
    } else {  // ready for the digits: outside the last bin the candidates agree above bit 34
      for (int k = threadIdx.x; k < 2 * kSelBins; k += kDmThreads) (&sel->hist[0][0])[k] = 0ull;
      if (threadIdx.x == 0) {
        sel->done[2] = 0u;
        out[0] = out[1] = 0.0;
      }
    }
  }
}

// One digit of the crossing candidate among n: bits [lo, lo + width) of the radius, or, once that is known, of the index.
// Passes take turns between the two histograms; the last block to finish finds the crossing bin and clears its own.
__global__ void __launch_bounds__(kDmThreads) k_dm_select_digit(const float4* __restrict__ pm, unsigned n,
                                                                const double* __restrict__ total_mass, double frac,
                                                                RadiusSelect* sel,
                                                                const unsigned long long* __restrict__ list_key,
                                                                const unsigned* __restrict__ list_idx, int pass, bool on_key,
                                                                int lo, int width, bool last, double* __restrict__ out) {
  __shared__ unsigned long long h[kSelBins];
  __shared__ int s_last;
  const double M = *total_mass, scale = sel_scale(M);
  const unsigned long long pk = sel->pk;
  const unsigned pi = sel->pi;
  const int top = lo + width;
  unsigned long long* hist = sel->hist[pass & 1];
  for (int k = threadIdx.x; k < kSelBins; k += kDmThreads) h[k] = 0ull;
  __syncthreads();
  const unsigned stride = gridDim.x * kDmThreads;
  for (unsigned i0 = blockIdx.x * kDmThreads; i0 < n; i0 += stride) {
    const unsigned i = i0 + threadIdx.x;
    unsigned bin = 0xffffffffu;
    unsigned long long w = 0ull;
    if (i < n) {
      const unsigned long long k = list_key[i];
      const unsigned x = list_idx[i];
      const bool in = on_key ? top >= 64 || (k >> top) == (pk >> top) : k == pk && (top >= 32 || (x >> top) == (pi >> top));
      if (in) {
        bin = (on_key ? (unsigned)(k >> lo) : x >> lo) & ((1u << width) - 1u);
        w = sel_weight(pm[x].w, scale);
      }
    }
    if (bin != 0xffffffffu) sel_add(h, bin, w);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kSelBins; k += kDmThreads)
    if (h[k]) atomicAdd(&hist[k], h[k]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&sel->done[2], 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int k = threadIdx.x; k < kSelBins; k += kDmThreads) {
    h[k] = __ldcg(&hist[k]);
    hist[k] = 0ull;
  }
  __syncthreads();
  unsigned long long base = sel->base[1];
  const unsigned bin = sel_cross(h, false, base, sel_target(frac, M, scale));
  if (threadIdx.x != 0) return;
  sel->done[2] = 0u;
  sel->base[1] = base;
  if (on_key) sel->pk = (top < 64 ? pk >> top << top : 0ull) | (unsigned long long)bin << lo;
  else sel->pi = pi | bin << lo;
  if (last) {
    out[0] = __longlong_as_double((long long)pk);  // (whole since the pass before)
    out[1] = scale > 0.0 ? (double)(base + sel_weight(pm[pi | bin << lo].w, scale)) / scale : 0.0;
  }
}

// ---- 3. orbit classification ----------------------------------------------------------------------------
// 0 escapes, 1 disk, 2 remnant: main.rs:232-247 (variant 0) or orbit.rs:91-116 (variant 1).
__device__ __forceinline__ int classify(int variant, double px, double py, double pz, double vx, double vy,
                                        double vz, double mu, double r_rem) {
  const double r = __dsqrt_rn(dsq3(px, py, pz));
  const double v2 = dsq3(vx, vy, vz);
  const double hx = __dsub_rn(__dmul_rn(py, vz), __dmul_rn(pz, vy));
  const double hy = __dsub_rn(__dmul_rn(pz, vx), __dmul_rn(px, vz));
  const double hz = __dsub_rn(__dmul_rn(px, vy), __dmul_rn(py, vx));
  const double h2 = dsq3(hx, hy, hz);
  if (variant == 0 && r == 0.0) return 2;
  if (variant == 1 && !(r > 0.0)) return 0;
  const double energy = __dsub_rn(__dmul_rn(0.5, v2), __ddiv_rn(mu, r));
  if (energy >= 0.0) return 0;
  const double hl = __dsqrt_rn(h2);  // variant 1 multiplies by |h| twice: ((2E·|h|)·|h|)/μ²
  const double num = variant == 0 ? __dmul_rn(__dmul_rn(2.0, energy), h2)
                                  : __dmul_rn(__dmul_rn(__dmul_rn(2.0, energy), hl), hl);
  const double q = __ddiv_rn(num, __dmul_rn(mu, mu));
  const double e = __dsqrt_rn(fmax(__dadd_rn(1.0, q), 0.0));
  const double a = __ddiv_rn(-mu, __dmul_rn(2.0, energy));
  return __dmul_rn(a, __dsub_rn(1.0, e)) > r_rem ? 1 : 2;
}

// Categories: 0 target disk, 1 impactor disk, 2 target remnant, 3 impactor remnant, 4/5 escaping.
__global__ void __launch_bounds__(kDmThreads) k_dm_classify(State st, unsigned off, unsigned m, unsigned chunk,
                                                            int variant, double G, const double* __restrict__ scal,
                                                            unsigned char* __restrict__ cat,
                                                            double* __restrict__ part, unsigned* __restrict__ bcnt,
                                                            unsigned* __restrict__ cnt) {
  __shared__ double s[kDmThreads / 32][kDmVals];
  double a[kDmVals] = {0, 0, 0, 0, 0, 0, 0, 0};
  const double cx = scal[S_COM], cy = scal[S_COM + 1], cz = scal[S_COM + 2];
  const double ux = scal[S_VCOM], uy = scal[S_VCOM + 1], uz = scal[S_VCOM + 2];
  const double mu = G * scal[S_MREM], r_rem = scal[S_RREM];
  const unsigned b0 = blockIdx.x * chunk, b1 = min(m, b0 + chunk);
  float extent = 0.0f;  // of the disk particles from the centre, along an axis
#pragma unroll 2
  for (unsigned i = b0 + threadIdx.x; i < b1; i += kDmThreads) {
    const unsigned t = off + i;
    const float3 p = pos_f32(st, t);
    const float4 v = st.vel_u[t];
    const double dx = __dsub_rn((double)p.x, cx), dy = __dsub_rn((double)p.y, cy), dz = __dsub_rn((double)p.z, cz);
    const int c = classify(variant, dx, dy, dz, __dsub_rn((double)v.x, ux), __dsub_rn((double)v.y, uy),
                           __dsub_rn((double)v.z, uz), mu, r_rem);
    const int k = (c == 1 ? 0 : c == 2 ? 2 : 4) + (st.prov[t] == 0u ? 0 : 1);
    cat[i] = (unsigned char)k;
    const double mm = st.mass[t];
#pragma unroll
    for (int j = 0; j < 6; ++j) a[j] += j == k ? mm : 0.0;
    if (c == 1) {
      a[6] += (double)st.pos_h[t].w;
      a[7] += 1.0;
      extent = fmaxf(extent, __double2float_ru(fmax(fabs(dx), fmax(fabs(dy), fabs(dz)))));
    }
  }
  extent = warp_max(extent);
  if ((threadIdx.x & 31) == 0 && extent > 0.0f) atomicMax(&cnt[C_CELLBITS], __float_as_uint(extent));
  block_sum(a, s);
  if (threadIdx.x == 0) {
    for (int k = 0; k < kDmVals; ++k) part[blockIdx.x * kDmVals + k] = a[k];
    bcnt[blockIdx.x] = (unsigned)a[7];
  }
}

// Cells an edge just above the linking length wide: a linked pair differs by at most one cell per axis even after
// the f32 subtraction of the tool's distance.
__device__ __forceinline__ double inv_cell(double link) { return 1.0 / (link * (1.0 + 0x1p-20)); }
// Bits of a cell coordinate that hold every disk particle, from the largest distance along an axis from the centre: the
// sort reads no more digits than the disk's extent needs (27-30 bits of key for a ring, three passes instead of seven).
__device__ __forceinline__ int cell_bits(float extent, double link) {
  const double cells = (double)extent * inv_cell(link) + 1.0;
  int b = 1;
  while (b < kCellBits && !(cells < (double)(1u << (b - 1)))) ++b;
  return b;
}

__global__ void __launch_bounds__(1024) k_dm_classify_final(const double* __restrict__ part, int nb, unsigned m,
                                                            int variant, double link_factor,
                                                            unsigned* __restrict__ bcnt, double* __restrict__ scal,
                                                            unsigned* __restrict__ cnt, double* __restrict__ out) {
  __shared__ unsigned s_warp[33];
  __shared__ double t[kDmVals];
  const int w = threadIdx.x >> 5;
  if (w < kDmVals) {
    const double v = warp_sum_column(part, nb, w);
    if ((threadIdx.x & 31) == 0) t[w] = v;
  }
  unsigned total;
  const unsigned c = threadIdx.x < (unsigned)nb ? bcnt[threadIdx.x] : 0u;
  const unsigned o = block_exclusive_scan(c, s_warp, total);  // synchronises the block
  if (threadIdx.x < (unsigned)nb) bcnt[threadIdx.x] = o;
  if (threadIdx.x == 0) {
    cnt[C_NDISK] = total;
    const double r_rem = scal[S_RREM];
    scal[S_RHOREM] = scal[S_MREM] / (4.0 / 3.0 * kPiD * (r_rem * r_rem * r_rem));
    for (int k = 0; k < 6; ++k) scal[S_CAT + k] = t[k];
    const double mean_h = variant == 0 ? (total ? t[6] / (double)total : 0.0) : scal[S_CAT + 7] / (double)m;
    scal[S_LINK] = link_factor * mean_h;
    cnt[C_CELLBITS] = (unsigned)cell_bits(__uint_as_float(cnt[C_CELLBITS]), link_factor * mean_h);
    const double disk = t[0] + t[1];
    out[0] = disk > 0.0 ? 100.0 * t[0] / disk : 0.0;
    out[1] = disk;
    for (int k = 0; k < 6; ++k) out[2 + k] = t[k];
    out[8] = scal[S_RREM];
    out[9] = scal[S_MREM];
    for (int k = 10; k < 15; ++k) out[k] = 0.0;
    out[15] = (double)total;
  }
}

// ---- 4. friends-of-friends over the disk ----------------------------------------------------------------
__device__ __forceinline__ unsigned cell_coord(double x, double c, double inv_cs, int bits) {
  const double q = floor((x - c) * inv_cs) + (double)(1u << (bits - 1));
  const unsigned top = (1u << bits) - 1u;
  if (!(q > 0.0)) return 0u;  // clamping only merges far cells: linked pairs stay within one cell per axis
  return q >= (double)top ? top : (unsigned)q;
}
__device__ __forceinline__ unsigned long long cell_key(unsigned ix, unsigned iy, unsigned iz, int bits) {
  return ((unsigned long long)ix << (2 * bits)) | ((unsigned long long)iy << bits) | (unsigned long long)iz;
}
// Order-preserving compaction of the disk particles (block b writes from its offset in chunk order, a thread its own run
// of the chunk: one scan a block).
__global__ void __launch_bounds__(kDmThreads) k_dm_compact(State st, const float* __restrict__ rho, unsigned off,
                                                           unsigned m, unsigned chunk, int bits,
                                                           const unsigned char* __restrict__ cat,
                                                           const unsigned* __restrict__ boff,
                                                           const double* __restrict__ scal, float4* __restrict__ dpos,
                                                           float4* __restrict__ dvel, float2* __restrict__ drp,
                                                           unsigned long long* __restrict__ keys,
                                                           unsigned* __restrict__ vals) {
  __shared__ unsigned s_warp[33];
  const double cx = scal[S_COM], cy = scal[S_COM + 1], cz = scal[S_COM + 2];
  const double inv_cs = inv_cell(scal[S_LINK]);
  const unsigned b0 = blockIdx.x * chunk, b1 = min(m, b0 + chunk);
  const unsigned per = chunk / kDmThreads, i0 = b0 + threadIdx.x * per, i1 = min(b1, i0 + per);
  unsigned mine = 0u, total;
  for (unsigned i = i0; i < i1; ++i) mine += cat[i] < 2 ? 1u : 0u;
  unsigned o = boff[blockIdx.x] + block_exclusive_scan(mine, s_warp, total);
  if (!mine) return;
  for (unsigned i = i0; i < i1; ++i) {
    if (cat[i] >= 2) continue;
    const unsigned t = off + i;
    const float3 p = pos_f32(st, t);
    const float4 v = st.vel_u[t];
    dpos[o] = make_float4(p.x, p.y, p.z, st.pos_h[t].w);
    dvel[o] = make_float4(v.x, v.y, v.z, st.mass[t]);
    drp[o] = make_float2(rho[t], __uint_as_float(st.prov[t]));
    keys[o] = cell_key(cell_coord(p.x, cx, inv_cs, bits), cell_coord(p.y, cy, inv_cs, bits),
                       cell_coord(p.z, cz, inv_cs, bits), bits);
    vals[o] = o;
    ++o;
  }
}

// A sort's waits ran out: its result is no permutation, nothing that follows may use it, and the call returns the error.
__device__ __forceinline__ bool unsorted(const unsigned* cnt) { return (cnt[C_ERR] & kFlagSortTimeout) != 0u; }

__global__ void k_dm_gather(unsigned n, const unsigned* __restrict__ order, const float4* __restrict__ p0,
                            const float4* __restrict__ v0, const float2* __restrict__ r0, float4* __restrict__ p1,
                            float4* __restrict__ v1, float2* __restrict__ r1, unsigned* __restrict__ parent,
                            unsigned* __restrict__ gcnt, const unsigned* __restrict__ cnt) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || unsorted(cnt)) return;
  const unsigned j = order[i];
  p1[i] = p0[j];
  v1[i] = v0[j];
  r1[i] = r0[j];
  if (parent) {
    parent[i] = i;
    gcnt[i] = 0u;
  }
}

// A node's rank, a fixed shuffle of the indices (multiplication by an odd number): roots are hooked by rank, since the
// particles are sorted in space and hooking by index makes chains across a whole ring. And the node of a rank.
__device__ __forceinline__ unsigned uf_rank(unsigned x) { return x * 2654435761u; }
__device__ __forceinline__ unsigned uf_node(unsigned r) { return r * 244002641u; }

// Root of x with path halving. A parent's rank is below its child's and the walk strictly falls, so it ends.
__device__ __forceinline__ unsigned uf_find(unsigned* parent, unsigned x) {
  volatile unsigned* p = parent;
  unsigned nx = p[x];
  while (nx != x) {
    const unsigned nn = p[nx];
    if (nn != nx) p[x] = nn;  // nn is an ancestor of x
    x = nx;
    nx = nn;
  }
  return x;
}

// Unites the groups of a and b, which were seen as roots. A root is hooked under a node of lower rank, wherever that
// node's own root is by then: ranks fall along every path, so no cycle can form.
__device__ __forceinline__ bool uf_unite(unsigned* parent, unsigned a, unsigned b) {
  for (int k = 0; k < kUnionTries; ++k) {
    if (a == b) return true;
    const bool up = uf_rank(a) > uf_rank(b);
    const unsigned hi = up ? a : b, lo = up ? b : a;
    if (atomicCAS(&parent[hi], hi, lo) == hi) return true;  // a failed hook means hi gained a parent
    a = uf_find(parent, hi);
    b = uf_find(parent, lo);
  }
  return false;
}

__device__ __forceinline__ double pair_d2(int variant, float4 a, float4 b) {
  if (variant == 0)  // main.rs:823: f32 difference, widened, squared
    return dsq3((double)__fsub_rn(a.x, b.x), (double)__fsub_rn(a.y, b.y), (double)__fsub_rn(a.z, b.z));
  return dsq3(__dsub_rn((double)a.x, (double)b.x), __dsub_rn((double)a.y, (double)b.y),
              __dsub_rn((double)a.z, (double)b.z));
}

__device__ __forceinline__ unsigned lower_bound_u64(const unsigned long long* k, unsigned n, unsigned long long x) {
  unsigned lo = 0, hi = n;
  while (lo < hi) {
    const unsigned mid = (lo + hi) >> 1;
    if (k[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// One warp per particle a: lanes 0-8 find the starts of the nine (x, y) columns' z-runs in the sorted cell keys, lanes
// 9-17 their ends; then the warp scans the runs' partners after a as one sequence, 32 at a time; a linked partner whose
// root differs from a's is united. Bound by the latency of the unions of one ring-wide group, whose roots change under
// many warps at once: searches and scan alone take 19 µs for 22,840 particles, with the unions hooked by index, each
// lane's partner under a's root by turns, 145 µs, by rank under the batch's lowest root 64-79.
__global__ void __launch_bounds__(kDmThreads) k_dm_link(unsigned n, int variant, int bits,
                                                        const unsigned long long* __restrict__ skeys,
                                                        const float4* __restrict__ dpos,
                                                        const double* __restrict__ scal,
                                                        unsigned* __restrict__ parent, unsigned* __restrict__ cnt) {
  if (unsorted(cnt)) return;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
  const unsigned top = (1u << bits) - 1u;
  const double link = scal[S_LINK], link2 = link * link;
  bool ok = true;
  for (unsigned a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; a + 1u < n; a += nwarps) {
    const unsigned long long ka = skeys[a], knext = skeys[a + 1u];
    const float4 pa = dpos[a];
    const unsigned ix = (unsigned)(ka >> (2 * bits)), iy = (unsigned)(ka >> bits) & top, iz = (unsigned)ka & top;
    const bool high = lane >= 9u;
    const unsigned col = high ? lane - 9u : lane;
    unsigned at = 0u;  // first partner of the column, or the one past its last
    if (lane < 18u) {
      const int cx = (int)ix + (int)(col / 3u) - 1, cy = (int)iy + (int)(col % 3u) - 1;
      if (cx >= 0 && cx <= (int)top && cy >= 0 && cy <= (int)top) {
        const unsigned long long lo = cell_key((unsigned)cx, (unsigned)cy, iz ? iz - 1u : 0u, bits);
        const unsigned long long hi = cell_key((unsigned)cx, (unsigned)cy, iz < top ? iz + 1u : top, bits);
        if (hi >= knext)  // partners come after a in the order, so each pair is tested once
          at = max(lower_bound_u64(skeys, n, high ? hi + 1ull : lo), a + 1u);
      }
    }
    const unsigned end = __shfl_down_sync(SPH_FULL_MASK, at, 9);
    const unsigned len = lane < 9u ? end - at : 0u;
    unsigned upto = len;  // partners in this column and those before it
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const unsigned t = __shfl_up_sync(SPH_FULL_MASK, upto, o);
      if (lane >= (unsigned)o) upto += t;
    }
    const unsigned total = __shfl_sync(SPH_FULL_MASK, upto, 8);
    const unsigned shift = at - (upto - len);  // partner k of the sequence is particle k + its column's shift
    unsigned ra = total ? uf_find(parent, a) : a;
    for (unsigned k0 = 0; k0 < total; k0 += 32u) {
      const unsigned k = k0 + lane;
      unsigned j = 0u;
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        const unsigned before = __shfl_sync(SPH_FULL_MASK, upto - len, c), sh = __shfl_sync(SPH_FULL_MASK, shift, c);
        const unsigned count = __shfl_sync(SPH_FULL_MASK, len, c);
        if (k - before < count) j = k + sh;
      }
      const bool linked = k < total && pair_d2(variant, pa, dpos[j]) <= link2;
      if (!__any_sync(SPH_FULL_MASK, linked)) continue;
      // all that is linked goes under the batch's root of lowest rank: the lanes hook different roots, one of them a's
      const unsigned rb = linked ? uf_find(parent, j) : ra;
      const unsigned low = uf_node(__reduce_min_sync(SPH_FULL_MASK, min(uf_rank(rb), uf_rank(ra))));
      if (linked && rb != ra && rb != low) ok &= uf_unite(parent, rb, low);
      if (lane == 0u && ra != low) ok &= uf_unite(parent, ra, low);
      ra = low;
    }
  }
  if (!ok) atomicOr(&cnt[C_ERR], 1u);
}

__global__ void k_dm_roots(unsigned n, unsigned* __restrict__ parent, unsigned* __restrict__ gcnt,
                           unsigned long long* __restrict__ keys, unsigned* __restrict__ vals,
                           const unsigned* __restrict__ cnt) {
  const unsigned a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n || unsorted(cnt)) return;
  const unsigned r = uf_find(parent, a);
  atomicAdd(&gcnt[r], 1u);
  keys[a] = r;
  vals[a] = a;
}

// ---- 5. clumps ------------------------------------------------------------------------------------------
__global__ void k_dm_clumps(unsigned n, const unsigned long long* __restrict__ skeys,
                            const unsigned* __restrict__ order, const unsigned* __restrict__ gcnt,
                            uint4* __restrict__ clump, unsigned* __restrict__ cnt) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || unsorted(cnt)) return;
  const unsigned r = (unsigned)skeys[i];
  if (i > 0 && (unsigned)skeys[i - 1] == r) return;
  const unsigned s = gcnt[r];
  if (s < 2u) return;
  const unsigned c = atomicAdd(&cnt[C_NCLUMP], 1u);
  clump[c] = make_uint4(i, s, order[i], 0u);  // (the sort is stable: the group's smallest index)
}

// A clump's mass, centre of mass, volume and target mass, then its internal kinetic energy, by `threads` threads of which
// this is the rank-th; sum() adds eight values over them and gives every thread the result (the order is fixed).
template <class Sum>
__device__ __forceinline__ void clump_stats(uint4 cl, unsigned rank, unsigned threads, int variant,
                                            const float4* __restrict__ dpos, const float4* __restrict__ dvel,
                                            const float2* __restrict__ drp, double* __restrict__ o, Sum sum) {
  double a[kDmVals] = {0, 0, 0, 0, 0, 0, 0, 0}, target = 0.0;
#pragma unroll 4
  for (unsigned j = rank; j < cl.y; j += threads) {
    const unsigned t = cl.x + j;
    const float4 p = dpos[t], v = dvel[t];
    const float2 rp = drp[t];
    const double mm = v.w;
    a[0] += mm;
    a[1] += (double)v.x * mm;
    a[2] += (double)v.y * mm;
    a[3] += (double)v.z * mm;
    a[4] += (double)p.x * mm;
    a[5] += (double)p.y * mm;
    a[6] += (double)p.z * mm;
    const double rho = variant == 0 ? (double)rp.x : (double)fmaxf(rp.x, 1.0f);  // gpu_sph.rs:450
    a[7] += mm / rho;
    target += __float_as_uint(rp.y) == 0u ? mm : 0.0;
  }
  sum(a);
  const double cvx = a[1] / a[0], cvy = a[2] / a[0], cvz = a[3] / a[0];
  double b[kDmVals] = {0, target, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (unsigned j = rank; j < cl.y; j += threads) {
    const float4 v = dvel[cl.x + j];
    b[0] += 0.5 * (double)v.w * dsq3((double)v.x - cvx, (double)v.y - cvy, (double)v.z - cvz);
  }
  sum(b);
  if (rank == 0) {
    o[0] = a[0];
    o[1] = a[4] / a[0];
    o[2] = a[5] / a[0];
    o[3] = a[6] / a[0];
    o[4] = a[7];
    o[5] = b[1];
    o[6] = b[0];
  }
}

// Most clumps have a few members and one has most of the disk: a block of 1,024 threads for each of the larger ones, then
// a warp for each of the rest (a block of 256 for every clump took 37 µs for a disk of 22,840 particles, this 24).
constexpr unsigned kWarpClump = 128;
__global__ void __launch_bounds__(1024) k_dm_clump_stats(const unsigned* __restrict__ cnt,
                                                         const uint4* __restrict__ clump, int variant,
                                                         const float4* __restrict__ dpos,
                                                         const float4* __restrict__ dvel,
                                                         const float2* __restrict__ drp, double* __restrict__ cstat) {
  __shared__ double s[32][kDmVals], s_total[kDmVals];
  const unsigned ncl = cnt[C_NCLUMP];
  for (unsigned c = blockIdx.x; c < ncl; c += gridDim.x) {
    const uint4 cl = clump[c];
    if (cl.y <= kWarpClump) continue;
    clump_stats(cl, threadIdx.x, blockDim.x, variant, dpos, dvel, drp, cstat + (size_t)c * 8, [&](double* v) {
      block_sum(v, s);
      if (threadIdx.x == 0)
        for (int k = 0; k < kDmVals; ++k) s_total[k] = v[k];
      __syncthreads();
      for (int k = 0; k < kDmVals; ++k) v[k] = s_total[k];
      __syncthreads();
    });
  }
  const unsigned warps = gridDim.x * (blockDim.x >> 5);
  for (unsigned c = blockIdx.x + gridDim.x * (threadIdx.x >> 5); c < ncl; c += warps) {
    const uint4 cl = clump[c];
    if (cl.y > kWarpClump) continue;
    clump_stats(cl, threadIdx.x & 31u, 32u, variant, dpos, dvel, drp, cstat + (size_t)c * 8, [](double* v) {
      for (int k = 0; k < kDmVals; ++k) v[k] = warp_sum(v[k]);
    });
  }
}

// Self-potential units: the 128 × 128 tile pairs (i >= j) of a clump's lower pair triangle, T(T+1)/2 for
// T = ceil(members / 128). Exclusive 64-bit prefix over the clumps; the total goes to cnt[C_UNITS64..+1].
__device__ __forceinline__ unsigned long long clump_units(unsigned members) {
  const unsigned long long t = (members + kPeRows - 1) / kPeRows;
  return t * (t + 1ull) / 2ull;
}

__global__ void __launch_bounds__(1024) k_dm_unit_scan(unsigned* __restrict__ cnt, const uint4* __restrict__ clump,
                                                       unsigned long long* __restrict__ uoff) {
  __shared__ unsigned long long s_warp[33];
  const unsigned ncl = cnt[C_NCLUMP];
  const unsigned per = (ncl + blockDim.x - 1) / blockDim.x;
  const unsigned c0 = threadIdx.x * per;
  unsigned long long sum = 0;
  for (unsigned k = 0; k < per; ++k)
    if (c0 + k < ncl) sum += clump_units(clump[c0 + k].y);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(SPH_FULL_MASK, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[w] = incl;
  __syncthreads();
  if (w == 0) {
    const unsigned long long x = lane < nw ? s_warp[lane] : 0ull;
    unsigned long long xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(SPH_FULL_MASK, xi, o);
      if (lane >= o) xi += t;
    }
    if (lane < nw) s_warp[lane] = xi - x;
    if (lane == 31) s_warp[32] = xi;
  }
  __syncthreads();
  unsigned long long run = s_warp[w] + incl - sum;
  for (unsigned k = 0; k < per; ++k)
    if (c0 + k < ncl) {
      uoff[c0 + k] = run;
      run += clump_units(clump[c0 + k].y);
    }
  if (threadIdx.x == 0) {
    uoff[ncl] = s_warp[32];
    *reinterpret_cast<unsigned long long*>(cnt + C_UNITS64) = s_warp[32];
  }
}

// One 128 × 128 tile pair of a clump per unit: row tile j (thread t owns member a = 128 j + t) against column
// tile i >= j staged in shared memory; on the diagonal only b > a. upe[unit] = Σ_a m_a Σ_b m_b / r_ab with the
// reference's pair distance (floored, variant 0; softened, variant 1).
__global__ void __launch_bounds__(kPeRows) k_dm_pe(const unsigned* __restrict__ cnt, const uint4* __restrict__ clump,
                                                   const unsigned long long* __restrict__ uoff, int variant,
                                                   double floor_r, double soft2, const float4* __restrict__ dpos,
                                                   const float4* __restrict__ dvel, double* __restrict__ upe) {
  __shared__ float4 sp[kPeRows];
  __shared__ double s_red[kPeRows / 32];
  const unsigned ncl = cnt[C_NCLUMP];
  const unsigned long long units = *reinterpret_cast<const unsigned long long*>(cnt + C_UNITS64);
  for (unsigned long long u = blockIdx.x; u < units; u += gridDim.x) {
    unsigned lo = 0, hi = ncl;  // the clump holding unit u: the last c with uoff[c] <= u
    while (hi - lo > 1) {
      const unsigned mid = (lo + hi) >> 1;
      if (uoff[mid] <= u) lo = mid;
      else hi = mid;
    }
    const uint4 cl = clump[lo];
    const unsigned long long k = u - uoff[lo];
    unsigned long long ti = (unsigned long long)((sqrt(8.0 * (double)k + 1.0) - 1.0) * 0.5);
    while (ti > 0 && ti * (ti + 1ull) / 2ull > k) --ti;            // the estimate is off by at most one
    while ((ti + 1ull) * (ti + 2ull) / 2ull <= k) ++ti;
    const unsigned i = (unsigned)ti, j = (unsigned)(k - ti * (ti + 1ull) / 2ull);
    const unsigned ia = j * kPeRows + threadIdx.x, ib = i * kPeRows + threadIdx.x;
    __syncthreads();  // the previous unit's readers are done with sp
    if (ib < cl.y) {
      float4 q = dpos[cl.x + ib];
      q.w = dvel[cl.x + ib].w;
      sp[threadIdx.x] = q;
    }
    __syncthreads();
    double acc = 0.0;
    if (ia < cl.y) {
      const float4 pa = dpos[cl.x + ia];
      const unsigned nb = min((unsigned)kPeRows, cl.y - i * kPeRows);
      double row = 0.0;
      // 1 / max(r, floor) = min(1/r, 1/floor) and 1 / sqrt(r² + s²) from one f64 reciprocal square root
      // (within an ulp of the divided form): the pair loop is bound by f64 issue, and this halves it
      const double inv_floor = 1.0 / floor_r;
      for (unsigned jj = i == j ? threadIdx.x + 1u : 0u; jj < nb; ++jj) {
        const float4 q = sp[jj];
        const double d2 = pair_d2(variant, pa, q);
        const double ir = variant == 0 ? fmin(rsqrt(d2), inv_floor) : rsqrt(__dadd_rn(d2, soft2));
        row += (double)q.w * ir;
      }
      acc = (double)dvel[cl.x + ia].w * row;
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < kPeRows / 32; ++w) t += s_red[w];
      upe[u] = t;
    }
  }
}

// One block per clump: its self-potential sum Σ_units, in a fixed order, into cstat[c][7].
__global__ void __launch_bounds__(kDmThreads) k_dm_pe_reduce(const unsigned* __restrict__ cnt,
                                                             const unsigned long long* __restrict__ uoff,
                                                             const double* __restrict__ upe,
                                                             double* __restrict__ cstat) {
  __shared__ double s[kDmThreads / 32][kDmVals];
  const unsigned ncl = cnt[C_NCLUMP];
  for (unsigned c = blockIdx.x; c < ncl; c += gridDim.x) {
    double a[kDmVals] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (unsigned long long u = uoff[c] + threadIdx.x; u < uoff[c + 1]; u += kDmThreads) a[0] += upe[u];
    block_sum(a, s);
    if (threadIdx.x == 0) cstat[(size_t)c * 8 + 7] = a[0];
  }
}

// Boundness, the Roche gate and the heaviest bound clump outside it (ties: the smaller root).
__global__ void __launch_bounds__(kDmThreads) k_dm_select(const unsigned* __restrict__ cnt,
                                                          const uint4* __restrict__ clump,
                                                          const double* __restrict__ cstat,
                                                          const double* __restrict__ scal, int variant, double G,
                                                          double roche, double rho_fallback, double* __restrict__ out) {
  __shared__ double s_m[kDmThreads / 32], s_e[kDmThreads / 32];
  __shared__ unsigned s_root[kDmThreads / 32], s_n[kDmThreads / 32], s_bound[kDmThreads / 32], s_cl[kDmThreads / 32];
  const unsigned ncl = cnt[C_NCLUMP];
  const double cx = scal[S_COM], cy = scal[S_COM + 1], cz = scal[S_COM + 2];
  const double r_rem = scal[S_RREM], rho_rem = scal[S_RHOREM];
  double bm = 0.0, be = 0.0;
  unsigned broot = 0xffffffffu, bn = 0, nb = 0, nc = 0;
  for (unsigned c = threadIdx.x; c < ncl; c += blockDim.x) {
    const double* st = cstat + (size_t)c * 8;
    const double M = st[0];
    if (variant == 1 && !(M > 0.0)) continue;  // accretion.rs:121 skips massless groups
    ++nc;
    const double pe = -G * st[7];
    const bool bound = st[6] + pe < 0.0;
    const double rho_c = st[4] > 0.0 ? M / st[4] : rho_fallback;
    const double d_roche = roche * r_rem * cbrt(rho_rem / rho_c);
    const double dx = st[1] - cx, dy = st[2] - cy, dz = st[3] - cz;
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    nb += bound ? 1u : 0u;
    const uint4 cl = clump[c];
    if (bound && dist > d_roche && (M > bm || (M == bm && M > 0.0 && cl.z < broot))) {
      bm = M;
      be = st[5];
      broot = cl.z;
      bn = cl.y;
    }
  }
  // the best of each warp, then of the warps (the larger mass, the smaller root: any order gives the same)
  const auto better = [&](double m, double e, unsigned root, unsigned n) {
    if (m > bm || (m == bm && m > 0.0 && root < broot)) {
      bm = m;
      be = e;
      broot = root;
      bn = n;
    }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    better(__shfl_xor_sync(SPH_FULL_MASK, bm, o), __shfl_xor_sync(SPH_FULL_MASK, be, o),
           __shfl_xor_sync(SPH_FULL_MASK, broot, o), __shfl_xor_sync(SPH_FULL_MASK, bn, o));
    nb += __shfl_xor_sync(SPH_FULL_MASK, nb, o);
    nc += __shfl_xor_sync(SPH_FULL_MASK, nc, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_m[w] = bm;
    s_e[w] = be;
    s_root[w] = broot;
    s_n[w] = bn;
    s_bound[w] = nb;
    s_cl[w] = nc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kDmThreads / 32; ++k) {
      nb += s_bound[k];
      nc += s_cl[k];
      better(s_m[k], s_e[k], s_root[k], s_n[k]);
    }
    out[10] = bm;
    out[11] = bm > 0.0 ? 100.0 * be / bm : 0.0;
    out[12] = (double)bn;
    out[13] = (double)nc;
    out[14] = (double)nb;
  }
}


// ---------------------------------------------------------------------------------------------------------
// Relaxed-body assembly: body_bulk (gpu_sph.rs:260-293) and assemble_from_relaxed_n (gpu_sph.rs:309-339).
// A body's bulk: the centre of mass of its particles, the radius holding 98 % of their mass about it, then twice
// the same over the particles within 1.5 × that radius of that centre (stray particles left by the relaxation
// do not drag the centre). The assembly recentres each source body (prov k) on its bulk centre, places it at
// offset k moving at vel k + spin k × (r − centre), keeps every other field, and drops particles whose prov has
// no placement.
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool bb_take(const State& st, unsigned t, unsigned prov, int clip,
                                        const double* __restrict__ bb) {
  if (st.prov[t] != prov) return false;
  if (!clip) return true;
  const float3 p = pos_f32(st, t);
  const double r = __dsqrt_rn(dsq3(__dsub_rn((double)p.x, bb[BB_C]), __dsub_rn((double)p.y, bb[BB_C + 1]),
                                   __dsub_rn((double)p.z, bb[BB_C + 2])));
  return r <= 1.5 * bb[BB_R];
}

__global__ void __launch_bounds__(kDmThreads) k_bb_count(State st, unsigned n, unsigned chunk, unsigned prov,
                                                         int clip, const double* __restrict__ bb,
                                                         double* __restrict__ part, unsigned* __restrict__ bcnt,
                                                         RadiusSelect* __restrict__ sel) {
  __shared__ double s[kDmThreads / 32][kDmVals];
  double a[kDmVals] = {0, 0, 0, 0, 0, 0, 0, 0};
  const unsigned b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  unsigned cnt = 0;
  float amax = 0.0f;
  for (unsigned base = b0; base < b1; base += kDmThreads) {
    const unsigned t = base + threadIdx.x;
    const bool take = t < b1 && bb_take(st, t, prov, clip, bb);
    if (take) {
      const float3 p = pos_f32(st, t);
      const double mm = st.mass[t];
      a[0] += mm;
      a[1] += (double)p.x * mm;
      a[2] += (double)p.y * mm;
      a[3] += (double)p.z * mm;
      amax = fmaxf(amax, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
    }
    cnt += (unsigned)__syncthreads_count(take);
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) atomicMax(&sel->amax, __float_as_uint(amax));
  block_sum(a, s);
  if (threadIdx.x == 0) {
    for (int k = 0; k < kDmVals; ++k) part[blockIdx.x * kDmVals + k] = a[k];
    bcnt[blockIdx.x] = cnt;
  }
}

// Sums of the selection (centre of mass, zero for a massless one: gpu_sph.rs:266) and the block offsets.
__global__ void __launch_bounds__(1024) k_bb_scan(const double* __restrict__ part, int nb, int first,
                                                  unsigned* __restrict__ bcnt, double* __restrict__ bb,
                                                  unsigned* __restrict__ cnt) {
  __shared__ unsigned s_warp[33];
  __shared__ double t[kDmVals];
  const int w = threadIdx.x >> 5;
  if (w < 4) {
    const double v = warp_sum_column(part, nb, w);
    if ((threadIdx.x & 31) == 0) t[w] = v;
  }
  unsigned total;
  const unsigned c = threadIdx.x < (unsigned)nb ? bcnt[threadIdx.x] : 0u;
  const unsigned o = block_exclusive_scan(c, s_warp, total);
  if (threadIdx.x < (unsigned)nb) bcnt[threadIdx.x] = o;
  if (threadIdx.x == 0) {
    cnt[C_SEL] = total;
    const double mm = t[0];
    for (int k = 0; k < 3; ++k) bb[BB_CN + k] = mm > 0.0 ? t[1 + k] / mm : 0.0;
    bb[BB_MN] = mm;
    if (first) bb[BB_M] = mm;
  }
}

__global__ void __launch_bounds__(kDmThreads) k_bb_write(State st, unsigned n, unsigned chunk, unsigned prov,
                                                         int clip, const double* __restrict__ bb,
                                                         const unsigned* __restrict__ boff, float4* __restrict__ pm) {
  __shared__ unsigned s_warp[33];
  const unsigned b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  unsigned run = boff[blockIdx.x];
  for (unsigned base = b0; base < b1; base += kDmThreads) {
    const unsigned t = base + threadIdx.x;
    const unsigned f = (t < b1 && bb_take(st, t, prov, clip, bb)) ? 1u : 0u;
    unsigned total;
    const unsigned o = run + block_exclusive_scan(f, s_warp, total);
    if (f) {
      const float3 p = pos_f32(st, t);
      pm[o] = make_float4(p.x, p.y, p.z, st.mass[t]);
    }
    run += total;
  }
}

__global__ void k_bb_commit(double* __restrict__ bb) {
  for (int k = 0; k < 3; ++k) bb[BB_C + k] = bb[BB_CN + k];
  bb[BB_R] = bb[BB_RN];
}

// Assembly: count the kept particles per block (original order), then write them transformed.
__global__ void __launch_bounds__(kDmThreads) k_asm_count(const P48x* __restrict__ aos, unsigned n, unsigned chunk,
                                                          unsigned np, unsigned* __restrict__ bcnt) {
  const unsigned b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  unsigned cnt = 0;
  for (unsigned base = b0; base < b1; base += kDmThreads) {
    const unsigned i = base + threadIdx.x;
    cnt += (unsigned)__syncthreads_count(i < b1 && aos[i].prov < np);
  }
  if (threadIdx.x == 0) bcnt[blockIdx.x] = cnt;
}

__global__ void __launch_bounds__(1024) k_u32_offsets(unsigned* __restrict__ bcnt, int nb, unsigned* __restrict__ total_out) {
  __shared__ unsigned s_warp[33];
  unsigned total;
  const unsigned c = threadIdx.x < (unsigned)nb ? bcnt[threadIdx.x] : 0u;
  const unsigned o = block_exclusive_scan(c, s_warp, total);
  if (threadIdx.x < (unsigned)nb) bcnt[threadIdx.x] = o;
  if (threadIdx.x == 0) *total_out = total;
}

__global__ void __launch_bounds__(kDmThreads) k_asm_write(const P48x* __restrict__ aos, unsigned n, unsigned chunk,
                                                          unsigned np, const double* __restrict__ place,
                                                          const unsigned* __restrict__ boff, P48x* __restrict__ dst,
                                                          unsigned* __restrict__ minh_key) {
  __shared__ unsigned s_warp[33];
  const unsigned b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  unsigned run = boff[blockIdx.x];
  unsigned hk = 0xffffffffu;
  for (unsigned base = b0; base < b1; base += kDmThreads) {
    const unsigned i = base + threadIdx.x;
    P48x p;
    unsigned f = 0u;
    if (i < b1) {
      p = aos[i];
      f = p.prov < np ? 1u : 0u;
    }
    unsigned total;
    const unsigned o = run + block_exclusive_scan(f, s_warp, total);
    if (f) {
      const double* pl = place + (size_t)p.prov * 12;  // offset, vel, spin, centre
      const double lx = __dsub_rn((double)p.px, pl[9]), ly = __dsub_rn((double)p.py, pl[10]),
                   lz = __dsub_rn((double)p.pz, pl[11]);
      const double qx = __dadd_rn(lx, pl[0]), qy = __dadd_rn(ly, pl[1]), qz = __dadd_rn(lz, pl[2]);
      const double sx = pl[6], sy = pl[7], sz = pl[8];
      const double vx = __dadd_rn(pl[3], __dsub_rn(__dmul_rn(sy, lz), __dmul_rn(ly, sz)));
      const double vy = __dadd_rn(pl[4], __dsub_rn(__dmul_rn(sz, lx), __dmul_rn(lz, sx)));
      const double vz = __dadd_rn(pl[5], __dsub_rn(__dmul_rn(sx, ly), __dmul_rn(lx, sy)));
      P48x q = p;
      q.px = (float)qx;
      q.py = (float)qy;
      q.pz = (float)qz;
      q.vx = (float)vx;
      q.vy = (float)vy;
      q.vz = (float)vz;
      dst[o] = q;
      hk = min(hk, float_key(p.h));
    }
    run += total;
  }
  hk = warp_min(hk);
  if ((threadIdx.x & 31) == 0 && hk != 0xffffffffu) atomicMin(minh_key, hk);
}

int bits_of(unsigned v) {
  int b = 0;
  while (b < 32 && (v >> b)) ++b;
  return b;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Carve the workspace for m particles from one allocation.
bool work_reserve(DiskWork* w, int m, cudaStream_t s) {
  if (w->cap >= m && w->base) return true;
  if (w->base) cudaFree(w->base);
  w->base = nullptr;
  w->cap = 0;
  const size_t n = (size_t)(m < 1 ? 1 : m), half = n / 2 + 2;
  size_t sz = 0;
  auto take = [&](size_t bytes) {
    const size_t o = sz;
    sz += align256(bytes);
    return o;
  };
  const size_t o_k0 = take(8 * n), o_k1 = take(8 * n), o_v0 = take(4 * n), o_v1 = take(4 * n);
  const size_t o_sort = take(sort_work_bytes((int)n)), o_part = take(8 * kDmBlocks * kDmVals);
  const size_t o_sel = take(sizeof(RadiusSelect)), o_scal = take(8 * S_COUNT), o_cnt = take(4 * C_COUNT);
  const size_t o_bcnt = take(4 * kDmBlocks), o_cat = take(n);
  const size_t o_pm = take(16 * n), o_p0 = take(16 * n), o_p1 = take(16 * n), o_u0 = take(16 * n), o_u1 = take(16 * n);
  const size_t o_r0 = take(8 * n), o_r1 = take(8 * n), o_par = take(4 * n), o_g = take(4 * n);
  const size_t o_cl = take(16 * half), o_uo = take(8 * (half + 1)), o_cs = take(64 * half);
  const size_t o_out = take(8 * 16), o_bb = take(8 * 16), o_pl = take(8 * 12 * kMaxPlacements);
  void* base = nullptr;
  if (cudaMalloc(&base, sz) != cudaSuccess) return false;
  if (cudaMemsetAsync((char*)base + o_sort, 0, sort_work_bytes((int)n), s) != cudaSuccess) {
    cudaFree(base);
    return false;
  }
  char* b = (char*)base;
  w->base = base;
  w->cap = (int)n;
  w->keys[0] = (unsigned long long*)(b + o_k0);
  w->keys[1] = (unsigned long long*)(b + o_k1);
  w->vals[0] = (unsigned*)(b + o_v0);
  w->vals[1] = (unsigned*)(b + o_v1);
  w->sort_work = b + o_sort;
  w->part = (double*)(b + o_part);
  w->sel = (RadiusSelect*)(b + o_sel);
  w->scal = (double*)(b + o_scal);
  w->cnt = (unsigned*)(b + o_cnt);
  w->bcnt = (unsigned*)(b + o_bcnt);
  w->cat = (unsigned char*)(b + o_cat);
  w->pm = (float4*)(b + o_pm);
  w->dpos[0] = (float4*)(b + o_p0);
  w->dpos[1] = (float4*)(b + o_p1);
  w->dvel[0] = (float4*)(b + o_u0);
  w->dvel[1] = (float4*)(b + o_u1);
  w->drp[0] = (float2*)(b + o_r0);
  w->drp[1] = (float2*)(b + o_r1);
  w->parent = (unsigned*)(b + o_par);
  w->gcnt = (unsigned*)(b + o_g);
  w->clump = (uint4*)(b + o_cl);
  w->uoff = (unsigned long long*)(b + o_uo);
  w->cstat = (double*)(b + o_cs);
  w->out = (double*)(b + o_out);
  w->bb = (double*)(b + o_bb);
  w->place = (double*)(b + o_pl);
  return true;
}

// Radius of the point whose running mass, in radius order about `centre`, first reaches frac·(*total)
// (out[0]) and that running mass (out[1]); every pointer is device memory; n >= 1. sel: its counters zero, its amax set.
// Leaves the number of candidates in w->cnt[C_MANY] where it takes launch_radius_digits to tell them apart (0: it does not).
int launch_radius_crossing(DiskWork* w, const float4* pm, unsigned n, const double* centre, const double* total,
                           double frac, double* out, cudaStream_t s) {
  const unsigned chunk = ((n + kDmBlocks - 1) / kDmBlocks + kDmThreads - 1) / kDmThreads * kDmThreads;
  const unsigned nb = (n + chunk - 1) / chunk;
  unsigned long long *keys = w->keys[0], *list = w->keys[1];
  k_dm_select_radius<0><<<nb, kDmThreads, 0, s>>>(pm, n, chunk, centre, total, frac, keys, w->sel, list, w->vals[0], out,
                                                    w->cnt);
  k_dm_select_radius<1><<<nb, kDmThreads, 0, s>>>(pm, n, chunk, centre, total, frac, keys, w->sel, list, w->vals[0], out,
                                                    w->cnt);
  k_dm_select_radius<2><<<nb, kDmThreads, 0, s>>>(pm, n, chunk, centre, total, frac, keys, w->sel, list, w->vals[0], out,
                                                    w->cnt);
  return 3;
}

// The crossing point among the `many` candidates that launch_radius_crossing left (its C_MANY): three digits of the radius,
// unless it is one, and two of the index for up to 2^24 points. By one block, in nine digits of all, a measurement of 1,000,000 points
// at one radius took 284 ms and of a shell of them in f32 61 ms; this way 0.27 and 0.30. The bulk radius of a lattice ball of
// 903,939 points (some 1,000 candidates) took 1,143 µs and takes 401.
int launch_radius_digits(DiskWork* w, const float4* pm, unsigned n, unsigned many, const double* total, double frac,
                         double* out, cudaStream_t s) {
  const unsigned count = many & ~(kSelWhole | kSelEqual), blocks = (count + kDmThreads - 1) / kDmThreads;
  int pass = 0;
  const auto digits = [&](bool on_key, int top) {
    while (top > 0) {
      const int width = top < kSelBits ? top : kSelBits;
      top -= width;
      k_dm_select_digit<<<blocks < kDmBlocks ? blocks : kDmBlocks, kDmThreads, 0, s>>>(
          pm, count, total, frac, w->sel, w->keys[1], w->vals[0], pass++, on_key, top, width, !on_key && top == 0, out);
    }
  };
  digits(true, many & kSelEqual ? 0 : many & kSelWhole ? 64 : 34);
  digits(false, bits_of(n));
  return pass;
}

}  // namespace

void disk_work_free(DiskWork* w) {
  if (!w) return;
  if (w->base) cudaFree(w->base);
  if (w->upe) cudaFree(w->upe);
  delete w;
}

int disk_measure(const Dev& d, unsigned off, unsigned m, const DiskCfg& c, DiskWork*& w, double* out,
                 unsigned long long* launches, const char** err, cudaStream_t s) {
  std::memset(out, 0, 16 * sizeof(double));
  *launches = 0;
  if (m == 0) return 0;
  if (!w) w = new DiskWork();
  if (!work_reserve(w, (int)m, s)) {
    *err = "disk measure: workspace allocation failed";
    return -3;
  }
  const State& st = d.s();
  unsigned long long L = 0;
  const unsigned chunk = ((m + kDmBlocks - 1) / kDmBlocks + kDmThreads - 1) / kDmThreads * kDmThreads;
  const int nb = (int)((m + chunk - 1) / chunk);
  cudaMemsetAsync(w->cnt, 0, 4 * C_COUNT, s);
  cudaMemsetAsync(w->sel, 0, sizeof(RadiusSelect), s);
  k_dm_moments<<<nb, kDmThreads, 0, s>>>(st, off, m, chunk, w->part, w->pm, w->sel);
  k_dm_moments_final<<<1, kDmThreads, 0, s>>>(w->part, nb, w->scal);
  L += 2;
  L += launch_radius_crossing(w, w->pm, m, w->scal + S_COM, w->scal + S_M, c.remnant_frac, w->scal + S_RREM, s);
  unsigned flags[C_COUNT];
  const auto classify = [&] {
    k_dm_classify<<<nb, kDmThreads, 0, s>>>(st, off, m, chunk, c.variant, c.G, w->scal, w->cat, w->part, w->bcnt, w->cnt);
    k_dm_classify_final<<<1, 1024, 0, s>>>(w->part, nb, m, c.variant, c.link_factor, w->bcnt, w->scal, w->cnt, w->out);
    L += 2;
    cudaMemcpyAsync(flags, w->cnt, sizeof(flags), cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
  };
  cudaError_t e = classify();
  if (e == cudaSuccess && flags[C_MANY]) {  // the remnant radius was still open
    L += launch_radius_digits(w, w->pm, m, flags[C_MANY], w->scal + S_M, c.remnant_frac, w->scal + S_RREM, s);
    cudaMemsetAsync(w->cnt, 0, sizeof(flags), s);
    e = classify();
  }
  if (e != cudaSuccess) {
    *err = cudaGetErrorString(e);
    return -2;
  }
  const unsigned nd = flags[C_NDISK];
  const int bits = (int)flags[C_CELLBITS];
  int src = 0;
  if (nd >= 2) {
    k_dm_compact<<<nb, kDmThreads, 0, s>>>(st, d.rho, off, m, chunk, bits, w->cat, w->bcnt, w->scal, w->dpos[0],
                                           w->dvel[0], w->drp[0], w->keys[0], w->vals[0]);
    L += 1;
    L += launch_radix_sort(w->keys, w->vals, (int)nd, 3 * bits, w->sort_work, d.sort_polls, w->cnt + C_ERR, src, s);
    const unsigned gb = (nd + 255) / 256;
    k_dm_gather<<<gb, 256, 0, s>>>(nd, w->vals[src], w->dpos[0], w->dvel[0], w->drp[0], w->dpos[1], w->dvel[1],
                                   w->drp[1], w->parent, w->gcnt, w->cnt);
    const unsigned lb = (nd + 7) / 8;  // one warp per particle, grid-strided over at most 16 blocks per SM
    k_dm_link<<<lb < 2368u ? lb : 2368u, kDmThreads, 0, s>>>(nd, c.variant, bits, w->keys[src], w->dpos[1], w->scal,
                                                             w->parent, w->cnt);
    k_dm_roots<<<gb, 256, 0, s>>>(nd, w->parent, w->gcnt, w->keys[0], w->vals[0], w->cnt);
    L += 3;
    L += launch_radix_sort(w->keys, w->vals, (int)nd, bits_of(nd), w->sort_work, d.sort_polls, w->cnt + C_ERR, src, s);
    k_dm_gather<<<gb, 256, 0, s>>>(nd, w->vals[src], w->dpos[1], w->dvel[1], w->drp[1], w->dpos[0], w->dvel[0],
                                   w->drp[0], nullptr, nullptr, w->cnt);
    k_dm_clumps<<<gb, 256, 0, s>>>(nd, w->keys[src], w->vals[src], w->gcnt, w->clump, w->cnt);
    const unsigned cb = nd / 2 < 1184u ? nd / 2 : 1184u;  // clumps <= nd / 2; blocks stride over them
    const unsigned sb = nd / 2 < 296u ? nd / 2 : 296u;  // two blocks of 1,024 threads per SM
    k_dm_clump_stats<<<sb, 1024, 0, s>>>(w->cnt, w->clump, c.variant, w->dpos[0], w->dvel[0], w->drp[0], w->cstat);
    k_dm_unit_scan<<<1, 1024, 0, s>>>(w->cnt, w->clump, w->uoff);
    L += 4;
    // the self-potential's unit count sizes its partial sums: read it back once
    unsigned long long units = 0;
    cudaMemcpyAsync(&units, w->cnt + C_UNITS64, 8, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      *err = cudaGetErrorString(e);
      return -2;
    }
    if (units > kMaxUnits) {
      *err = "disk measure: a clump's self-potential needs more than 2^28 tile pairs (a clump of ~3M particles)";
      return -5;
    }
    if (units > w->upe_cap) {
      if (w->upe) cudaFree(w->upe);
      w->upe = nullptr;
      w->upe_cap = 0;
      const unsigned long long cap = units + units / 2 + 1024;
      if (cudaMalloc(&w->upe, 8 * cap) != cudaSuccess) {
        *err = "disk measure: self-potential workspace allocation failed";
        return -3;
      }
      w->upe_cap = cap;
    }
    if (units) {
      const unsigned pb = units < 4736ull ? (unsigned)units : 4736u;  // 32 blocks per SM, grid-strided
      k_dm_pe<<<pb, kPeRows, 0, s>>>(w->cnt, w->clump, w->uoff, c.variant, c.pe_floor, c.pe_soft * c.pe_soft,
                                     w->dpos[0], w->dvel[0], w->upe);
      k_dm_pe_reduce<<<cb, kDmThreads, 0, s>>>(w->cnt, w->uoff, w->upe, w->cstat);
      L += 2;
    }
    k_dm_select<<<1, kDmThreads, 0, s>>>(w->cnt, w->clump, w->cstat, w->scal, c.variant, c.G, c.roche,
                                         c.rho_fallback, w->out);
    L += 1;
  }
  cudaMemcpyAsync(out, w->out, 16 * sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(flags, w->cnt, sizeof(flags), cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    *err = cudaGetErrorString(e);
    return -2;
  }
  *launches = L;
  if (flags[C_ERR] & kFlagSortTimeout) {
    *err = "disk measure: a sort's waits ran out";
    return -4;
  }
  if (flags[C_ERR]) {
    *err = "disk measure: a union-find hook gave up after its retry limit";
    return -5;
  }
  return 0;
}


namespace {

int reserve_or_fail(DiskWork*& w, unsigned m, const char** err, cudaStream_t s) {
  if (!w) w = new DiskWork();
  if (!work_reserve(w, (int)(m ? m : 1u), s)) {
    *err = "body measurement: workspace allocation failed";
    return -3;
  }
  return 0;
}

int sync_or_fail(cudaStream_t s, const char** err) {
  cudaError_t e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    *err = cudaGetErrorString(e);
    return -2;
  }
  return 0;
}

// body_bulk of one provenance into w->bb; on return out5 = {cx, cy, cz, mass, radius} (host).
int body_bulk_impl(const Dev& d, unsigned prov, DiskWork* w, double* out5, unsigned long long* L,
                   const char** err, cudaStream_t s) {
  const unsigned n = (unsigned)d.n;
  const State& st = d.s();
  const unsigned chunk = ((n + kDmBlocks - 1) / kDmBlocks + kDmThreads - 1) / kDmThreads * kDmThreads;
  const int nb = (int)((n + chunk - 1) / chunk);
  cudaMemsetAsync(w->bb, 0, 16 * sizeof(double), s);
  for (int round = 0; round < 3; ++round) {
    const int clip = round > 0;
    cudaMemsetAsync(w->sel, 0, sizeof(RadiusSelect), s);
    k_bb_count<<<nb, kDmThreads, 0, s>>>(st, n, chunk, prov, clip, w->bb, w->part, w->bcnt, w->sel);
    k_bb_scan<<<1, 1024, 0, s>>>(w->part, nb, round == 0, w->bcnt, w->bb, w->cnt);
    unsigned sel = 0;
    cudaMemcpyAsync(&sel, w->cnt + C_SEL, 4, cudaMemcpyDeviceToHost, s);
    *L += 2;
    if (int rc = sync_or_fail(s, err)) return rc;
    if (sel == 0) break;  // nothing of this body (round 0), or nothing inside the clip sphere: keep the last
    k_bb_write<<<nb, kDmThreads, 0, s>>>(st, n, chunk, prov, clip, w->bb, w->bcnt, w->pm);
    *L += 1 + launch_radius_crossing(w, w->pm, sel, w->bb + BB_CN, w->bb + BB_MN, 0.98, w->bb + BB_RN, s);
    unsigned many = 0;
    if (sel > (unsigned)kSelBrute) {
      cudaMemcpyAsync(&many, w->cnt + C_MANY, 4, cudaMemcpyDeviceToHost, s);
      if (int rc = sync_or_fail(s, err)) return rc;
    }
    if (many) *L += launch_radius_digits(w, w->pm, sel, many, w->bb + BB_MN, 0.98, w->bb + BB_RN, s);
    k_bb_commit<<<1, 1, 0, s>>>(w->bb);
    *L += 1;
  }
  double bb[16];
  cudaMemcpyAsync(bb, w->bb, sizeof(bb), cudaMemcpyDeviceToHost, s);
  if (int rc = sync_or_fail(s, err)) return rc;
  out5[0] = bb[BB_C];
  out5[1] = bb[BB_C + 1];
  out5[2] = bb[BB_C + 2];
  out5[3] = bb[BB_M];
  out5[4] = bb[BB_R];
  return 0;
}

}  // namespace

int body_bulk(const Dev& d, unsigned prov, DiskWork*& w, double* out5, unsigned long long* launches,
              const char** err, cudaStream_t s) {
  *launches = 0;
  for (int k = 0; k < 5; ++k) out5[k] = 0.0;
  if (d.n == 0) return 0;
  if (int rc = reserve_or_fail(w, (unsigned)d.n, err, s)) return rc;
  return body_bulk_impl(d, prov, w, out5, launches, err, s);
}

int assemble_n(const Dev& d, const double* placements, unsigned np, void* dst, unsigned* n_out, float* min_h,
               DiskWork*& w, unsigned long long* launches, const char** err, cudaStream_t s) {
  *launches = 0;
  *n_out = 0;
  *min_h = __builtin_inff();
  if (np > kMaxPlacements) {
    *err = "assemble: at most 256 placements";
    return -1;
  }
  const unsigned n = (unsigned)d.n;
  if (n == 0 || np == 0) return 0;
  if (int rc = reserve_or_fail(w, n, err, s)) return rc;
  unsigned long long L = 0;
  double place[kMaxPlacements * 12];
  for (unsigned k = 0; k < np; ++k) {
    double bulk[5];
    if (int rc = body_bulk_impl(d, k, w, bulk, &L, err, s)) return rc;
    for (int j = 0; j < 9; ++j) place[k * 12 + j] = placements[k * 9 + j];
    for (int j = 0; j < 3; ++j) place[k * 12 + 9 + j] = bulk[j];
  }
  cudaMemcpyAsync(w->place, place, sizeof(double) * 12 * np, cudaMemcpyHostToDevice, s);
  launch_to_aos(d, s);  // the state in original order, as the 48-byte records the reference assembles from
  const unsigned chunk = ((n + kDmBlocks - 1) / kDmBlocks + kDmThreads - 1) / kDmThreads * kDmThreads;
  const int nb = (int)((n + chunk - 1) / chunk);
  cudaMemsetAsync(w->cnt + C_MINH, 0xff, 4, s);
  k_asm_count<<<nb, kDmThreads, 0, s>>>((const P48x*)d.aos, n, chunk, np, w->bcnt);
  k_u32_offsets<<<1, 1024, 0, s>>>(w->bcnt, nb, w->cnt + C_SEL);
  k_asm_write<<<nb, kDmThreads, 0, s>>>((const P48x*)d.aos, n, chunk, np, w->place, w->bcnt, (P48x*)dst,
                                        w->cnt + C_MINH);
  L += 4;
  unsigned cnts[C_COUNT];
  cudaMemcpyAsync(cnts, w->cnt, sizeof(cnts), cudaMemcpyDeviceToHost, s);
  if (int rc = sync_or_fail(s, err)) return rc;
  *n_out = cnts[C_SEL];
  if (cnts[C_MINH] != 0xffffffffu) {  // the order-preserving key back to the float
    const unsigned k = cnts[C_MINH];
    const unsigned b = (k >> 31) ? (k ^ 0x80000000u) : ~k;
    std::memcpy(min_h, &b, 4);
  }
  *launches = L;
  return 0;
}

}  // namespace sphb
