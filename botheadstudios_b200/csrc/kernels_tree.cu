// LBVH construction on B200: bounding box → 30-bit Morton keys → LSD radix sort (kernels_sort.cu) → state
// permutation → links and moments (bottom-up in one pass; for the per-particle walk Karras nodes, then moments).
//
// Reference: shaders/bh_gravity.wgsl (cs_bbox :68, cs_morton :100, cs_tree :135, cs_com :201) and the CPU
// sort of crates/engine/src/gpu_gravity.rs:336-368. The sort order is (Morton code, original index), made
// exact by a stable radix sort of the codes laid out in original-index order, so the permutation, the leaf
// codes and the Karras topology are bit-identical to the reference's. A batch of impacts prefixes the code with the impact
// (segment) index: every impact is quantised in its own box, sorted into its own contiguous range and
// built into its own subtree, exactly as if it were alone.
#include <cuda/atomic>

#include "sph_kernels.cuh"

namespace sphb {

// ---------------------------------------------------------------------------------------------------
// Segment table set-up: the first particle of every leaf (leaves are K-particle buckets counted from the
// start of their segment; the last bucket of a segment may be partial).
// ---------------------------------------------------------------------------------------------------
// The walk groups are consecutive runs of `per` (= 32/K) leaves of one impact, so a warp holds 32 Morton-consecutive
// particles of one impact (the walk splits a run where consecutive particles are far apart). Against maximal LBVH
// subtrees of <= 32 particles (which left ~22 % of the lanes idle) this is 10 % faster at 1M with the same gravity
// error. Both tables depend on the impacts' sizes alone, so they are written once for each upload (segs[k].pad: the
// impact's first group).
__global__ void k_leaf_start(const Seg* __restrict__ segs, int nseg, int K, int L, int n, int per,
                             unsigned* __restrict__ leaf_start, uint2* __restrict__ groups) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > L) return;
  if (c == L) {
    leaf_start[L] = (unsigned)n;
    return;
  }
  int lo = 0, hi = nseg - 1;  // last segment whose first leaf is <= c
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].loff <= (unsigned)c) lo = mid;
    else hi = mid - 1;
  }
  const unsigned local = (unsigned)c - segs[lo].loff;
  leaf_start[c] = segs[lo].off + local * (unsigned)K;
  if (local % (unsigned)per == 0u)
    groups[segs[lo].pad + local / (unsigned)per] = make_uint2((unsigned)c, min((unsigned)(c + per), segs[lo + 1].loff) - 1u);
}

int launch_segments(const Dev& d, cudaStream_t s) {
  k_leaf_start<<<(d.L + 1 + 255) / 256, 256, 0, s>>>(d.segs, d.nseg, d.K, d.L, d.n, group_leaves(d.K), d.leaf_start,
                                                     d.groups);
  return 1;
}

__global__ void k_segments_single(Seg* segs, int n, int L, float soft2, double dt) {
  write_single_segment(segs, n, L, soft2, dt);
}

int launch_segments_single(const Dev& d, float soft2, double dt, cudaStream_t s) {
  k_segments_single<<<1, 1, 0, s>>>(d.segs, d.n, d.L, soft2, dt);
  return 1 + launch_segments(d, s);
}

// ---------------------------------------------------------------------------------------------------
// Bounding box per segment (cs_bbox): order-preserving u32 keys, reduced per block (seg_bbox_commit).
// ---------------------------------------------------------------------------------------------------
__global__ void k_bbox_reset(Seg* segs, int nseg) {
  const int k = threadIdx.x;
  if (k >= nseg) return;
  for (int a = 0; a < 3; ++a) {
    segs[k].bbox[a] = 0xffffffffu;
    segs[k].bbox[3 + a] = 0u;
  }
}

__global__ void k_bbox(const float4* __restrict__ pos, const unsigned* __restrict__ seg, int n, Seg* segs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  unsigned sg = kNoSeg;
  if (i < n) {
    const float4 p = pos[i];
    lo[0] = hi[0] = float_key(p.x);
    lo[1] = hi[1] = float_key(p.y);
    lo[2] = hi[2] = float_key(p.z);
    sg = seg[i];
  }
  seg_bbox_commit(lo, hi, sg, segs);
}

static int launch_bbox(const Dev& d, cudaStream_t s) {
  k_bbox_reset<<<1, kMaxSegments, 0, s>>>(d.segs, d.nseg);
  k_bbox<<<(d.n + 255) / 256, 256, 0, s>>>(d.s().pos_h, d.s().seg, d.n, d.segs);
  return 2;
}

// ---------------------------------------------------------------------------------------------------
// Permutation of the particle state into the new order; leaf cluster codes (gpu_gravity.rs:366). After a sort whose waits
// ran out the particles stay where they are and the leaves are coded in that order: any order gives a valid tree, with
// larger boxes, so what follows stays in bounds and its results stay good.
// ---------------------------------------------------------------------------------------------------
__global__ void k_permute(int n, int L, const unsigned* __restrict__ order,
                          const unsigned long long* __restrict__ skeys, const unsigned* __restrict__ leaf_start,
                          State in, State out, float4* __restrict__ body,
                          unsigned long long* __restrict__ leaf_codes, const SortEnd* __restrict__ end,
                          const Seg* __restrict__ segs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const bool sorted = !end || end->epoch != end->failed;
  const unsigned o = sorted ? order[t] : (unsigned)t;
  const float4 p = in.pos_h[o];
  const float m = in.mass[o];
  out.pos_h[t] = p;
  out.vel_u[t] = in.vel_u[o];
  out.x[t] = in.x[o];
  out.y[t] = in.y[o];
  out.z[t] = in.z[o];
  out.mass[t] = m;
  out.mat[t] = in.mat[o];
  out.prov[t] = in.prov[o];
  out.id[t] = in.id[o];
  out.seg[t] = in.seg[o];
  body[t] = make_float4(p.x, p.y, p.z, m);
  if (t < L) {
    const unsigned first = leaf_start[t];
    if (sorted) {
      leaf_codes[t] = skeys[first];
    } else {
      const unsigned sg = in.seg[first];
      leaf_codes[t] = (unsigned long long)sg << 30 | ((unsigned)t - segs[sg].loff);
    }
  }
}

// The sort order is (segment, code, original index): the sort is stable and starts out in original-index order
// (kernels_sort.cu). Each particle is quantised in its own segment's box.
int launch_sort_permute(Dev& d, bool need_bbox, cudaStream_t s) {
  const int n = d.n;
  const int box = need_bbox ? launch_bbox(d, s) : 0;
  const State& in = d.st[d.cur];
  const State& out = d.st[d.cur ^ 1];
  int src = 0;
  const SortEnd* end;
  const int sorts = launch_morton_sort(d, src, end, s);
  // vals[src] = old slot of each sorted position; keys[src] = sorted keys
  k_permute<<<(n + 255) / 256, 256, 0, s>>>(n, d.L, d.vals[src], d.keys[src], d.leaf_start, in, out, d.body,
                                            d.leaf_codes, end, d.segs);
  d.cur ^= 1;
  d.sorted = src;
  return box + sorts + 1;
}

// ---------------------------------------------------------------------------------------------------
// Karras 2012 internal nodes over the leaf cluster codes (cs_tree, bh_gravity.wgsl:114-184): the per-particle walk's
// tree, top-down with the reference's split of equal codes. (The group walk's tree is built with its moments below.)
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned code_seg(unsigned long long c) { return (unsigned)(c >> 30); }

// Leaf codes are segment << 30 | Morton code: one impact's leaves share the top bits, so each impact is one
// subtree. Equal codes (always within one impact) are told apart by the leaf index counted from the impact's
// first leaf, so an impact's subtree is the tree it would get alone. With one segment every delta is the
// reference's plus 32 (bh_gravity.wgsl:114-120), which leaves every comparison unchanged.
__device__ __forceinline__ int kdelta(const unsigned long long* __restrict__ codes, const Seg* __restrict__ segs,
                                      int L, int i, int j) {
  if (j < 0 || j >= L) return -1;
  const unsigned long long ci = codes[i], cj = codes[j];
  if (ci == cj) {
    const unsigned base = segs[code_seg(ci)].loff;
    return 64 + __clz(((unsigned)i - base) ^ ((unsigned)j - base));
  }
  return __clzll(ci ^ cj);
}

// Leaves [first, last] are exactly one segment.
__device__ __forceinline__ bool whole_segment(const unsigned long long* __restrict__ codes, int L, int first,
                                              int last) {
  const unsigned sg = code_seg(codes[first]);
  return code_seg(codes[last]) == sg && (first == 0 || code_seg(codes[first - 1]) != sg) &&
         (last == L - 1 || code_seg(codes[last + 1]) != sg);
}

__global__ void k_karras(const unsigned long long* __restrict__ codes, int L, unsigned* __restrict__ left,
                         unsigned* __restrict__ right, unsigned* __restrict__ parent,
                         Seg* __restrict__ segs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L - 1) {
    if (L == 1 && i == 0) segs[0].root = 0u;  // a single leaf is the root
    return;
  }
  const int d = kdelta(codes, segs, L, i, i + 1) > kdelta(codes, segs, L, i, i - 1) ? 1 : -1;
  const int dmin = kdelta(codes, segs, L, i, i - d);
  int lmax = 2;
  while (kdelta(codes, segs, L, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2)
    if (kdelta(codes, segs, L, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int first = min(i, j), last = max(i, j);
  int split = first;
  const unsigned long long fc = codes[first], lc = codes[last];
  if (fc == lc) {
    // the reference's split of a run of equal codes (bh_gravity.wgsl:159-160); it can disagree with the
    // index-extended ranges the children compute for themselves, so such trees may be invalid
    split = (first + last) >> 1;
  } else {
    const int cpfx = __clzll(fc ^ lc);
    int step = last - first;
    for (;;) {
      step = (step + 1) >> 1;
      const int ns = split + step;
      if (ns < last && __clzll(fc ^ codes[ns]) > cpfx) split = ns;
      if (step <= 1) break;
    }
  }
  const unsigned lidx = (split == first) ? (unsigned)(L - 1 + split) : (unsigned)split;
  const unsigned ridx = (split + 1 == last) ? (unsigned)(L - 1 + split + 1) : (unsigned)(split + 1);
  left[i] = lidx;
  right[i] = ridx;
  parent[lidx] = (unsigned)i;
  parent[ridx] = (unsigned)i;
  // segment roots: the node spanning exactly one impact (a leaf when the impact has one leaf)
  if (whole_segment(codes, L, first, last)) segs[code_seg(fc)].root = (unsigned)i;
  if (split == first && whole_segment(codes, L, first, first)) segs[code_seg(fc)].root = lidx;
  if (split + 1 == last && whole_segment(codes, L, last, last)) segs[code_seg(lc)].root = ridx;
}

// ---------------------------------------------------------------------------------------------------
// Bottom-up moments (cs_com, bh_gravity.wgsl:201-241), single pass: each leaf thread sums its bucket, then climbs; the
// first child to arrive at a parent stops, the second merges. Nothing waits: the climb is bounded by the tree height.
// An arrival is an acq_rel device-scope atomic, so the second one sees the sibling's node data (the ordering that
// WGSL could not express and that made the reference fall back to a 33-dispatch sweep).
// Node data: com.xyz/mass (mass-weighted merge, same f32 operations as the reference), AABB with the
// subtree's max smoothing length, the opening radius size/θ + |centre − COM| (size: the largest side for the
// group walk, the diagonal for the reference's per-particle walk) and, optionally, the
// traceless quadrupole about the COM (parallel-axis merge).
// ---------------------------------------------------------------------------------------------------
struct NodeRec {
  float4 com, lo, hi, q0;  // com.xyz and mass; box min and max h; box max and opening radius; Qxx Qyy Qzz Qxy
  float2 q1;               // Qxz Qyz
};

struct NodeArrays {
  float4 *com, *lo, *hi, *q0, *q1;
};

__device__ __forceinline__ float opening_radius(const float lo[3], const float hi[3], float4 com, float theta, int side_mac) {
  const float ex = fsub(hi[0], lo[0]), ey = fsub(hi[1], lo[1]), ez = fsub(hi[2], lo[2]);
  const float size = side_mac ? fmaxf(fmaxf(ex, ey), ez) : fsqrt(dot3_exact(ex, ey, ez));
  const float cx = fsub(fmul(0.5f, fadd(lo[0], hi[0])), com.x), cy = fsub(fmul(0.5f, fadd(lo[1], hi[1])), com.y),
              cz = fsub(fmul(0.5f, fadd(lo[2], hi[2])), com.z);
  return fadd(fdiv(size, theta), fsqrt(dot3_exact(cx, cy, cz)));
}

template <bool QUAD>
__device__ __forceinline__ NodeRec merge_nodes(const NodeRec& l, const NodeRec& r, float theta, int side_mac) {
  NodeRec o;
  const float4 cl = l.com, cr = r.com;
  const float mm = fadd(cl.w, cr.w);
  o.com = make_float4(mm > 0.0f ? fdiv(fadd(fmul(cl.x, cl.w), fmul(cr.x, cr.w)), mm) : 0.0f,
                      mm > 0.0f ? fdiv(fadd(fmul(cl.y, cl.w), fmul(cr.y, cr.w)), mm) : 0.0f,
                      mm > 0.0f ? fdiv(fadd(fmul(cl.z, cl.w), fmul(cr.z, cr.w)), mm) : 0.0f, mm);
  const float bl[3] = {fminf(l.lo.x, r.lo.x), fminf(l.lo.y, r.lo.y), fminf(l.lo.z, r.lo.z)};
  const float bh[3] = {fmaxf(l.hi.x, r.hi.x), fmaxf(l.hi.y, r.hi.y), fmaxf(l.hi.z, r.hi.z)};
  o.lo = make_float4(bl[0], bl[1], bl[2], fmaxf(l.lo.w, r.lo.w));
  o.hi = make_float4(bh[0], bh[1], bh[2], opening_radius(bl, bh, o.com, theta, side_mac));
  o.q0 = make_float4(0, 0, 0, 0);
  o.q1 = make_float2(0, 0);
  if (QUAD) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const NodeRec& c = k ? r : l;
      const float sx = c.com.x - o.com.x, sy = c.com.y - o.com.y, sz = c.com.z - o.com.z, w = c.com.w;
      const float s2 = sx * sx + sy * sy + sz * sz;
      o.q0.x += c.q0.x + w * (3.0f * sx * sx - s2);
      o.q0.y += c.q0.y + w * (3.0f * sy * sy - s2);
      o.q0.z += c.q0.z + w * (3.0f * sz * sz - s2);
      o.q0.w += c.q0.w + w * 3.0f * sx * sy;
      o.q1.x += c.q1.x + w * 3.0f * sx * sz;
      o.q1.y += c.q1.y + w * 3.0f * sy * sz;
    }
  }
  return o;
}

template <bool QUAD>
__device__ __forceinline__ void store_node(const NodeArrays& n, unsigned node, const NodeRec& r) {
  n.com[node] = r.com;
  n.lo[node] = r.lo;
  n.hi[node] = r.hi;
  if (QUAD) {
    n.q0[node] = r.q0;
    n.q1[node] = make_float4(r.q1.x, r.q1.y, 0.0f, 0.0f);
  }
}

// A node another block may have written (past the L1).
template <bool QUAD>
__device__ __forceinline__ NodeRec load_node(const NodeArrays& n, unsigned node) {
  NodeRec r;
  r.com = __ldcg(&n.com[node]);
  r.lo = __ldcg(&n.lo[node]);
  r.hi = __ldcg(&n.hi[node]);
  r.q0 = make_float4(0, 0, 0, 0);
  r.q1 = make_float2(0, 0);
  if (QUAD) {
    r.q0 = __ldcg(&n.q0[node]);
    const float4 b = __ldcg(&n.q1[node]);
    r.q1 = make_float2(b.x, b.y);
  }
  return r;
}

// Traceless quadrupole of the particles [a, b) about `com`.
template <typename Body>
__device__ __forceinline__ void leaf_quadrupole(Body body, unsigned a, unsigned b, float4 com, float4& q0, float2& q1) {
  float qxx = 0, qyy = 0, qzz = 0, qxy = 0, qxz = 0, qyz = 0;
  for (unsigned s = a; s < b; ++s) {
    const float4 p = body(s);
    const float dx = p.x - com.x, dy = p.y - com.y, dz = p.z - com.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    qxx += p.w * (3.0f * dx * dx - r2);
    qyy += p.w * (3.0f * dy * dy - r2);
    qzz += p.w * (3.0f * dz * dz - r2);
    qxy += p.w * 3.0f * dx * dy;
    qxz += p.w * 3.0f * dx * dz;
    qyz += p.w * 3.0f * dy * dz;
  }
  q0 = make_float4(qxx, qyy, qzz, qxy);
  q1 = make_float2(qxz, qyz);
}

// The leaf holding particles [a, b): body(s) is a particle's position and mass, h(s) its smoothing length.
template <bool QUAD, typename Body, typename H>
__device__ __forceinline__ NodeRec leaf_record(Body body, H h, unsigned a, unsigned b, float theta, int side_mac) {
  float m = 0.0f, mx = 0.0f, my = 0.0f, mz = 0.0f, hmax = 0.0f;
  float lo[3] = {1.0e30f, 1.0e30f, 1.0e30f}, hi[3] = {-1.0e30f, -1.0e30f, -1.0e30f};
  for (unsigned s = a; s < b; ++s) {
    const float4 p = body(s);
    m = fadd(m, p.w);
    mx = fadd(mx, fmul(p.x, p.w));
    my = fadd(my, fmul(p.y, p.w));
    mz = fadd(mz, fmul(p.z, p.w));
    lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
    hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
    hmax = fmaxf(hmax, h(s));
  }
  NodeRec r;
  r.com = make_float4(m > 0.0f ? fdiv(mx, m) : 0.0f, m > 0.0f ? fdiv(my, m) : 0.0f, m > 0.0f ? fdiv(mz, m) : 0.0f, m);
  r.lo = make_float4(lo[0], lo[1], lo[2], hmax);
  r.hi = make_float4(hi[0], hi[1], hi[2], opening_radius(lo, hi, r.com, theta, side_mac));
  r.q0 = make_float4(0, 0, 0, 0);
  r.q1 = make_float2(0, 0);
  if (QUAD) leaf_quadrupole(body, a, b, r.com, r.q0, r.q1);
  return r;
}

// The per-particle walk's moments over the links of k_karras.
template <bool QUAD>
__global__ void k_leaf_climb(const float4* __restrict__ body, const float4* __restrict__ pos_h,
                             const unsigned* __restrict__ leaf_start, int L, const unsigned* __restrict__ left,
                             const unsigned* __restrict__ right, const unsigned* __restrict__ parent,
                             unsigned* __restrict__ counters, NodeArrays nodes, float theta) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L) return;
  const int li = L - 1 + c;
  store_node<QUAD>(nodes, (unsigned)li,
                   leaf_record<QUAD>([&](unsigned s) { return body[s]; }, [&](unsigned s) { return pos_h[s].w; },
                                     leaf_start[c], leaf_start[c + 1], theta, 0));
  unsigned node = parent[li];
  while (node != SPH_NO_PARENT) {
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> cnt(counters[node]);
    const unsigned arrived = cnt.fetch_add(1u, cuda::memory_order_acq_rel);
    if (arrived == 0u) return;  // the sibling subtree finishes this node
    store_node<QUAD>(nodes, node, merge_nodes<QUAD>(load_node<QUAD>(nodes, left[node]), load_node<QUAD>(nodes, right[node]),
                                                    theta, 0));
    node = parent[node];
  }
}

// ---------------------------------------------------------------------------------------------------
// The group walk's tree, links and moments in one bottom-up pass (Apetrei 2014, "Fast and Simple Agglomerative LBVH
// Construction"): a finished node [l, r] is a left child when its leaves share more key bits with r + 1 than with
// l − 1, so it meets its sibling at the slot of the split, r or l − 1, and the second to arrive merges. Keys are the
// leaf codes extended by the leaf's index (kdelta), so the tree is the one of Karras 2012 with index-extended keys,
// in his numbering: a left child has the index of its last leaf, a right child of its first, the root is 0.
// The slot carries what the sibling needs of this side: its other end and the key bits shared across that end; a
// climb reads no codes and no links.
//
// Bound by the chain of levels: meeting in memory costs ~1.2-2 µs a level, in shared memory ~0.3 µs. So a block takes a
// run of about 128 leaves and merges in shared memory every node that lies in the run. The run ends where, of the 64
// places around the 128th leaf, the fewest key bits are shared, so a node that crosses an end holds 64 leaves at
// least: log2(L/64) levels or so go through memory, where runs of exactly 128 leaves would send half of all paths
// there near the bottom. A block also stages its particles in shared memory. Links and moments as two passes
// (top-down links, every level of the moments in memory, 7 launches with their resets) took 66 µs at 10,240 particles,
// 70 at 65,536, 78 at 262,144, 103 at 1,048,576 and 195 at 4,194,304; this takes 28, 31, 34, 56 and 126.
// ---------------------------------------------------------------------------------------------------
constexpr int TB_RUN = 128, TB_SLACK = 32;
constexpr int TB_THREADS = TB_RUN + 2 * TB_SLACK;  // the longest run

struct TreeSmem {
  NodeRec rec[2 * TB_THREADS];           // the block's leaves, then its nodes
  unsigned long long slot[TB_THREADS];   // the meeting places inside the run
};

// A staged particle's place: one in 17 records is skipped, so that 8 leaves' particles lie in different banks.
__device__ __forceinline__ unsigned tb_at(unsigned i) { return i + (i >> 4); }

// What the first child to arrive leaves for its sibling: its far end, and the key bits (+1) shared across that end.
__device__ __forceinline__ unsigned long long tb_word(unsigned end, int delta) {
  return 1ull << 63 | (unsigned long long)(unsigned)(delta + 1) << 32 | end;
}

// The start of run b (of nb), and the key bits shared across it. Called by whole warps.
__device__ __forceinline__ void tb_edge(const unsigned long long* __restrict__ codes, const Seg* __restrict__ segs, int L,
                                        int nb, int b, int& at, int& delta) {
  if (b == 0 || b == nb) {
    at = b == 0 ? 0 : L;
    delta = -1;
    return;
  }
  unsigned best = 0xffffffffu;  // shared bits << 8 | place: the fewest bits, then the first place
#pragma unroll
  for (int k = (int)(threadIdx.x & 31); k < 2 * TB_SLACK; k += 32) {
    const int c = b * TB_RUN - TB_SLACK + k;
    if (c < L) best = min(best, (unsigned)kdelta(codes, segs, L, c - 1, c) << 8 | (unsigned)k);
  }
  best = warp_min(best);
  at = b * TB_RUN - TB_SLACK + (int)(best & 255u);
  delta = (int)(best >> 8);
}

template <bool QUAD>
__global__ void __launch_bounds__(TB_THREADS) k_tree_build(
    const float4* __restrict__ body, const float4* __restrict__ pos_h, const unsigned* __restrict__ leaf_start, int L,
    const unsigned long long* __restrict__ codes, Seg* __restrict__ segs, unsigned* __restrict__ left,
    unsigned* __restrict__ right, unsigned* __restrict__ parent, unsigned long long* __restrict__ slots,
    NodeArrays nodes, float theta, int half, float4* __restrict__ hcom, float4* __restrict__ hq0,
    float2* __restrict__ hq1, float2* __restrict__ hrc, int staged) {
  extern __shared__ __align__(16) unsigned char tb_raw[];
  __shared__ int s_at[2], s_delta[2];
  const int w = threadIdx.x >> 5;
  if (w < 2) {
    int at, delta;
    tb_edge(codes, segs, L, (int)gridDim.x, (int)blockIdx.x + w, at, delta);
    if ((threadIdx.x & 31) == 0) {
      s_at[w] = at;
      s_delta[w] = delta;
    }
  }
  __syncthreads();
  const int c0 = s_at[0], c1 = s_at[1], c = c0 + (int)threadIdx.x;
  const int edge = max(s_delta[0], s_delta[1]);  // nodes that share more key bits than this lie in the run
  // the run's particles (first use of the shared memory), `staged` records and smoothing lengths
  float4* sb = reinterpret_cast<float4*>(tb_raw);
  float* sh = reinterpret_cast<float*>(sb + staged);
  const unsigned p0 = leaf_start[c0], p1 = leaf_start[c1];
  for (unsigned i = threadIdx.x; i < p1 - p0; i += TB_THREADS) {
    sb[tb_at(i)] = body[p0 + i];
    sh[tb_at(i)] = pos_h[p0 + i].w;
  }
  const bool have = c < c1;
  int dl = -1, dr = -1;
  if (have) {
    dl = kdelta(codes, segs, L, c, c - 1);
    dr = kdelta(codes, segs, L, c, c + 1);
  }
  __syncthreads();
  NodeRec me;
  if (have) {
    const unsigned s0 = leaf_start[c] - p0, s1 = leaf_start[c + 1] - p0;
    auto at = [&](unsigned s) { return sb[tb_at(s)]; };
    me = leaf_record<QUAD>(at, [&](unsigned s) { return sh[tb_at(s)]; }, s0, s1, theta, 1);
    if (half > 0) {
      // the leaf's two halves as multipoles of their own (the far field of the group walk): COM, mass, the
      // traceless quadrupole about that COM, and the opening radius largest side/θ + |centre − COM|
      float rcs[2] = {0.0f, 0.0f};
      for (int b = 0; b < 2; ++b) {
        const unsigned a0 = s0 + b * half, a1 = min(s0 + (b + 1) * half, s1);
        float hm = 0.0f, hx = 0.0f, hy = 0.0f, hz = 0.0f;
        float l3[3] = {1.0e30f, 1.0e30f, 1.0e30f}, u3[3] = {-1.0e30f, -1.0e30f, -1.0e30f};
        for (unsigned s = a0; s < a1; ++s) {
          const float4 q = at(s);
          hm += q.w;
          hx = fmaf(q.x, q.w, hx);
          hy = fmaf(q.y, q.w, hy);
          hz = fmaf(q.z, q.w, hz);
          l3[0] = fminf(l3[0], q.x); l3[1] = fminf(l3[1], q.y); l3[2] = fminf(l3[2], q.z);
          u3[0] = fmaxf(u3[0], q.x); u3[1] = fmaxf(u3[1], q.y); u3[2] = fmaxf(u3[2], q.z);
        }
        const float inv = hm > 0.0f ? 1.0f / hm : 0.0f;
        const float4 hc = make_float4(hx * inv, hy * inv, hz * inv, hm);
        if (a1 > a0) {
          const float ex = u3[0] - l3[0], ey = u3[1] - l3[1], ez = u3[2] - l3[2];
          const float size = fmaxf(fmaxf(ex, ey), ez);
          const float cx = 0.5f * (l3[0] + u3[0]) - hc.x, cy = 0.5f * (l3[1] + u3[1]) - hc.y,
                      cz = 0.5f * (l3[2] + u3[2]) - hc.z;
          rcs[b] = size / theta + sqrtf(cx * cx + cy * cy + cz * cz);
        }
        float4 q0 = make_float4(0, 0, 0, 0);
        float2 q1 = make_float2(0, 0);
        if (QUAD) leaf_quadrupole(at, a0, a1, hc, q0, q1);
        hcom[2 * c + b] = hc;
        hq0[2 * c + b] = q0;
        hq1[2 * c + b] = q1;
      }
      hrc[c] = make_float2(rcs[0], rcs[1]);
    }
  }
  __syncthreads();  // the particles are done with: the run's nodes take their place
  TreeSmem& S = *reinterpret_cast<TreeSmem*>(tb_raw);
  S.slot[threadIdx.x] = 0ull;
  __syncthreads();
  if (!have) return;
  const unsigned leaf0 = (unsigned)(L - 1);
  unsigned l = (unsigned)c, r = (unsigned)c, lchild = 0u, rchild = 0u;
  int dn = 64;  // key bits shared by all of the node's leaves
  for (;;) {
    const bool root = l == 0u && r == leaf0, is_left = dr > dl;
    const unsigned node = l == r ? leaf0 + l : (root || !is_left) ? l : r;
    store_node<QUAD>(nodes, node, me);
    if (l != r) {
      left[node] = lchild;
      right[node] = rchild;
      parent[lchild] = node;
      parent[rchild] = node;
    }
    // the node of exactly one impact: keys of different impacts share at most 33 of their 64 bits
    if (dl <= 33 && dr <= 33 && dn > 33) segs[code_seg(codes[l])].root = node;
    if (root) {
      parent[node] = SPH_NO_PARENT;
      return;
    }
    const unsigned split = is_left ? r : l - 1u;
    const unsigned long long word = is_left ? tb_word(l, dl) : tb_word(r, dr);
    dn = is_left ? dr : dl;
    const bool inside = dn > edge;
    unsigned long long got;
    if (inside) {
      S.rec[(l == r ? 0u : (unsigned)TB_THREADS) + (l == r ? l : node) - (unsigned)c0] = me;
      __threadfence_block();
      got = atomicExch(&S.slot[split - (unsigned)c0], word);
      if (!got) return;  // the sibling finishes the parent
      __threadfence_block();
    } else {
      // a sibling that is there already is taken without publishing this side (its record is in registers)
      cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> slot(slots[split]);
      got = slot.load(cuda::memory_order_acquire);
      if (!got) got = slot.exchange(word, cuda::memory_order_acq_rel);
      if (!got) return;
      slots[split] = 0ull;  // ready for the next build
    }
    const unsigned end = (unsigned)got;
    const int far = (int)((unsigned)(got >> 32) & 0x7fffffffu) - 1;
    const unsigned first = is_left ? split + 1u : split;  // the sibling's leaf at the split
    const bool leaf = end == first;
    const unsigned sib = leaf ? leaf0 + first : first;
    const NodeRec o = inside ? S.rec[(leaf ? 0u : (unsigned)TB_THREADS) + first - (unsigned)c0] : load_node<QUAD>(nodes, sib);
    if (is_left) {
      me = merge_nodes<QUAD>(me, o, theta, 1);
      lchild = node;
      rchild = sib;
      r = end;
      dr = far;
    } else {
      me = merge_nodes<QUAD>(o, me, theta, 1);
      lchild = sib;
      rchild = node;
      l = end;
      dl = far;
    }
  }
}

template <bool QUAD>
static void tree_build(const Dev& d, const NodeArrays& nodes, float theta, int half, cudaStream_t s) {
  const int most = TB_THREADS * d.K, staged = most + (most >> 4) + 1;
  const size_t part = (size_t)staged * (sizeof(float4) + sizeof(float));
  const size_t smem = part > sizeof(TreeSmem) ? part : sizeof(TreeSmem);
  static SmemLimit attr;
  smem_limit(k_tree_build<QUAD>, (TB_THREADS * 34 + 1) * 20, attr);  // leaves of 32
  k_tree_build<QUAD><<<(d.L + TB_RUN - 1) / TB_RUN, TB_THREADS, smem, s>>>(
      d.body, d.s().pos_h, d.leaf_start, d.L, d.leaf_codes, d.segs, d.left, d.right, d.parent, d.slots, nodes, theta, half,
      d.hcom, d.hq0, d.hq1, d.hrc, staged);
}

int launch_tree(const Dev& d, const Cfg& c, float theta, cudaStream_t s) {
  const int L = d.L;
  const NodeArrays nodes{d.ncom, d.nbmin, d.nbmax, d.nq0, d.nq1};
  if (c.mac == 0) {
    const int half = half_leaf(d, c);
    if (c.quad) tree_build<true>(d, nodes, theta, half, s);
    else tree_build<false>(d, nodes, theta, half, s);
    return 1;
  }
  // the reference's split of equal codes can leave nodes without a parent: they read as such
  cudaMemsetAsync(d.parent, 0xff, sizeof(unsigned) * (2 * (size_t)L - 1), s);
  if (L > 1) cudaMemsetAsync(d.counters, 0, sizeof(unsigned) * (L - 1), s);
  k_karras<<<(L + 255) / 256, 256, 0, s>>>(d.leaf_codes, L, d.left, d.right, d.parent, d.segs);
  const State& st = d.s();
  if (c.quad)
    k_leaf_climb<true><<<(L + 127) / 128, 128, 0, s>>>(d.body, st.pos_h, d.leaf_start, L, d.left, d.right, d.parent,
                                                       d.counters, nodes, theta);
  else
    k_leaf_climb<false><<<(L + 127) / 128, 128, 0, s>>>(d.body, st.pos_h, d.leaf_start, L, d.left, d.right, d.parent,
                                                        d.counters, nodes, theta);
  return 2;
}

// Far leaves are split in the group walk when a half holds at least 8 particles: one quadrupole evaluation
// (~50 instructions) then replaces 8 pairwise ones (~14 each); halves of 4 would not pay.
int half_leaf(const Dev& d, const Cfg& c) {
  return (c.mac == 0 && c.gravity == 0 && d.K >= 16 && d.hcom) ? d.K / 2 : 0;
}

}  // namespace sphb
