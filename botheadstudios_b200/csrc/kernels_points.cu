// Barnes-Hut gravity of a point set (no smoothing lengths) over the LBVH: every point walks with its own
// opening decisions, a block walks for 32 of them.
//
// The group walk decides for the bounding box of a group it keeps together; points carry no smoothing length that
// says which of them belong together, so here the "group" is a single point: a node is accepted when
// sqrt(|com − p|² + ε²) >= side/θ + |centre − com| and its box does not contain the point, a leaf that is not
// accepted is summed pairwise, and (leaves of >= 16) each half of one is accepted or summed by its own moments.
// A point's accelerations depend on no other point's walk.
//
// A block owns 32 Morton-consecutive points: lane l of each of its 8 warps holds point l. The points share one
// stack of (node, lanes that need it) in shared memory; a round pops up to 128 nodes, stages their records with
// one load per thread, and each warp takes every 8th of them: all lanes evaluate the opening test for their own
// point, the lanes that accept add the multipole, and the children go back on the stack with the lanes that
// opened the node. Neighbouring points open nearly the same nodes, so a node costs one staging and one test for
// 32 points, where a walk for each point alone (a warp whose 32 points are 32 groups of one) repeats both 32 times:
// 16,001 points in 16-point leaves with quadrupoles: a call took 3,394 µs that way (3,305 µs of them in the walk) and
// takes 265 µs (202 in the walk). Bound by latency below about 20,000 points (rounds of dependent loads, hence 8 warps for 32 points)
// and by issue above.
#include "sph_kernels.cuh"

namespace sphb {

constexpr int PT_WARPS = 8;
constexpr int PT_ROUND = 128;   // nodes popped in one round
// (node, lanes) entries. A round leaves at most as many entries on the stack as it popped for each level below, so
// the 2,048 that full rounds may fill last for 16 levels of trees opened throughout; above that a round pops 32 and
// the rest lasts for 64 more.
constexpr int PT_STACK = 4096;

struct PointSmem {
  uint2 stack[PT_STACK];
  float4 com[PT_ROUND], bmin[PT_ROUND], bmax[PT_ROUND], q0[PT_ROUND];
  float2 q1[PT_ROUND];
  uint2 link[PT_ROUND];            // children of an internal node, source range of a leaf
  uint2 node[PT_ROUND];            // the popped entries
  unsigned open[PT_ROUND];         // lanes that opened the node
  float4 src[PT_WARPS][32];        // a warp's leaf sources in pairs: (x0 x1 y0 y1)(z0 z1 m0 m1)
  float4 sum[PT_WARPS][32];
  int sp;
};

struct PointAcc {
  float x = 0.f, y = 0.f, z = 0.f, phi = 0.f;
};

// The multipole (com, M), Q about its com, softened, at offset d = com − p with r2 = |d|² + ε²:
// a = d (G M/R³ + 5/2 eᵀQe/R⁵) − Q e/R⁴, φ = −G M/R − ½ eᵀQe/R³, e = d/R (Q·e stays in f32 range in SI units).
template <bool QUAD>
__device__ __forceinline__ void point_multipole(float dx, float dy, float dz, float r2, float gm, float G, float4 q0,
                                                float2 q1, PointAcc& a) {
  const float ri = rsqrt_ftz(r2), ri2 = ri * ri;
  const float mr = gm * ri;
  float c = mr * ri2;
  if (QUAD) {
    const float ex = dx * ri, ey = dy * ri, ez = dz * ri;
    const float qx = G * fmaf(q0.x, ex, fmaf(q0.w, ey, q1.x * ez));
    const float qy = G * fmaf(q0.w, ex, fmaf(q0.y, ey, q1.y * ez));
    const float qz = G * fmaf(q1.x, ex, fmaf(q1.y, ey, q0.z * ez));
    const float eqe = fmaf(ex, qx, fmaf(ey, qy, ez * qz));
    const float ri4 = ri2 * ri2;
    c = fmaf(2.5f * eqe, ri4 * ri, c);
    a.x = fmaf(-ri4, qx, a.x);
    a.y = fmaf(-ri4, qy, a.y);
    a.z = fmaf(-ri4, qz, a.z);
    a.phi = fmaf(-0.5f * eqe, ri2 * ri, a.phi);
  }
  a.x = fmaf(c, dx, a.x);
  a.y = fmaf(c, dy, a.y);
  a.z = fmaf(c, dz, a.z);
  a.phi -= mr;
}

template <bool QUAD>
__global__ void __launch_bounds__(PT_WARPS * 32) k_point_walk(
    const float4* __restrict__ body, int n, int L, const unsigned* __restrict__ leaf_start,
    const Seg* __restrict__ segs, const unsigned* __restrict__ left, const unsigned* __restrict__ right,
    const float4* __restrict__ ncom, const float4* __restrict__ nbmin, const float4* __restrict__ nbmax,
    const float4* __restrict__ nq0, const float4* __restrict__ nq1, DevParams* P, float4* __restrict__ out,
    int stack_cap, int half, const float4* __restrict__ hcom, const float4* __restrict__ hq0,
    const float2* __restrict__ hq1, const float2* __restrict__ hrc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PointSmem& S = *reinterpret_cast<PointSmem*>(smem_raw);
  const int tid = threadIdx.x, w = tid >> 5;
  const unsigned lane = tid & 31u;
  const int t = blockIdx.x * 32 + (int)lane;
  const bool valid = t < n;
  const float4 p = body[valid ? t : n - 1];
  const float G = P->G, soft2 = segs[0].soft2;
  const unsigned leaf0 = (unsigned)(L - 1);
  const unsigned all = __ballot_sync(SPH_FULL_MASK, valid);
  PointAcc a;
  if (tid == 0) {
    S.stack[0] = make_uint2(segs[0].root, all);
    S.sp = 1;
  }
  __syncthreads();
  int sp = 1;
  while (sp > 0) {
    const int take = min(sp, sp > PT_STACK / 2 ? 32 : PT_ROUND), base = sp - take;
    // thread i stages the opening record of node i, thread 128 + i its multipole and links
    const int i = tid & (PT_ROUND - 1);
    if (i < take) {
      const uint2 e = S.stack[base + i];
      if (tid < PT_ROUND) {
        S.node[i] = e;
        S.com[i] = ncom[e.x];
        S.bmin[i] = nbmin[e.x];
        S.bmax[i] = nbmax[e.x];
      } else {
        if (QUAD) {
          S.q0[i] = nq0[e.x];
          const float4 b = nq1[e.x];
          S.q1[i] = make_float2(b.x, b.y);
        }
        S.link[i] = e.x >= leaf0 ? make_uint2(leaf_start[e.x - leaf0], leaf_start[e.x - leaf0 + 1])
                                 : make_uint2(left[e.x], right[e.x]);
        S.open[i] = 0u;
      }
    }
    __syncthreads();
    for (int k = w; k < take; k += PT_WARPS) {
      const uint2 e = S.node[k];
      const bool in = (e.y >> lane) & 1u;
      const float4 c = S.com[k], lo = S.bmin[k], hi = S.bmax[k];
      const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, soft2)));
      const float ro = hi.w * 1.00001f;
      const bool near = lo.x <= p.x && hi.x >= p.x && lo.y <= p.y && hi.y >= p.y && lo.z <= p.z && hi.z >= p.z;
      const bool accept = in && !near && dx * dx + dy * dy + dz * dz + soft2 >= ro * ro;
      if (accept) point_multipole<QUAD>(dx, dy, dz, r2, G * c.w, G, QUAD ? S.q0[k] : c, QUAD ? S.q1[k] : make_float2(0.f, 0.f), a);
      const unsigned more = __ballot_sync(SPH_FULL_MASK, in && !accept);
      if (!more) continue;
      if (e.x < leaf0) {
        if (lane == 0) S.open[k] = more;
        continue;
      }
      // a leaf some lanes cannot accept: its sources, staged in pairs, each half by its own moments if it has any
      const unsigned s0 = S.link[k].x, s1 = S.link[k].y, cl = e.x - leaf0;
      float4 b = make_float4(3.0e18f, 3.0e18f, 3.0e18f, 0.0f);  // padding: massless and far away
      if (s0 + lane < s1) b = body[s0 + lane];
      float* f = reinterpret_cast<float*>(&S.src[w][0]) + 8 * (lane >> 1) + (lane & 1u);
      f[0] = b.x;
      f[2] = b.y;
      f[4] = b.z;
      f[6] = G * b.w;
      __syncwarp();
      const bool need = in && !accept;
      const unsigned step = half > 0 ? (unsigned)half : 32u;
      for (unsigned h = 0, a0 = 0; s0 + a0 < s1; ++h, a0 += step) {
        bool pairs = need;
        if (half > 0) {
          const float4 hc = hcom[2u * cl + h];
          const float2 rc = hrc[cl];
          const float ux = hc.x - p.x, uy = hc.y - p.y, uz = hc.z - p.z;
          const float rh = (h ? rc.y : rc.x) * 1.00001f;
          const bool far = need && !near && ux * ux + uy * uy + uz * uz + soft2 >= rh * rh;
          if (far)
            point_multipole<QUAD>(ux, uy, uz, fmaf(ux, ux, fmaf(uy, uy, fmaf(uz, uz, soft2))), G * hc.w, G,
                                  hq0[2u * cl + h], hq1[2u * cl + h], a);
          pairs = need && !far;
        }
        if (pairs) {
          const int k1 = (int)((min(a0 + step, s1 - s0) + 1u) >> 1);
          const int self = t - (int)s0;  // this point's place among the leaf's sources, if it is one of them
          float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx, sp2 = sx;
          const float2 npx = make_float2(-p.x, -p.x), npy = make_float2(-p.y, -p.y), npz = make_float2(-p.z, -p.z),
                       e2 = make_float2(soft2, soft2);
#pragma unroll 4
          for (int q = (int)(a0 >> 1); q < k1; ++q) {
            const float4 xy = S.src[w][2 * q], zm = S.src[w][2 * q + 1];
            const float2 ex = __fadd2_rn(make_float2(xy.x, xy.y), npx);
            const float2 ey = __fadd2_rn(make_float2(xy.z, xy.w), npy);
            const float2 ez = __fadd2_rn(make_float2(zm.x, zm.y), npz);
            const float2 d2 = __ffma2_rn(ex, ex, __ffma2_rn(ey, ey, __ffma2_rn(ez, ez, e2)));
            const bool s_a = self == 2 * q, s_b = self == 2 * q + 1;  // the point itself adds nothing
            const float2 ri = make_float2(rsqrt_ftz(s_a ? 1.0f : d2.x), rsqrt_ftz(s_b ? 1.0f : d2.y));
            const float2 gm = __fmul2_rn(make_float2(s_a ? 0.0f : zm.z, s_b ? 0.0f : zm.w), ri);
            const float2 g = __fmul2_rn(__fmul2_rn(gm, ri), ri);
            sx = __ffma2_rn(g, ex, sx);
            sy = __ffma2_rn(g, ey, sy);
            sz = __ffma2_rn(g, ez, sz);
            sp2 = __fadd2_rn(sp2, gm);
          }
          a.x += sx.x + sx.y;
          a.y += sy.x + sy.y;
          a.z += sz.x + sz.y;
          a.phi -= sp2.x + sp2.y;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    // the opened nodes' children, in the order of the round, on top of what is left of the stack
    if (w == 0) {
      int add = 0;
      unsigned om[PT_ROUND / 32];
      int at[PT_ROUND / 32];
#pragma unroll
      for (int r = 0; r < PT_ROUND / 32; ++r) {
        const int k = 32 * r + (int)lane;
        om[r] = k < take ? S.open[k] : 0u;
        const unsigned bal = __ballot_sync(SPH_FULL_MASK, om[r] != 0u);
        at[r] = base + 2 * (add + __popc(bal & ((1u << lane) - 1u)));
        add += __popc(bal);
      }
      if (base + 2 * add <= stack_cap) {
#pragma unroll
        for (int r = 0; r < PT_ROUND / 32; ++r)
          if (om[r]) {
            const uint2 ch = S.link[32 * r + lane];
            S.stack[at[r]] = make_uint2(ch.x, om[r]);
            S.stack[at[r] + 1] = make_uint2(ch.y, om[r]);
          }
        if (lane == 0) S.sp = base + 2 * add;
      } else if (lane == 0) {  // the children that do not fit are skipped and the flag says so
        atomicOr(&P->flags, kFlagStackOverflow);
        S.sp = base;
      }
    }
    __syncthreads();
    sp = S.sp;
  }
  S.sum[w][lane] = make_float4(a.x, a.y, a.z, a.phi);
  __syncthreads();
  if (w == 0 && valid) {
    float4 r = S.sum[0][lane];
#pragma unroll
    for (int k = 1; k < PT_WARPS; ++k) {
      const float4 v = S.sum[k][lane];
      r.x += v.x;
      r.y += v.y;
      r.z += v.z;
      r.w += v.w;
    }
    out[t] = r;
  }
}

template <bool QUAD>
static void point_walk(const Dev& d, const Cfg& c, cudaStream_t s) {
  static SmemLimit attr;
  smem_limit(k_point_walk<QUAD>, (int)sizeof(PointSmem), attr);
  k_point_walk<QUAD><<<(d.n + 31) / 32, PT_WARPS * 32, sizeof(PointSmem), s>>>(
      d.body, d.n, d.L, d.leaf_start, d.segs, d.left, d.right, d.ncom, d.nbmin, d.nbmax, d.nq0, d.nq1, d.P, d.grav,
      c.walk_stack > 0 && c.walk_stack < PT_STACK ? c.walk_stack : PT_STACK, half_leaf(d, c), d.hcom, d.hq0, d.hq1,
      d.hrc);
}

// Gravity only, for point sets without SPH (one impact, h = 0): accelerations and potentials.
int launch_gravity_points(const Dev& d, const Cfg& c, cudaStream_t s) {
  if (c.quad) point_walk<true>(d, c, s);
  else point_walk<false>(d, c, s);
  return 1;
}

}  // namespace sphb
