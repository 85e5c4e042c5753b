// mrmg_pen.cu -- smoothed path-penetration cost of sphere-arm paths and its
// gradient through forward kinematics.
//
// There is no counterpart in the reference; the consumer is path shortcutting
// and repair (robot_mode_shortcut, planners/shortcutting.py:87-244).  For a
// path w[0..T-1] (each a full joint vector):
//
//   cost = sum_t sum_pairs softplus(beta (margin - d)) / (beta scale)
//        + smooth_w * sum_t |w[t+1] - w[t]|^2
//
// over every sphere-box pair (d = box signed distance of the centre minus the
// radius) and every pair of spheres on different robots (d = centre distance
// minus both radii).  With beta = 1 this is softplus(margin - d) / scale.
//
// One CTA per segment of 32 (cost) or 16 (gradient, where two CTAs then fit an
// SM) consecutive waypoints of one path, one waypoint per lane or per pair of
// half-warp lanes: forward kinematics runs per segment (a warp or half warp
// walks one robot's chain for its waypoints) and is recomputed, not stored, when
// the gradient is asked for.  Few segments: a cluster of CTAs shares each.  The gradient of a joint angle theta_k follows the geometric Jacobian:
// with o, z the origin and z axis of frame k-1 and g_s = dcost/dc_s,
//   dcost/dtheta_k = z . sum_{s beyond joint k} (c_s - o) x g_s = z . M,
// accumulated from the tip back: M is moved from one joint's origin to the next,
// M += (o' - o) x G with G = sum g_s, so its lever arms stay short (about the world's
// origin, z . (M - o x G) loses digits to the difference).  FP32 throughout; per-lane sums are
// compensated and segment totals are added in FP64 in a fixed order, so the
// cost and gradient are deterministic (no atomics: with the gradient, each
// inter-robot pair is evaluated from both sides).
#include <algorithm>

#include "mrmg_internal.cuh"

namespace mrmg {
namespace {

constexpr int kMaxSplit = 8;              // CTAs that share a segment, at most (a portable cluster)
// a CTA's fixed work over a whole segment's pair work: a part that does not depend
// on the scene, and what is worth this many pairs per waypoint
constexpr double kFixedShare = 0.05, kFixedPairs = 3000.0;

__host__ __device__ inline size_t al4(size_t n) { return (n + 3) & ~(size_t)3; }

// shared memory layout, in floats (every region a multiple of 16 bytes).
// The gradient regions cover the Sg spheres and Rg robots whose gradients
// the launch computes (all of them, or one group of robots of a scene too
// large for one CTA's shared memory).
template <int SEG>
struct PenLayout {
  size_t C, G, OZ, W, QG, sph, box, br, part, total;
  // tasks: pair tasks where a cluster shares the segment (their costs are kept one by one), else 0
  __host__ __device__ PenLayout(int S, int B, int D, bool grad, int warps, int tasks, int Sg, int Rg) {
    size_t o = 0;
    C = o;   o += (size_t)S * 3 * SEG;                          // sphere centres [S/2][3][SEG][2]
    G = o;   o += grad ? (size_t)Sg * 3 * SEG : 0;              // dcost/dcentre  [Sg*3][SEG]
    OZ = o;  o += grad ? (size_t)Rg * kMaxLinks * 6 * SEG : 0;  // frame origin, z axis [Rg][L][6][SEG]
    W = o;   o += al4((size_t)(SEG + 2) * D);                   // waypoints t0-1 .. t0+SEG
    QG = o;  o += grad ? al4((size_t)SEG * D) : 0;              // obstacle gradient [SEG][D]
    sph = o; o += (size_t)S * 4;
    box = o; o += (size_t)((B + 1) / 2) * 12;                    // pairs of boxes [(B+1)/2][6][2]
    br = o;  o += al4((size_t)S);                               // beta log2(e) radius
    part = o; o += (size_t)32 * (tasks > 2 * warps ? tasks : 2 * warps);
    total = o;
  }
};

// place of coordinate i of sphere s, waypoint `wl`, among the centres:
// spheres 2j and 2j + 1 side by side, read as one packed pair
template <int SEG>
__device__ __forceinline__ int cen(int s, int i, int wl) { return (((s >> 1) * 3 + i) * SEG + wl) * 2 + (s & 1); }

__host__ __device__ inline int pen_first_sphere(const PenDev& pd, int R, int r) { return r < R ? pd.lk[r][0] : pd.S; }

// the CTAs of a cluster: size, this CTA's rank, barrier, and stores to the same
// shared-memory place of CTA `rank`
__device__ __forceinline__ int cluster_size() { int v; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(v)); return v; }
__device__ __forceinline__ int cluster_rank() { int v; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v)); return v; }
// (not the .aligned forms: half warps come from branches of their own)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_st(float* p, int rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr(p, rank)), "f"(v) : "memory");
}

// MUFU approximations (PTX): 2^x, log2, sqrt, 1/sqrt, 1/x
__device__ __forceinline__ float ex2a(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float lg2a(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float sqrta(float x) { float y; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rsqa(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcpa(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// Pair terms in base-2 units.  With x2 = beta log2(e) (margin - d) and
// e = 2^-|x2|:  softplus(beta (margin - d)) = ln 2 * (max(x2, 0) + log2(1 + e))
// and sigmoid(beta (margin - d)) = 1 / (1 + e) for x2 >= 0, e / (1 + e) else.
// K folds the constant part: x2 = K - beta log2(e) * (distance).
//
// One sphere is evaluated against two partners (boxes or spheres, .x and .y) in
// packed FP32x2 arithmetic: one add / multiply / FMA instruction does both, and
// the partners' data are read as pairs (broadcasting a scalar into a packed
// operand would cost moves); min/max, abs and the special functions stay per
// component.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }

// one sphere of a task: minus its centre, the constant of x2 and its sums
struct Side {
  float2 nx, ny, nz;   // minus the centre, broadcast
  float2 K;            // beta log2(e) (margin + radius), broadcast
  float2 ps;           // sums of log2(1 + 2^x2) (without DIRECT: of max(x2, 0) + log2(1 + e))
  float2 pr;           // product of the 1 + e not yet in ps, less 1
  float2 gx, gy, gz;   // scale * dcost / dcentre
};

// Floor of the squared distances whose reciprocal root is taken: added to the
// last product of the sum, it leaves every square above 1e-22 m^2 unchanged.
constexpr float kTiny2 = 1e-30f;
// x2 of a partner that is not there: -infinity, so e = 0 for any beta
#define MRMG_PEN_NONE __int_as_float(0xff800000)
// the sphere of radius -infinity that makes a robot's count even: its pairs get
// MRMG_PEN_NONE for beta times the radius
__device__ __forceinline__ bool empty_sphere(float radius) { return radius < -3.402823466e38f; }

// Pairs whose 1 + e are multiplied before one log2 is taken of the product:
// log2 is an eighth of an FMA on this part (measured 16 against 128 per clock
// and SM) and the sum of log2(1 + e) is the log2 of the product.  The product is
// kept less 1, so pairs far apart (e below half an ulp of 1) still count.  With
// DIRECT every factor is at most 1 + 2^kDirectMax, so kProd of them stay below
// 2^113; without, at most 2.
constexpr int kProd = 16;
constexpr float kDirectMax = 7.f;

// softplus (base 2) of x2 into the product; e and 1 + e for the sigmoid.
// DIRECT (every x2 of the scene is at most kDirectMax): e = 2^x2, no |x2|, no max.
template <bool COST, bool DIRECT>
__device__ __forceinline__ void soft2(Side& a, float2 x2, float2* e, float2* ope) {
  *e = DIRECT ? make_float2(ex2a(x2.x), ex2a(x2.y)) : make_float2(ex2a(-fabsf(x2.x)), ex2a(-fabsf(x2.y)));
  *ope = add2(*e, bc2(1.f));
  if (COST) {
    a.pr = fma2(a.pr, *ope, *e);   // (1 + p)(1 + e) - 1
    if (!DIRECT) a.ps = add2(a.ps, make_float2(fmaxf(x2.x, 0.f), fmaxf(x2.y, 0.f)));
  }
}

// sigmoids of the four pairs of a step from two reciprocals:
// 1/a = b * (1 / (a b)), 1/b = a * (1 / (a b))
template <bool DIRECT>
__device__ __forceinline__ void sigmoid4(float2 x0, float2 e0, float2 o0, float2 x1, float2 e1, float2 o1, float2* w0,
                                         float2* w1) {
  const float2 m = mul2(o0, o1);
  const float2 r = make_float2(rcpa(m.x), rcpa(m.y));
  const float2 i0 = mul2(r, o1), i1 = mul2(r, o0);
  *w0 = mul2(e0, i0);
  *w1 = mul2(e1, i1);
  if (!DIRECT) {
    *w0 = make_float2(x0.x >= 0.f ? i0.x : w0->x, x0.y >= 0.f ? i0.y : w0->y);
    *w1 = make_float2(x1.x >= 0.f ? i1.x : w1->x, x1.y >= 0.f ? i1.y : w1->y);
  }
}

// log2(1 + p): the series of the logarithm below 1/64 (its first left-out term
// is p^4 / 5 < 1.2e-8 of the value)
template <bool COST>
__device__ __forceinline__ void flush_product(Side& a) {
  if (COST) {
    const float2 p = a.pr;
    const float2 t = fma2(fma2(fma2(p, bc2(-0.25f), bc2(0.33333333f)), p, bc2(-0.5f)), p, bc2(1.f));
    const float2 s = mul2(mul2(p, bc2(1.44269504f)), t);
    const float2 l = make_float2(lg2a(1.f + p.x), lg2a(1.f + p.y));
    a.ps = add2(a.ps, make_float2(p.x < 0.015625f ? s.x : l.x, p.y < 0.015625f ? s.y : l.y));
    a.pr = bc2(0.f);
  }
}

// a sphere whose centre lies inside a box (every max(|d| - h, 0) zero): its
// signed distance max_k(|d_k| - h_k), and the unit vector along that axis
__device__ __forceinline__ float inside_box(float dx, float dy, float dz, float hx, float hy, float hz, float* gx,
                                            float* gy, float* gz) {
  const float ax = fabsf(dx) - hx, ay = fabsf(dy) - hy, az = fabsf(dz) - hz;
  const bool bx = ax >= ay && ax >= az, by = !bx && ay >= az;
  *gx = bx ? copysignf(1.f, dx) : 0.f;
  *gy = by ? copysignf(1.f, dy) : 0.f;
  *gz = (!bx && !by) ? copysignf(1.f, dz) : 0.f;
  return fmaxf(ax, fmaxf(ay, az));
}

__device__ __forceinline__ float2 beyond2(float2 d, float2 h) {   // max(|d| - h, 0)
  return make_float2(fmaxf(fabsf(d.x) - h.x, 0.f), fmaxf(fabsf(d.y) - h.y, 0.f));
}
__device__ __forceinline__ float2 sign2(float2 m, float2 d) { return make_float2(copysignf(m.x, d.x), copysignf(m.y, d.y)); }

template <bool V>
struct Flag { static constexpr bool value = V; };

// two boxes: centres and half extents
struct Box2 {
  float2 cx, cy, cz, hx, hy, hz;
};

// x2 of a sphere against two boxes; with GRAD also u, inv: the gradient of the
// distance is -u * inv (the vector from the centre to the box over its length)
template <bool GRAD>
__device__ __forceinline__ float2 box_x2(const Side& a, const Box2& b, float2 nbl, float2 K, float2* ux, float2* uy,
                                         float2* uz, float2* inv) {
  const float2 dx = add2(b.cx, a.nx), dy = add2(b.cy, a.ny), dz = add2(b.cz, a.nz);
  *ux = beyond2(dx, b.hx);
  *uy = beyond2(dy, b.hy);
  *uz = beyond2(dz, b.hz);
  float2 sdf;
  if (!GRAD) {
    const float2 u2 = fma2(*ux, *ux, fma2(*uy, *uy, mul2(*uz, *uz)));
    sdf = make_float2(sqrta(u2.x), sqrta(u2.y));
    if (__builtin_expect(fminf(u2.x, u2.y) == 0.f, 0)) {   // a centre inside a box (seldom): the negative part
      float gx, gy, gz;
      if (u2.x == 0.f) sdf.x = fminf(inside_box(dx.x, dy.x, dz.x, b.hx.x, b.hy.x, b.hz.x, &gx, &gy, &gz), 0.f);
      if (u2.y == 0.f) sdf.y = fminf(inside_box(dx.y, dy.y, dz.y, b.hx.y, b.hy.y, b.hz.y, &gx, &gy, &gz), 0.f);
    }
  } else {
    const float2 u2 = fma2(*ux, *ux, fma2(*uy, *uy, fma2(*uz, *uz, bc2(kTiny2))));
    *inv = make_float2(rsqa(u2.x), rsqa(u2.y));
    sdf = mul2(u2, *inv);
    *ux = sign2(*ux, dx);
    *uy = sign2(*uy, dy);
    *uz = sign2(*uz, dz);
    if (__builtin_expect(fminf(u2.x, u2.y) <= kTiny2, 0)) {   // a centre inside a box (seldom)
      if (u2.x <= kTiny2) {
        sdf.x = inside_box(dx.x, dy.x, dz.x, b.hx.x, b.hy.x, b.hz.x, &ux->x, &uy->x, &uz->x);
        inv->x = 1.f;
      }
      if (u2.y <= kTiny2) {
        sdf.y = inside_box(dx.y, dy.y, dz.y, b.hx.y, b.hy.y, b.hz.y, &ux->y, &uy->y, &uz->y);
        inv->y = 1.f;
      }
    }
  }
  return fma2(nbl, sdf, K);
}

// x2 of a sphere against two spheres (centres x, y, z); v: from the centre to theirs
template <bool GRAD>
__device__ __forceinline__ float2 sphere_x2(const Side& a, float2 x, float2 y, float2 z, float2 nbl, float2 K, float2* vx,
                                            float2* vy, float2* vz, float2* inv) {
  *vx = add2(x, a.nx);
  *vy = add2(y, a.ny);
  *vz = add2(z, a.nz);
  if (!GRAD) {
    const float2 d2 = fma2(*vx, *vx, fma2(*vy, *vy, mul2(*vz, *vz)));
    return fma2(nbl, make_float2(sqrta(d2.x), sqrta(d2.y)), K);
  }
  const float2 d2 = fma2(*vx, *vx, fma2(*vy, *vy, fma2(*vz, *vz, bc2(kTiny2))));
  *inv = make_float2(rsqa(d2.x), rsqa(d2.y));
  return fma2(nbl, mul2(d2, *inv), K);
}

__device__ __forceinline__ void pull(Side& a, float2 w, float2 inv, float2 ux, float2 uy, float2 uz) {
  const float2 f = mul2(w, inv);
  a.gx = fma2(f, ux, a.gx);
  a.gy = fma2(f, uy, a.gy);
  a.gz = fma2(f, uz, a.gz);
}

// both spheres of a task against two boxes
template <bool COST, bool GRAD, bool DIRECT>
__device__ __forceinline__ void box_step(Side& a, Side& b, const Box2& bx, float2 nbl, float2 Ka, float2 Kb) {
  float2 ax, ay, az, ai, cx, cy, cz, ci, ea, oa, ec, oc;
  const float2 xa = box_x2<GRAD>(a, bx, nbl, Ka, &ax, &ay, &az, &ai);
  const float2 xc = box_x2<GRAD>(b, bx, nbl, Kb, &cx, &cy, &cz, &ci);
  soft2<COST, DIRECT>(a, xa, &ea, &oa);
  soft2<COST, DIRECT>(b, xc, &ec, &oc);
  if (GRAD) {
    float2 wa, wc;
    sigmoid4<DIRECT>(xa, ea, oa, xc, ec, oc, &wa, &wc);
    pull(a, wa, ai, ax, ay, az);
    pull(b, wc, ci, cx, cy, cz);
  }
}

// both spheres of a task against two spheres of another robot
template <bool COST, bool GRAD, bool DIRECT>
__device__ __forceinline__ void sphere_step(Side& a, Side& b, float2 x, float2 y, float2 z, float2 br, float2 nbl) {
  float2 ax, ay, az, ai, cx, cy, cz, ci, ea, oa, ec, oc;
  const float2 xa = sphere_x2<GRAD>(a, x, y, z, nbl, add2(a.K, br), &ax, &ay, &az, &ai);
  const float2 xc = sphere_x2<GRAD>(b, x, y, z, nbl, add2(b.K, br), &cx, &cy, &cz, &ci);
  soft2<COST, DIRECT>(a, xa, &ea, &oa);
  soft2<COST, DIRECT>(b, xc, &ec, &oc);
  if (GRAD) {
    float2 wa, wc;
    sigmoid4<DIRECT>(xa, ea, oa, xc, ec, oc, &wa, &wc);
    pull(a, wa, ai, ax, ay, az);
    pull(b, wc, ci, cx, cy, cz);
  }
}

__device__ __forceinline__ void acc2(float& h, float& l, float v) {
  float s, e;
  two_sum(h, v, &s, &e);
  h = s;
  l += e;
}

// Bound: issue slots (cost: 15 warp instructions per 32 pairs, 83 % of them
// used) and, with the gradient, the FMA and special-function pipes together
// (18 instructions; 17 and 16 of 27 cycles per 32 pairs).  512 paths of 256
// waypoints, four arms, 50 boxes: cost 1.55 -> 1.22 ms, gradient 3.63 -> 2.76
// ms, both 4.03 -> 3.03 ms, against one log2 and one reciprocal per pair, two
// spheres per packed instruction and 32-waypoint gradient CTAs (one per SM).
// The sphere loop unrolled by 1, 2, 4 or 8: cost 1.31, 1.31, 1.24, 1.23 ms, the
// gradient unchanged; the box loop by 1 or 2: gradient 2.80, 2.76 ms, both 3.09,
// 3.06 ms.  SHARED (clusters): 12 paths of 45 waypoints, 20 boxes: cost 47 us,
// gradient 46 us, both 56 us; with the joint gradients of each CTA's own spheres
// added up over the CTAs (whose bits then depend on the split) 47, 46 and 56 us,
// with sphere gradients fetched behind the barrier, not stored before it, 52, 49
// and 60 us.
template <int SEG, bool COST, bool GRAD, bool DIRECT, bool SHARED>
__global__ void __launch_bounds__(GRAD && SEG == 16 ? 384 : 512, GRAD && SEG == 32 ? 1 : 2)
    pen_kernel(ArmDev a, PenDev pd, PenParams pp, const float* __restrict__ paths, int T, int nseg,
               const float* __restrict__ gout, double* __restrict__ seg_cost, float* __restrict__ wp_cost,
               float* __restrict__ grad, int gr0, int gr1) {
  extern __shared__ __align__(16) float smf[];
  const int S = pd.S, B = pd.B, R = a.R, D = a.D;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NW = blockDim.x >> 5;
  // HV half warps (or whole ones) hold the same SEG waypoints: this lane's
  // waypoint, and its share of a warp's partners and robots
  constexpr int HV = 32 / SEG;
  const int wl = lane & (SEG - 1), half = HV > 1 ? lane / SEG : 0;
  // SHARED: the CTAs of a cluster share one segment: each runs its kinematics and
  // a share of the pair tasks
  const int split = SHARED ? cluster_size() : 1, rank = SHARED ? cluster_rank() : 0;
  if (SHARED) cluster_arrive();   // (waited for before the first store to another CTA)
  const long long sidx = blockIdx.x / split;
  const long long p = sidx / nseg;
  const int seg = (int)(sidx - p * nseg);
  const int t0 = seg * SEG;
  // the gradient of this launch: robots [gr0, gr1), their spheres [s_lo, s_hi)
  // and joints [j_lo, j_hi) (robots' joints are contiguous in robot order)
  const int s_lo = pen_first_sphere(pd, R, gr0), s_hi = pen_first_sphere(pd, R, gr1);
  const int j_lo = a.q_off[gr0], j_hi = gr1 < R ? a.q_off[gr1] : D;
  const PenLayout<SEG> L(S, B, D, GRAD, NW, SHARED ? pd.NTK : 0, s_hi - s_lo, gr1 - gr0);
  float* C = smf + L.C;
  float* Gs = smf + L.G;
  float* OZ = smf + L.OZ;
  float* W = smf + L.W;
  float* QG = smf + L.QG;
  float4* sph = (float4*)(smf + L.sph);
  float2* box = (float2*)(smf + L.box);
  float* br = smf + L.br;
  const int NTK = pd.NTK;
  float* part = smf + L.part;

  // ---- stage tables and the segment's waypoints (rows t0-1 .. t0+SEG)
  for (int i = tid; i < S; i += blockDim.x) {
    sph[i] = pd.sph[i];
    br[i] = empty_sphere(sph[i].w) ? MRMG_PEN_NONE : pp.beta * 1.4426950408889634f * sph[i].w;
  }
  for (int i = tid; i < 6 * ((B + 1) / 2); i += blockDim.x) {   // pair i / 6: centre x, y, z, half extent x, y, z
    const int b = 2 * (i / 6), k = i % 6, c = b + 1 < B ? b + 1 : b;
    const float* f = (const float*)pd.box;
    box[i] = make_float2(f[8 * b + (k < 3 ? k : k + 1)], f[8 * c + (k < 3 ? k : k + 1)]);
  }
  {
    const float* src = paths + (size_t)p * T * D;
    const int n = (SEG + 2) * D;
    for (int i = tid; i < n; i += blockDim.x) {
      const int t = t0 - 1 + i / D;
      W[i] = (t >= 0 && t < T) ? src[(long long)(t0 - 1) * D + i] : 0.f;
    }
  }
  if (GRAD)
    for (int i = tid; i < SEG * D; i += blockDim.x) QG[i] = 0.f;
  __syncthreads();

  // ---- forward kinematics: (half) warp r walks robot r's chain, lane = waypoint
  if (HV * warp + half < R) {
    const int r = HV * warp + half;
    const float* q = W + (wl + 1) * D;
    int jo = a.q_off[r];
    float m[9], o[3];
    {
      const float4 b0 = a.base32[3 * r], b1 = a.base32[3 * r + 1], b2 = a.base32[3 * r + 2];
      if (a.base_kind[r] == 1) {
        float sn, cs;
        sincosf(a.off32 ? q[jo + 2] + a.off32[jo + 2].x : q[jo + 2], &sn, &cs);
        m[0] = cs * b0.x - sn * b1.x; m[1] = cs * b0.y - sn * b1.y; m[2] = cs * b0.z - sn * b1.z;
        m[3] = sn * b0.x + cs * b1.x; m[4] = sn * b0.y + cs * b1.y; m[5] = sn * b0.z + cs * b1.z;
        m[6] = b2.x; m[7] = b2.y; m[8] = b2.z;
        o[0] = q[jo] + (cs * b0.w - sn * b1.w);
        o[1] = q[jo + 1] + (sn * b0.w + cs * b1.w);
        o[2] = b2.w;
        jo += 3;
      } else {
        m[0] = b0.x; m[1] = b0.y; m[2] = b0.z; m[3] = b1.x; m[4] = b1.y; m[5] = b1.z;
        m[6] = b2.x; m[7] = b2.y; m[8] = b2.z;
        o[0] = b0.w; o[1] = b1.w; o[2] = b2.w;
      }
    }
    const int nl = a.nl[r];
    for (int k = 0; k <= nl; k++) {
      if (k > 0) {
        if (GRAD && r >= gr0 && r < gr1) {
          float* oz = OZ + (size_t)(((r - gr0) * kMaxLinks + (k - 1)) * 6) * SEG + wl;
          oz[0] = o[0]; oz[SEG] = o[1]; oz[2 * SEG] = o[2];
          oz[3 * SEG] = m[2]; oz[4 * SEG] = m[5]; oz[5 * SEG] = m[8];
        }
        const float4 h = a.dh32[r * kMaxLinks + k - 1];   // a, d, cos(alpha), sin(alpha)
        float sn, cs;
        sincosf(a.off32 ? q[jo + k - 1] + a.off32[jo + k - 1].x : q[jo + k - 1], &sn, &cs);
        const float sca = sn * h.z, cca = cs * h.z, ssa = sn * h.w, csa = cs * h.w;
        const float ac = h.x * cs, as = h.x * sn;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const float r0 = m[3 * i], r1 = m[3 * i + 1], r2 = m[3 * i + 2];
          m[3 * i] = r0 * cs + r1 * sn;
          m[3 * i + 1] = (r1 * cca - r0 * sca) + r2 * h.w;
          m[3 * i + 2] = (r0 * ssa - r1 * csa) + r2 * h.z;
          o[i] += (r0 * ac + r1 * as) + r2 * h.y;
        }
      }
      for (int s = pd.lk[r][k]; s < pd.lk[r][k + 1]; s++) {
        const float4 l = sph[s];
#pragma unroll
        for (int i = 0; i < 3; i++)
          C[cen<SEG>(s, i, wl)] = o[i] + ((m[3 * i] * l.x + m[3 * i + 1] * l.y) + m[3 * i + 2] * l.z);
      }
    }
  }
  __syncthreads();

  // ---- pair terms.  A task is two spheres of one robot against every box and
  // every sphere of the other robots, by one warp (SEG 16: its halves take every
  // other pair of partners).  With the gradient, each
  // inter-robot pair is evaluated from both sides, so a task owns its spheres'
  // gradients outright (no atomics, a fixed summation order); the cost counts
  // each pair once (the partners on later robots).  Tasks are dealt zig-zag
  // over the warps.
  const float bl = pp.beta * 1.4426950408889634f;   // beta log2(e)
  const float blm = bl * pp.margin;
  float acc_h = 0.f, acc_l = 0.f;
  const int VW = NW * split, vw = warp * split + rank;   // the cluster's warps, dealt over its CTAs
  if (SHARED) cluster_wait();   // every CTA runs
  // The sums of a segment do not depend on how many CTAs share it, so a path's
  // cost and gradient have the same bits alone and in any batch: each CTA gets every
  // sphere's gradient, the first one every task's cost, and adds them up as a CTA
  // alone does.
  auto put = [&](int s, int i, float v) {   // dcost/dcentre, coordinate i of sphere s
    float* g = Gs + (3 * (s - s_lo) + i) * SEG + wl;
    if (!SHARED) *g = v;
    else
      for (int r = 0; r < split; r++) cluster_st(g, r, v);
  };
  for (int base = 0, turn = 0; base < NTK; base += VW, turn ^= 1) {
    const int tk = turn ? base + VW - 1 - vw : base + vw;
    if (tk >= NTK) continue;
    const int2 task = __ldg(&pd.task[tk]);   // the robot's first sphere, the next robot's first
    const int i0 = 2 * tk, i1 = i0 + 1;
    if (GRAD && !COST && (i0 < s_lo || i0 >= s_hi)) continue;   // another group's robot
    auto side = [&](int i) {
      Side d;
      d.nx = bc2(-C[cen<SEG>(i, 0, wl)]);
      d.ny = bc2(-C[cen<SEG>(i, 1, wl)]);
      d.nz = bc2(-C[cen<SEG>(i, 2, wl)]);
      d.K = bc2(empty_sphere(sph[i].w) ? MRMG_PEN_NONE : fmaf(bl, sph[i].w, blm));
      d.ps = d.pr = d.gx = d.gy = d.gz = bc2(0.f);
      return d;
    };
    Side a = side(i0), b = side(i1);
    const float2 nbl = bc2(-bl);
    const float4* b4 = (const float4*)box;
    auto boxes = [&](int k, float2 Ka, float2 Kb) {
      const float4 u = b4[3 * k], v = b4[3 * k + 1], w = b4[3 * k + 2];
      const Box2 bx{make_float2(u.x, u.y), make_float2(u.z, u.w), make_float2(v.x, v.y),
                    make_float2(v.z, v.w), make_float2(w.x, w.y), make_float2(w.z, w.w)};
      box_step<COST, GRAD, DIRECT>(a, b, bx, nbl, Ka, Kb);
    };
    const int nb2 = B / 2, even = nb2 & ~(HV - 1);
#pragma unroll 2
    for (int k = 0; k < even; k += HV) {
      boxes(k + half, a.K, b.K);
      if (COST && (k / HV) % kProd == kProd - 1) {
        flush_product<COST>(a);
        flush_product<COST>(b);
      }
    }
    if (B > 2 * even) {   // the boxes left: a place without a box adds nothing
      const int k = even + half, left = B - 2 * k;   // of this half's pair: both there when 2 or more, the first when 1
      const float kx = left > 0 ? 0.f : MRMG_PEN_NONE, ky = left > 1 ? 0.f : MRMG_PEN_NONE;
      boxes(left > 0 ? k : even, add2(a.K, make_float2(kx, ky)), add2(b.K, make_float2(kx, ky)));
    }
    flush_product<COST>(a);
    flush_product<COST>(b);
    const float2* C2 = (const float2*)C + wl;
    const float2* br2 = (const float2*)br;
    auto spheres = [&](auto with_cost, int j, float2 r) {
      sphere_step<decltype(with_cost)::value, GRAD, DIRECT>(a, b, C2[(3 * j) * SEG], C2[(3 * j + 1) * SEG],
                                                            C2[(3 * j + 2) * SEG], r, nbl);
    };
    const float2 none = bc2(MRMG_PEN_NONE);
    {   // the later robots' spheres
      const int j0 = task.y / 2, j1 = S / 2, je = j0 + ((j1 - j0) & ~(HV - 1));
#pragma unroll 4
      for (int j = j0; j < je; j += HV) {
        spheres(Flag<COST>(), j + half, br2[j + half]);
        if (COST && ((j - j0) / HV) % kProd == kProd - 1) {
          flush_product<COST>(a);
          flush_product<COST>(b);
        }
      }
      if (HV > 1 && je < j1) spheres(Flag<COST>(), je, half ? none : br2[je]);
      flush_product<COST>(a);
      flush_product<COST>(b);
    }
    if (GRAD) {   // the earlier robots' (the cost has counted them)
      const int z = task.x / 2, ze = z & ~(HV - 1);
#pragma unroll 4
      for (int j = 0; j < ze; j += HV) spheres(Flag<false>(), j + half, br2[j + half]);
      if (HV > 1 && ze < z) spheres(Flag<false>(), ze, half ? none : br2[ze]);
      const float is = pp.inv_scale;
      const float g[3] = {a.gx.x + a.gx.y, a.gy.x + a.gy.y, a.gz.x + a.gz.y};
      const float h[3] = {b.gx.x + b.gx.y, b.gy.x + b.gy.y, b.gz.x + b.gz.y};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        if (HV == 1) {
          put(i0, i, is * g[i]);
          put(i1, i, is * h[i]);
        } else {   // both halves' sums: half 0 stores the first sphere's, half 1 the second's
          const float mine = half ? h[i] : g[i], other = half ? g[i] : h[i];
          put(i0 + half, i, is * (mine + __shfl_xor_sync(MRMG_FULL, other, SEG & 31)));
        }
      }
    }
    if (COST) {
      const float v = (a.ps.x + a.ps.y) + (b.ps.x + b.ps.y);
      if (SHARED) cluster_st(part + tk * 32 + lane, 0, v);
      else acc2(acc_h, acc_l, v);
    }
  }
  if (SHARED) {
    cluster_arrive();   // every CTA's tasks are done
    cluster_wait();
    if (COST && rank == 0)
      for (int base = 0, turn = 0; base < NTK; base += NW, turn ^= 1) {
        const int tk = turn ? base + NW - 1 - warp : base + warp;
        if (tk < NTK) acc2(acc_h, acc_l, part[tk * 32 + lane]);
      }
  }
  if (COST && rank == 0) {   // (where tasks' costs lie in `part`, these are places of this warp's own tasks)
    part[warp * 32 + lane] = acc_h;
    part[(2 * NW - 1 - warp) * 32 + lane] = acc_l;
  }
  __syncthreads();

  double csum = 0.0;   // warp 0 of the first CTA: the pair terms of waypoint t0 + wl
  if (COST && warp == 0 && rank == 0) {
    for (int w = 0; w < NW; w++) csum += (double)part[w * 32 + lane] + (double)part[(2 * NW - 1 - w) * 32 + lane];
    if (HV > 1) csum += __shfl_xor_sync(MRMG_FULL, csum, SEG & 31);
  }
  if (GRAD) {
    // ---- joint gradients from the sphere gradients, tip to base
    if (gr0 + HV * warp + half < gr1) {
      const int r = gr0 + HV * warp + half;
      const int nl = a.nl[r];
      int jo = a.q_off[r] + (a.base_kind[r] == 1 ? 3 : 0);
      // sums of g and of the moments, compensated: the rounding of the pair terms
      // is then what is left of the error
      float G[3] = {0.f, 0.f, 0.f}, M[3] = {0.f, 0.f, 0.f}, Gl[3] = {0.f, 0.f, 0.f}, Ml[3] = {0.f, 0.f, 0.f};
      float o[3] = {0.f, 0.f, 0.f};   // the point M is about: the joint's frame origin
      float* qg = QG + wl * D;
      const bool planar = a.base_kind[r] == 1;
      const int b0 = a.q_off[r];
      for (int k = nl; k >= (planar ? 0 : 1); k--) {
        const float* oz = OZ + (size_t)(((r - gr0) * kMaxLinks + (k - 1)) * 6) * SEG + wl;
        float d[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const float n = k > 0 ? oz[i * SEG] : (i < 2 ? W[(wl + 1) * D + b0 + i] : 0.f);
          d[i] = o[i] - n;
          o[i] = n;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const int j = (i + 1) % 3, l = (i + 2) % 3;
          acc2(M[i], Ml[i], d[j] * (G[l] + Gl[l]) - d[l] * (G[j] + Gl[j]));
        }
        float gs[3] = {0.f, 0.f, 0.f}, ms[3] = {0.f, 0.f, 0.f};   // this link's spheres
        for (int s = pd.lk[r][k]; s < pd.lk[r][k + 1]; s++) {
          float c[3], g[3];
#pragma unroll
          for (int i = 0; i < 3; i++) {
            c[i] = C[cen<SEG>(s, i, wl)] - o[i];
            g[i] = Gs[(3 * (s - s_lo) + i) * SEG + wl];
          }
#pragma unroll
          for (int i = 0; i < 3; i++) {
            const int j = (i + 1) % 3, l = (i + 2) % 3;
            gs[i] += g[i];
            ms[i] += c[j] * g[l] - c[l] * g[j];
          }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          acc2(G[i], Gl[i], gs[i]);
          acc2(M[i], Ml[i], ms[i]);
        }
        if (k > 0)
          qg[jo + k - 1] = oz[3 * SEG] * (M[0] + Ml[0]) + oz[4 * SEG] * (M[1] + Ml[1]) + oz[5 * SEG] * (M[2] + Ml[2]);
      }
      if (planar) {
        qg[b0] = G[0] + Gl[0];
        qg[b0 + 1] = G[1] + Gl[1];
        qg[b0 + 2] = M[2] + Ml[2];
      }
    }
  }

  const int t = t0 + wl;
  if (COST && warp == 0 && rank == 0) {
    double c = csum;
    c *= 0.69314718055994531 * (double)pp.inv_beta * (double)pp.inv_scale;   // ln 2 / (beta scale)
    if (t + 1 < T) {
      const float* w0 = W + (wl + 1) * D;
      const float* w1 = W + (wl + 2) * D;
      float sh = 0.f, sl = 0.f;
      for (int k = 0; k < D; k++) {
        const float dv = w1[k] - w0[k];
        acc2(sh, sl, dv * dv);
      }
      c += (double)pp.smooth_w * ((double)sh + (double)sl);
    }
    if (t >= T || half) c = 0.0;   // the second half holds copies
    if (wp_cost && t < T && !half) wp_cost[(size_t)p * T + t] = (float)c;
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(MRMG_FULL, c, o);
    if (lane == 0 && seg_cost) seg_cost[(size_t)p * nseg + seg] = c;
  }

  if (GRAD) {
    __syncthreads();
    // ---- add the smoothness gradient, scale by dL/dcost, write coalesced
    const float go = gout ? gout[p] : 1.f;
    const float sw2 = 2.f * pp.smooth_w;
    const int n = SEG * D, share = (n + split - 1) / split;   // each CTA writes a share of the rows
    float* dst = grad + ((size_t)p * T + t0) * D;
    for (int i = rank * share + tid; i < min(n, (rank + 1) * share); i += blockDim.x) {
      const int tt = t0 + i / D;
      if (tt >= T) break;
      const int j = i - (i / D) * D;
      if (j < j_lo || j >= j_hi) continue;   // another group's joint
      const float wc = W[i + D];
      float gsm = 0.f;
      if (tt > 0) gsm += sw2 * (wc - W[i]);
      if (tt + 1 < T) gsm -= sw2 * (W[i + 2 * D] - wc);
      dst[i] = go * (QG[i] + gsm);
    }
  }
}

__global__ void pen_sum_kernel(const double* __restrict__ seg, long long P, int nseg, double* __restrict__ cost) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    double c = 0.0;
    for (int s = 0; s < nseg; s++) c += seg[p * nseg + s];
    cost[p] = c;
  }
}

// CTAs per segment: a segment's pair tasks go to a cluster of `s` CTAs where the
// segments alone leave SMs idle.  Modelled time: rounds of a CTA per SM (two on one
// SM take as long as one after the other), each paying the fixed part (tables,
// kinematics, joint gradients) and its share of the pairs per waypoint.  24
// segments on 152 SMs, four arms, 50 boxes: one CTA each 81 us, clusters of 8 50 us
// (cost kernel).  Against the best of 1, 2, 4 and 8 on 189 calls (seven scenes of 56
// to 304 spheres, 1 to 200 paths) the choice loses 0.5 %; rounds of all resident
// CTAs and a fixed part of a tenth lost 5.4 % (200 segments of two mobile robots 55
// us, a CTA each 52).
int pen_split(long long segs, int num_sms, double pairs) {
  const double fixed = kFixedShare + kFixedPairs / std::max(pairs, 1.0);
  int best = 1;
  double best_t = 0.0;
  for (int s = 1; s <= kMaxSplit; s *= 2) {
    const double t = (double)((segs * s + num_sms - 1) / num_sms) * (fixed + 1.0 / s);
    if (s == 1 || t < best_t) {
      best = s;
      best_t = t;
    }
  }
  return best;
}

template <int SEG>
size_t smem_bytes(const ArmDev& a, const PenDev& pd, int grad, int warps, int tasks, int gr0, int gr1) {
  return PenLayout<SEG>(pd.S, pd.B, a.D, grad != 0, warps, tasks,
                        pen_first_sphere(pd, a.R, gr1) - pen_first_sphere(pd, a.R, gr0), gr1 - gr0)
             .total * sizeof(float);
}

template <int SEG, bool COST, bool GRAD, bool DIRECT, bool SHARED>
cudaError_t launch_one(const ArmDev& a, const PenDev& pd, const PenParams& pp, const float* paths, long long P, int T,
                       const float* gout, double* seg, float* wp, float* grad, int warps, int split, int gr0, int gr1,
                       cudaStream_t st) {
  const size_t smem = smem_bytes<SEG>(a, pd, GRAD, warps, SHARED ? pd.NTK : 0, gr0, gr1);
  auto kernel = pen_kernel<SEG, COST, GRAD, DIRECT, SHARED>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int nseg = pen_segments(T, SEG);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(P * nseg * split));
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = split;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = SHARED ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a, pd, pp, paths, T, nseg, gout, seg, wp, grad, gr0, gr1);
}

// One launch covers every path unless its grid would pass the limit of
// 2^31 - 1 CTAs.
template <int SEG, bool COST, bool GRAD>
cudaError_t launch_form(const ArmDev& a, const PenDev& pd, const PenParams& pp, const float* paths, long long P, int T,
                        const float* gout, double* seg, float* wp, float* grad, int warps, int gr0, int gr1,
                        int num_sms, size_t smem_sm, cudaStream_t st) {
  // the largest x2 of any pair: centres coincide, or lie deepest in a box
  const bool direct = pp.beta * 1.4426951f * (pp.margin + pd.reach) <= kDirectMax;
  const int nseg = pen_segments(T, SEG);
  // (with the gradient each pair of spheres is evaluated from both sides)
  const double pairs = (double)pd.S * (pd.B + (double)pd.S * (a.R - 1) / a.R * (GRAD ? 1.0 : 0.5));
  int split = pen_split(P * nseg, num_sms, pairs);
  // (1 KB per CTA is the system's; a cluster keeps its tasks' costs in shared memory too)
  while (split > 1 && smem_bytes<SEG>(a, pd, GRAD, warps, pd.NTK, gr0, gr1) + 1024 > smem_sm)
    split /= 2;
  const long long step = std::max(1ll, 0x7fffffffll / ((long long)nseg * split));
  cudaError_t e = cudaSuccess;
  for (long long p0 = 0; p0 < P && e == cudaSuccess; p0 += step) {
    const long long n = std::min(step, P - p0);
    const size_t wp0 = (size_t)p0 * T;
    const float* w = paths + wp0 * a.D;
    const float* go = gout ? gout + p0 : nullptr;
    double* sg = seg ? seg + p0 * nseg : nullptr;
    float* wc = wp ? wp + wp0 : nullptr;
    float* g = grad ? grad + wp0 * a.D : nullptr;
    auto launch = direct ? (split > 1 ? launch_one<SEG, COST, GRAD, true, true> : launch_one<SEG, COST, GRAD, true, false>)
                         : (split > 1 ? launch_one<SEG, COST, GRAD, false, true> : launch_one<SEG, COST, GRAD, false, false>);
    e = launch(a, pd, pp, w, n, T, go, sg, wc, g, warps, split, gr0, gr1, st);
  }
  return e;
}

}  // namespace

size_t pen_smem_bytes(const ArmDev& a, const PenDev& pd, int grad, int warps, int gr0, int gr1) {
  return smem_bytes<32>(a, pd, grad, warps, 0, gr0, gr1);
}

int pen_grad_groups(const ArmDev& a, const PenDev& pd, int warps, size_t smem_max, int* bounds) {
  // joints must be contiguous in robot order for the groups' joint ranges
  int jo = 0;
  for (int r = 0; r < a.R; r++) {
    if (a.q_off[r] != jo) return a.R == 1 || pen_smem_bytes(a, pd, 1, warps, 0, a.R) <= smem_max ? 1 : 0;
    jo += (a.base_kind[r] == 1 ? 3 : 0) + a.nl[r];
  }
  if (jo != a.D) return pen_smem_bytes(a, pd, 1, warps, 0, a.R) <= smem_max ? 1 : 0;
  // fewest groups of consecutive robots (balanced by count) whose gradient regions fit
  for (int ng = 1; ng <= a.R; ng++) {
    bool ok = true;
    for (int g = 0; g <= ng; g++) bounds[g] = g * a.R / ng;
    for (int g = 0; g < ng && ok; g++) ok = pen_smem_bytes(a, pd, 1, warps, bounds[g], bounds[g + 1]) <= smem_max;
    if (ok) return ng;
  }
  return 0;
}

cudaError_t pen_launch(const ArmDev& a, const PenDev& pd, const PenParams& pp, const float* paths, long long P, int T,
                       const float* gout, double* seg, double* cost, float* wp_cost, float* grad, int warps,
                       int n_groups, const int* bounds, int num_sms, size_t smem_sm, cudaStream_t st) {
  if (P <= 0) return cudaSuccess;
  const bool want_cost = cost || wp_cost;
  // gradient form: half-warp segments where two of their CTAs fit an SM
  const int gw = std::min(warps, kPenGradWarps);
  const bool halves = grad && n_groups <= 1 && 2 * (smem_bytes<16>(a, pd, 1, gw, 0, 0, a.R) + 1024) <= smem_sm;
  cudaError_t e = cudaSuccess;
  int nseg = pen_segments(T, 32);   // segments whose costs are summed
  if (grad && n_groups <= 1 && halves) {
    nseg = pen_segments(T, 16);
    if (want_cost)
      e = launch_form<16, true, true>(a, pd, pp, paths, P, T, gout, seg, wp_cost, grad, gw, 0, a.R, num_sms, smem_sm, st);
    else
      e = launch_form<16, false, true>(a, pd, pp, paths, P, T, gout, nullptr, nullptr, grad, gw, 0, a.R, num_sms, smem_sm, st);
  } else if (grad && n_groups <= 1) {
    if (want_cost)
      e = launch_form<32, true, true>(a, pd, pp, paths, P, T, gout, seg, wp_cost, grad, warps, 0, a.R, num_sms, smem_sm, st);
    else
      e = launch_form<32, false, true>(a, pd, pp, paths, P, T, gout, nullptr, nullptr, grad, warps, 0, a.R, num_sms, smem_sm, st);
  } else {
    if (want_cost || !grad)
      e = launch_form<32, true, false>(a, pd, pp, paths, P, T, gout, seg, wp_cost, nullptr, warps, 0, a.R, num_sms, smem_sm, st);
    for (int g = 0; grad && g < n_groups && e == cudaSuccess; g++)
      e = launch_form<32, false, true>(a, pd, pp, paths, P, T, gout, nullptr, nullptr, grad, warps, bounds[g],
                                       bounds[g + 1], num_sms, smem_sm, st);
  }
  if (e != cudaSuccess || !cost) return e;
  const int blocks = (int)std::min<long long>((P + 255) / 256, 4096);
  pen_sum_kernel<<<blocks, 256, 0, st>>>(seg, P, nseg, cost);
  return cudaGetLastError();
}

}  // namespace mrmg
