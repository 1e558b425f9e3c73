// Collision-distance drop-ins: world sphere ([B,K,M] and per-link reduced
// [B,N,M]), world capsule, self sphere and self capsule.
//
// Replaces the handlers of src/pyroffi/cuda_kernels/_collision_cuda_kernel.cu
// (CollisionWorldSphereFfi :507, ...ReducedFfi :673, CollisionWorldCapsuleFfi
// :843, CollisionSelfSphereFfi :1006, CollisionSelfCapsuleFfi :1114).
//
// B200 layout: every obstacle type is staged once per block into shared
// memory and handled by one kernel (no per-type launches, no graph cache).
// Output rows [.., M] are written by groups of lanes running over m, so each
// warp store covers contiguous 16-byte chunks of one row.  The reduced and
// the self-sphere kernels bring a block's configurations into shared memory
// once, the spheres that exist packed into pairs, and run on packed FP32x2
// arithmetic.  Both are bound by FP32 issue and the reciprocal square roots
// (one per sphere-obstacle or sphere-sphere pair), and take one Newton step on
// the root so the distances keep the accuracy of the IEEE square root.
#include <algorithm>

#include "pk_obstacles.cuh"

namespace pk {

// lanes that share one output row: enough to cover M with 4 columns each
static int lanes_per_row(int M) {
  int l = 1;
  while (l < 32 && l * 4 < M) l <<= 1;
  return l;
}

struct RowArgs {
  WorldArgs w;
  const float* centers;  // [3, B, K] SoA (sphere robot) or caps [7, B, N] (capsule robot)
  const float* radii;    // [B, K] (sphere robot)
  float* out;
  long long B;
  int K;                 // robot elements per configuration (spheres K, or links N)
  int N;                 // links (reduced kernel)
  int S;                 // spheres per link (reduced kernel)
  int lpr;               // lanes per row
  int stage;
};

__device__ __forceinline__ ObsView world_view(const RowArgs& a, float* smem) {
  if (a.stage) return stage_world(a.w, smem);
  ObsView ob;
  ob.sph = reinterpret_cast<const float4*>(a.w.spheres);
  ob.cap = a.w.capsules; ob.box = a.w.boxes; ob.hs = a.w.halfspaces;
  ob.Ms = a.w.Ms; ob.Mc = a.w.Mc; ob.Mb = a.w.Mb; ob.Mh = a.w.Mh;
  return ob;
}

// A block's robot spheres packed per link into pairs: the spheres that exist,
// moved to the front, spheres 2q and 2q + 1 of a link as float4 (x0, x1, y0, y1)
// and (z0, z1, -r0, -r1); the odd slot of an odd count with -r = 1e30, so its
// packed distances never win a minimum, wherever the obstacles are.
__host__ __device__ __forceinline__ int link_pair_count(int S) { return (S + 1) >> 1; }

// Packs `nc` configurations into dst (link n of configuration c at c * cstride
// + n * lstride float4), sphere (c, s, n) read by centre(c, s, n) and radius(c,
// s, n), consecutive threads taking consecutive links; counts[c * N + n] pairs.
// NaN and negative radii are left out: neither can win a minimum.
template <class Centre, class Radius>
__device__ __forceinline__ void pack_link_pairs(float4* dst, int* counts, int nc, int N, int S, int cstride,
                                                int lstride, Centre centre, Radius radius) {
  for (int g = threadIdx.x; g < nc * N; g += blockDim.x) {
    const int c = g / N, n = g - c * N;
    float* d = reinterpret_cast<float*>(dst + (size_t)c * cstride + (size_t)n * lstride);
    int cnt = 0;
    auto put = [&](float3 p, float r) {
      float* e = d + (cnt >> 1) * 8 + (cnt & 1);
      e[0] = p.x; e[2] = p.y; e[4] = p.z; e[6] = -r;
      ++cnt;
    };
    // (the centre is read before the radius is known, so that the loads of
    // several spheres are in flight together)
#pragma unroll 4
    for (int s = 0; s < S; ++s) {
      const float r = radius(c, s, n);
      const float3 p = centre(c, s, n);
      if (r >= 0.f) put(p, r);
    }
    counts[g] = (cnt + 1) >> 1;
    if (cnt & 1) put(make_float3(0.f, 0.f, 0.f), -1e30f);
  }
}

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// Signed distances of the sphere pair (A, B) to the sphere at -(nx, ny, nz),
// its radius negated in nro: |c - o| - (r + r_o).
__device__ __forceinline__ float2 pair_sphere_dist(float4 A, float4 B, float2 nx, float2 ny, float2 nz, float2 nro) {
  const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nx), dy = __fadd2_rn(make_float2(A.z, A.w), ny),
               dz = __fadd2_rn(make_float2(B.x, B.y), nz);
  float2 d2 = __ffma2_rn(dz, dz, dup2(1e-30f));
  d2 = __ffma2_rn(dy, dy, d2);
  d2 = __ffma2_rn(dx, dx, d2);
  return __fadd2_rn(root_newton2(d2, make_float2(rsqrt_approx(d2.x), rsqrt_approx(d2.y))),
                    __fadd2_rn(make_float2(B.z, B.w), nro));
}

// ... to the box b: d_sphere_box on packed FP32x2.
__device__ __forceinline__ float2 pair_box_dist(float4 A, float4 B, const float (&b)[15]) {
  const float2 dx = __fadd2_rn(make_float2(A.x, A.y), dup2(-b[0]));
  const float2 dy = __fadd2_rn(make_float2(A.z, A.w), dup2(-b[1]));
  const float2 dz = __fadd2_rn(make_float2(B.x, B.y), dup2(-b[2]));
  float2 q[3], m[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float2 l = __fmul2_rn(dx, dup2(b[3 + 3 * i]));
    l = __ffma2_rn(dy, dup2(b[4 + 3 * i]), l);
    l = __ffma2_rn(dz, dup2(b[5 + 3 * i]), l);
    q[i] = make_float2(fabsf(l.x) - b[12 + i], fabsf(l.y) - b[12 + i]);
    m[i] = make_float2(fmaxf(q[i].x, 0.f), fmaxf(q[i].y, 0.f));
  }
  float2 x = __fmul2_rn(m[0], m[0]);
  x = __ffma2_rn(m[1], m[1], x);
  x = __ffma2_rn(m[2], m[2], x);
  const float2 xe = __fadd2_rn(x, dup2(1e-30f));
  const float2 out = root_newton2(x, make_float2(rsqrt_approx(xe.x), rsqrt_approx(xe.y)));
  const float2 in = make_float2(fminf(fmaxf(fmaxf(q[0].x, q[1].x), q[2].x), 0.f),
                                fminf(fmaxf(fmaxf(q[0].y, q[1].y), q[2].y), 0.f));
  return __fadd2_rn(__fadd2_rn(out, in), make_float2(B.z, B.w));
}

struct LinkRowArgs {
  WorldArgs w;
  const float* centers;  // [3, B, S * N]
  const float* radii;    // [B, S * N]
  float* out;            // [B, N, M]
  long long B;
  int N, S, cpb, stage;
};

__host__ __device__ inline size_t link_rows_smem(int cpb, int N, int S) {
  return ((sizeof(float4) * 2 * (size_t)N * link_pair_count(S) + sizeof(int) * (size_t)N) * cpb + 15) & ~size_t(15);
}

// Per-link minimum over the spheres of every link: [B, N, M].  The lanes walk
// the (row, obstacle) pairs of one obstacle kind at a time, rows being the
// (configuration, link) pairs of the block, so they stay full whatever the
// counts and never mix kinds; a lane holds its obstacle (four, for spheres,
// nq columns apart so that loads and stores are consecutive over the lanes)
// in registers while it runs over the link's sphere pairs.  gridDim.y blocks
// share the pairs of their configurations.
__global__ void __launch_bounds__(256, 3) link_rows_kernel(LinkRowArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = a.N, S = a.S, SP = link_pair_count(S);
  float4* centres = reinterpret_cast<float4*>(smem_raw);
  int* counts = reinterpret_cast<int*>(centres + (size_t)a.cpb * 2 * N * SP);
  const long long b0 = (long long)blockIdx.x * a.cpb;
  const int nc = (int)min((long long)a.cpb, a.B - b0);
  const long long K = (long long)S * N, BK = a.B * K;
  const float* cen = a.centers + b0 * K;
  const float* rad = a.radii + b0 * K;
  pack_link_pairs(centres, counts, nc, N, S, 2 * N * SP, 2 * SP,
                  [&](int c, int s, int n) {
                    const long long q = c * K + (long long)s * N + n;
                    return make_float3(__ldg(cen + q), __ldg(cen + BK + q), __ldg(cen + 2 * BK + q));
                  },
                  [&](int c, int s, int n) { return __ldg(rad + c * K + (long long)s * N + n); });
  ObsView ob;
  if (a.stage) {
    ob = stage_world(a.w, reinterpret_cast<float*>(smem_raw + link_rows_smem(a.cpb, N, S)));
  } else {
    ob.sph = reinterpret_cast<const float4*>(a.w.spheres);
    ob.cap = a.w.capsules; ob.box = a.w.boxes; ob.hs = a.w.halfspaces;
    ob.Ms = a.w.Ms; ob.Mc = a.w.Mc; ob.Mb = a.w.Mb; ob.Mh = a.w.Mh;
  }
  __syncthreads();
  const int M = a.w.total(), rows = nc * N, tid = blockIdx.y * blockDim.x + threadIdx.x, T = gridDim.y * blockDim.x;
  float* out = a.out + b0 * N * (long long)M;

  const int nq = (ob.Ms + 3) >> 2;
  for (int e = tid; e < rows * nq; e += T) {
    const int row = e / nq, q0 = e - row * nq;
    float2 nx[4], ny[4], nz[4], nro[4];
    float d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 o = ob.sph[min(q0 + u * nq, ob.Ms - 1)];
      nx[u] = dup2(-o.x); ny[u] = dup2(-o.y); nz[u] = dup2(-o.z); nro[u] = dup2(-o.w);
      d[u] = 1e9f;
    }
    const float4* pr = centres + (size_t)row * 2 * SP;
    const int np = counts[row];
    for (int q = 0; q < np; ++q) {
      const float4 A = pr[2 * q], B = pr[2 * q + 1];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 t = pair_sphere_dist(A, B, nx[u], ny[u], nz[u], nro[u]);
        d[u] = fminf(d[u], fminf(t.x, t.y));
      }
    }
    float* o = out + (long long)row * M + q0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * nq < ob.Ms) __stcs(o + u * nq, d[u]);
  }
  int base = ob.Ms;
  for (int e = tid; e < rows * ob.Mc; e += T) {
    const int row = e / ob.Mc, m = e - row * ob.Mc;
    const float* cp = ob.cap + 7 * m;
    const float ax = cp[0], ay = cp[1], az = cp[2], vx = cp[3] - ax, vy = cp[4] - ay, vz = cp[5] - az, rc = cp[6];
    const float len2 = vx * vx + vy * vy + vz * vz;
    const float il2 = len2 > 1e-12f ? 1.f / len2 : 0.f;
    auto dist = [&](float x, float y, float z, float nr) {
      const float t = fmaxf(0.f, fminf(1.f, ((x - ax) * vx + (y - ay) * vy + (z - az) * vz) * il2));
      const float px = ax + t * vx - x, py = ay + t * vy - y, pz = az + t * vz - z;
      const float d2 = px * px + py * py + pz * pz;
      return root_newton(d2, rsqrt_approx(d2 + 1e-30f)) + (nr - rc);
    };
    const float4* pr = centres + (size_t)row * 2 * SP;
    const int np = counts[row];
    float d = 1e9f;
    for (int q = 0; q < np; ++q) {
      const float4 A = pr[2 * q], B = pr[2 * q + 1];
      d = fminf(d, fminf(dist(A.x, A.z, B.x, B.z), dist(A.y, A.w, B.y, B.w)));
    }
    __stcs(out + (long long)row * M + base + m, d);
  }
  base += ob.Mc;
  for (int e = tid; e < rows * ob.Mb; e += T) {
    const int row = e / ob.Mb, m = e - row * ob.Mb;
    float b[15];
#pragma unroll
    for (int i = 0; i < 15; ++i) b[i] = ob.box[15 * m + i];
    const float4* pr = centres + (size_t)row * 2 * SP;
    const int np = counts[row];
    float d = 1e9f;
    for (int q = 0; q < np; ++q) {
      const float2 t = pair_box_dist(pr[2 * q], pr[2 * q + 1], b);
      d = fminf(d, fminf(t.x, t.y));
    }
    __stcs(out + (long long)row * M + base + m, d);
  }
  base += ob.Mb;
  for (int e = tid; e < rows * ob.Mh; e += T) {
    const int row = e / ob.Mh, m = e - row * ob.Mh;
    const float* h = ob.hs + 6 * m;
    const float4* pr = centres + (size_t)row * 2 * SP;
    const int np = counts[row];
    float d = 1e9f;
    for (int q = 0; q < np; ++q) {
      const float4 A = pr[2 * q], B = pr[2 * q + 1];
      d = fminf(d, d_sphere_halfspace(make_float3(A.x, A.z, B.x), -B.z, h));
      if (B.w <= 0.f) d = fminf(d, d_sphere_halfspace(make_float3(A.y, A.w, B.y), -B.w, h));  // not the odd slot
    }
    __stcs(out + (long long)row * M + base + m, d);
  }
}

// MODE 0: per-sphere rows [B,K,M]; MODE 1: per-link min over s [B,N,M];
// MODE 2: capsule robot rows [B,N,M].
template <int MODE>
__global__ void __launch_bounds__(256) world_rows_kernel(RowArgs a) {
  extern __shared__ __align__(16) float smem_f[];
  const ObsView ob = world_view(a, smem_f);
  __syncthreads();
  const int M = a.w.total();
  const int lpr = a.lpr;
  const int rows_per_block = blockDim.x / lpr;
  const int sub = threadIdx.x / lpr, sl = threadIdx.x - sub * lpr;
  const long long R = a.B * (long long)a.K;  // rows (b, k) or (b, n)
  const long long row = (long long)blockIdx.x * rows_per_block + sub;
  if (row >= R) return;
  const long long b = row / a.K;
  const int k = (int)(row - b * a.K);
  float* orow = a.out + row * (long long)M;
  const bool vec4 = ((M & 3) == 0) && ((reinterpret_cast<uintptr_t>(a.out) & 15) == 0);

  if (MODE == 0) {
    const long long BK = a.B * (long long)a.K;
    const float r = __ldg(a.radii + row);
    const float3 c = make_float3(__ldg(a.centers + row), __ldg(a.centers + BK + row),
                                 __ldg(a.centers + 2 * BK + row));
    if (vec4) {
      for (int m0 = sl * 4; m0 < M; m0 += lpr * 4) {
        float4 d;
        if (r < 0.f) {
          d = make_float4(1e9f, 1e9f, 1e9f, 1e9f);
        } else {
          d.x = obstacle_dist(ob, m0, c, r);
          d.y = obstacle_dist(ob, m0 + 1, c, r);
          d.z = obstacle_dist(ob, m0 + 2, c, r);
          d.w = obstacle_dist(ob, m0 + 3, c, r);
        }
        __stcs(reinterpret_cast<float4*>(orow + m0), d);
      }
    } else {
      for (int m0 = sl; m0 < M; m0 += lpr) orow[m0] = (r < 0.f) ? 1e9f : obstacle_dist(ob, m0, c, r);
    }
  } else if (MODE == 1) {
    // row = (b, n); sphere k = s*N + n
    const long long BK = a.B * (long long)a.S * a.N;
    const long long kb = b * (long long)a.S * a.N + k;
    for (int m0 = sl * 4; m0 < M; m0 += lpr * 4) {
      float d0 = 1e9f, d1 = 1e9f, d2 = 1e9f, d3 = 1e9f;
      for (int s = 0; s < a.S; ++s) {
        const long long q = kb + (long long)s * a.N;
        const float r = __ldg(a.radii + q);
        if (r < 0.f) continue;
        const float3 c = make_float3(__ldg(a.centers + q), __ldg(a.centers + BK + q),
                                     __ldg(a.centers + 2 * BK + q));
        d0 = fminf(d0, obstacle_dist(ob, m0, c, r));
        if (m0 + 1 < M) d1 = fminf(d1, obstacle_dist(ob, m0 + 1, c, r));
        if (m0 + 2 < M) d2 = fminf(d2, obstacle_dist(ob, m0 + 2, c, r));
        if (m0 + 3 < M) d3 = fminf(d3, obstacle_dist(ob, m0 + 3, c, r));
      }
      if (vec4) {
        __stcs(reinterpret_cast<float4*>(orow + m0), make_float4(d0, d1, d2, d3));
      } else {
        orow[m0] = d0;
        if (m0 + 1 < M) orow[m0 + 1] = d1;
        if (m0 + 2 < M) orow[m0 + 2] = d2;
        if (m0 + 3 < M) orow[m0 + 3] = d3;
      }
    }
  } else {
    // capsule robot: caps [7, B, N] SoA; row = (b, n)
    float cap[7];
#pragma unroll
    for (int c = 0; c < 7; ++c) cap[c] = __ldg(a.centers + (long long)c * R + row);
    for (int m0 = sl; m0 < M; m0 += lpr) {
      int m = m0;
      float d;
      if (m < ob.Ms) {
        // sphere-capsule with the world sphere as the sphere argument
        const float4 s = ob.sph[m];
        d = d_sphere_capsule(make_float3(s.x, s.y, s.z), s.w, cap);
      } else if ((m -= ob.Ms) < ob.Mc) {
        d = d_capsule_capsule(cap, ob.cap + 7 * m);
      } else if ((m -= ob.Mc) < ob.Mb) {
        d = d_capsule_box(cap, ob.box + 15 * m);
      } else {
        m -= ob.Mb;
        d = d_capsule_halfspace(cap, ob.hs + 6 * m);
      }
      orow[m0] = d;
    }
  }
}

// Self-collision, sphere robot: centers [B,S,N,3], radii [B,S,N]; one thread
// per (b, p), the block's configurations next to each other in a warp: they
// share the pair and mostly its sphere counts, so the warp's loops agree.  The
// packed links take an odd number of float4, a configuration 1 more than a
// multiple of 8, so the eight 16-byte reads of a quarter warp mostly hit
// different banks.
__host__ __device__ inline int self_pairs_cstride(int N, int S) {
  return ((N * (2 * link_pair_count(S) + 1) + 6) & ~7) + 1;
}
__host__ __device__ inline size_t self_pairs_smem(int cpb, int N, int S) {
  return (sizeof(float4) * (size_t)self_pairs_cstride(N, S) + sizeof(int) * (size_t)N) * cpb;
}

__global__ void __launch_bounds__(256, 4) self_pairs_kernel(const float* __restrict__ centers,
                                                            const float* __restrict__ radii,
                                                            const int* __restrict__ pair_i,
                                                            const int* __restrict__ pair_j, float* __restrict__ out,
                                                            long long B, int S, int N, int P, int cpb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int LS = 2 * link_pair_count(S) + 1, CS = self_pairs_cstride(N, S);
  float4* sph = reinterpret_cast<float4*>(smem_raw);
  int* counts = reinterpret_cast<int*>(sph + (size_t)cpb * CS);
  const long long b0 = (long long)blockIdx.x * cpb;
  const int nc = (int)min((long long)cpb, B - b0);
  const long long SN = (long long)S * N;
  pack_link_pairs(sph, counts, nc, N, S, CS, LS,
                  [&](int c, int s, int n) {
                    const float* q = centers + 3 * ((b0 + c) * SN + (long long)s * N + n);
                    return make_float3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
                  },
                  [&](int c, int s, int n) { return __ldg(radii + (b0 + c) * SN + (long long)s * N + n); });
  __syncthreads();
  for (int g = threadIdx.x; g < nc * P; g += blockDim.x) {
    const int p = g / nc, c = g - p * nc;
    const int li = __ldg(pair_i + p), lj = __ldg(pair_j + p);
    float dmin = 1e9f;
    if (li >= 0 && li < N && lj >= 0 && lj < N) {  // else an invalid link index: no pair
      const float4* Ai = sph + (size_t)c * CS + (size_t)li * LS;
      const float4* Bj = sph + (size_t)c * CS + (size_t)lj * LS;
      const int na = counts[c * N + li], nb = counts[c * N + lj];
      // two spheres of li against the pairs of lj (the odd slot of li not taken)
      for (int q = 0; q < na; ++q) {
        const float4 A = Ai[2 * q], Av = Ai[2 * q + 1];
        const float2 x0 = dup2(-A.x), y0 = dup2(-A.z), z0 = dup2(-Av.x), r0 = dup2(Av.z);
        const float2 x1 = dup2(-A.y), y1 = dup2(-A.w), z1 = dup2(-Av.y), r1 = dup2(Av.w);
        const bool two = Av.w <= 0.f;
        for (int k = 0; k < nb; ++k) {
          const float4 Bq = Bj[2 * k], Bv = Bj[2 * k + 1];
          const float2 t0 = pair_sphere_dist(Bq, Bv, x0, y0, z0, r0);
          const float2 t1 = pair_sphere_dist(Bq, Bv, x1, y1, z1, r1);
          dmin = fminf(dmin, fminf(t0.x, t0.y));
          if (two) dmin = fminf(dmin, fminf(t1.x, t1.y));
        }
      }
    }
    out[(b0 + c) * P + p] = dmin;
  }
}

// The same with one sphere at a time from unpacked spheres, for robots whose
// packed links do not fit in shared memory.
__global__ void __launch_bounds__(256) self_sphere_kernel(const float* __restrict__ centers,
                                                          const float* __restrict__ radii,
                                                          const int* __restrict__ pair_i,
                                                          const int* __restrict__ pair_j,
                                                          float* __restrict__ out, long long B, int S,
                                                          int N, int P, int cpb) {
  extern __shared__ __align__(16) float4 sph[];  // [cpb][S*N] (x,y,z,r)
  const int SN = S * N;
  const long long b0 = (long long)blockIdx.x * cpb;
  const int nc = (int)min((long long)cpb, B - b0);
  for (int g = threadIdx.x; g < nc * SN; g += blockDim.x) {
    const long long e = b0 * SN + g;
    sph[g] = make_float4(__ldg(centers + 3 * e), __ldg(centers + 3 * e + 1), __ldg(centers + 3 * e + 2),
                         __ldg(radii + e));
  }
  __syncthreads();
  for (int g = threadIdx.x; g < nc * P; g += blockDim.x) {
    const int c = g / P, p = g - c * P;
    const int li = __ldg(pair_i + p), lj = __ldg(pair_j + p);
    const float4* base = sph + c * SN;
    float dmin = 1e9f;
    if (li < 0 || li >= N || lj < 0 || lj >= N) {  // invalid link index: no pair
      out[(b0 + c) * P + p] = dmin;
      continue;
    }
    for (int si = 0; si < S; ++si) {
      const float4 A = base[si * N + li];
      if (A.w < 0.f) continue;
      for (int sj = 0; sj < S; ++sj) {
        const float4 Bq = base[sj * N + lj];
        if (Bq.w < 0.f) continue;
        dmin = fminf(dmin, d_sphere_sphere(make_float3(A.x, A.y, A.z), A.w, Bq.x, Bq.y, Bq.z, Bq.w));
      }
    }
    out[(b0 + c) * P + p] = dmin;
  }
}

__global__ void __launch_bounds__(256) self_capsule_kernel(const float* __restrict__ caps,
                                                           const int* __restrict__ pair_i,
                                                           const int* __restrict__ pair_j,
                                                           float* __restrict__ out, long long B, int N,
                                                           int P) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= B * P) return;
  const long long b = idx / P;
  const int p = (int)(idx - b * P);
  const int li = __ldg(pair_i + p), lj = __ldg(pair_j + p);
  if (li < 0 || li >= N || lj < 0 || lj >= N) {  // invalid link index: no pair
    out[idx] = 1e9f;
    return;
  }
  float A[7], Bc[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    A[c] = __ldg(caps + (b * N + li) * 7 + c);
    Bc[c] = __ldg(caps + (b * N + lj) * 7 + c);
  }
  out[idx] = d_capsule_capsule(A, Bc);
}

static const size_t kWorldSmemLimit = 128 * 1024;

static int check_world(const WorldArgs& w) {
  PK_CHECK_ARG(w.Ms >= 0 && w.Mc >= 0 && w.Mb >= 0 && w.Mh >= 0, "negative obstacle count");
  PK_CHECK_ARG((w.Ms == 0 || w.spheres) && (w.Mc == 0 || w.capsules) && (w.Mb == 0 || w.boxes) &&
                   (w.Mh == 0 || w.halfspaces),
               "null world buffer");
  return PK_OK;
}

template <int MODE>
static int launch_rows(cudaStream_t stream, RowArgs a) {
  const int M = a.w.total();
  a.lpr = lanes_per_row(M);
  const size_t wbytes = sizeof(float) * a.w.smem_floats();
  a.stage = wbytes <= kWorldSmemLimit ? 1 : 0;
  PK_CHECK_ARG(a.stage || a.w.spheres == nullptr ||
                   (reinterpret_cast<uintptr_t>(a.w.spheres) & 15) == 0,
               "world_spheres must be 16-byte aligned when the world exceeds shared memory");
  const int threads = 256;
  const int rpb = threads / a.lpr;
  const long long rows = a.B * (long long)a.K;
  const long long blocks = (rows + rpb - 1) / rpb;
  PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
  const size_t smem = a.stage ? wbytes : 0;
  if (int st = set_smem_limit((const void*)world_rows_kernel<MODE>, smem)) return st;
  world_rows_kernel<MODE><<<(unsigned)blocks, threads, smem, stream>>>(a);
  return cuda_status(cudaGetLastError(), "world_rows_kernel launch");
}

}  // namespace pk

using namespace pk;

extern "C" int pk_collision_world_sphere(void* stream, const float* centers, const float* radii,
                                         const float* world_spheres, const float* world_capsules,
                                         const float* world_boxes, const float* world_halfspaces,
                                         float* out, int64_t B, int32_t K, int32_t Ms, int32_t Mc,
                                         int32_t Mb, int32_t Mh) {
  PK_CHECK_ARG(B >= 0 && K >= 0, "negative extent");
  WorldArgs w{world_spheres, world_capsules, world_boxes, world_halfspaces, Ms, Mc, Mb, Mh};
  if (int st = check_world(w)) return st;
  if (B == 0 || K == 0 || w.total() == 0) return PK_OK;
  PK_CHECK_ARG(centers && radii && out, "null buffer");
  RowArgs a{};
  a.w = w; a.centers = centers; a.radii = radii; a.out = out; a.B = B; a.K = K;
  return launch_rows<0>((cudaStream_t)stream, a);
}

extern "C" int pk_collision_world_sphere_reduced(void* stream, const float* centers,
                                                 const float* radii, const float* world_spheres,
                                                 const float* world_capsules,
                                                 const float* world_boxes,
                                                 const float* world_halfspaces, float* out,
                                                 int64_t B, int32_t K, int32_t Ms, int32_t Mc,
                                                 int32_t Mb, int32_t Mh, int64_t n) {
  PK_CHECK_ARG(B >= 0 && K >= 0 && n >= 0, "negative extent");
  WorldArgs w{world_spheres, world_capsules, world_boxes, world_halfspaces, Ms, Mc, Mb, Mh};
  if (int st = check_world(w)) return st;
  if (B == 0 || n == 0 || w.total() == 0) return PK_OK;
  PK_CHECK_ARG(n <= K || K == 0, "n=%lld exceeds K=%d", (long long)n, K);
  PK_CHECK_ARG(centers && radii && out, "null buffer");
  RowArgs a{};
  a.w = w; a.centers = centers; a.radii = radii; a.out = out; a.B = B;
  a.N = (int)n; a.S = (int)(K / n); a.K = (int)n;
  // centers are [3, B, K]: the SoA plane stride is B*K even when K != S*N.
  // Sphere (b, s, n) sits at b*K + s*N + n; the kernel addresses b*S*N, so
  // require K == S*N as the reference does (its K / N truncation).
  PK_CHECK_ARG((long long)a.S * n == K, "K=%d is not a multiple of n=%lld", K, (long long)n);
  // The packed per-link rows wherever one configuration's spheres fit in
  // shared memory; the row kernel for larger robots.  2,048 configurations, 30
  // links x 4-12 spheres, 268 obstacles of four kinds, with the self pairs of
  // pk_collision_self_sphere: 1167 -> 212 us for both.
  LinkRowArgs r{w, centers, radii, out, B, a.N, a.S, 1, 0};
  const size_t wbytes = sizeof(float) * w.smem_floats();
  // obstacles are read once per work unit into registers, so only a small
  // world is worth a copy; unaligned spheres cannot be read as float4 in place
  const bool aligned = w.spheres == nullptr || (reinterpret_cast<uintptr_t>(w.spheres) & 15) == 0;
  r.stage = wbytes <= 48 * 1024 || (!aligned && wbytes <= kWorldSmemLimit);
  const size_t wsm = r.stage ? wbytes : 0;
  // a block counts its (row, obstacle) pairs of a kind (quads, for spheres) in
  // 32 bits, with room for the step past the last one
  constexpr long long kMostSplits = 1024;
  const long long most = (1LL << 31) - 256 * kMostSplits;
  const long long quads = (Ms + 3LL) / 4, columns = quads + Mc + Mb + Mh;
  const long long wide = std::max({quads, (long long)Mc, (long long)Mb, (long long)Mh});
  if (link_rows_smem(1, r.N, r.S) + wsm <= 200 * 1024 && (r.stage || aligned) && n * wide <= most) {
    // as many configurations per block (at most 8) as leave three blocks for
    // every SM and fit half of its shared memory
    r.cpb = 8;
    while (r.cpb > 1 && ((B + r.cpb - 1) / r.cpb < 3 * 148 || link_rows_smem(r.cpb, r.N, r.S) + wsm > 100 * 1024 ||
                         r.cpb * n * wide > most))
      r.cpb >>= 1;
    // The row kernel stays the faster one, once the batch fills the GPU,
    // - for few obstacles, which use a packed sphere once or in too few lanes:
    //   20,000 configurations of 3 links x 100 spheres among 5 capsules 200 us
    //   (packed 334), among 8 spheres 118 (348), 1 sphere 86 (149); 7 x 8, 1
    //   sphere 22 (34); 100 x 3, 1 sphere 78 (99), but 8 spheres 170 (123);
    // - for links of one sphere, half of each pair, in a world that it can
    //   stage in a third of an SM and this one cannot at all: 2,048
    //   configurations of 64 x 1 among 4,100 spheres 1,066 us (1,142).
    const long long work = B * n * columns;
    const bool few = columns == 1 ? work > 100000 || work * r.S > 4000000
                                  : r.cpb * n * columns < 256 && work > 100000;
    const bool half = r.S == 1 && !r.stage && wbytes <= 75 * 1024 && work > 100000000;
    if (!few && !half) {
      const size_t smem = link_rows_smem(r.cpb, r.N, r.S) + wsm;
      const long long blocks = (B + r.cpb - 1) / r.cpb;
      PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
      // the columns of a few configurations are split over as many blocks as
      // fill the GPU, those of a large world over four times as many, so that no
      // last wave of long blocks leaves it idle (each packs its configurations):
      // one configuration of 64 links x 1 sphere, 5,000 obstacles 109 us in one
      // block, 37 in the row kernel; 2,048 with 4,100 obstacles 1,213 and 1,067
      const long long pairs = r.cpb * n * wide, want = (pairs >= 32768 ? 4 : 1) * 3 * 148;
      const long long splits = std::max(1LL, std::min({(want + blocks - 1) / blocks, pairs / 1024, kMostSplits}));
      if (int st = set_smem_limit((const void*)link_rows_kernel, smem)) return st;
      link_rows_kernel<<<dim3((unsigned)blocks, (unsigned)splits), 256, smem, (cudaStream_t)stream>>>(r);
      return cuda_status(cudaGetLastError(), "link_rows_kernel launch");
    }
  }
  return launch_rows<1>((cudaStream_t)stream, a);
}

extern "C" int pk_collision_world_capsule(void* stream, const float* caps,
                                          const float* world_spheres, const float* world_capsules,
                                          const float* world_boxes, const float* world_halfspaces,
                                          float* out, int64_t B, int32_t N, int32_t Ms, int32_t Mc,
                                          int32_t Mb, int32_t Mh) {
  PK_CHECK_ARG(B >= 0 && N >= 0, "negative extent");
  WorldArgs w{world_spheres, world_capsules, world_boxes, world_halfspaces, Ms, Mc, Mb, Mh};
  if (int st = check_world(w)) return st;
  if (B == 0 || N == 0 || w.total() == 0) return PK_OK;
  PK_CHECK_ARG(caps && out, "null buffer");
  RowArgs a{};
  a.w = w; a.centers = caps; a.out = out; a.B = B; a.K = N;
  return launch_rows<2>((cudaStream_t)stream, a);
}

extern "C" int pk_collision_self_sphere(void* stream, const float* centers, const float* radii,
                                        const int32_t* pair_i, const int32_t* pair_j, float* out,
                                        int64_t B, int32_t S, int32_t N, int32_t P) {
  PK_CHECK_ARG(B >= 0 && S >= 0 && N >= 0 && P >= 0, "negative extent");
  if (B == 0 || P == 0) return PK_OK;
  PK_CHECK_ARG(centers && radii && pair_i && pair_j && out, "null buffer");
  // Packed links wherever a configuration's fit in shared memory, but for few
  // pairs of links of up to three spheres, which do not repay the packing:
  // 100,000 configurations of 64 links x 1 sphere, 1 pair 46 us (packed 72), 100
  // pairs 108 (123), 500 pairs 331 (304); 100 x 3, 20 pairs 231 (314), 100 pairs
  // 394 (384); 30 x 2, 5 pairs 45 (61).  With four spheres or more the packed
  // kernel is the faster one from one pair on.
  const bool few = S <= 3 && (long long)P * S < 2LL * N && (size_t)S * N * sizeof(float4) <= 96 * 1024;
  if (!few && self_pairs_smem(1, N, S) <= 200 * 1024) {
    // as for the reduced rows; 16 configurations of a small robot
    int cpb = 16;
    while (cpb > 1 &&
           ((B + cpb - 1) / cpb < 3 * 148 || self_pairs_smem(cpb, N, S) > (cpb > 8 ? 20 : 56) * 1024))
      cpb >>= 1;
    const size_t smem = self_pairs_smem(cpb, N, S);
    const long long blocks = (B + cpb - 1) / cpb;
    PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
    if (int st = set_smem_limit((const void*)self_pairs_kernel, smem)) return st;
    self_pairs_kernel<<<(unsigned)blocks, 256, smem, (cudaStream_t)stream>>>(centers, radii, pair_i, pair_j, out, B, S,
                                                                              N, P, cpb);
    return cuda_status(cudaGetLastError(), "self_pairs_kernel launch");
  }
  const int SN = S * N;
  int cpb = 64;
  while (cpb > 1 && (size_t)cpb * SN * sizeof(float4) > 96 * 1024) cpb >>= 1;
  PK_CHECK_CAP((size_t)cpb * SN * sizeof(float4) <= 96 * 1024, "S*N=%d too large", SN);
  const size_t smem = (size_t)cpb * SN * sizeof(float4);
  const long long blocks = (B + cpb - 1) / cpb;
  PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
  if (int st = set_smem_limit((const void*)self_sphere_kernel, smem)) return st;
  self_sphere_kernel<<<(unsigned)blocks, 256, smem, (cudaStream_t)stream>>>(centers, radii, pair_i,
                                                                             pair_j, out, B, S, N, P, cpb);
  return cuda_status(cudaGetLastError(), "self_sphere_kernel launch");
}

extern "C" int pk_collision_self_capsule(void* stream, const float* caps, const int32_t* pair_i,
                                         const int32_t* pair_j, float* out, int64_t B, int32_t N,
                                         int32_t P) {
  PK_CHECK_ARG(B >= 0 && N >= 0 && P >= 0, "negative extent");
  if (B == 0 || P == 0) return PK_OK;
  PK_CHECK_ARG(caps && pair_i && pair_j && out, "null buffer");
  const long long total = B * (long long)P;
  const long long blocks = (total + 255) / 256;
  PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
  self_capsule_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(caps, pair_i, pair_j, out, B,
                                                                            N, P);
  return cuda_status(cudaGetLastError(), "self_capsule_kernel launch");
}
