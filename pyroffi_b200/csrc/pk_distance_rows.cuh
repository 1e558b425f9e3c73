// Distance rows of a block of configurations against the obstacle world:
// per-sphere rows [., K, M] or per-link minima [., N, M], from robot sphere
// centres in shared memory.  Shared by the fused FK -> distance kernel
// (pk_fk.cu) and the drop-in distance kernels (pk_collision.cu).
#pragma once

#include "pk_obstacles.cuh"

namespace pk {

// Robot spheres of one block, in shared memory.  Per-sphere rows (PER_LINK
// false): float4 (x, y, z, r) of sphere k of configuration c at
// centres[c * N * S + k], r < 0 marking padding.  Per-link rows: the spheres
// that exist, in pairs (see link_pair_count), link k's pairs of configuration
// c counted in pairs[c * pair_stride + k] (pair_stride 0: the same for every
// configuration).
struct RowSpheres {
  const float4* centres;
  const int* pairs;
  int pair_stride;
  int N, S;
};

// sqrt(x) of x >= 1e-30 (or x = 0 with `tiny` added) from the approximate
// reciprocal square root; PRECISE adds one Newton step on the root, which
// leaves it within an ulp of the correctly rounded value (the approximation
// alone is a few ulp off).
template <bool PRECISE>
__device__ __forceinline__ float root_of(float x, float y) {
  const float s = x * y;
  if (!PRECISE) return s;
  return fmaf(fmaf(-s, s, x), 0.5f * y, s);
}
template <bool PRECISE>
__device__ __forceinline__ float2 root_of2(float2 x, float2 y) {
  const float2 s = __fmul2_rn(x, y);
  if (!PRECISE) return s;
  const float2 e = __ffma2_rn(make_float2(-s.x, -s.y), s, x);
  return __ffma2_rn(e, __fmul2_rn(y, make_float2(0.5f, 0.5f)), s);
}

// |c - o| for a robot sphere centre c and obstacle sphere o.
template <bool PRECISE = false>
__device__ __forceinline__ float centre_dist(float4 c, float4 o) {
  const float dx = c.x - o.x, dy = c.y - o.y, dz = c.z - o.z;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, 1e-30f)));
  return root_of<PRECISE>(d2, rsqrt_approx(d2));
}

// One obstacle held in registers by a lane: kind 0 sphere (x, y, z, r),
// 1 capsule (p1, p2, r, 1/|p2 - p1|^2 or 0), 2 box (centre, axis columns,
// half-lengths), 3 halfspace (n, n . p0, p0).
struct ObsReg {
  int kind;
  float p[15];
};

__device__ __forceinline__ ObsReg load_obstacle(const ObsView& ob, int m) {
  ObsReg o;
#pragma unroll
  for (int i = 0; i < 15; ++i) o.p[i] = 0.f;
  if (m < ob.Ms) {
    o.kind = 0;
    const float4 s = ob.sph[m];
    o.p[0] = s.x; o.p[1] = s.y; o.p[2] = s.z; o.p[3] = s.w;
    return o;
  }
  m -= ob.Ms;
  if (m < ob.Mc) {
    o.kind = 1;
#pragma unroll
    for (int i = 0; i < 7; ++i) o.p[i] = ob.cap[7 * m + i];
    const float vx = o.p[3] - o.p[0], vy = o.p[4] - o.p[1], vz = o.p[5] - o.p[2];
    const float len2 = vx * vx + vy * vy + vz * vz;
    o.p[7] = (len2 > 1e-12f) ? 1.f / len2 : 0.f;
    return o;
  }
  m -= ob.Mc;
  if (m < ob.Mb) {
    o.kind = 2;
#pragma unroll
    for (int i = 0; i < 15; ++i) o.p[i] = ob.box[15 * m + i];
    return o;
  }
  m -= ob.Mb;
  o.kind = 3;
  const float* h = ob.hs + 6 * m;
  o.p[0] = h[0]; o.p[1] = h[1]; o.p[2] = h[2];
  o.p[3] = h[3] * h[0] + h[4] * h[1] + h[5] * h[2];
  o.p[4] = h[3]; o.p[5] = h[4]; o.p[6] = h[5];
  return o;
}

// Signed distance from sphere (c, r) to a register obstacle of a known kind.
template <int KIND, bool PRECISE = false>
__device__ __forceinline__ float reg_dist(const ObsReg& o, float4 c) {
  if (KIND == 0) {
    return centre_dist<PRECISE>(c, make_float4(o.p[0], o.p[1], o.p[2], 0.f)) - (c.w + o.p[3]);
  } else if (KIND == 1) {
    const float vx = o.p[3] - o.p[0], vy = o.p[4] - o.p[1], vz = o.p[5] - o.p[2];
    float t = ((c.x - o.p[0]) * vx + (c.y - o.p[1]) * vy + (c.z - o.p[2]) * vz) * o.p[7];
    t = fmaxf(0.f, fminf(1.f, t));
    const float px = fmaf(t, vx, o.p[0]) - c.x, py = fmaf(t, vy, o.p[1]) - c.y, pz = fmaf(t, vz, o.p[2]) - c.z;
    const float d2 = px * px + py * py + pz * pz;
    return root_of<PRECISE>(d2, rsqrt_approx(d2 + 1e-30f)) - (c.w + o.p[6]);
  } else if (KIND == 2) {
    const float dx = c.x - o.p[0], dy = c.y - o.p[1], dz = c.z - o.p[2];
    const float q1 = fabsf(dx * o.p[3] + dy * o.p[4] + dz * o.p[5]) - o.p[12];
    const float q2 = fabsf(dx * o.p[6] + dy * o.p[7] + dz * o.p[8]) - o.p[13];
    const float q3 = fabsf(dx * o.p[9] + dy * o.p[10] + dz * o.p[11]) - o.p[14];
    const float m1 = fmaxf(q1, 0.f), m2 = fmaxf(q2, 0.f), m3 = fmaxf(q3, 0.f);
    const float d2 = m1 * m1 + m2 * m2 + m3 * m3;
    return root_of<PRECISE>(d2, rsqrt_approx(d2 + 1e-30f)) + fminf(fmaxf(fmaxf(q1, q2), q3), 0.f) - c.w;
  } else {
    if (PRECISE) return (c.x - o.p[4]) * o.p[0] + (c.y - o.p[5]) * o.p[1] + (c.z - o.p[6]) * o.p[2] - c.w;
    return c.x * o.p[0] + c.y * o.p[1] + c.z * o.p[2] - o.p[3] - c.w;
  }
}

// Per-link rows read each link's spheres in pairs, so that the sphere-quad
// loop runs on packed FP32x2 arithmetic: the link's spheres that exist (radius
// >= 0), packed to the front, and for spheres 2q and 2q + 1 of them, link k,
// configuration c, float4 A = (x0, x1, y0, y1) and B = (z0, z1, -r0, -r1) at
// centres[((c * N + k) * SP + q) * 2 + {0, 1}], SP = ceil(S / 2).  The odd slot
// of an odd count is stored at 1e18 with -r = 1: its packed distances
// (~1.7e18) never win the minimum, and the scalar rows skip it by its radius.
__host__ __device__ __forceinline__ int link_pair_count(int S) { return (S + 1) >> 1; }

// Signed distances of the sphere pair (A, B) in the link-pair layout to a
// register box: reg_dist<2> on packed FP32x2, the projections written as
// fma(dz, a_z, fma(dy, a_y, dx * a_x)).
template <bool PRECISE>
__device__ __forceinline__ float2 box_dist2(const ObsReg& o, float4 A, float4 B) {
  const float2 dx = __fadd2_rn(make_float2(A.x, A.y), make_float2(-o.p[0], -o.p[0]));
  const float2 dy = __fadd2_rn(make_float2(A.z, A.w), make_float2(-o.p[1], -o.p[1]));
  const float2 dz = __fadd2_rn(make_float2(B.x, B.y), make_float2(-o.p[2], -o.p[2]));
  float2 q[3], m[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float ax = o.p[3 + 3 * i], ay = o.p[4 + 3 * i], az = o.p[5 + 3 * i], h = o.p[12 + i];
    float2 l = __fmul2_rn(dx, make_float2(ax, ax));
    l = __ffma2_rn(dy, make_float2(ay, ay), l);
    l = __ffma2_rn(dz, make_float2(az, az), l);
    q[i] = make_float2(fabsf(l.x) - h, fabsf(l.y) - h);
    m[i] = make_float2(fmaxf(q[i].x, 0.f), fmaxf(q[i].y, 0.f));
  }
  float2 x = __fmul2_rn(m[0], m[0]);
  x = __ffma2_rn(m[1], m[1], x);
  x = __ffma2_rn(m[2], m[2], x);
  const float2 xe = __fadd2_rn(x, make_float2(1e-30f, 1e-30f));
  const float2 out = root_of2<PRECISE>(x, make_float2(rsqrt_approx(xe.x), rsqrt_approx(xe.y)));
  const float2 in = make_float2(fminf(fmaxf(fmaxf(q[0].x, q[1].x), q[2].x), 0.f),
                                fminf(fmaxf(fmaxf(q[0].y, q[1].y), q[2].y), 0.f));
  return __fadd2_rn(__fadd2_rn(out, in), make_float2(B.z, B.w));
}

// Rows of one configuration against one register obstacle (a single column
// m per lane): per-sphere rows (R = K) or per-link minima (R = N).  Returns
// the lane's minimum; stores go to o, o + M, ... when `store`.
template <bool PER_LINK, int KIND, bool PRECISE>
__device__ __forceinline__ float single_rows(const ObsReg& ob, const float4* cc, const int* pairs, int S, int R,
                                             float* o, int M, bool store) {
  float vmin = 1e9f;
  const int SP = link_pair_count(S);
  for (int k = 0; k < R; ++k) {
    float d = 1e9f;
    if (PER_LINK) {
      const int np = pairs[k];
      for (int q = 0; q < np; ++q) {
        const float4 A = cc[(k * SP + q) * 2], B = cc[(k * SP + q) * 2 + 1];
        if (KIND == 2) {
          // boxes on packed FP32x2 over the sphere pair; the odd slot is far
          // away and masked by its radius
          const float2 t = box_dist2<PRECISE>(ob, A, B);
          if (B.z <= 0.f) d = fminf(d, t.x);
          if (B.w <= 0.f) d = fminf(d, t.y);
        } else {
          const float4 c0 = make_float4(A.x, A.z, B.x, -B.z), c1 = make_float4(A.y, A.w, B.y, -B.w);
          if (c0.w >= 0.f) d = fminf(d, reg_dist<KIND, PRECISE>(ob, c0));
          if (c1.w >= 0.f) d = fminf(d, reg_dist<KIND, PRECISE>(ob, c1));
        }
      }
    } else {
      const float4 ce = cc[k];
      if (ce.w >= 0.f) d = reg_dist<KIND, PRECISE>(ob, ce);
    }
    vmin = fminf(vmin, d);
    if (store) o[(long long)k * M] = d;
  }
  return vmin;
}

// Distance rows of one block.  Block row (c, k) is configuration c and
// robot sphere k (R = K, output [B, K, M]) or link k (R = N, PER_LINK,
// output [B, N, M] = min over the link's S spheres); the M columns are the
// obstacles.  Columns come in two kinds of tile:
//  * sphere quads: the first Ms4 = 4 * floor(Ms / 4) columns; a lane owns
//    4 consecutive sphere obstacles in registers, lpr lanes cover a row
//    (lpr * 4 >= Ms4 when that is small, so short rows pack 32 / lpr rows per
//    warp) and rows stream past as shared-memory broadcasts; 16-byte
//    streaming stores;
//  * singles: the remaining columns (sphere tail, capsules, boxes,
//    halfspaces), one obstacle per lane in registers, 32 consecutive columns
//    per tile, coalesced 4-byte stores.
// Work units (tile, chunk of configurations) are spread over the warps.
// After each configuration the warp reduces its minimum by shuffles and
// folds it into cmin[c] with one atomic.  Padding spheres (radius < 0) give
// 1e9 in [B, K, M] and are skipped in the per-link minimum (a link without
// spheres gives 1e9).
template <bool PER_LINK, bool PRECISE = false>
__device__ __forceinline__ void distance_rows(const RowSpheres& rs, const ObsView& ob, int* cmin, long long b0,
                                              int nc, float* out, bool do_min) {
  const int N = rs.N, S = rs.S, K = N * S;
  const int SP = link_pair_count(S);
  const int CK = PER_LINK ? 2 * N * SP : K;  // float4 per configuration
  const int M = ob.Ms + ob.Mc + ob.Mb + ob.Mh;
  const int R = PER_LINK ? N : K;
  if (M == 0 || R == 0 || nc == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int Ms4 = ob.Ms & ~3;
  const int quads = Ms4 >> 2;
  int lpr = 1;
  while (lpr < 32 && lpr < quads) lpr <<= 1;
  const int rpw = 32 / lpr;
  const int sub = lane / lpr, sl = lane - sub * lpr;
  const int ntq = (quads + lpr - 1) / lpr;
  const int nts = (M - Ms4 + 31) / 32;
  const int nt = ntq + nts;
  int nchunk = min(nc, max(1, (16 * nwarps + nt - 1) / nt));
  const int cchunk = (nc + nchunk - 1) / nchunk;
  nchunk = (nc + cchunk - 1) / cchunk;
  const bool vec = out && ((M & 3) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);

  for (int u = warp; u < nt * nchunk; u += nwarps) {
    const int tile = u % nt, chunk = u / nt;
    const bool is_quad = tile < ntq;
    const int m0 = is_quad ? 4 * (tile * lpr + sl) : Ms4 + 32 * (tile - ntq) + lane;
    const bool active = is_quad ? (m0 < Ms4) : (m0 < M);
    const bool store = out != nullptr && active;
    float4 o0 = make_float4(0.f, 0.f, 0.f, 0.f), o1 = o0, o2 = o0, o3 = o0;
    ObsReg single;
    single.kind = -1;
    if (is_quad && active) {
      o0 = ob.sph[m0]; o1 = ob.sph[m0 + 1]; o2 = ob.sph[m0 + 2]; o3 = ob.sph[m0 + 3];
    } else if (!is_quad && active) {
      single = load_obstacle(ob, m0);
    }
    // negated obstacle centres, duplicated for the packed per-link loop
    const float2 nx0 = make_float2(-o0.x, -o0.x), ny0 = make_float2(-o0.y, -o0.y), nz0 = make_float2(-o0.z, -o0.z);
    const float2 nx1 = make_float2(-o1.x, -o1.x), ny1 = make_float2(-o1.y, -o1.y), nz1 = make_float2(-o1.z, -o1.z);
    const float2 nx2 = make_float2(-o2.x, -o2.x), ny2 = make_float2(-o2.y, -o2.y), nz2 = make_float2(-o2.z, -o2.z);
    const float2 nx3 = make_float2(-o3.x, -o3.x), ny3 = make_float2(-o3.y, -o3.y), nz3 = make_float2(-o3.z, -o3.z);
    const int c1 = min(nc, (chunk + 1) * cchunk);
    for (int c = chunk * cchunk; c < c1; ++c) {
      float vmin = 1e9f;
      const float4* cc = rs.centres + c * CK;
      const int* pairs = PER_LINK ? rs.pairs + c * rs.pair_stride : nullptr;
      if (is_quad && active) {
        // quad rows k = sub, sub + rpw, ...; output pointer advanced only when storing
        float* o = store ? out + ((b0 + c) * R + sub) * (long long)M + m0 : nullptr;
        const long long ostep = store ? (long long)rpw * M : 0;
        for (int k = sub; k < R; k += rpw, o += ostep) {
          float4 d;
          if (PER_LINK) {
            // two spheres per packed op: |c - o| = d2 * rsqrt(d2), d2 = dx^2 + dy^2 + dz^2 + 1e-30
            // (the scalar centre_dist, operation for operation), minus r
            d = make_float4(1e9f, 1e9f, 1e9f, 1e9f);
            const float4* pr = cc + k * SP * 2;
            const int np = pairs[k];
#pragma unroll 2
            for (int q = 0; q < np; ++q) {
              const float4 A = pr[2 * q], B = pr[2 * q + 1];
              const float2 cx = make_float2(A.x, A.y), cy = make_float2(A.z, A.w), cz = make_float2(B.x, B.y);
              const float2 nr = make_float2(B.z, B.w);
              auto one = [&](const float2& nx, const float2& ny, const float2& nz, float& acc) {
                const float2 dx = __fadd2_rn(cx, nx), dy = __fadd2_rn(cy, ny), dz = __fadd2_rn(cz, nz);
                float2 d2 = __ffma2_rn(dz, dz, make_float2(1e-30f, 1e-30f));
                d2 = __ffma2_rn(dy, dy, d2);
                d2 = __ffma2_rn(dx, dx, d2);
                const float2 t = __fadd2_rn(root_of2<PRECISE>(d2, make_float2(rsqrt_approx(d2.x), rsqrt_approx(d2.y))), nr);
                acc = fminf(acc, fminf(t.x, t.y));
              };
              one(nx0, ny0, nz0, d.x);
              one(nx1, ny1, nz1, d.y);
              one(nx2, ny2, nz2, d.z);
              one(nx3, ny3, nz3, d.w);
            }
            if (np) {
              d.x -= o0.w; d.y -= o1.w; d.z -= o2.w; d.w -= o3.w;
            } else {
              d = make_float4(1e9f, 1e9f, 1e9f, 1e9f);
            }
          } else {
            const float4 ce = cc[k];
            if (ce.w >= 0.f) {
              d.x = centre_dist(ce, o0) - (ce.w + o0.w);
              d.y = centre_dist(ce, o1) - (ce.w + o1.w);
              d.z = centre_dist(ce, o2) - (ce.w + o2.w);
              d.w = centre_dist(ce, o3) - (ce.w + o3.w);
            } else {
              d = make_float4(1e9f, 1e9f, 1e9f, 1e9f);
            }
          }
          vmin = fminf(vmin, fminf(fminf(d.x, d.y), fminf(d.z, d.w)));
          if (store) {
            if (vec) {
              __stcs(reinterpret_cast<float4*>(o), d);
            } else {
              o[0] = d.x; o[1] = d.y; o[2] = d.z; o[3] = d.w;
            }
          }
        }
      } else if (active) {
        float* o = store ? out + (b0 + c) * R * (long long)M + m0 : nullptr;
        switch (single.kind) {
          case 0: vmin = single_rows<PER_LINK, 0, PRECISE>(single, cc, pairs, S, R, o, M, store); break;
          case 1: vmin = single_rows<PER_LINK, 1, PRECISE>(single, cc, pairs, S, R, o, M, store); break;
          case 2: vmin = single_rows<PER_LINK, 2, PRECISE>(single, cc, pairs, S, R, o, M, store); break;
          default: vmin = single_rows<PER_LINK, 3, PRECISE>(single, cc, pairs, S, R, o, M, store); break;
        }
      }
      if (do_min) {
        vmin = warp_min(vmin);
        if (lane == 0) atomicMin(&cmin[c], float_to_ordered(vmin));
      }
    }
  }
}

}  // namespace pk
