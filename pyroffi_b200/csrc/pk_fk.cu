// Forward kinematics and the fused FK -> spheres -> world-distance kernel.
//
// pk_fk_cuda replaces the reference's "fk_cuda" XLA FFI target
// (src/pyroffi/cuda_kernels/_fk_cuda_kernel.cu:236-471).  One thread owns one
// configuration; the robot description is staged per block in shared memory
// (topological order) and the joint poses leave through a per-warp shared
// tile in contiguous runs.  No model data is cached across
// calls, so there is no pointer-keyed constant upload and no host sync.
#include <algorithm>

#include "pk_obstacles.cuh"

namespace pk {

// ---------------------------------------------------------------------------
// FK: out[b, j, :] = world pose of joint j (original joint order)
// ---------------------------------------------------------------------------

// One thread per configuration, bound by HBM writes (28 bytes per joint) when
// enough configurations are in flight.  A warp computes kFkChunk joints of its
// 32 configurations, keeps their poses in its own staging tile (component-major,
// 33 floats per row: conflict-free both ways) and writes them out as contiguous
// runs of kFkChunk * 28 bytes per configuration before it goes on, so the
// shared memory does not grow with the robot and every SM holds 24 warps (a
// whole robot's poses per thread, 104 KB per block for 29 joints, left 6).  A
// parent of an earlier chunk is read back from the output rows, which this
// warp has written.  100,003 configurations of the 29-joint humanoid:
// 178 -> 76 us (0.52 -> 1.2 TB/s), 71 with the joint values loaded a joint ahead.
constexpr int kFkChunk = 8;
constexpr int kFkTile = kFkChunk * 7;  // floats per configuration and chunk

__global__ void __launch_bounds__(128, 6) fk_kernel(ModelArgs m, const float* __restrict__ cfg, float* out,
                                                 long long batch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  JointTable& jt = *reinterpret_cast<JointTable*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float* tile = reinterpret_cast<float*>(smem_raw + sizeof(JointTable)) + wid * kFkTile * 33;
  load_joint_table(jt, m);

  const long long b0 = ((long long)blockIdx.x * (blockDim.x >> 5) + wid) * 32;
  if (b0 >= batch) return;
  const int rows = (int)min(32LL, batch - b0);
  const bool live = lane < rows;
  const int n = jt.n, nj7 = n * 7;
  const float* c = cfg + (b0 + (live ? lane : 0)) * m.n_act;
  float* row = out + (b0 + (live ? lane : 0)) * nj7;
  const PoseSlots ps{tile + lane, 33};
  Pose prev = pose_identity();
  // the joint values one joint ahead: their loads are the only long waits
  auto value = [&](int i) {
    const int src = i < n ? jt.src[i] : -1;
    return src < 0 ? 0.f : __ldg(c + src);
  };
  float q_next = value(0);
  for (int i0 = 0; i0 < n; i0 += kFkChunk) {
    const int cn = min(kFkChunk, n - i0);
#pragma unroll 1
    for (int i = i0; i < i0 + cn; ++i) {
      const float q = q_next * jt.mul[i] + jt.off[i];
      q_next = value(i + 1);
      const Pose Tpc = joint_local(jt, i, q);
      const int p = jt.psorted[i];
      Pose Tw;
      if (p < 0) {
        Tw = Tpc;
      } else if (p == i - 1) {
        Tw = pose_compose(prev, Tpc);
      } else if (p >= i0) {
        Tw = pose_compose(ps.load(p - i0), Tpc);
      } else {
        const volatile float* g = row + jt.orig[p] * 7;  // written by this warp, before its last __syncwarp
        Tw = pose_compose(Pose{g[0], g[1], g[2], g[3], g[4], g[5], g[6]}, Tpc);
      }
      ps.store(i - i0, Tw);
      prev = Tw;
    }
    __syncwarp();
    // element e = lane + 32 k of the tile, row-major [32][kFkTile]: 4 rows
    // every 7 steps, so a lane's seven columns repeat
    float* dst = out + b0 * nj7;
#pragma unroll 1
    for (int k = 0; k < 7; ++k) {
      const int e = lane + 32 * k;
      const int r0 = e / kFkTile, col = e - r0 * kFkTile;
      if (col >= cn * 7) continue;
      const int jj = col / 7;
      const float* from = tile + col * 33 + r0;
      float* to = dst + r0 * nj7 + jt.orig[i0 + jj] * 7 + (col - jj * 7);
      if (rows == 32) {
#pragma unroll
        for (int g = 0; g < 8; ++g) to[4 * g * nj7] = from[4 * g];
      } else {
        for (int r = r0; r < rows; r += 4, from += 4, to += 4 * nj7) *to = *from;
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Fused FK -> link poses -> sphere centres -> world distances
// ---------------------------------------------------------------------------

struct FusedArgs {
  ModelArgs m;
  WorldArgs w;
  const float* cfg;
  const int* parent_joint;  // [N]
  const float* link_spheres;  // [N, S, 4]
  float* min_dist;          // [B] or null
  float* link_poses;        // [B, N, 7] or null
  float* dist_bkm;          // [B, K, M] or null
  float* dist_bnm;          // [B, N, M] or null (min over each link's spheres)
  float* centres_out;       // [B, K, 4] or null (world centre and radius, k = s*N + n)
  long long batch;
  int N, S;
  int cpb;                  // configurations per block
  int stage_world;          // obstacles in shared memory
};

// |c - o| for a robot sphere centre c and obstacle sphere o.
__device__ __forceinline__ float centre_dist(float4 c, float4 o) {
  const float dx = c.x - o.x, dy = c.y - o.y, dz = c.z - o.z;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, 1e-30f)));
  return d2 * rsqrt_approx(d2);
}

// One obstacle held in registers by a lane: kind 0 sphere (x, y, z, r),
// 1 capsule (p1, p2, r, 1/|p2 - p1|^2 or 0), 2 box (centre, axis columns,
// half-lengths), 3 halfspace (n, n . p0).
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
  return o;
}

// Signed distance from sphere (c, r) to a register obstacle of a known kind.
template <int KIND>
__device__ __forceinline__ float reg_dist(const ObsReg& o, float4 c) {
  if (KIND == 0) {
    return centre_dist(c, make_float4(o.p[0], o.p[1], o.p[2], 0.f)) - (c.w + o.p[3]);
  } else if (KIND == 1) {
    const float vx = o.p[3] - o.p[0], vy = o.p[4] - o.p[1], vz = o.p[5] - o.p[2];
    float t = ((c.x - o.p[0]) * vx + (c.y - o.p[1]) * vy + (c.z - o.p[2]) * vz) * o.p[7];
    t = fmaxf(0.f, fminf(1.f, t));
    const float px = fmaf(t, vx, o.p[0]) - c.x, py = fmaf(t, vy, o.p[1]) - c.y, pz = fmaf(t, vz, o.p[2]) - c.z;
    return sqrt_fast(px * px + py * py + pz * pz) - (c.w + o.p[6]);
  } else if (KIND == 2) {
    const float dx = c.x - o.p[0], dy = c.y - o.p[1], dz = c.z - o.p[2];
    const float q1 = fabsf(dx * o.p[3] + dy * o.p[4] + dz * o.p[5]) - o.p[12];
    const float q2 = fabsf(dx * o.p[6] + dy * o.p[7] + dz * o.p[8]) - o.p[13];
    const float q3 = fabsf(dx * o.p[9] + dy * o.p[10] + dz * o.p[11]) - o.p[14];
    const float m1 = fmaxf(q1, 0.f), m2 = fmaxf(q2, 0.f), m3 = fmaxf(q3, 0.f);
    return sqrt_fast(m1 * m1 + m2 * m2 + m3 * m3) + fminf(fmaxf(fmaxf(q1, q2), q3), 0.f) - c.w;
  } else {
    return c.x * o.p[0] + c.y * o.p[1] + c.z * o.p[2] - o.p[3] - c.w;
  }
}

// Per-link rows read each link's spheres in pairs, so that the sphere-quad
// loop runs on packed FP32x2 arithmetic: for spheres 2q and 2q + 1 of link k
// of configuration c, float4 A = (x0, x1, y0, y1) and B = (z0, z1, -r0, -r1)
// at cc[((c * N + k) * SP + q) * 2 + {0, 1}], SP = ceil(S / 2).  A padding
// sphere (radius < 0, or the odd slot) is stored at 1e18 with -r = 1: its
// packed distances (~1.7e18) never win the minimum, and the scalar rows skip
// it by its radius.
__device__ __forceinline__ int link_pair_count(int S) { return (S + 1) >> 1; }

// Signed distances of the sphere pair (A, B) in the link-pair layout to a
// register box: reg_dist<2> on packed FP32x2, the projections written as
// fma(dz, a_z, fma(dy, a_y, dx * a_x)).
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
  const float2 out = __fmul2_rn(x, make_float2(rsqrt_approx(xe.x), rsqrt_approx(xe.y)));
  const float2 in = make_float2(fminf(fmaxf(fmaxf(q[0].x, q[1].x), q[2].x), 0.f),
                                fminf(fmaxf(fmaxf(q[0].y, q[1].y), q[2].y), 0.f));
  return __fadd2_rn(__fadd2_rn(out, in), make_float2(B.z, B.w));
}

// Rows of one configuration against one register obstacle (a single column
// m per lane): per-sphere rows (R = K) or per-link minima (R = N).  Returns
// the lane's minimum; stores go to o, o + M, ... when `store`.
template <bool PER_LINK, int KIND>
__device__ __forceinline__ float single_rows(const ObsReg& ob, const float4* cc, int N, int S, int R,
                                             float* o, int M, bool store) {
  float vmin = 1e9f;
  for (int k = 0; k < R; ++k) {
    float d = 1e9f;
    if (PER_LINK) {
      const int SP = (S + 1) >> 1;
      for (int q = 0; q < SP; ++q) {
        const float4 A = cc[(k * SP + q) * 2], B = cc[(k * SP + q) * 2 + 1];
        if (KIND == 2) {
          // boxes on packed FP32x2 over the sphere pair; padding spheres are
          // far away and masked by their radius
          const float2 t = box_dist2(ob, A, B);
          if (B.z <= 0.f) d = fminf(d, t.x);
          if (B.w <= 0.f) d = fminf(d, t.y);
        } else {
          const float4 c0 = make_float4(A.x, A.z, B.x, -B.z), c1 = make_float4(A.y, A.w, B.y, -B.w);
          if (c0.w >= 0.f) d = fminf(d, reg_dist<KIND>(ob, c0));
          if (c1.w >= 0.f) d = fminf(d, reg_dist<KIND>(ob, c1));
        }
      }
    } else {
      const float4 ce = cc[k];
      if (ce.w >= 0.f) d = reg_dist<KIND>(ob, ce);
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
template <bool PER_LINK>
__device__ __forceinline__ void distance_rows(const FusedArgs& a, const ObsView& ob,
                                              const float4* centres, const int* lany, int* cmin, long long b0,
                                              int nc, float* out, bool do_min) {
  const int N = a.N, S = a.S, K = N * S;
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
      const float4* cc = centres + c * CK;
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
#pragma unroll 2
            for (int q = 0; q < SP; ++q) {
              const float4 A = pr[2 * q], B = pr[2 * q + 1];
              const float2 cx = make_float2(A.x, A.y), cy = make_float2(A.z, A.w), cz = make_float2(B.x, B.y);
              const float2 nr = make_float2(B.z, B.w);
              auto one = [&](const float2& nx, const float2& ny, const float2& nz, float& acc) {
                const float2 dx = __fadd2_rn(cx, nx), dy = __fadd2_rn(cy, ny), dz = __fadd2_rn(cz, nz);
                float2 d2 = __ffma2_rn(dz, dz, make_float2(1e-30f, 1e-30f));
                d2 = __ffma2_rn(dy, dy, d2);
                d2 = __ffma2_rn(dx, dx, d2);
                const float2 t = __fadd2_rn(__fmul2_rn(d2, make_float2(rsqrt_approx(d2.x), rsqrt_approx(d2.y))), nr);
                acc = fminf(acc, fminf(t.x, t.y));
              };
              one(nx0, ny0, nz0, d.x);
              one(nx1, ny1, nz1, d.y);
              one(nx2, ny2, nz2, d.z);
              one(nx3, ny3, nz3, d.w);
            }
            if (lany[k]) {
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
          case 0: vmin = single_rows<PER_LINK, 0>(single, cc, N, S, R, o, M, store); break;
          case 1: vmin = single_rows<PER_LINK, 1>(single, cc, N, S, R, o, M, store); break;
          case 2: vmin = single_rows<PER_LINK, 2>(single, cc, N, S, R, o, M, store); break;
          default: vmin = single_rows<PER_LINK, 3>(single, cc, N, S, R, o, M, store); break;
        }
      }
      if (do_min) {
        vmin = warp_min(vmin);
        if (lane == 0) atomicMin(&cmin[c], float_to_ordered(vmin));
      }
    }
  }
}

// MINB: resident blocks per SM the register budget is sized for.  4 (64
// registers, small spills) keeps more configurations in flight, which
// shortens small batches; 3 (80 registers) suits the arithmetic-bound rows of
// a large world.
template <int MINB>
__global__ void __launch_bounds__(256, MINB) fk_sphere_collision_kernel(FusedArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  JointTable& jt = *reinterpret_cast<JointTable*>(smem_raw);
  unsigned char* p = smem_raw + sizeof(JointTable);
  const int cpb = a.cpb, N = a.N, S = a.S, K = N * S;
  const int M = a.w.total();
  const int SP = link_pair_count(S);
  float4* centres = reinterpret_cast<float4*>(p);          // [cpb][K], or [cpb][N][SP][2] in link pairs
  p += sizeof(float4) * (size_t)cpb * max(K, 2 * N * SP);
  int* lany = reinterpret_cast<int*>(p);                    // [N] link has a sphere
  p += sizeof(int) * (size_t)((N + 3) & ~3);
  float* lp = reinterpret_cast<float*>(p);                  // [cpb][N][7]
  p += sizeof(float) * (size_t)cpb * N * 7;
  int* cmin = reinterpret_cast<int*>(p);                    // [cpb]
  p += sizeof(int) * (size_t)((cpb + 3) & ~3);
  float* slots = reinterpret_cast<float*>(p);               // FK pose slots [n_j*7][cpb+1]
  p += sizeof(float) * (size_t)a.m.n_joints * 7 * (cpb + 1);
  p = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15));

  load_joint_table(jt, a.m);
  ObsView ob;
  if (a.stage_world) {
    ob = stage_world(a.w, reinterpret_cast<float*>(p));
  } else {
    ob.sph = reinterpret_cast<const float4*>(a.w.spheres);
    ob.cap = a.w.capsules; ob.box = a.w.boxes; ob.hs = a.w.halfspaces;
    ob.Ms = a.w.Ms; ob.Mc = a.w.Mc; ob.Mb = a.w.Mb; ob.Mh = a.w.Mh;
  }

  const long long b0 = (long long)blockIdx.x * cpb;
  const int nc = (int)min((long long)cpb, a.batch - b0);
  const int tid = threadIdx.x, T = blockDim.x;

  // phase 1: FK, one thread per configuration
  if (tid < nc) {
    PoseSlots ps{slots + tid, cpb + 1};
    const float* c = a.cfg + (b0 + tid) * a.m.n_act;
    fk_thread(jt, [&](int i) { return __ldg(c + i); }, ps);
    for (int n = 0; n < N; ++n) {
      const int pj = a.parent_joint[n];
      Pose T_l = (pj < 0 || pj >= jt.n) ? pose_identity() : ps.load(jt.sorted_of[pj]);
      float* d = lp + ((size_t)tid * N + n) * 7;
      d[0] = T_l.w; d[1] = T_l.x; d[2] = T_l.y; d[3] = T_l.z;
      d[4] = T_l.tx; d[5] = T_l.ty; d[6] = T_l.tz;
    }
  }
  for (int c = tid; c < cpb; c += T) cmin[c] = float_to_ordered(1e9f);
  __syncthreads();

  // link poses out (coalesced)
  if (a.link_poses) {
    float* dst = a.link_poses + b0 * N * 7;
    const int tot = nc * N * 7;
    for (int g = tid; g < tot; g += T) dst[g] = lp[g];
  }

  // phase 2: sphere centres, per sphere (k = s*N + n) or in link pairs
  auto world_centre = [&](int c, int n, int s) {
    const float4 ls = *reinterpret_cast<const float4*>(a.link_spheres + ((size_t)n * S + s) * 4);
    const float* q = lp + ((size_t)c * N + n) * 7;
    const Pose Tl{q[0], q[1], q[2], q[3], q[4], q[5], q[6]};
    const float3 w = pose_apply(Tl, make_float3(ls.x, ls.y, ls.z));
    return make_float4(w.x, w.y, w.z, ls.w);
  };
  auto write_pairs = [&]() {
    const int K2 = 2 * N * SP;
    for (int g = tid; g < nc * K2; g += T) {
      const int c = g / K2, r = g - c * K2;
      const int n = r / (2 * SP), s = r - n * 2 * SP;
      float4 w = s < S ? world_centre(c, n, s) : make_float4(0.f, 0.f, 0.f, -1.f);
      if (!(w.w >= 0.f)) w = make_float4(1e18f, 1e18f, 1e18f, -1.f);
      float* d = reinterpret_cast<float*>(centres + (size_t)c * K2 + ((size_t)n * SP + (s >> 1)) * 2);
      const int h = s & 1;
      d[h] = w.x; d[2 + h] = w.y; d[4 + h] = w.z; d[6 + h] = -w.w;
    }
  };
  if (a.centres_out) {
    float4* dst = reinterpret_cast<float4*>(a.centres_out) + b0 * K;
    for (int g = tid; g < nc * K; g += T) {
      const int c = g / K, k = g - c * K;
      const int s = k / N, n = k - s * N;
      __stcs(dst + g, world_centre(c, n, s));
    }
  }
  const bool per_link = a.dist_bnm || !a.dist_bkm;
  if (per_link)
    for (int n = tid; n < N; n += T) {
      int any = 0;
      for (int s = 0; s < S; ++s) any |= a.link_spheres[((size_t)n * S + s) * 4 + 3] >= 0.f;
      lany[n] = any;
    }
  if (a.dist_bkm) {
    for (int g = tid; g < nc * K; g += T) {
      const int c = g / K, k = g - c * K;
      const int s = k / N, n = k - s * N;
      centres[g] = world_centre(c, n, s);
    }
  } else {
    write_pairs();
  }
  __syncthreads();

  // phase 3: distances (per-sphere rows, per-link rows, or the minimum only)
  // (the per-link pass gives the minimum when only that, or nothing, is requested)
  if (a.dist_bkm) {
    distance_rows<false>(a, ob, centres, lany, cmin, b0, nc, a.dist_bkm, true);
    if (per_link) {
      __syncthreads();
      write_pairs();
      __syncthreads();
    }
  }
  if (per_link) distance_rows<true>(a, ob, centres, lany, cmin, b0, nc, a.dist_bnm, !a.dist_bkm);
  __syncthreads();
  if (a.min_dist)
    for (int c = tid; c < nc; c += T) a.min_dist[b0 + c] = ordered_to_float(cmin[c]);
}

static size_t fk_smem_bytes(int threads) {
  return sizeof(JointTable) + sizeof(float) * (size_t)(threads / 32) * kFkTile * 33;
}

}  // namespace pk

using namespace pk;

static int check_model(const int32_t* parent_idx, int n_act, int n_joints) {
  PK_CHECK_ARG(n_joints >= 0 && n_act >= 0, "negative joint count");
  PK_CHECK_CAP(n_joints <= PK_MAX_JOINTS, "n_joints=%d exceeds %d", n_joints, PK_MAX_JOINTS);
  (void)parent_idx;
  return PK_OK;
}

extern "C" int pk_fk_cuda(void* stream, const float* cfg, const float* twists,
                          const float* parent_tf, const int32_t* parent_idx,
                          const int32_t* act_idx, const float* mimic_mul, const float* mimic_off,
                          const int32_t* mimic_act_idx, const int32_t* topo_inv,
                          const int32_t* fk_level_starts, const int32_t* fk_level_joints,
                          float* out, int64_t batch, int32_t n_act, int32_t n_joints,
                          int32_t n_levels) {
  PK_CHECK_ARG(batch >= 0, "negative batch");
  if (int st = check_model(parent_idx, n_act, n_joints)) return st;
  PK_CHECK_CAP(n_levels <= PK_MAX_JOINTS, "n_levels=%d exceeds %d", n_levels, PK_MAX_JOINTS);
  (void)fk_level_starts;
  (void)fk_level_joints;  // the depth schedule is implied by parent_idx/topo_inv here
  if (batch == 0 || n_joints == 0) return PK_OK;
  PK_CHECK_ARG(cfg && twists && parent_tf && parent_idx && act_idx && mimic_mul && mimic_off &&
                   mimic_act_idx && topo_inv && out,
               "null buffer");
  // one-warp blocks while they all fit on the GPU at once spread a small batch
  // over the SMs; four-warp blocks share the staged robot otherwise
  const int threads = batch <= 148 * 32 ? 32 : 128;
  const size_t smem = fk_smem_bytes(threads);
  if (int st = set_smem_limit((const void*)fk_kernel, smem)) return st;
  ModelArgs m{twists, parent_tf, parent_idx, act_idx, mimic_mul, mimic_off, mimic_act_idx,
              topo_inv, n_joints, n_act};
  const long long blocks = (batch + threads - 1) / threads;
  PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
  fk_kernel<<<(unsigned)blocks, threads, smem, (cudaStream_t)stream>>>(m, cfg, out, batch);
  return cuda_status(cudaGetLastError(), "fk_kernel launch");
}

extern "C" int pk_fk_sphere_collision(
    void* stream, const float* cfg, const float* twists, const float* parent_tf,
    const int32_t* parent_idx, const int32_t* act_idx, const float* mimic_mul,
    const float* mimic_off, const int32_t* mimic_act_idx, const int32_t* topo_inv,
    const int32_t* parent_joint_indices, const float* link_spheres, const float* world_spheres,
    const float* world_capsules, const float* world_boxes, const float* world_halfspaces,
    float* min_dist, float* link_poses, float* dist_bkm, float* dist_bnm, float* sphere_centers, int64_t batch,
    int32_t n_act,
    int32_t n_joints, int32_t n_links, int32_t S, int32_t Ms, int32_t Mc, int32_t Mb,
    int32_t Mh) {
  PK_CHECK_ARG(batch >= 0 && n_links >= 0 && S >= 0 && Ms >= 0 && Mc >= 0 && Mb >= 0 && Mh >= 0,
               "negative extent");
  if (int st = check_model(parent_idx, n_act, n_joints)) return st;
  if (batch == 0) return PK_OK;
  PK_CHECK_ARG(cfg && twists && parent_tf && parent_idx && act_idx && mimic_mul && mimic_off &&
                   mimic_act_idx && topo_inv && parent_joint_indices,
               "null model buffer");
  PK_CHECK_ARG(n_links == 0 || S == 0 || link_spheres, "null link_spheres");
  PK_CHECK_ARG((Ms == 0 || world_spheres) && (Mc == 0 || world_capsules) &&
                   (Mb == 0 || world_boxes) && (Mh == 0 || world_halfspaces),
               "null world buffer");
  PK_CHECK_ARG(link_spheres == nullptr || (reinterpret_cast<uintptr_t>(link_spheres) & 15) == 0,
               "link_spheres must be 16-byte aligned");
  PK_CHECK_ARG(sphere_centers == nullptr || (reinterpret_cast<uintptr_t>(sphere_centers) & 15) == 0,
               "sphere_centers must be 16-byte aligned");
  WorldArgs w{world_spheres, world_capsules, world_boxes, world_halfspaces, Ms, Mc, Mb, Mh};
  const int K = n_links * S;
  const int threads = 256;
  int cpb = 32;
  auto smem_for = [&](int c, bool stage) {
    const size_t per_cfg = std::max((size_t)K, 2 * (size_t)n_links * (size_t)((S + 1) / 2));
    size_t b = sizeof(JointTable) + sizeof(float4) * (size_t)c * per_cfg + sizeof(int) * (size_t)((n_links + 3) & ~3) +
               sizeof(float) * (size_t)c * n_links * 7 + sizeof(int) * (size_t)((c + 3) & ~3) +
               sizeof(float) * (size_t)n_joints * 7 * (c + 1) + 16;
    if (stage) b += sizeof(float) * w.smem_floats();
    return b;
  };
  const size_t limit = 200 * 1024;
  // Sphere obstacles are read once per work unit into registers, so only a
  // small world is worth a shared-memory copy; a large one is read through L1.
  bool stage = smem_for(1, true) <= limit && sizeof(float) * w.smem_floats() <= 48 * 1024;
  PK_CHECK_ARG(stage || world_spheres == nullptr || (reinterpret_cast<uintptr_t>(world_spheres) & 15) == 0,
               "world_spheres must be 16-byte aligned");
  while (cpb > 1 && smem_for(cpb, stage) > limit) cpb >>= 1;
  // enough blocks to fill every SM a few times over
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  while (cpb > 1 && (batch + cpb - 1) / cpb < 4LL * sms) cpb >>= 1;
  PK_CHECK_CAP(smem_for(cpb, stage) <= limit, "robot too large for the fused kernel");
  const size_t smem = smem_for(cpb, stage);
  // register budget: 4 blocks per SM below 1,024 obstacles, 3 for the arithmetic-bound rows of larger worlds
  auto kern = (Ms + Mc + Mb + Mh >= 1024) ? fk_sphere_collision_kernel<3> : fk_sphere_collision_kernel<4>;
  if (int st = set_smem_limit((const void*)kern, smem)) return st;
  FusedArgs a;
  a.m = ModelArgs{twists, parent_tf, parent_idx, act_idx, mimic_mul, mimic_off, mimic_act_idx,
                  topo_inv, n_joints, n_act};
  a.w = w;
  a.cfg = cfg;
  a.parent_joint = parent_joint_indices;
  a.link_spheres = link_spheres;
  a.min_dist = min_dist;
  a.link_poses = link_poses;
  a.dist_bkm = dist_bkm;
  a.dist_bnm = dist_bnm;
  a.centres_out = sphere_centers;
  a.batch = batch;
  a.N = n_links;
  a.S = S;
  a.cpb = cpb;
  a.stage_world = stage ? 1 : 0;
  const long long blocks = (batch + cpb - 1) / cpb;
  PK_CHECK_CAP(blocks < (1LL << 31), "batch too large");
  kern<<<(unsigned)blocks, threads, smem, (cudaStream_t)stream>>>(a);
  return cuda_status(cudaGetLastError(), "fk_sphere_collision_kernel launch");
}
