// All-pairs interaction, FP32 pair math with FP64 accumulation, every unordered
// particle pair once: the symmetric pair engine (the FP32 hot path).
//
// Reference: the pair physics of INTERACT (src/interaction/interaction_utils.h:363-407)
// with KERNEL (src/interaction/highorder.h:48-60), summed over all unordered
// pairs of a system by __interaction::interact (src/interaction/interaction.cpp:95-108).
// The pair algebra and the tile-pair classes are pair_f32.cu's (its file
// comment derives them); what differs is that a pair's distance, kernel
// factors, alpha_i x alpha_j and triple product are formed once and added to
// both particles.
//
// Symmetric forms.  Far (x' = x - c, beta = alpha x x', d = x'_i - x'_j):
//   u_i   += m (alpha_j x d),       u_j   -= m (alpha_i x d)
//   W_i    = sum m beta_j, Q_i = sum m alpha_j, G_i = sum g d
//   W_j    = sum m beta_i, Q_j = sum m alpha_i, N_j = sum g d = -G_j
//   with t~ = alpha_j.beta_i + alpha_i.beta_j (= -alpha_i.(alpha_j x d)) and
//   g = -fh t, so u = A (Q x x' - W), dalpha = alpha x (A Q) + 3 A G on either side.
// Near (hi/lo differences): u_i += q (alpha_j x d), u_j -= q (alpha_i x d), and
// one vector s = q (alpha_i x alpha_j) + 3 F t d + 15 nu Dp (v_i alpha_j -
// v_j alpha_i), antisymmetric in (i, j): dalpha_i += s, dalpha_j -= s.  The
// diffusion vector is formed as v_i w + (v_i mu - v_j) alpha_i - v_j lo_i from
// the w = alpha_j - mu alpha_i that alpha_i x alpha_j is formed from, accurate for
// nearly equal strengths and volumes whatever mu's rounding (14 operations; from
// alpha_j - alpha_i in hi and lo 20, and 3 % more time on near tiles).
//
// Layout.  A warp computes a 128 x 128 tile pair (I, J): each lane holds R
// targets of I (4 on far tiles, 2 on near ones) and their sums in registers,
// and 32 sources of J at a time sit in shared memory, one per lane.  At step k
// lane l takes source l ^ k (bank-conflict-free), and the sums of that source
// travel with it by shuffle (9 floats far, 6 near), so after 32 steps every
// source has met all the warp's targets and its sums are back at its own lane.
// Sums are FP32 over 32 sources (near, small systems) or 128 (far, large
// ones) on the target's side and over 128 (64 near) targets on the source's,
// then folded into FP64.
//
// What bounds it: register-file reads of the FMA pipe.  A far step of one
// target is 37 FMA-pipe operations and one MUFU for two interactions (the
// one-sided packed loop: 28 for one); 23 of them read three different
// registers, at about two reads per cycle and lane.  The step's 3 loads, 9
// shuffles and address are shared by four targets; with two the shared-memory
// pipe (21 of its cycles per step) would be the limit.  One right-hand side of
// the ring pair at N = 131,072: 13.9 ms (1,236 G interactions/s) against 18.4 ms
// one-sided; 20,011 unordered particles (near tile pairs only, mixed radii)
// 0.83 ms against 1.48.
//
// Compiled without contraction of multiply-adds (every FMA is written out), so
// that the kernels of the launch shapes below round alike and a system's result
// does not depend on which of them runs it.
//
// Work items.  Large systems: a block of four warps takes a group of 4 tiles
// (512 particles) against a run of groups; in round r warp w computes tile w
// against tile (w + r) % 4 of the group, so no two warps add to one source's
// FP64 sums at a time and their order is fixed.  Small systems: one tile pair
// per block, each warp 32 of its sources (launches of few tile pairs: eight warps,
// in one block or a cluster of two).  An item writes its target-side sums
// once and its source-side sums per group, each to a slot of its own; a
// separate kernel sums a particle's slots in a fixed order, so results do not
// depend on scheduling.
#include "pair_scalars.cuh"
#include "pair_sym.cuh"

namespace pawan {
namespace {

constexpr int kBlocks = 3;          // per SM: 168 registers, no spills (four blocks of 128 ran 4 % slower)
constexpr int kStageBytes = 1792;   // per warp: 3 x float4[32], float2[32]

struct Stage {
  float4 *s0, *s1, *s2;
  float2 *s3;
};

__device__ __forceinline__ Stage stage_of(char *base) {
  Stage s;
  s.s0 = reinterpret_cast<float4 *>(base);
  s.s1 = reinterpret_cast<float4 *>(base + 512);
  s.s2 = reinterpret_cast<float4 *>(base + 1024);
  s.s3 = reinterpret_cast<float2 *>(base + 1536);
  return s;
}

// Particles past the end: far from everything (as a source and as a target on
// opposite sides, so that they never coincide), zero strength and volume; every
// product they enter is exactly zero.
constexpr float kPadSource = 1e18f, kPadTarget = -1e18f;

enum FarClass { FAR_Z = 0, FAR_NZ = 1, FAR_SER = 2 };

struct FarTarget {
  float x, y, z;     // x' = x - c
  float ax, ay, az;  // strength (hi)
  float bx, by, bz;  // beta = alpha x x'
  float h, v;
};

struct Sums9 {
  float wx, wy, wz, qx, qy, qz, gx, gy, gz;
};

__device__ __forceinline__ void rotate(Sums9 &a, int m) {
  a.wx = __shfl_xor_sync(kFull, a.wx, m);
  a.wy = __shfl_xor_sync(kFull, a.wy, m);
  a.wz = __shfl_xor_sync(kFull, a.wz, m);
  a.qx = __shfl_xor_sync(kFull, a.qx, m);
  a.qy = __shfl_xor_sync(kFull, a.qy, m);
  a.qz = __shfl_xor_sync(kFull, a.qz, m);
  a.gx = __shfl_xor_sync(kFull, a.gx, m);
  a.gy = __shfl_xor_sync(kFull, a.gy, m);
  a.gz = __shfl_xor_sync(kFull, a.gz, m);
}

// Adds a pair's weight m to the W and Q sums of both particles, or of one.
template <int SIDE>
__device__ __forceinline__ void add_wq(const FarTarget &T, const float4 &s, const float4 &e, float m, Sums9 &a,
                                       Sums9 &b) {
  if (SIDE != SIDE_J) {
    a.wx = fmaf(m, e.x, a.wx);
    a.wy = fmaf(m, e.y, a.wy);
    a.wz = fmaf(m, e.z, a.wz);
    a.qx = fmaf(m, s.x, a.qx);
    a.qy = fmaf(m, s.y, a.qy);
    a.qz = fmaf(m, s.z, a.qz);
  }
  if (SIDE != SIDE_I) {
    b.wx = fmaf(m, T.bx, b.wx);
    b.wy = fmaf(m, T.by, b.wy);
    b.wz = fmaf(m, T.bz, b.wz);
    b.qx = fmaf(m, T.ax, b.qx);
    b.qy = fmaf(m, T.ay, b.qy);
    b.qz = fmaf(m, T.az, b.qz);
  }
}

// t~ = alpha_j.beta_i + alpha_i.beta_j
__device__ __forceinline__ float far_t(const FarTarget &T, const float4 &s, const float4 &e) {
  return fmaf(T.az, e.z, fmaf(T.ay, e.y, fmaf(T.ax, e.x,
         fmaf(s.z, T.bz, fmaf(s.y, T.by, s.x * T.bx)))));
}

// 32 sources of a far tile with the Z terms against R targets per lane.  kap:
// the diffusion factor in the units of the G sums (5 nu, or 80 nu / h with one
// radius).
template <int SIDE, bool UNI, bool DIFF, int KERN, int R>
__device__ __forceinline__ void far_block_z(const Stage &st, int lane, const FarTarget (&T)[R], float hu,
                                            float kap, Sums9 (&a)[R], Sums9 &b) {
  const float s2u = 2.f * hu, c240 = -480.f * hu;
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += 2) {
    const int base = lane ^ kk;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float4 p = st.s0[base ^ u], s = st.s1[base ^ u], e = st.s2[base ^ u];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float dx = T[r].x - p.x, dy = T[r].y - p.y, dz = T[r].z - p.z;
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const float ri = rsqrtf(r2);
        float m, fh, dp;
        if (KERN == KERNEL_GAUSSIAN)
          gauss_scalars(T[r].h + p.w, r2, ri, m, fh, dp);
        else if (UNI)
          kernel_scalars_uniform(hu, c240, rsqrtf(r2 + s2u), ri, m, fh, dp);
        else
          kernel_scalars(T[r].h + p.w, rsqrtf(r2 + (T[r].h + p.w)), ri, m, fh, dp);
        const float g = -fh * far_t(T[r], s, e);
        add_wq<SIDE>(T[r], s, e, m, a[r], b);
        if (DIFF) {
          const float kd = kap * dp;
          const float gx = fmaf(kd, fmaf(T[r].v, s.x, -s.w * T[r].ax), g * dx);
          const float gy = fmaf(kd, fmaf(T[r].v, s.y, -s.w * T[r].ay), g * dy);
          const float gz = fmaf(kd, fmaf(T[r].v, s.z, -s.w * T[r].az), g * dz);
          if (SIDE != SIDE_J) {
            a[r].gx += gx;
            a[r].gy += gy;
            a[r].gz += gz;
          }
          if (SIDE != SIDE_I) {
            b.gx += gx;
            b.gy += gy;
            b.gz += gz;
          }
        } else {
          if (SIDE != SIDE_J) {
            a[r].gx = fmaf(g, dx, a[r].gx);
            a[r].gy = fmaf(g, dy, a[r].gy);
            a[r].gz = fmaf(g, dz, a[r].gz);
          }
          if (SIDE != SIDE_I) {
            b.gx = fmaf(g, dx, b.gx);
            b.gy = fmaf(g, dy, b.gy);
            b.gz = fmaf(g, dz, b.gz);
          }
        }
      }
      // lane l holds the sums of source l ^ k and next takes l ^ (k + 1)
      const int k = kk + u;
      if (SIDE != SIDE_I) rotate(b, (k ^ (k + 1)) & 31);
    }
  }
}

// Weight m and 1/rho^2 of two pairs without the Z terms, from rho^2 and (unless
// UNI) sigma^2.
template <int CLS, bool UNI, int KERN>
__device__ __forceinline__ float2 far_weights(float2 r2, float2 sig2, float hu, float2 &ri2) {
  const float2 one2 = make_float2(1.f, 1.f), half2 = make_float2(0.5f, 0.5f), nhalf2 = make_float2(-0.5f, -0.5f);
  const float2 h2 = make_float2(hu, hu), nh2 = make_float2(-hu, -hu), s2u2 = make_float2(2.f * hu, 2.f * hu);
  const float2 ri = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  ri2 = __fmul2_rn(ri, ri);
  if (CLS == FAR_SER && KERN == KERNEL_GAUSSIAN) return __fmul2_rn(ri, ri2);
  if (CLS == FAR_SER && UNI)
    return __fmul2_rn(__fmul2_rn(__fmul2_rn(ri, ri2), __ffma2_rn(nh2, ri2, one2)), ri2);
  if (CLS == FAR_SER) {
    const float2 eps = __fmul2_rn(sig2, ri2);
    return __fmul2_rn(__fmul2_rn(__fmul2_rn(eps, ri), ri2), __ffma2_rn(nhalf2, eps, one2));
  }
  const float2 sr = __fadd2_rn(r2, UNI ? s2u2 : sig2);
  const float2 y = make_float2(rcp_approx(sr.x), rcp_approx(sr.y));
  if (UNI) return __fmul2_rn(__fmul2_rn(__ffma2_rn(__fmul2_rn(h2, y), y, y), ri), ri2);
  const float2 ph = __ffma2_rn(__fmul2_rn(__fmul2_rn(half2, sig2), y), y, y);
  return __fmul2_rn(__fmul2_rn(__fmul2_rn(ph, sig2), ri), ri2);
}

// The same without the Z terms (FAR_NZ, FAR_SER), R even: two targets per
// FP32x2 instruction where no source operand enters (distance, kernel factors),
// scalar FMAs for the rest.  The loop is held by register-file reads -- an FMA
// of three different registers takes 1.5 issue slots, one of an FP32x2 pair
// half -- which is what the packing saves: 1,435 G interactions/s against 1,340
// of the scalar loop in a loop of its own on one B200, 1,210 against 1,150 in
// this kernel on the ring pair at N = 131,072.
template <int SIDE, int CLS, bool UNI, int KERN, int R, int UNROLL>
__device__ __forceinline__ void far_block(const Stage &st, int lane, const FarTarget (&T)[R], float hu,
                                          Sums9 (&a)[R], Sums9 &b) {
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += UNROLL) {
    const int base = lane ^ kk;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const float4 p = st.s0[base ^ u], s = st.s1[base ^ u], e = st.s2[base ^ u];
#pragma unroll
      for (int r = 0; r < R; r += 2) {
        const FarTarget &X = T[r], &Y = T[r + 1];
        const float2 dx = make_float2(X.x - p.x, Y.x - p.x), dy = make_float2(X.y - p.y, Y.y - p.y),
                     dz = make_float2(X.z - p.z, Y.z - p.z);
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        float2 ri2;
        const float2 m = far_weights<CLS, UNI, KERN>(r2, make_float2(X.h + p.w, Y.h + p.w), hu, ri2);
        const float2 g = __fmul2_rn(__fmul2_rn(m, ri2), make_float2(far_t(X, s, e), far_t(Y, s, e)));
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float gq = q ? g.y : g.x, ex = q ? dx.y : dx.x, ey = q ? dy.y : dy.x, ez = q ? dz.y : dz.x;
          Sums9 &c = a[r + q];
          add_wq<SIDE>(T[r + q], s, e, q ? m.y : m.x, c, b);
          if (SIDE != SIDE_J) {
            c.gx = fmaf(gq, ex, c.gx);
            c.gy = fmaf(gq, ey, c.gy);
            c.gz = fmaf(gq, ez, c.gz);
          }
          if (SIDE != SIDE_I) {
            b.gx = fmaf(gq, ex, b.gx);
            b.gy = fmaf(gq, ey, b.gy);
            b.gz = fmaf(gq, ez, b.gz);
          }
        }
      }
      const int k = kk + u;
      if (SIDE != SIDE_I) rotate(b, (k ^ (k + 1)) & 31);
    }
  }
}

// The sources' sums of a tile pair alone: each lane keeps four sources and their
// sums in registers and meets the 128 targets in shared memory (t: 4 x 32 of
// (x', h), (strength, volume), (beta)), in the order in which the travelling sums
// of far_block meet them -- the same terms added in the same order, without the
// shuffles.  The last rank of eight at N = 131,072, whose items are mostly of this
// kind: 2.48 ms, 2.73 with the sums travelling (one-sided kernel 2.40).
template <int CLS, bool UNI, int KERN>
__device__ __forceinline__ void far_block_sources(const float4 *t, int lane, const FarTarget (&S)[4], float hu,
                                                  Sums9 (&b)[4]) {
#pragma unroll 1
  for (int k = 0; k < 32; ++k) {
    const float4 *const at = t + (lane ^ k);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 x = at[96 * r], ta = at[96 * r + 32], tb = at[96 * r + 64];
      const FarTarget T{x.x, x.y, x.z, ta.x, ta.y, ta.z, tb.x, tb.y, tb.z, x.w, ta.w};
#pragma unroll
      for (int q = 0; q < 4; q += 2) {
        const FarTarget &X = S[q], &Y = S[q + 1];
        const float2 dx = make_float2(T.x - X.x, T.x - Y.x), dy = make_float2(T.y - X.y, T.y - Y.y),
                     dz = make_float2(T.z - X.z, T.z - Y.z);
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        float2 ri2;
        const float2 m = far_weights<CLS, UNI, KERN>(r2, make_float2(T.h + X.h, T.h + Y.h), hu, ri2);
        float2 ft;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const FarTarget &Z = S[q + o];
          (o ? ft.y : ft.x) = far_t(T, make_float4(Z.ax, Z.ay, Z.az, 0.f), make_float4(Z.bx, Z.by, Z.bz, 0.f));
        }
        const float2 g = __fmul2_rn(__fmul2_rn(m, ri2), ft);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const float gq = o ? g.y : g.x, ex = o ? dx.y : dx.x, ey = o ? dy.y : dy.x, ez = o ? dz.y : dz.x;
          Sums9 &c = b[q + o], unused;
          add_wq<SIDE_J>(T, x, x, o ? m.y : m.x, unused, c);
          c.gx = fmaf(gq, ex, c.gx);
          c.gy = fmaf(gq, ey, c.gy);
          c.gz = fmaf(gq, ez, c.gz);
        }
      }
    }
  }
}

// FP32 far sums of one particle into its six FP64 sums acc[k * stride]:
// u += As2 (Q x x' - W), dalpha += alpha x (As2 Q) + g3 G, with alpha = hi + lo.
__device__ __forceinline__ void fold_far(const Sums9 &s, float x, float y, float z, float ax, float ay,
                                         float az, float lx, float ly, float lz, double As2, double g3,
                                         double *acc, int stride) {
  const double Qx = As2 * s.qx, Qy = As2 * s.qy, Qz = As2 * s.qz;
  const double xp = x, yp = y, zp = z;
  const double px = (double)ax + (double)lx, py = (double)ay + (double)ly, pz = (double)az + (double)lz;
  acc[0] += fma(-As2, (double)s.wx, fma(Qy, zp, -Qz * yp));
  acc[stride] += fma(-As2, (double)s.wy, fma(Qz, xp, -Qx * zp));
  acc[2 * stride] += fma(-As2, (double)s.wz, fma(Qx, yp, -Qy * xp));
  acc[3 * stride] += fma(g3, (double)s.gx, fma(py, Qz, -pz * Qy));
  acc[4 * stride] += fma(g3, (double)s.gy, fma(pz, Qx, -px * Qz));
  acc[5 * stride] += fma(g3, (double)s.gz, fma(px, Qy, -py * Qx));
}

// Particle i of a tile relative to the centre c, with its beta; `away` when there
// is none.
__device__ __forceinline__ FarTarget far_particle(const SymSeg &sg, int i, float cx, float cy, float cz, float away) {
  FarTarget T{away, away, away, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 1.f, 0.f};
  if (i < sg.n) {
    const float4 p = sg.pos32[i], q = sg.vor32[i];
    const float x = p.x - cx, y = p.y - cy, z = p.z - cz;
    T = FarTarget{x, y, z, q.x, q.y, q.z, fmaf(q.y, z, -q.z * y), fmaf(q.z, x, -q.x * z), fmaf(q.x, y, -q.y * x),
                  p.w, q.w};
  }
  return T;
}

// far_block_sources over a whole tile pair; t: shared memory of 6 KB of the warp's own.
template <int CLS, bool UNI, int KERN>
__device__ __forceinline__ void far_pair_sources(const SymSeg &sg, int I, int J, float cx, float cy, float cz, float hu,
                                                 float4 *t, int lane, double *accJ) {
  const double As2 = UNI ? kInv4Pi * 2.0 * (double)hu : kInv4Pi;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const FarTarget T = far_particle(sg, I * kT + 32 * r + lane, cx, cy, cz, kPadTarget);
    t[96 * r + lane] = make_float4(T.x, T.y, T.z, T.h);
    t[96 * r + 32 + lane] = make_float4(T.ax, T.ay, T.az, T.v);
    t[96 * r + 64 + lane] = make_float4(T.bx, T.by, T.bz, 0.f);
  }
  FarTarget S[4];
  Sums9 b[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    S[q] = far_particle(sg, J * kT + 32 * q + lane, cx, cy, cz, kPadSource);
    b[q] = Sums9{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  }
  __syncwarp();
  far_block_sources<CLS, UNI, KERN>(t, lane, S, hu, b);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = J * kT + 32 * q + lane;
    const float4 l = j < sg.n ? sg.vorlo[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    fold_far(b[q], S[q].x, S[q].y, S[q].z, S[q].ax, S[q].ay, S[q].az, l.x, l.y, l.z, As2, -3.0 * As2,
             accJ + 32 * q + lane, kT);
  }
}

// A far tile pair: sub-blocks [k0, k1) of 32 sources of tile J against all
// targets of tile I, R per lane and pass.  accI: the warp's [6][128] target
// sums; accJ: [6][128] source sums of tile J.
template <int SIDE, int CLS, bool UNI, bool DIFF, int KERN, int R, int UNROLL>
__device__ __forceinline__ void far_pair(const SymSeg &sg, int I, int J, int k0, int k1, int ta, int tb,
                                         float cx, float cy, float cz, float hu, const Stage &st, int lane,
                                         double *accI, double *accJ) {
  if constexpr (SIDE == SIDE_J && CLS != FAR_Z) {
    if (k1 - k0 == 4) {  // (a constant where this is inlined; accI is the warp's, and not used for sums)
      far_pair_sources<CLS, UNI, KERN>(sg, I, J, cx, cy, cz, hu, reinterpret_cast<float4 *>(accI), lane, accJ);
      return;
    }
  }
  if (R == 4) {  // one pass over all targets
    if (ta > 0) return;
    tb = kT;
  }
  const double As2 = UNI ? kInv4Pi * 2.0 * (double)hu : kInv4Pi;
  const float kap = (CLS == FAR_Z && DIFF) ? (float)(UNI ? 80.0 * sg.nu / (double)hu : 5.0 * sg.nu) : 0.f;
  const float4 *pos = sg.pos32;
  const float4 *vor = sg.vor32;
  const float4 *vlo = sg.vorlo;
  const int n = sg.n;
#pragma unroll 1
  for (int t0 = ta; t0 < tb; t0 += 32 * R) {
    FarTarget T[R];
    Sums9 a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      T[r] = far_particle(sg, I * kT + t0 + 32 * r + lane, cx, cy, cz, kPadTarget);
      a[r] = Sums9{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    }
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int j = J * kT + 32 * k + lane;
      float4 p = make_float4(kPadSource, kPadSource, kPadSource, 1.f), q = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 l = q, e = q;
      if (j < n) {
        p = pos[j];
        q = vor[j];
        l = vlo[j];
        p.x -= cx;
        p.y -= cy;
        p.z -= cz;
        e = make_float4(fmaf(q.y, p.z, -q.z * p.y), fmaf(q.z, p.x, -q.x * p.z), fmaf(q.x, p.y, -q.y * p.x), 0.f);
      }
      e.w = l.x;
      st.s0[lane] = p;
      st.s1[lane] = q;
      st.s2[lane] = e;
      st.s3[lane] = make_float2(l.y, l.z);
      __syncwarp();
      Sums9 b{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if constexpr (CLS == FAR_Z)
        far_block_z<SIDE, UNI, DIFF, KERN, R>(st, lane, T, hu, kap, a, b);
      else
        far_block<SIDE, CLS, UNI, KERN, R, UNROLL>(st, lane, T, hu, a, b);
      if (SIDE != SIDE_I) {
        const float4 pj = st.s0[lane], qj = st.s1[lane], ej = st.s2[lane];
        const float2 lj = st.s3[lane];
        fold_far(b, pj.x, pj.y, pj.z, qj.x, qj.y, qj.z, ej.w, lj.x, lj.y, As2, -3.0 * As2,
                 accJ + 32 * k + lane, kT);
      }
      __syncwarp();
    }
    if (SIDE == SIDE_J) continue;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = I * kT + t0 + 32 * r + lane;
      const float4 l = i < n ? vlo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      fold_far(a[r], T[r].x, T[r].y, T[r].z, T[r].ax, T[r].ay, T[r].az, l.x, l.y, l.z, As2, 3.0 * As2,
               accI + t0 + 32 * r + lane, kT);
    }
  }
}

struct NearTarget {
  float xh, yh, zh, xl, yl, zl;  // position hi, lo
  float ax, ay, az, lx, ly, lz;  // strength hi, lo
  float iaa;                     // 1 / |alpha_hi|^2 (0 for alpha = 0)
  float cx, cy, cz;              // alpha_lo x alpha_hi
  float h, v;
};

struct Sums6 {
  float ux, uy, uz, sx, sy, sz;
};

__device__ __forceinline__ void rotate(Sums6 &a, int m) {
  a.ux = __shfl_xor_sync(kFull, a.ux, m);
  a.uy = __shfl_xor_sync(kFull, a.uy, m);
  a.uz = __shfl_xor_sync(kFull, a.uz, m);
  a.sx = __shfl_xor_sync(kFull, a.sx, m);
  a.sy = __shfl_xor_sync(kFull, a.sy, m);
  a.sz = __shfl_xor_sync(kFull, a.sz, m);
}

// 32 sources of a near tile against R targets per lane.  DIAG: both tiles are
// the same one, every ordered pair is visited and only the targets' sums are
// kept; the pair of a particle with itself falls on step 0 of target `self`
// (no target when it is outside 0..R-1).  kap: the diffusion factor in the
// units of the s sums (15 nu, or 240 nu / h with one radius).
template <int SIDE, bool UNI, bool DIAG, bool DIFF, int KERN, int R>
__device__ __forceinline__ void near_block(const Stage &st, int lane, const NearTarget (&T)[R], int self,
                                           float hu, float kap, Sums6 (&a)[R], Sums6 &b) {
  // steps per iteration (the Gaussian scalars' code is four times as long): against
  // four, two and eight take 1 % more on near tiles
  constexpr int kUnroll = KERN == KERNEL_GAUSSIAN ? 2 : 4;
  const float s2u = 2.f * hu, c240 = -480.f * hu;
#pragma unroll 1
  for (int kk = 0; kk < 32; kk += kUnroll) {
    const int base = lane ^ kk;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      // (hi position, h), (lo position, volume), (strength, lo.x), (lo.y, lo.z)
      const float4 p = st.s0[base ^ u], pl = st.s1[base ^ u], s = st.s2[base ^ u];
      const float2 l = st.s3[base ^ u];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float dx = (T[r].xh - p.x) + (T[r].xl - pl.x);
        const float dy = (T[r].yh - p.y) + (T[r].yl - pl.y);
        const float dz = (T[r].zh - p.z) + (T[r].zl - pl.z);
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const float ri = rsqrtf(r2);
        float q, fh, dp;
        if (KERN == KERNEL_GAUSSIAN)
          gauss_scalars(T[r].h + p.w, r2, ri, q, fh, dp);
        else if (UNI)
          kernel_scalars_uniform(hu, c240, rsqrtf(r2 + s2u), ri, q, fh, dp);
        else
          kernel_scalars(T[r].h + p.w, rsqrtf(r2 + (T[r].h + p.w)), ri, q, fh, dp);
        // alpha_j x d, and alpha_i x alpha_j from the hi/lo strengths
        const float cx = fmaf(s.y, dz, -s.z * dy);
        const float cy = fmaf(s.z, dx, -s.x * dz);
        const float cz = fmaf(s.x, dy, -s.y * dx);
        float wx, wy, wz, mu, vx, vy, vz;
        projection_cross(T[r].ax, T[r].ay, T[r].az, T[r].iaa, T[r].cx, T[r].cy, T[r].cz, s.x, s.y, s.z,
                         s.w, l.x, l.y, wx, wy, wz, mu, vx, vy, vz);
        const float t = fmaf(dz, wz, fmaf(dy, wy, dx * wx));
        const float ft = 3.0f * fh * t;
        float sx = fmaf(ft, dx, q * wx);
        float sy = fmaf(ft, dy, q * wy);
        float sz = fmaf(ft, dz, q * wz);
        if (DIFF) {
          const float kd = kap * dp, kv = kd * T[r].v, ka = kd * fmaf(T[r].v, mu, -pl.w), kl = -kd * pl.w;
          sx = fmaf(kv, vx, fmaf(ka, T[r].ax, fmaf(kl, T[r].lx, sx)));
          sy = fmaf(kv, vy, fmaf(ka, T[r].ay, fmaf(kl, T[r].ly, sy)));
          sz = fmaf(kv, vz, fmaf(ka, T[r].az, fmaf(kl, T[r].lz, sz)));
        }
        if (DIAG && u == 0) {
          const bool own = kk == 0 && r == self;
          q = own ? 0.f : q;
          sx = own ? 0.f : sx;
          sy = own ? 0.f : sy;
          sz = own ? 0.f : sz;
        }
        if (SIDE != SIDE_J) {
          a[r].ux = fmaf(q, cx, a[r].ux);
          a[r].uy = fmaf(q, cy, a[r].uy);
          a[r].uz = fmaf(q, cz, a[r].uz);
          a[r].sx += sx;
          a[r].sy += sy;
          a[r].sz += sz;
        }
        if (!DIAG && SIDE != SIDE_I) {
          // alpha_i x d; subtracted at the fold
          b.ux = fmaf(q, fmaf(T[r].ay, dz, -T[r].az * dy), b.ux);
          b.uy = fmaf(q, fmaf(T[r].az, dx, -T[r].ax * dz), b.uy);
          b.uz = fmaf(q, fmaf(T[r].ax, dy, -T[r].ay * dx), b.uz);
          b.sx += sx;
          b.sy += sy;
          b.sz += sz;
        }
      }
      const int k = kk + u;
      if (!DIAG && SIDE != SIDE_I) rotate(b, (k ^ (k + 1)) & 31);
    }
  }
}

// (product and sum rounded apart: two passes over the targets add up alike
// whether one warp or two make them)
__device__ __forceinline__ void fold_near(const Sums6 &s, double As2, double *acc, int stride) {
  acc[0] += As2 * s.ux;
  acc[stride] += As2 * s.uy;
  acc[2 * stride] += As2 * s.uz;
  acc[3 * stride] += As2 * s.sx;
  acc[4 * stride] += As2 * s.sy;
  acc[5 * stride] += As2 * s.sz;
}

template <int SIDE, bool UNI, bool DIAG, bool DIFF, int KERN>
__device__ __forceinline__ void near_pair(const SymSeg &sg, int I, int J, int k0, int k1, int ta, int tb,
                                          float hu, const Stage &st, int lane, double *accI, double *accJ) {
  constexpr int R = 2;
  const double As2 = UNI ? kInv4Pi * 2.0 * (double)hu : kInv4Pi;
  const float kap = DIFF ? (float)(UNI ? 240.0 * sg.nu / (double)hu : 15.0 * sg.nu) : 0.f;
  const int n = sg.n;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int t0 = ta; t0 < tb; t0 += 32 * R) {
    NearTarget T[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = I * kT + t0 + 32 * r + lane;
      float4 p = make_float4(kPadTarget, kPadTarget, kPadTarget, 1.f), pl = zero, q = zero, l = zero;
      if (i < n) {
        p = sg.pos32[i];
        pl = sg.poslo[i];
        q = sg.vor32[i];
        l = sg.vorlo[i];
      }
      const float aa = fmaf(q.z, q.z, fmaf(q.y, q.y, q.x * q.x));
      T[r] = NearTarget{p.x, p.y, p.z, pl.x, pl.y, pl.z, q.x, q.y, q.z, l.x, l.y, l.z,
                        aa > 0.f ? 1.0f / aa : 0.f, fmaf(l.y, q.z, -l.z * q.y),
                        fmaf(l.z, q.x, -l.x * q.z), fmaf(l.x, q.y, -l.y * q.x), p.w, q.w};
    }
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int j = J * kT + 32 * k + lane;
      float4 p = make_float4(kPadSource, kPadSource, kPadSource, 1.f), pl = zero, q = zero, l = zero;
      if (j < n) {
        p = sg.pos32[j];
        pl = sg.poslo[j];
        q = sg.vor32[j];
        l = sg.vorlo[j];
      }
      st.s0[lane] = p;
      st.s1[lane] = make_float4(pl.x, pl.y, pl.z, q.w);
      st.s2[lane] = make_float4(q.x, q.y, q.z, l.x);
      st.s3[lane] = make_float2(l.y, l.z);
      __syncwarp();
      Sums6 a[R], b{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = b;
      near_block<SIDE, UNI, DIAG, DIFF, KERN, R>(st, lane, T, k - t0 / 32, hu, kap, a, b);
      if (SIDE != SIDE_J) {
#pragma unroll
        for (int r = 0; r < R; ++r) fold_near(a[r], As2, accI + t0 + 32 * r + lane, kT);
      }
      if (!DIAG && SIDE != SIDE_I) fold_near(b, -As2, accJ + 32 * k + lane, kT);
      __syncwarp();
    }
  }
}

// One tile pair (I <= J), sub-blocks [k0, k1) of J's sources and the targets [ta,
// tb) of I (all of them, when ta is 0, in the classes of one pass), in the class that
// the two tiles' boxes allow.  The classes and their bounds are pair_f32.cu's;
// the far formulation is centred on the smaller of the two boxes, whose
// half-diagonal bounds |x'_i| + |x'_j| by 3 |d| for every pair.
template <int SIDE, bool DIFF, int KERN, int UNROLL>
__device__ __forceinline__ void tile_pair(const SymSeg &sg, int I, int J, int k0, int k1, int ta, int tb,
                                          const Stage &st, int lane, double *accI, double *accJ) {
  const float4 alo = sg.boxes[2 * I], ahi = sg.boxes[2 * I + 1];
  const float4 blo = sg.boxes[2 * J], bhi = sg.boxes[2 * J + 1];
  const bool uni = KERN == KERNEL_HIGHORDER && alo.w == ahi.w && blo.w == bhi.w && alo.w == blo.w;
  const float hu = alo.w;
  if (SIDE == SIDE_BOTH && I == J) {  // (a tile pair of one side has tiles of two processes)
    if (uni)
      near_pair<SIDE_BOTH, true, true, DIFF, KERN>(sg, I, J, k0, k1, ta, tb, hu, st, lane, accI, accJ);
    else
      near_pair<SIDE_BOTH, false, true, DIFF, KERN>(sg, I, J, k0, k1, ta, tb, hu, st, lane, accI, accJ);
    return;
  }
  const float gap2 = box_gap2(alo, ahi, blo, bhi);
  const float da = box_half_diag2(alo, ahi), db = box_half_diag2(blo, bhi);
  const bool first = da < db;
  const bool far = gap2 > 0.f && gap2 >= sg.near2 && gap2 >= (first ? da : db);
  if (!far) {
    if (uni)
      near_pair<SIDE, true, false, DIFF, KERN>(sg, I, J, k0, k1, ta, tb, hu, st, lane, accI, accJ);
    else
      near_pair<SIDE, false, false, DIFF, KERN>(sg, I, J, k0, k1, ta, tb, hu, st, lane, accI, accJ);
    return;
  }
  const float4 lo = first ? alo : blo, hi = first ? ahi : bhi;
  const float cx = 0.5f * (lo.x + hi.x), cy = 0.5f * (lo.y + hi.y), cz = 0.5f * (lo.z + hi.z);
  const float sig2max = ahi.w + bhi.w;
  if (KERN == KERNEL_GAUSSIAN) {
    if (gap2 >= 49.f * sig2max)
      far_pair<SIDE, FAR_SER, false, DIFF, KERN, 4, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
    else
      far_pair<SIDE, FAR_Z, false, DIFF, KERN, 2, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
    return;
  }
  if (gap2 >= 256.f * sig2max) {
    if (uni)
      far_pair<SIDE, FAR_SER, true, DIFF, KERN, 4, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
    else
      far_pair<SIDE, FAR_SER, false, DIFF, KERN, 4, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
  } else if (gap2 >= 36.f * sig2max) {
    if (uni)
      far_pair<SIDE, FAR_NZ, true, DIFF, KERN, 4, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
    else
      far_pair<SIDE, FAR_NZ, false, DIFF, KERN, 4, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
  } else {
    if (uni)
      far_pair<SIDE, FAR_Z, true, DIFF, KERN, 2, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
    else
      far_pair<SIDE, FAR_Z, false, DIFF, KERN, 2, UNROLL>(sg, I, J, k0, k1, ta, tb, cx, cy, cz, hu, st, lane, accI, accJ);
  }
}

template <bool DIFF, int KERN, int UNROLL>
struct Pair32 {
  static constexpr int kStageBytes = ::pawan::kStageBytes;
  template <int SIDE>
  static __device__ __forceinline__ void tile_pair(const SymSeg &sg, int I, int J, int k0, int k1, int ta, int tb,
                                                   char *st, int lane, double *accI, double *accJ) {
    ::pawan::tile_pair<SIDE, DIFF, KERN, UNROLL>(sg, I, J, k0, k1, ta, tb, stage_of(st), lane, accI, accJ);
  }
};

// Steps of the far loop per iteration: four where the registers and the code
// (two far classes instead of six) leave room, the Gaussian kernel's single tile
// pairs (N = 32,000 1,021 -> 993 us).  In groups four spill (65,536 particles 3.69
// -> 3.98 ms), and with the default kernel's classes they gain 1 % at 32,768 and
// lose 2-5 % at 2,100 to 4,096.
template <bool DIFF, int KERN>
using TilePair32 = Pair32<DIFF, KERN, KERN == KERNEL_GAUSSIAN ? 4 : 2>;

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, kBlocks)
    sym_f32_group_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                         const int *__restrict__ jbase, double *__restrict__ slots) {
  group_item<Pair32<DIFF, KERN, 2>>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, kBlocks)
    sym_f32_tile_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                        const int *__restrict__ jbase, double *__restrict__ slots) {
  tile_item<TilePair32<DIFF, KERN>>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(Spread<1>::threads, 1)
    sym_f32_wide_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                        const int *__restrict__ jbase, double *__restrict__ slots) {
  spread_item<TilePair32<DIFF, KERN>, 1>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(Spread<2>::threads, 2)
    sym_f32_spread_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                          const int *__restrict__ jbase, double *__restrict__ slots) {
  spread_item<TilePair32<DIFF, KERN>, 2>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, kBlocks)
    sym_f32_group_sided_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                               const int *__restrict__ jbase, double *__restrict__ slots) {
  sided_item<Pair32<DIFF, KERN, 2>, true>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, kBlocks)
    sym_f32_tile_sided_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                              const int *__restrict__ jbase, double *__restrict__ slots) {
  sided_item<TilePair32<DIFF, KERN>, false>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
SymKernel select_k(int shape, bool sided) {
  if (sided) return shape == SYM_GROUP ? &sym_f32_group_sided_kernel<DIFF, KERN> : &sym_f32_tile_sided_kernel<DIFF, KERN>;
  return shape == SYM_GROUP  ? &sym_f32_group_kernel<DIFF, KERN>
         : shape == SYM_TILE ? &sym_f32_tile_kernel<DIFF, KERN>
         : shape == SYM_WIDE ? &sym_f32_wide_kernel<DIFF, KERN>
                             : &sym_f32_spread_kernel<DIFF, KERN>;
}

SymKernel select(int shape, bool sided, bool diffusion, int kernel) {
  if (kernel == KERNEL_GAUSSIAN)
    return diffusion ? select_k<true, KERNEL_GAUSSIAN>(shape, sided) : select_k<false, KERNEL_GAUSSIAN>(shape, sided);
  return diffusion ? select_k<true, KERNEL_HIGHORDER>(shape, sided) : select_k<false, KERNEL_HIGHORDER>(shape, sided);
}

}  // namespace

cudaError_t sym_f32_occupancy(bool diffusion, int kernel, int *blocks_per_sm) {
  return sym_occupancy(select(SYM_GROUP, false, diffusion, kernel), sym_smem_bytes(SYM_GROUP, kStageBytes), blocks_per_sm);
}

cudaError_t launch_sym_f32(bool group, bool sided, bool diffusion, int kernel, const SymItem *items, int n_items,
                           int sm_count, const SymSeg *segs, const int *jbase, double *slots, cudaStream_t s) {
  // Up to one tile pair per SM a launch lasts as long as one tile pair's chain of
  // steps: eight warps take it in less time than four, and two SMs in less than
  // one (two warps a scheduler issue at 0.8 per cycle, one alone at 0.6).  One
  // right-hand side as an RK4 stage runs it, wide / spread: n = 64 13.5 / 10.9 us,
  // 512 16.2 / 13.0, 1,408 17.5 / 14.5.  With more than two blocks per SM-pair the
  // clusters are not placed evenly: 2,048 19.1 / 21.8 (four warps: 24.6).
  const int shape = group                     ? SYM_GROUP
                    : sided                   ? SYM_TILE
                    : 2 * n_items <= sm_count ? SYM_SPREAD
                    : n_items <= sm_count     ? SYM_WIDE
                                              : SYM_TILE;
  return sym_launch(select(shape, sided, diffusion, kernel), shape, kStageBytes, items, n_items, segs, jbase, slots, s);
}

}  // namespace pawan
