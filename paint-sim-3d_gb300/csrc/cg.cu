// cg.cu — the implicit hydrostatic steps of a frame (film.wgsl:895-1302,
// dispatched by Film::encode_frame, src/film/mod.rs:1373-1408): per step a
// Jacobi-preconditioned conjugate-gradient solve of the hydrostatic flow of
// the frame over the active tiles, then the flux it implies and a mass
// rescale.
//
// Layout of the work (one film alone or many in a packed launch):
//  - kp_cg_setup: the face mobilities cg_m (and, with the implicit capillary
//    term, cg_t / cg_t2, the weighted Laplacians of h and of the hold level);
//  - kp_cg_init: diagonal, right-hand side, residual, first direction;
//  - kp_cg_solve: every iteration in one cooperative launch whose blocks walk
//    the active tiles that hold paint: phase a forms the search direction
//    p_k = r / d + beta p_{k-1} of the tile and its halo on the fly (so the
//    reference's cg_iter_c needs no pass of its own) and computes q = A p_k,
//    phase b updates r; after each phase the blocks meet, and the tiles'
//    partials are summed and the film's scalars updated: of a film alone by
//    every block for itself, of several by one group of threads a film, after
//    which the blocks meet again.  With the
//    implicit capillary term (off by default) the iterations are separate
//    launches instead (kp_cg_lap_p, kp_cg_iter_a, kp_cg_iter_b and
//    kp_cg_scalars), which also form the Laplacian of the direction;
//  - kp_cg_finish: the flux of the step into acc, the new h into a side plane
//    (neighbours read h as of before the dispatch), the final direction into
//    cg_p; kp_cg_rescale: the mass correction and the h commit.
// Each sum over a film (p.q, r.z, the mass change) is a per-tile tree sum
// and the film's total of them in tile order; in the once-per-step kernels it
// is formed by the last block to finish (an atomic count, no waiting).  A
// neighbour in an inactive tile is read as the reference reads it: its cg_m and
// cg_p as the last step that covered it left them.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "film_kernels.h"

namespace cfk {

namespace {

__device__ __forceinline__ float kappa(const cf_params& P) {  // film.wgsl:925-927
  return P.front[3] * P.phys[0] * P.g[2] * P.inv_dx * P.inv_dx;
}
__device__ __forceinline__ float hold_u(const Film& F, const cf_params& P, uint32_t c) {  // film.wgsl:929-933
  float hold = 0.f;
  if (F.hh[c] > 0.f) hold = hold_level(P, nose_dist(F, c));
  return F.m[c] - hold;
}

// film.wgsl:895-923: the mobility of a face (the face's flow index as in face())
template <int MODE>
__device__ float face_mob(const Film& F, const cf_params& P, uint32_t ca, uint32_t cb, float2 gcap, float2 ghyd,
                          float2 gtilt, bool diag) {
  const float ha = F.hh[ca], hb = F.hh[cb];
  if (fminf(ha, hb) <= 0.f) return 0.f;
  const float hf = 0.5f * (ha + hb);
  const float rax = rmu<MODE>(F, ca), ray = rtau<MODE>(F, ca);
  const float rbx = rmu<MODE>(F, cb), rby = rtau<MODE>(F, cb);
  const float wa = ha / (ha + hb);
  const float wb = 1.0f - wa;
  const float mu = expf(wa * logf(fmaxf(rax, 1e-4f)) + wb * logf(fmaxf(rbx, 1e-4f)));
  const float ty = wa * ray + wb * rby;
  const float na = rn<MODE>(F, ca), nb = rn<MODE>(F, cb);
  const float nf = na == nb ? na : wa * na + wb * nb;
  const float thin = fminf(ha, hb) / hf;
  const float fcap = thin * thin * thin;
  float2 yc = make_float2(gcap.x * fcap, gcap.y * fcap);  // yield_cap (film.wgsl:44-49)
  {
    const float gcl = sqrtf(yc.x * yc.x + yc.y * yc.y);
    const float gc_max = P.phys[1] / (1e-3f * 1e-3f);
    if (!(ty <= 0.f || gcl <= gc_max)) {
      const float sc = gc_max / gcl;
      yc.x = yc.x * sc;
      yc.y = yc.y * sc;
    }
  }
  const float2 gg = make_float2(yc.x + ghyd.x + gtilt.x, yc.y + ghyd.y + gtilt.y);
  const float gmag = sqrtf(gg.x * gg.x + gg.y * gg.y);
  float ydep = hf;  // yield_depth (film.wgsl:89-92)
  if (ty > 0.f) ydep = gg.x >= 0.f ? ha : hb;
  float qq, qy, qup;
  hb_flux(gmag, ydep, mu, ty, nf, qq, qy, qup);
  if (qq <= 0.f) return 0.f;
  float mob = fminf(fmaxf(qq / gmag - P.misc[3], 0.f), P.front[2]);
  if (fminf(ha, hb) < 0.5f * fmaxf(ha, hb)) {
    if (diag) return 0.f;
    const uint32_t tgt = hb > ha ? ca : cb;
    mob = mob / powf((float)max(feeders(F, P, tgt), 1u), 0.7f);
  }
  return mob;
}

// film.wgsl:994-1010: neighbour k of (i, j) and the weighted mobility of the
// face to it; faces 4..7 belong to the lower-left neighbours
__device__ __forceinline__ bool cg_nb(const Film& F, int k, int i, int j, uint32_t& nc, float& mw) {
  const uint32_t c = idx(F, i, j);
  nc = 0u;
  mw = 0.f;
  const int W = (int)F.w, H = (int)F.h;
  switch (k) {
    case 0: if (i + 1 < W) { nc = idx(F, i + 1, j); mw = W_AXIS * F.cg_m[c].x; } break;
    case 1: if (j + 1 < H) { nc = idx(F, i, j + 1); mw = W_AXIS * F.cg_m[c].y; } break;
    case 2: if (i + 1 < W && j + 1 < H) { nc = idx(F, i + 1, j + 1); mw = W_DIAG_LAP * F.cg_m[c].z; } break;
    case 3: if (i + 1 < W && j > 0) { nc = idx(F, i + 1, j - 1); mw = W_DIAG_LAP * F.cg_m[c].w; } break;
    case 4: if (i > 0) { nc = idx(F, i - 1, j); mw = W_AXIS * F.cg_m[nc].x; } break;
    case 5: if (j > 0) { nc = idx(F, i, j - 1); mw = W_AXIS * F.cg_m[nc].y; } break;
    case 6: if (i > 0 && j > 0) { nc = idx(F, i - 1, j - 1); mw = W_DIAG_LAP * F.cg_m[nc].z; } break;
    default: if (i > 0 && j + 1 < H) { nc = idx(F, i - 1, j + 1); mw = W_DIAG_LAP * F.cg_m[nc].w; } break;
  }
  return mw > 0.f;
}

// film.wgsl:1023-1043: sum over wet active neighbours of w (v(n) - v(c))
template <class Src>
__device__ __forceinline__ float lap_w(const Film& F, int i, int j, uint32_t c, Src v) {
  const float vc = v(c);
  float acc_v = 0.f;
  for (int dj = -1; dj <= 1; ++dj)
    for (int di = -1; di <= 1; ++di) {
      if (di == 0 && dj == 0) continue;
      const int x = i + di, y = j + dj;
      if (x < 0 || y < 0 || x >= (int)F.w || y >= (int)F.h) continue;
      if (!cell_active(F, x, y)) continue;
      const uint32_t n = idx(F, x, y);
      if (F.hh[n] <= 0.f) continue;
      const float w = (di != 0 && dj != 0) ? W_DIAG_LAP : W_AXIS;
      acc_v += w * (v(n) - vc);
    }
  return acc_v;
}
// film.wgsl:1045-1064
__device__ __forceinline__ float lap_diag(const Film& F, int i, int j) {
  float s1 = 0.f, s2 = 0.f;
  for (int dj = -1; dj <= 1; ++dj)
    for (int di = -1; di <= 1; ++di) {
      if (di == 0 && dj == 0) continue;
      const int x = i + di, y = j + dj;
      if (x < 0 || y < 0 || x >= (int)F.w || y >= (int)F.h) continue;
      if (!cell_active(F, x, y)) continue;
      if (F.hh[idx(F, x, y)] <= 0.f) continue;
      const float w = (di != 0 && dj != 0) ? W_DIAG_LAP : W_AXIS;
      s1 += w;
      s2 += w * w;
    }
  return s1 * s1 + s2;
}

// The sum of a 256-thread block's values (the shader sums its workgroup
// with a tree, film.wgsl:1099-1107; this is a tree too, by warp shuffles, then
// over the 8 warps): every thread gets the total.
__device__ __forceinline__ float block_tree(float* sv, float v) {
  const uint32_t li = threadIdx.y * 16u + threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // sv may still be read by a previous call
  if ((li & 31u) == 0u) sv[li >> 5] = v;
  __syncthreads();
  float t = sv[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) t += sv[w];
  return t;
}

// Writes this block's tile partial(s), then reports whether it is the last
// block of the film to do so (the caller then sums the film's partials).  The
// count is two-level: a counter per group of 32 tiles, and the film's counter
// taken only by each group's last block, so no address takes more than a few
// hundred atomics per launch (one counter per film serialised 16 k atomics at
// 2048^2, tens of microseconds per launch).
__device__ __forceinline__ bool last_block(const Film& F, uint32_t t, float part, float part2) {
  __shared__ uint32_t s_last;
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    F.cg_part[t] = part;
    F.cg_part2[t] = part2;
    __threadfence();
    const uint32_t nt = F.tw * F.th, g = t >> 5, ng = (nt + 31u) >> 5;
    const uint32_t in_group = min(32u, nt - (g << 5));
    s_last = 0u;
    if (atomicAdd(&F.cg_cnt[g], 1u) == in_group - 1u) {
      F.cg_cnt[g] = 0u;  // every block of the group has counted
      __threadfence();
      s_last = atomicAdd(&F.cg->blocks_done, 1u) == ng - 1u ? 1u : 0u;
    }
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last != 0u;
}

// The film's total of the tile partials, by the last block: each thread's
// strided sum over the tiles in order, then the tree (as total_parts,
// film.wgsl:1157-1168, over every tile; inactive tiles add 0).
__device__ __forceinline__ float film_total(const Film& F, const float* part, float* sv) {
  const uint32_t li = threadIdx.y * 16u + threadIdx.x, nt = F.tw * F.th;
  float v = 0.f;
  for (uint32_t t = li; t < nt; t += 256u) v += __ldcg(part + t);
  return block_tree(sv, v);
}

#define CG_ARGS const Film* __restrict__ films, const uint2* __restrict__ tiles, uint32_t ntiles
#define CG_TILE                                                          \
  if (blockIdx.x >= ntiles) return;                                      \
  const uint2 pe_ = tile_entry(tiles, blockIdx.x);                       \
  const Film& F = films[pe_.x];                                          \
  const DevParams& D = *F.P;                                             \
  const cf_params& P = D.p;                                              \
  const uint32_t t = pe_.y;                                              \
  const int i = (int)((t % F.tw) * 16u + threadIdx.x);                   \
  const int j = (int)((t / F.tw) * 16u + threadIdx.y);                   \
  const bool tile_on = (F.tile_flags[t] & ACTIVE) != 0u;                 \
  const bool cell_on = tile_on && i < (int)F.w && j < (int)F.h;          \
  const uint32_t c = cell_on ? idx(F, i, j) : 0u;                        \
  (void)c;

// film.wgsl:935-987 (+ cg_lap_h, film.wgsl:1073-1078, when the implicit
// capillary term is on)
template <int MODE>
__global__ void __launch_bounds__(256) kp_cg_setup(CG_ARGS, uint32_t step) {
  CG_TILE
  if (step >= D.implicit_steps || !cell_on) return;
  float4 mob = make_float4(0.f, 0.f, 0.f, 0.f);
  if (P.front3[0] == 0.f && (F.tile_flags[t] & 1u) == 0u) {  // a dry cell's faces have no mobility
    F.cg_m[c] = mob;
    return;
  }
  const float2 p00 = pres_at(F, i, j);
  const float2 gxy = make_float2(P.phys[0] * P.g[0], P.phys[0] * P.g[1]);
  const float s2 = 0.70710678f;
  if (i + 1 < (int)F.w && cell_active(F, i + 1, j)) {
    const float2 p10 = pres_at(F, i + 1, j);
    const float2 gm = make_float2(-(p10.x - p00.x) * P.inv_dx, -(p10.y - p00.y) * P.inv_dx);
    const float2 a = pres_wet(F, i, j + 1, p00), b = pres_wet(F, i + 1, j + 1, p10);
    const float2 cc = pres_wet(F, i, j - 1, p00), d = pres_wet(F, i + 1, j - 1, p10);
    const float2 pt = make_float2(a.x + b.x - cc.x - d.x, a.y + b.y - cc.y - d.y);
    const float2 gt = make_float2(-pt.x * 0.25f * P.inv_dx, -pt.y * 0.25f * P.inv_dx);
    mob.x = face_mob<MODE>(F, P, c, idx(F, i + 1, j), make_float2(gm.x, gt.x), make_float2(gm.y, gt.y), gxy, false);
  }
  if (j + 1 < (int)F.h && cell_active(F, i, j + 1)) {
    const float2 p01 = pres_at(F, i, j + 1);
    const float2 gm = make_float2(-(p01.x - p00.x) * P.inv_dx, -(p01.y - p00.y) * P.inv_dx);
    const float2 a = pres_wet(F, i + 1, j, p00), b = pres_wet(F, i + 1, j + 1, p01);
    const float2 cc = pres_wet(F, i - 1, j, p00), d = pres_wet(F, i - 1, j + 1, p01);
    const float2 pt = make_float2(a.x + b.x - cc.x - d.x, a.y + b.y - cc.y - d.y);
    const float2 gt = make_float2(-pt.x * 0.25f * P.inv_dx, -pt.y * 0.25f * P.inv_dx);
    mob.y = face_mob<MODE>(F, P, c, idx(F, i, j + 1), make_float2(gm.x, gt.x), make_float2(gm.y, gt.y),
                           make_float2(gxy.y, gxy.x), false);
  }
  if (i + 1 < (int)F.w && j + 1 < (int)F.h && cell_active(F, i + 1, j + 1)) {
    const float2 p11 = pres_at(F, i + 1, j + 1);
    const float2 ga = make_float2(-(p11.x - p00.x) * P.inv_dx * s2, -(p11.y - p00.y) * P.inv_dx * s2);
    const float2 pa = pres_wet(F, i + 1, j, p00), pb = pres_wet(F, i, j + 1, p11);
    const float2 gp = make_float2(-(pa.x - pb.x) * P.inv_dx * s2, -(pa.y - pb.y) * P.inv_dx * s2);
    const float2 gt = make_float2((gxy.x + gxy.y) * s2, (gxy.x - gxy.y) * s2);
    mob.z = face_mob<MODE>(F, P, c, idx(F, i + 1, j + 1), make_float2(ga.x, gp.x), make_float2(ga.y, gp.y), gt,
                           true);
  }
  if (i + 1 < (int)F.w && j > 0 && cell_active(F, i + 1, j - 1)) {
    const float2 p1m = pres_at(F, i + 1, j - 1);
    const float2 ga = make_float2(-(p1m.x - p00.x) * P.inv_dx * s2, -(p1m.y - p00.y) * P.inv_dx * s2);
    const float2 pa = pres_wet(F, i + 1, j, p00), pb = pres_wet(F, i, j - 1, p1m);
    const float2 gp = make_float2(-(pa.x - pb.x) * P.inv_dx * s2, -(pa.y - pb.y) * P.inv_dx * s2);
    const float2 gt = make_float2((gxy.x - gxy.y) * s2, (gxy.x + gxy.y) * s2);
    mob.w = face_mob<MODE>(F, P, c, idx(F, i + 1, j - 1), make_float2(ga.x, gp.x), make_float2(ga.y, gp.y), gt,
                           true);
  }
  F.cg_m[c] = mob;
  if (P.front3[0] != 0.f) {  // cg_lap_h
    F.cg_t[c] = lap_w(F, i, j, c, [&](uint32_t n) { return F.hh[n]; });
    F.cg_t2[c] = lap_w(F, i, j, c, [&](uint32_t n) { return hold_u(F, P, n); });
  }
}

// The matrix weights of a cell's own faces (film.wgsl:1083-1094): kappa times
// the weighted mobility.
__device__ __forceinline__ float4 face_weights(float k, float4 mob) {
  return make_float4(k * (W_AXIS * mob.x), k * (W_AXIS * mob.y), k * (W_DIAG_LAP * mob.z), k * (W_DIAG_LAP * mob.w));
}

// film.wgsl:1110-1141 and cg_reduce_init (film.wgsl:1170-1176).  The heights
// and hold potentials (an exp each) of the tile and a one-cell halo are
// evaluated once into shared memory, for the nine cells that read each; the
// terms of the implicit capillary part are left out where it is off (they add
// zero).  With LEAN (the solve follows) the faces' weights go to the flux
// plane, which the frame's substeps write afresh after the solve, and a tile
// without paint writes its x alone: nothing else of it is read.
template <bool LEAN>
__global__ void __launch_bounds__(256) kp_cg_init(CG_ARGS, uint32_t step) {
  CG_TILE
  if (step >= D.implicit_steps) return;
  __shared__ float sv[256];
  __shared__ float sh[18][18], su[18][18];
  float v = 0.f;
  if (LEAN && tile_on && (F.tile_flags[t] & 1u) == 0u) {
    if (cell_on) F.cg_x[c] = F.hh[c];
  } else if (tile_on) {
    const int li = (int)(threadIdx.y * 16u + threadIdx.x);
    const int x0 = (int)(t % F.tw) * 16 - 1, y0 = (int)(t / F.tw) * 16 - 1;
    for (int e = li; e < 18 * 18; e += 256) {
      const int x = x0 + e % 18, y = y0 + e / 18;
      if (x >= 0 && y >= 0 && x < (int)F.w && y < (int)F.h) {
        const uint32_t n = idx(F, x, y);
        sh[e / 18][e % 18] = F.hh[n];
        su[e / 18][e % 18] = hold_u(F, P, n);
      }
    }
    __syncthreads();
    if (cell_on) {
      const int lx = (int)threadIdx.x + 1, ly = (int)threadIdx.y + 1;
      const float k = kappa(P), hc = sh[ly][lx], uc = su[ly][lx];
      float diag = 1.0f, b = hc, ax = hc;
#pragma unroll
      for (int f = 0; f < 8; ++f) {
        uint32_t nc;
        float mw;
        if (cg_nb(F, f, i, j, nc, mw)) {
          // neighbour f of cg_nb: right, up, up-right, down-right, left, down, down-left, up-left
          const int di = f == 1 || f == 5 ? 0 : f < 4 ? 1 : -1;
          const int dj = f == 0 || f == 4 ? 0 : f == 1 || f == 2 || f == 7 ? 1 : -1;
          diag += k * mw;
          b += k * mw * (su[ly + dj][lx + di] - uc);
          ax += k * mw * (hc - sh[ly + dj][lx + di]);
        }
      }
      const float cc = P.front3[0];
      if (hc > 0.f && cc != 0.f) {
        diag += cc * lap_diag(F, i, j);
        b -= cc * lap_w(F, i, j, c, [&](uint32_t n) { return F.cg_t2[n]; });
        ax += cc * lap_w(F, i, j, c, [&](uint32_t n) { return F.cg_t[n]; });
      }
      const float r = b - ax;
      if (LEAN) {  // the solve's weights of the cell's own faces
        const float4 mob = F.cg_m[c];
        F.flux[c] = face_weights(k, mob);
      }
      F.cg_d[c] = diag;
      F.cg_x[c] = hc;
      F.cg_r[c] = r;
      F.cg_pa[c] = r / diag;
      v = r * r / diag;
    }
  }
  const float part = block_tree(sv, v);
  // cg_part2 is the solve's other set of partials: 0 for the tiles it leaves out
  if (last_block(F, t, part, 0.f)) {
    const float rz = film_total(F, F.cg_part, sv);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
      CgState& S = *F.cg;
      S.rz = rz; S.pq = 0.f; S.alpha = 0.f; S.beta = 0.f;
      S.s1x = rz; S.dv = 0.f; S.tv = 0.f; S.s0x = 0.f;
      S.blocks_done = 0u;
      S.failed = 0u;
    }
  }
}

// The search direction of iteration `it` at cell n: the init's one for it = 0,
// else r / d + beta p_{it-1} (film.wgsl:1150-1155); an inactive cell keeps the
// last one the reference left in cg_p.
__device__ __forceinline__ float dir_at(const Film& F, uint32_t n, bool active, uint32_t it, float beta,
                                        const float* prev) {
  if (!active) return F.cg_p[n];
  if (it == 0u) return prev[n];
  return F.cg_r[n] / F.cg_d[n] + beta * prev[n];
}

// cg_lap_p (film.wgsl:1066-1071), only with the implicit capillary term: it
// also forms the direction of the iteration (kp_cg_iter_a then reads it).
__global__ void __launch_bounds__(256) kp_cg_lap_p(CG_ARGS, uint32_t step, uint32_t it) {
  CG_TILE
  if (step >= D.implicit_steps || it >= D.implicit_iters || !cell_on) return;
  const float* prev = (it & 1u) || it == 0u ? F.cg_pa : F.cg_pb;  // p_{it-1}; the init's p for it = 0
  const float beta = F.cg->beta;
  auto p_of = [&](uint32_t n) {
    const int x = (int)(n % F.w), y = (int)(n / F.w);
    return dir_at(F, n, cell_active(F, x, y), it, beta, prev);
  };
  F.cg_t[c] = lap_w(F, i, j, c, p_of);
  F.cg_q[c] = p_of(c);  // the new direction, stored by kp_cg_iter_a
}

// cg_iter_a (film.wgsl:1109-1120, apply_a :1083-1094) and cg_reduce_a
// (film.wgsl:1214-1222) with the implicit capillary term; the direction of
// the iteration is the one kp_cg_lap_p formed (the fused cg_iter_c of the
// previous iteration).
__global__ void __launch_bounds__(256) kp_cg_iter_a(CG_ARGS, uint32_t step, uint32_t it) {
  CG_TILE
  if (step >= D.implicit_steps || it >= D.implicit_iters) return;
  __shared__ float sv[256];
  // p_it goes to cg_pa for even it, cg_pb for odd; p_{it-1} is in the other
  // (for it = 0 the init's direction, in cg_pa)
  const float* prev = (it & 1u) || it == 0u ? F.cg_pa : F.cg_pb;
  float* cur = (it & 1u) ? F.cg_pb : F.cg_pa;
  const float beta = F.cg->beta;
  float v = 0.f;
  if (cell_on) {
    const float pc = F.cg_q[c];
    const float k = kappa(P);
    float acc_v = pc;
    for (int f = 0; f < 8; ++f) {
      uint32_t nc;
      float mw;
      if (cg_nb(F, f, i, j, nc, mw)) {
        const int x = (int)(nc % F.w), y = (int)(nc / F.w);
        const float pn = dir_at(F, nc, cell_active(F, x, y), it, beta, prev);
        acc_v += k * mw * (pc - pn);
      }
    }
    if (F.hh[c] > 0.f && P.front3[0] != 0.f)
      acc_v += P.front3[0] * lap_w(F, i, j, c, [&](uint32_t n) { return F.cg_t[n]; });
    v = pc * acc_v;
    cur[c] = pc;  // other blocks read p_{it-1} from the other plane
    F.cg_q[c] = acc_v;
  }
  const float part = block_tree(sv, v);
  if (threadIdx.x == 0 && threadIdx.y == 0) F.cg_part[t] = part;  // summed by kp_cg_scalars
}

// cg_iter_b (film.wgsl:1122-1135) and cg_reduce_b (film.wgsl:1224-1232)
__global__ void __launch_bounds__(256) kp_cg_iter_b(CG_ARGS, uint32_t step, uint32_t it) {
  CG_TILE
  if (step >= D.implicit_steps || it >= D.implicit_iters) return;
  __shared__ float sv[256];
  const float* cur = (it & 1u) ? F.cg_pb : F.cg_pa;
  const float alpha = F.cg->alpha;
  float v = 0.f;
  if (cell_on) {
    const float r = F.cg_r[c] - alpha * F.cg_q[c];
    F.cg_x[c] = F.cg_x[c] + alpha * cur[c];
    F.cg_r[c] = r;
    v = r * r / F.cg_d[c];
  }
  const float part = block_tree(sv, v);
  if (threadIdx.x == 0 && threadIdx.y == 0) F.cg_part[t] = part;  // summed by kp_cg_scalars
}

// cg_reduce_a (film.wgsl:1214-1222) after kp_cg_iter_a, cg_reduce_b
// (:1224-1232) after kp_cg_iter_b: one block per film sums its tile partials
// (each thread's strided sum in tile order, then the tree) and updates the
// film's scalars.  A separate launch instead of a last-block count: at 2048^2
// the fence and atomics of 16 k blocks made the iteration kernels several
// times slower than their loads.
__global__ void __launch_bounds__(256) kp_cg_scalars(const Film* __restrict__ films, uint32_t nfilms, uint32_t step,
                                                     uint32_t it, int after_b) {
  if (blockIdx.x >= nfilms) return;
  const Film& F = films[blockIdx.x];
  const DevParams& D = *F.P;
  if (step >= D.implicit_steps || it >= D.implicit_iters) return;
  __shared__ float sv[256];
  const float total = film_total(F, F.cg_part, sv);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    CgState& S = *F.cg;
    if (!after_b) {
      S.pq = total;
      S.alpha = total > 0.f ? S.rz / total : 0.f;
      S.beta = 0.f;
    } else {
      S.beta = S.rz > 0.f ? total / S.rz : 0.f;
      S.rz = total;
    }
  }
}

// ---- the iterations without the implicit capillary term, in one launch ----
__device__ __forceinline__ uint32_t load_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// The solve's blocks: GROUPS groups of 256 threads, each with SPAN tiles of
// the table at a time, one cell of every tile a thread.  The loads of the
// tiles are in flight together and their sums are formed side by side: with
// one tile a group, most of a phase was the chain flags, loads, barrier, sum
// of one tile after the other.  One block an SM (64 registers), so that few
// blocks have to meet: a meet costs 2.6 us, a round of tiles in a phase 8 us.
// Frames in ms at GROUPS / SPAN / PER_SM, 1200x800 pours and 2048^2 pours: 4/2/1
// 13.6 and 8.8, 3/2/2 14.1 and 8.5, 4/1/2 14.2 and 9.1, 3/1/2 14.0 and 9.3; as
// three launches an iteration 16.3 and 16.4.
constexpr int GROUPS = 4, SPAN = 2, PER_SM = 1;
__device__ __forceinline__ void group_sync() {
  asm volatile("bar.sync %0, 256;" ::"r"(threadIdx.z + 1u) : "memory");
}
__device__ __forceinline__ bool lead_thread() { return threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0; }

// All blocks of a cooperative launch meet: what each wrote before is visible
// to all after.  `meet` counts the launch's meetings from 1.  Returns false
// when the wait ran out after `polls`: the caller leaves the solve.
// The wait polls the count of arrivals with relaxed loads and fences once: an
// acquiring poll empties the SM's L1 each time.
__device__ __forceinline__ bool blocks_meet(CgState* M, uint32_t& meet, uint32_t polls) {
  __shared__ uint32_t s_ok;
  ++meet;
  __syncthreads();
  if (lead_thread()) {
    uint32_t ok = 1u, k = 0;
    fence_gpu();
    atomicAdd(&M->met, 1u);
    while (load_relaxed(&M->met) < meet * gridDim.x) {
      if (k++ >= polls) {
        ok = 0u;
        break;
      }
    }
    fence_gpu();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0u;
}
// Every block calls this as its last act; the last to leave clears the
// meeting point for the next launch.
__device__ __forceinline__ void blocks_leave(CgState* M) {
  __syncthreads();
  if (lead_thread()) {
    fence_gpu();
    if (atomicAdd(&M->left, 1u) == gridDim.x - 1u) {
      M->met = 0u;
      M->left = 0u;
    }
  }
}

// The sum of a 256-thread group's values in block_tree's order, in its first
// thread.
__device__ __forceinline__ float group_tree(float* sv, float v) {
  const uint32_t li = threadIdx.y * 16u + threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((li & 31u) == 0u) sv[li >> 5] = v;
  group_sync();
  float t = sv[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) t += sv[w];
  return t;
}
// The partials of a group's SPAN tiles, each in block_tree's order: the sum
// of tile u in thread u.
__device__ __forceinline__ float span_trees(float (*sv)[8], float v[SPAN]) {
  const uint32_t li = threadIdx.y * 16u + threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int u = 0; u < SPAN; ++u) v[u] += __shfl_xor_sync(0xffffffffu, v[u], o);
  if ((li & 31u) == 0u) {
#pragma unroll
    for (int u = 0; u < SPAN; ++u) sv[u][li >> 5] = v[u];
  }
  group_sync();
  float t = 0.f;
  if (li < SPAN) {
    t = sv[li][0];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += sv[li][w];
  }
  return t;
}
// The film's total of the partials (film_total's order), by one group, in its
// first thread: 16 loads ahead of their sum.
__device__ __forceinline__ float group_total(const Film& F, const float* part, float* sv) {
  const uint32_t li = threadIdx.y * 16u + threadIdx.x, nt = F.tw * F.th;
  float v = 0.f;
  uint32_t t = li;
  for (; t + 15u * 256u < nt; t += 16u * 256u) {
    float p[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) p[k] = __ldcg(part + t + 256u * k);
#pragma unroll
    for (int k = 0; k < 16; ++k) v += p[k];
  }
  {
    float p[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) p[k] = t + 256u * k < nt ? __ldcg(part + t + 256u * k) : 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) v = t + 256u * k < nt ? v + p[k] : v;
  }
  return group_tree(sv, v);
}
// The scalars of a film after a phase (cg_reduce_a, cg_reduce_b).
struct SolveScalars {
  float rz, pq, alpha, beta;
  __device__ __forceinline__ void take(float total, bool after_b) {
    if (!after_b) {
      pq = total;
      alpha = total > 0.f ? rz / total : 0.f;
    } else {
      beta = rz > 0.f ? total / rz : 0.f;
      rz = total;
    }
  }
};

// Cell `item` of a tile's ring, as a position in its 18 x 18 box: rows 0 and
// 17, then columns 0 and 17.
constexpr int RING = 68;
__device__ __forceinline__ void ring_cell(int item, int& hx, int& hy) {
  hx = item < 36 ? item % 18 : ((item - 36) & 1) * 17;
  hy = item < 36 ? (item / 18) * 17 : 1 + (item - 36) / 2;
}
static_assert(SPAN * RING <= 256 && 9 * SPAN <= 32 && (SPAN & (SPAN - 1)) == 0, "one thread a ring cell, one lane a flag");

// A group's shared memory: the directions of each tile and its ring, the
// faces' weights of the tile and its ring but the right one, the warps' sums.
struct SolveGroup {
  float p[SPAN][18][18];
  float4 m[SPAN][18][17];
  float sv[SPAN][8];
};
constexpr size_t SOLVE_SMEM = sizeof(SolveGroup) * GROUPS;

// All iterations of an implicit step (cg_iter_a, cg_iter_b and their
// reductions, film.wgsl:1083-1135, 1214-1232), values and sums in the order of
// one launch per phase.
//
// Bound by memory, by the meetings on small films: per iteration a cell of a
// wet tile moves 60 bytes (a: z = r / d, p, the mobilities and x read, p, q and
// x written; b: r, q and d read, r and z written), against 76 with the
// direction formed from r and d, cg_p read for every cell and x updated from
// a second read of p.  b walks the tiles backwards, so that it begins with
// what a left in L2, and a in turn.  A tile without paint holds zeros
// throughout (no face of a dry cell has a mobility) and is left out: its
// partial is the init's 0, its directions are taken as 0.
// Every plane the launch writes is read past L1 (other SMs write it too).
// ONE: the launch's only film by value, so that its planes' addresses are
// operands from the constant bank (loaded from the film's record they took
// more instructions than the cells).
template <bool ONE>
__global__ void __launch_bounds__(256 * GROUPS, PER_SM)
    kp_cg_solve(const __grid_constant__ Film only, CG_ARGS, uint32_t nfilms, uint32_t step, uint32_t iters,
                uint32_t polls) {
  extern __shared__ __align__(16) unsigned char solve_smem[];
  __shared__ SolveScalars s_one;  // of a film alone
  SolveGroup& G = reinterpret_cast<SolveGroup*>(solve_smem)[threadIdx.z];
  const int li = (int)(threadIdx.y * 16u + threadIdx.x), lane = li & 31;
  constexpr uint32_t ON = ACTIVE | 1u;  // an active tile that holds paint
  // the blocks meet at the first film that takes the step (a film without
  // implicit steps has no CgState)
  uint32_t first = 0;
  while (first < nfilms && step >= (ONE ? only : films[first]).P->implicit_steps) ++first;
  if (first == nfilms) return;  // no film takes this step: the same for every block
  if (ONE) iters = min(iters, only.P->implicit_iters);
  CgState* M = ONE ? only.cg : films[first].cg;
  uint32_t meet = 0;
  const uint32_t q0 = blockIdx.x * GROUPS + threadIdx.z, dq = gridDim.x * GROUPS;
  const uint32_t nq = (ntiles + SPAN - 1u) / SPAN;
  if (ONE && lead_thread()) s_one = SolveScalars{M->rz, 0.f, 0.f, 0.f};
  // The film totals, then the scalars: every block forms those of a film
  // alone for itself (the partials are a few tens of KB in L2), so the blocks
  // meet once a phase; of several films, a group each, and a second meeting.
  auto reduce = [&](uint32_t it, bool after_b) {
    if (!blocks_meet(M, meet, polls)) return false;
    if (ONE) {
      if (threadIdx.z == 0) {
        const float total = group_total(only, after_b ? only.cg_part2 : only.cg_part, G.sv[0]);
        if (li == 0) {
          s_one.take(total, after_b);
          if (blockIdx.x == 0) {  // what the step's finish reads
            M->rz = s_one.rz;
            M->beta = s_one.beta;
          }
        }
      }
      __syncthreads();
      return true;
    }
    for (uint32_t f = q0; f < nfilms; f += dq) {
      const Film& F = films[f];
      if (step >= F.P->implicit_steps || it >= F.P->implicit_iters) continue;
      group_sync();  // the last sum in sv has been read
      const float total = group_total(F, after_b ? F.cg_part2 : F.cg_part, G.sv[0]);
      if (li == 0) {
        SolveScalars S{F.cg->rz, F.cg->pq, F.cg->alpha, F.cg->beta};
        S.take(total, after_b);
        F.cg->rz = S.rz;
        F.cg->pq = S.pq;
        F.cg->alpha = S.alpha;
        F.cg->beta = S.beta;
      }
    }
    return blocks_meet(M, meet, polls);
  };
  // Walks the spans of the table, the tiles of one film at a time:
  // body(F, span, tx, ty) with the mask of the span's tiles that belong to F
  // and take part, and the tile coordinates of tile u in lane u of each warp.
  auto each_span = [&](bool backwards, uint32_t it, auto body) {
    for (uint32_t qi = q0; qi < nq; qi += dq) {
      const uint32_t q = backwards ? nq - 1u - qi : qi, e = q * SPAN + (uint32_t)(lane & (SPAN - 1));
      if constexpr (ONE) {
        const int ty = (int)(e / only.tw), tx = (int)(e - (uint32_t)ty * only.tw);
        body(only, min(ntiles - q * SPAN, (uint32_t)SPAN) == SPAN ? (1u << SPAN) - 1u : (1u << (ntiles - q * SPAN)) - 1u,
             tx, ty);
      } else {
        uint2 pe = make_uint2(0u, 0u);
        bool take = e < ntiles;
        if (take) {
          pe = tile_entry(tiles, e);
          const DevParams& D = *films[pe.x].P;
          take = step < D.implicit_steps && it < D.implicit_iters;
        }
        const uint32_t tw = films[pe.x].tw;
        const int ty = (int)(pe.y / tw), tx = (int)(pe.y - (uint32_t)ty * tw);
        uint32_t todo = __ballot_sync(0xffffffffu, take) & ((1u << SPAN) - 1u);
        while (todo != 0u) {
          const uint32_t f = __shfl_sync(0xffffffffu, pe.x, __ffs(todo) - 1);
          const uint32_t span = todo & __ballot_sync(0xffffffffu, take && pe.x == f);
          todo &= ~span;
          body(films[f], span, tx, ty);
        }
      }
    }
  };
  // a's partials go to cg_part, b's to cg_part2: a block may be in b while
  // another still sums a's
  auto put_partials = [&](const Film& F, float* part, uint32_t on, int tx, int ty, float v[SPAN]) {
    const float s = span_trees(G.sv, v);
    if (li < SPAN && ((on >> li) & 1u)) part[(uint32_t)tx + (uint32_t)ty * F.tw] = s;
  };
  bool left_early = false;
  for (uint32_t it = 0; it < iters; ++it) {
    // p_it goes to cg_pa for even it, cg_pb for odd; p_{it-1} is in the other
    // (for it = 0 the init's direction, in cg_pa)
    const bool prev_a = (it & 1u) != 0u || it == 0u, cur_a = (it & 1u) == 0u;
    each_span(false, it, [&](const Film& F, uint32_t span, int tx, int ty) {
      // flags of the 3 x 3 tiles around tile u in lanes 9 u .. 9 u + 8
      uint32_t fl = 0u, on = 0u;  // on, bit u: tile u takes part and holds paint
      {
        const int u = lane / 9, m = lane % 9;
        const int nx = __shfl_sync(0xffffffffu, tx, u) + m % 3 - 1, ny = __shfl_sync(0xffffffffu, ty, u) + m / 3 - 1;
        if (u < SPAN && ((span >> u) & 1u) && nx >= 0 && ny >= 0 && nx < (int)F.tw && ny < (int)F.th)
          fl = F.tile_flags[nx + ny * (int)F.tw];
        const uint32_t b = __ballot_sync(0xffffffffu, (fl & ON) == ON);
#pragma unroll
        for (int v = 0; v < SPAN; ++v) on |= ((b >> (9 * v + 4)) & 1u) << v;
      }
      if (on == 0u) return;
      const int W = (int)F.w, H = (int)F.h;
      const float* prev = prev_a ? F.cg_pa : F.cg_pb;
      float* cur = cur_a ? F.cg_pa : F.cg_pb;
      const float beta = it == 0u ? 0.f : ONE ? s_one.beta : __ldcg(&F.cg->beta);
      const float alpha = it == 0u ? 0.f : ONE ? s_one.alpha : __ldcg(&F.cg->alpha);
      // the direction from the stored z = r / d and p_{it-1}: for it = 0 the
      // init's p (its z is not written yet)
      auto dir = [&](float z, float p) { return it == 0u ? p : fmaf(beta, p, z); };
      // Every load of the tiles and of the 68 cells around each goes out
      // before the first store to shared memory (the compiler cannot move a
      // load past one).  Cells outside the grid load cell 0 and take zeros.
      uint32_t c[SPAN];
      bool in[SPAN];
      float4 mv[SPAN];
      float pp[SPAN], zz[SPAN], xo[SPAN];
#pragma unroll
      for (int u = 0; u < SPAN; ++u) {
        const int i = __shfl_sync(0xffffffffu, tx, u) * 16 + (int)threadIdx.x;
        const int j = __shfl_sync(0xffffffffu, ty, u) * 16 + (int)threadIdx.y;
        in[u] = i < W && j < H && ((on >> u) & 1u);
        c[u] = in[u] ? idx(F, i, j) : 0u;
        mv[u] = F.flux[c[u]];
        pp[u] = __ldcg(prev + c[u]);
        zz[u] = __ldcg(F.cg_t + c[u]);
        xo[u] = __ldcg(F.cg_x + c[u]);
      }
      // the ring: cell li % 68 of tile li / 68
      const int ru = min(li / RING, SPAN - 1);
      const bool ring = li < SPAN * RING && ((on >> ru) & 1u) != 0u;
      int hx, hy;
      ring_cell(li % RING, hx, hy);
      float4 hm;
      float hp;
      {
        const int m = (hy == 0 ? 0 : hy == 17 ? 6 : 3) + (hx == 0 ? 0 : hx == 17 ? 2 : 1);
        const uint32_t f = __shfl_sync(0xffffffffu, fl, 9 * ru + m);
        const int x = __shfl_sync(0xffffffffu, tx, ru) * 16 - 1 + hx, y = __shfl_sync(0xffffffffu, ty, ru) * 16 - 1 + hy;
        const bool inr = ring && x >= 0 && y >= 0 && x < W && y < H, live = inr && (f & ON) == ON;
        const uint32_t n = inr ? idx(F, x, y) : 0u;
        if (ring) {
          hm = F.flux[n];
          hp = dir(__ldcg(F.cg_t + n), __ldcg(prev + n));
          if (!live) {
            hm = make_float4(0.f, 0.f, 0.f, 0.f);
            hp = 0.f;
            if (inr && (f & ACTIVE) == 0u) {  // as the last step that covered it left it
              hm = face_weights(kappa(F.P->p), F.cg_m[n]);
              hp = F.cg_p[n];
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < SPAN; ++u) {
        G.p[u][threadIdx.y + 1][threadIdx.x + 1] = in[u] ? dir(zz[u], pp[u]) : 0.f;
        G.m[u][threadIdx.y + 1][threadIdx.x + 1] = in[u] ? mv[u] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (ring) {
        G.p[ru][hy][hx] = hp;
        if (hx < 17) G.m[ru][hy][hx] = hm;
      }
      group_sync();
      float v[SPAN];
#pragma unroll
      for (int u = 0; u < SPAN; ++u) {
        const int lx = (int)threadIdx.x + 1, ly = (int)threadIdx.y + 1;
        const float(*sp)[18] = G.p[u];
        const float4(*sm)[17] = G.m[u];
        const float pc = sp[ly][lx];
        // the order of cg_nb (film.wgsl:994-1010), which leaves out the faces
        // without mobility (those across the grid's edge among them): their
        // weight is 0 and adds 0
        float acc_v = fmaf(mv[u].x, pc - sp[ly][lx + 1], pc);
        acc_v = fmaf(mv[u].y, pc - sp[ly + 1][lx], acc_v);
        acc_v = fmaf(mv[u].z, pc - sp[ly + 1][lx + 1], acc_v);
        acc_v = fmaf(mv[u].w, pc - sp[ly - 1][lx + 1], acc_v);
        acc_v = fmaf(sm[ly][lx - 1].x, pc - sp[ly][lx - 1], acc_v);
        acc_v = fmaf(sm[ly - 1][lx].y, pc - sp[ly - 1][lx], acc_v);
        acc_v = fmaf(sm[ly - 1][lx - 1].z, pc - sp[ly - 1][lx - 1], acc_v);
        acc_v = fmaf(sm[ly + 1][lx - 1].w, pc - sp[ly + 1][lx - 1], acc_v);
        v[u] = in[u] ? pc * acc_v : 0.f;
        if (in[u]) {
          cur[c[u]] = pc;  // other blocks read p_{it-1} from the other plane
          F.cg_q[c[u]] = acc_v;
          // cg_iter_b's x of the previous iteration, whose p is at hand here
          if (it != 0u) F.cg_x[c[u]] = fmaf(alpha, pp[u], xo[u]);
        }
      }
      put_partials(F, F.cg_part, on, tx, ty, v);
    });
    if (!reduce(it, false)) {
      left_early = true;
      break;
    }
    each_span(true, it, [&](const Film& F, uint32_t span, int tx, int ty) {
      const uint32_t fl = lane < SPAN && ((span >> lane) & 1u) ? F.tile_flags[(uint32_t)tx + (uint32_t)ty * F.tw] : 0u;
      const uint32_t on = __ballot_sync(0xffffffffu, (fl & ON) == ON);
      if (on == 0u) return;
      const float* cur = cur_a ? F.cg_pa : F.cg_pb;
      const float alpha = ONE ? s_one.alpha : __ldcg(&F.cg->alpha);
      const bool last = it + 1u == (ONE ? iters : F.P->implicit_iters);
      float d[SPAN], r[SPAN], w[SPAN], v[SPAN];
      uint32_t c[SPAN];
      bool in[SPAN];
#pragma unroll
      for (int u = 0; u < SPAN; ++u) {
        const int i = __shfl_sync(0xffffffffu, tx, u) * 16 + (int)threadIdx.x;
        const int j = __shfl_sync(0xffffffffu, ty, u) * 16 + (int)threadIdx.y;
        in[u] = i < (int)F.w && j < (int)F.h && ((on >> u) & 1u);
        c[u] = in[u] ? idx(F, i, j) : 0u;
        d[u] = F.cg_d[c[u]];
        r[u] = __ldcg(F.cg_r + c[u]);
        w[u] = __ldcg(F.cg_q + c[u]);
      }
#pragma unroll
      for (int u = 0; u < SPAN; ++u) {
        const float rn = fmaf(-alpha, w[u], r[u]);
        v[u] = 0.f;
        if (in[u]) {
          v[u] = __fmul_rn(rn, rn) / d[u];
          if (last) F.cg_x[c[u]] = fmaf(alpha, __ldcg(cur + c[u]), __ldcg(F.cg_x + c[u]));
          F.cg_r[c[u]] = rn;
          F.cg_t[c[u]] = rn / d[u];
        }
      }
      group_sync();  // the last span's sums have been read
      put_partials(F, F.cg_part2, on, tx, ty, v);
    });
    if (!reduce(it, true)) {
      left_early = true;
      break;
    }
  }
  // a wait ran out: every film that takes the step counts it and keeps its h
  // through the step (kp_cg_finish)
  if (left_early && lead_thread())
    for (uint32_t f = first; f < nfilms; ++f)
      if (step < films[f].P->implicit_steps) {
        atomicAdd(&films[f].stats->wait_timeouts, 1u);
        films[f].cg->failed = 1u;
      }
  blocks_leave(M);
}

// The SMs that work enqueued on `st` may run on: those of the stream's green
// context where it has one, else all of the device's `sms`.
uint32_t stream_sms(cudaStream_t st, uint32_t sms) {
  using GetCtx = CUresult (*)(CUstream, CUcontext*, CUgreenCtx*);
  using GetRes = CUresult (*)(CUgreenCtx, CUdevResource*, CUdevResourceType);
  static GetCtx get_ctx = nullptr;
  static GetRes get_res = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {  // through the runtime: the library does not link the driver library
    cudaDriverEntryPointQueryResult q{};
    void *c = nullptr, *r = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &c, 12050, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess &&
        cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", &r, 12040, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      get_ctx = reinterpret_cast<GetCtx>(c);
      get_res = reinterpret_cast<GetRes>(r);
    }
    cudaGetLastError();
  });
  CUcontext ctx = nullptr;
  CUgreenCtx green = nullptr;
  CUdevResource res;
  if (get_ctx == nullptr || get_ctx(st, &ctx, &green) != CUDA_SUCCESS || green == nullptr ||
      get_res(green, &res, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
    return sms;
  return std::min<uint32_t>(sms, std::max(res.sm.smCount, 1u));
}

// The grid of kp_cg_solve: every block that fits at once on the SMs the stream
// has (a larger cooperative launch is refused), no more than the tiles fill.
// The sums do not depend on it.
uint32_t solve_blocks(uint32_t ntiles, cudaStream_t st) {
  static std::mutex mu;
  static int per_device[64] = {}, sms_of[64] = {};  // blocks an SM, SMs
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1u;
  std::lock_guard<std::mutex> lock(mu);
  if (per_device[dev] == 0) {
    int sms = 0, a = 0, b = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(kp_cg_solve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLVE_SMEM);
    cudaFuncSetAttribute(kp_cg_solve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLVE_SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kp_cg_solve<true>, 256 * GROUPS, SOLVE_SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kp_cg_solve<false>, 256 * GROUPS, SOLVE_SMEM);
    per_device[dev] = std::max(std::min(a, b), 1);
    sms_of[dev] = std::max(sms, 1);
  }
  return std::min<uint32_t>((uint32_t)per_device[dev] * stream_sms(st, (uint32_t)sms_of[dev]),
                            (ntiles + GROUPS * SPAN - 1u) / (GROUPS * SPAN));
}

// cg_lap_u (film.wgsl:1080-1085), only with the implicit capillary term
__global__ void __launch_bounds__(256) kp_cg_lap_u(CG_ARGS, uint32_t step) {
  CG_TILE
  if (step >= D.implicit_steps || !cell_on) return;
  F.cg_t[c] = lap_w(F, i, j, c, [&](uint32_t n) { return F.cg_x[n] + hold_u(F, P, n); });
}

// film.wgsl:1227-1274 and cg_reduce_mass (film.wgsl:1190-1207).  The new h
// goes to cg_q (kp_cg_rescale commits it), so every read of a neighbour's h
// sees the h of before the dispatch.  The final direction of the solve (the
// reference's last cg_iter_c) is kept in cg_p for later steps' reads.  A film
// whose solve was left early keeps its h, acc and cg_p: the step is not taken
// (the mark is looked at before the stores, not ahead of the loads: 11 us less a
// step at 1200x800, 24 at 2048^2).
__global__ void __launch_bounds__(256) kp_cg_finish(CG_ARGS, uint32_t step) {
  CG_TILE
  if (step >= D.implicit_steps) return;
  __shared__ float sv[256];
  __shared__ __align__(16) float stv[256];
  __shared__ uint32_t s_moved;
  const uint32_t li = threadIdx.y * 16u + threadIdx.x;
  if (li == 0u) s_moved = 0u;
  __syncthreads();
  float dv = 0.f, tv = 0.f;
  if (cell_on) {
    const uint32_t last = D.implicit_iters - 1u;
    const float* plast = (last & 1u) ? F.cg_pb : F.cg_pa;
    // a tile without paint is left out of the solve: its direction stays 0
    const bool dry = P.front3[0] == 0.f && (F.tile_flags[t] & 1u) == 0u;
    const float dir = dry ? 0.f : F.cg_r[c] / F.cg_d[c] + F.cg->beta * plast[c];
    const float h0 = F.hh[c], hn = fmaxf(F.cg_x[c], 0.f);
    const float rg = P.phys[0] * P.g[2] * P.inv_dx;
    auto pot = [&](uint32_t n) { return F.cg_x[n] + hold_u(F, P, n); };  // film.wgsl:1227-1229
    const float pc = pot(c);
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 mob = F.cg_m[c];
    if (mob.x > 0.f) f.x = W_AXIS * mob.x * rg * (pc - pot(idx(F, i + 1, j)));
    if (mob.y > 0.f) f.y = W_AXIS * mob.y * rg * (pc - pot(idx(F, i, j + 1)));
    if (mob.z > 0.f) f.z = W_DIAG_FLUX * mob.z * rg * (pc - pot(idx(F, i + 1, j + 1))) * 0.70710678f;
    if (mob.w > 0.f) f.w = W_DIAG_FLUX * mob.w * rg * (pc - pot(idx(F, i + 1, j - 1))) * 0.70710678f;
    if (h0 > 0.f && P.front3[1] != 0.f) {
      const float kc = P.front3[1], tc = F.cg_t[c];
      auto wet_on = [&](int x, int y) { return F.hh[idx(F, x, y)] > 0.f && cell_active(F, x, y); };
      if (i + 1 < (int)F.w && wet_on(i + 1, j)) f.x += W_AXIS * kc * (F.cg_t[idx(F, i + 1, j)] - tc);
      if (j + 1 < (int)F.h && wet_on(i, j + 1)) f.y += W_AXIS * kc * (F.cg_t[idx(F, i, j + 1)] - tc);
      if (i + 1 < (int)F.w && j + 1 < (int)F.h && wet_on(i + 1, j + 1))
        f.z += W_DIAG_FLUX * kc * (F.cg_t[idx(F, i + 1, j + 1)] - tc) * 0.70710678f;
      if (i + 1 < (int)F.w && j > 0 && wet_on(i + 1, j - 1))
        f.w += W_DIAG_FLUX * kc * (F.cg_t[idx(F, i + 1, j - 1)] - tc) * 0.70710678f;
    }
    const float4 a = F.acc[c];
    const float fw = P.front[3];
    if (F.cg->failed == 0u) {
      F.cg_p[c] = dir;
      F.acc[c] = make_float4(a.x + f.x * fw, a.y + f.y * fw, a.z + f.z * fw, a.w + f.w * fw);
      F.cg_q[c] = hn;
      if (fabsf(hn - h0) > MOVE_EPS) s_moved = 1u;
    }
    dv = hn - h0;
    tv = hn;
  }
  stv[li] = tv;
  const float part = block_tree(sv, dv);  // its barriers also publish stv and s_moved
  float part2 = 0.f;
  if (li == 0u) {
    // thread 0's sequential sum (film.wgsl:1268-1272), its loads ahead of it
    const float4* q = reinterpret_cast<const float4*>(stv);
#pragma unroll 16
    for (int k = 0; k < 64; ++k) {
      const float4 a = q[k];
      part2 += a.x;
      part2 += a.y;
      part2 += a.z;
      part2 += a.w;
    }
    if (s_moved) F.tile_moved[t] = 1u;
  }
  if (last_block(F, t, part, part2)) {
    const float sdv = film_total(F, F.cg_part, sv);
    const float stot = film_total(F, F.cg_part2, stv);
    if (li == 0u) {
      CgState& S = *F.cg;
      S.dv = sdv;
      S.tv = stot;
      S.s0x = S.rz;
      S.blocks_done = 0u;
    }
  }
}

// cg_rescale (film.wgsl:1179-1188) with the commit of cg_finish's h
__global__ void __launch_bounds__(256) kp_cg_rescale(CG_ARGS, uint32_t step) {
  CG_TILE
  if (step >= D.implicit_steps || !cell_on) return;
  const float hn = F.cg_q[c];
  const CgState& S = *F.cg;
  if (S.failed != 0u) return;
  if (S.tv <= 0.f) {
    F.hh[c] = hn;
    return;
  }
  const float fr = 1.0f - S.dv / S.tv;
  F.hh[c] = fmaxf(hn * fr, 0.f);
}

}  // namespace

uint32_t launch_cg_step(const PackedFrame& V, int mode, uint32_t step, uint32_t iters, bool cap_implicit,
                        cudaStream_t st) {
  const Film* A = V.films;
  const uint2* T = V.tiles;
  const uint32_t nt = V.ntiles;
  const dim3 b(16, 16);
  uint32_t n = 0;
  if (mode == CF_PREC_REFERENCE) kp_cg_setup<CF_PREC_REFERENCE><<<nt, b, 0, st>>>(A, T, nt, step);
  else if (mode == CF_PREC_FP32) kp_cg_setup<CF_PREC_FP32><<<nt, b, 0, st>>>(A, T, nt, step);
  else kp_cg_setup<CF_PREC_BF16><<<nt, b, 0, st>>>(A, T, nt, step);
  n += 2;
  if (cap_implicit) {
    kp_cg_init<false><<<nt, b, 0, st>>>(A, T, nt, step);
    for (uint32_t it = 0; it < iters; ++it) {
      kp_cg_lap_p<<<nt, b, 0, st>>>(A, T, nt, step, it);
      kp_cg_iter_a<<<nt, b, 0, st>>>(A, T, nt, step, it);
      kp_cg_scalars<<<V.nfilms, b, 0, st>>>(A, V.nfilms, step, it, 0);
      kp_cg_iter_b<<<nt, b, 0, st>>>(A, T, nt, step, it);
      kp_cg_scalars<<<V.nfilms, b, 0, st>>>(A, V.nfilms, step, it, 1);
      n += 5;
    }
  } else {
    kp_cg_init<true><<<nt, b, 0, st>>>(A, T, nt, step);
    uint32_t nfilms = V.nfilms, ntiles = nt, polls = V.meet_polls;
    Film only = V.only != nullptr ? *V.only : Film{};
    void* args[] = {&only, &A, &T, &ntiles, &nfilms, &step, &iters, &polls};
    // an error stays with the runtime for the caller's check of the launches
    cudaLaunchCooperativeKernel(V.only != nullptr ? (const void*)kp_cg_solve<true> : (const void*)kp_cg_solve<false>,
                                dim3(solve_blocks(nt, st)), dim3(16, 16, GROUPS), args, SOLVE_SMEM, st);
    n += 1;
  }
  if (cap_implicit) { kp_cg_lap_u<<<nt, b, 0, st>>>(A, T, nt, step); ++n; }
  kp_cg_finish<<<nt, b, 0, st>>>(A, T, nt, step);
  kp_cg_rescale<<<nt, b, 0, st>>>(A, T, nt, step);
  return n + 2;
}

}  // namespace cfk
