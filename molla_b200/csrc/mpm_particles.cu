// mpm_particles.cu — the particle kernels of the B200 MLS-MPM substep.
//
// One substep of the reference (crates/molla-solvers/src/mpm.rs:2476-2551:
// reset_grid, p2g, grid_update, g2p, plasticity) runs as three launches
// (two for small groups, where the gather and scatter are fused):
//
//   grid_update(n)  acc[a] -> velocity, clears acc[b]               (grid sweep)
//   gather(n)       G2P(n) + F update + return mapping(n); writes the particle
//                   and, for the next substep, its 64-byte record in deposit
//                   form (mass, m v - fx.Bd, Bd = B dx with the APIC/stress
//                   matrix B = m C + 4/dx^2 S, S the fixed-corotated stress)
//   scatter(n+1)    27-node deposit of mass and momentum into acc[b]
//
// Both particle kernels are persistent over lists built by the last
// regrouping (a stable radix sort of the particles by base-cell key, in tiles
// of 4^3 base cells).  The gather's warps each take units (32..640 particles
// of a tile) with the tile's 8^3-node velocity block in shared memory; the
// scatter's CTAs take items (at most kStageMax particles of a tile), stage the
// records with TMA, link them into lists by their current base cell and
// accumulate into an 8^3-node shared block that is flushed to HBM with one
// float4 atomic per non-empty node.  They are separate kernels because the
// gather (SVD, return mapping) runs at 96 registers in warps that wait for
// nobody, while the scatter's steps need CTA barriers: split, each has its own
// shape, and the record's round trip through HBM is cheaper than the fused
// kernel's two CTAs an SM.  Up to kFusedMaxParticles the fused k_g2p2g keeps
// the records in shared memory and saves a launch per substep.  The SVD
// computed by the return mapping is reused for the next substep's stress; a
// step_n call whose records cannot be carried over from the last one opens
// with a record-only gather that computes it from F.
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "mpm_device.cuh"
#include "mpm_kernels.cuh"

namespace mpm {

namespace {

__device__ __forceinline__ int region_index(int lx, int ly, int lz) { return lx + kRsy * ly + kRsz * lz; }

// Regroup key of a particle from its base cell: ((scene tile offset + tile)
// << 6) | cell within the tile; base clamped to the grid.
__device__ __forceinline__ uint32_t base_key(const SceneDev& sc, const int* base) {
  uint32_t t[3], c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int b = base[a];
    b = b < 0 ? 0 : b;
    b = b > (int)sc.n - 1 ? (int)sc.n - 1 : b;
    t[a] = (uint32_t)b >> 2;
    c[a] = (uint32_t)b & 3u;
  }
  const uint32_t tile = t[0] + sc.w * (t[1] + sc.w * t[2]);
  return ((sc.key_off + tile) << kCellBits) | c[0] | (c[1] << 2) | (c[2] << 4);
}

// Gather for a particle whose stencil is not inside the staged 8^3 block
// (it left its tile since the last regrouping): 27 global reads with the
// reference's out-of-grid skip.  Kept out of line and rolled so that the
// unrolled shared-memory path stays small; it takes scalars and writes
// v (3) and G = sum w gv d^T (9) to out.
__device__ __noinline__ void gather_global(const float4* vel_pool, const SceneDev& sc,
                                           const uint32_t* tile_slot, float xp0, float xp1, float xp2,
                                           float* out) {
  const float xp[3] = {xp0, xp1, xp2};
  const int win[3] = {sc.winx, sc.winy, sc.winz};
  const float dx = sc.dx;
  float w[3][3], d[3][3];
  int base[3];
  for (int a = 0; a < 3; ++a) {
    const float bf = floorf(xp[a] - 0.5f);
    base[a] = (int)bf - win[a];
    const float fx = xp[a] - bf;
    quad_weights(fx, w[a]);
    for (int i = 0; i < 3; ++i) d[a][i] = ((float)i - fx) * dx;
  }
  float acc[12];
  for (int i = 0; i < 12; ++i) acc[i] = 0.f;
#pragma unroll 1
  for (int q = 0; q < 27; ++q) {
    const int i = q / 9, j = (q / 3) % 3, k = q % 3;
    const int64_t c = node_index(sc, tile_slot, base[0] + i, base[1] + j, base[2] + k);
    if (c < 0) continue;
    const float4 g = vel_pool[c];
    const float wt = w[0][i] * w[1][j] * w[2][k];
    const float gv[3] = {wt * g.x, wt * g.y, wt * g.z};
    for (int r = 0; r < 3; ++r) {
      acc[r] += gv[r];
      acc[3 + r] += gv[r] * d[0][i];
      acc[6 + r] += gv[r] * d[1][j];
      acc[9 + r] += gv[r] * d[2][k];
    }
  }
  for (int i = 0; i < 12; ++i) out[i] = acc[i];
}

// mbarrier + bulk-copy (TMA engine) helpers for the scatter's record stage.
__device__ __forceinline__ uint32_t smem_addr(const void* ptr) {
  return (uint32_t)__cvta_generic_to_shared(ptr);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Orders this CTA's earlier generic-proxy accesses of shared memory before
// later async-proxy (bulk copy) writes to it.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// 2-D TMA tile load (box of kStageBoxRows records) at coordinates (0, row)
// of the record tensor map, completing on `bar`.
__device__ __forceinline__ void tma_load_rows(void* dst, const CUtensorMap* map, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(row), "r"(smem_addr(bar))
      : "memory");
}
// 3-D TMA box (32 floats x 8 x 8: the 8^3 nodes of a velocity block) from
// coordinates (x, y, z); x is a multiple of four floats.
__device__ __forceinline__ void tma_load_box(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
      : "memory");
}
// Makes a tensor map in global memory, written by an earlier copy, visible to
// the TMA loads of this thread.
__device__ __forceinline__ void fence_tensormap(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Ampere-style asynchronous global -> shared copies (cp.async) of 4 or 16
// bytes; a thread waits for its own.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Waits for the phase of `bar` with the given parity to complete; gives up
// (returns false) after about one second.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > 1000000000ull) return false;
  }
  return true;
}

}  // namespace

// The particle inputs the gather stages in shared memory, in order: the
// position planes, the F planes, mass, volume and J_p (planes PX..PZ and
// F0..JP in plane order), then the meta word.
constexpr int kStagedInputs = 16;
static_assert(PY == PX + 1 && PZ == PX + 2 && MASS == F0 + 9 && VOL == F0 + 10 && JP == F0 + 11,
              "the staged planes are two runs of consecutive planes");
// A particle's inputs in that order, from a lane's column of the stage or
// straight from the pool.
struct StagedIn {
  const float* col;
  __device__ __forceinline__ float f(int q) const { return col[32 * q]; }
  __device__ __forceinline__ uint32_t mat() const { return __float_as_uint(f(kStagedInputs - 1)) & 7u; }
};
struct PoolIn {
  const PoolDev& p;
  uint32_t s;
  __device__ __forceinline__ float f(int q) const { return plane(p, q < 3 ? PX + q : F0 + q - 3)[s]; }
  __device__ __forceinline__ uint32_t mat() const { return p.meta[s] & 7u; }
};
constexpr int kInMass = 12, kInVol = 13, kInJp = 14;
// What particle_step tells the owner of its inputs: `late` before it reads the
// first of mass, volume, J_p and material, `early_read` when it has read x and F
// for the last time, `done` when it has read everything.
struct NoRefill {
  __device__ __forceinline__ void late() const {}
  __device__ __forceinline__ void early_read() const {}
  __device__ __forceinline__ void done() const {}
};
// Lattice x of a record that deposits nothing: outside every grid.
constexpr float kOffGrid = 1.0e30f;

// The uniform values of the unit a gather warp is on, kept in shared memory so
// that they hold no registers through the particle computation: the scene's
// status word, the 8^3 velocity block origin, whether this substep publishes v
// and C, and the unit's slot range.
struct GatherCtx {
  uint32_t* status;
  int rx, ry, rz;
  uint32_t publish_vc;
  uint32_t start, count;
  uint32_t tiles;  // sparse storage: the tiles the unit's records touch (block_tiles)
};

// One particle: G2P + F update + return mapping (MODE != kRecord) and the
// scatter record (MODE != kG2P), returned in rec.  ctx holds the unit's
// uniform values; vblock is the staged 8^3-node velocity block of its tile
// (origin node ctx.rx, ctx.ry, ctx.rz).  Inputs are read when they are needed
// (mass, volume, J_p and material would hold four registers through the G2P
// and the SVD).
template <int MODE, bool WRITE_KEYS, bool SPARSE, bool FIXED, class SR, class IN, class REFILL>
__device__ __forceinline__ void particle_step(const PoolDev& p, const SceneDev& sc, uint32_t s, GatherCtx& ctx,
                                              const float4* __restrict__ vblock, SR stol, int sweeps,
                                              const IN in, const REFILL refill, float4 (&rec)[4]) {
  constexpr bool kGather = MODE != kRecord;
  constexpr bool kScatter = MODE != kG2P;
  float x, y, z, F[9], jp;
  float v[3], C[9];
  bool ok = true;
  SvdOut<SR> svd;
  if constexpr (kGather) {
    // ---- g2p (mpm.wgsl:1242-1353) ----
    const float xp[3] = {lattice_pos(in.f(0), sc.ox, sc.inv_dx), lattice_pos(in.f(1), sc.oy, sc.inv_dx),
                         lattice_pos(in.f(2), sc.oz, sc.inv_dx)};
    {
      float w[3][3], d[3][3];
      int base[3];
      const int win[3] = {sc.winx, sc.winy, sc.winz};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float bf = floorf(xp[a] - 0.5f);
        base[a] = (int)bf - win[a];
        const float fx = xp[a] - bf;
        quad_weights(fx, w[a]);
#pragma unroll
        for (int i = 0; i < 3; ++i) d[a][i] = ((float)i - fx) * sc.dx;
      }
      const int lx0 = base[0] - ctx.rx, ly0 = base[1] - ctx.ry, lz0 = base[2] - ctx.rz;
      const bool inside = (unsigned)lx0 <= (unsigned)(kRegion - 3) && (unsigned)ly0 <= (unsigned)(kRegion - 3) &&
                          (unsigned)lz0 <= (unsigned)(kRegion - 3);
      // Separable accumulation: v = sum w gv; G = sum (w gv) d^T.
      float vs[3] = {0.f, 0.f, 0.f};
      float G[9];
      if (inside) {
        const float4* __restrict__ blk = &vblock[lx0 + 8 * ly0 + 64 * lz0];
        if constexpr ((sizeof(SR) == 4 || !SPARSE) && !FIXED) {
          // In pairs, one instruction for two sums (16M particles x 16 substeps
          // 38.2 -> 37.6 ms in the FP64 form, 4M x 12 6.63 -> 6.43 in the FP32
          // form); the sparse FP64 form has no registers left for them (184
          // bytes of spills).
          // The sums over k, then j, then i of the products with the weights
          // (and, for one axis at a time, with the offset d), the components in
          // pairs: (x, y) of sum w gv, z of it beside z of sum w d_z gv, (x, y)
          // of the latter.
          float2 v01 = make_float2(0.f, 0.f), v2z2 = v01, z01 = v01, x01 = v01, y01 = v01;
          float x2 = 0.f, y2 = 0.f;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            float2 s01 = make_float2(0.f, 0.f), s2t2 = s01, t01 = s01, u01 = s01;
            float u2 = 0.f;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              float2 a01 = make_float2(0.f, 0.f), a2b2 = a01, b01 = a01;
#pragma unroll
              for (int kk = 0; kk < 3; ++kk) {
                const float4 g = blk[i + 8 * j + 64 * kk];
                const float wk = w[2][kk], wd = wk * d[2][kk];
                const float2 gxy = make_float2(g.x, g.y);
                a01 = fma2(make_float2(wk, wk), gxy, a01);
                a2b2 = fma2(make_float2(wk, wd), make_float2(g.z, g.z), a2b2);
                b01 = fma2(make_float2(wd, wd), gxy, b01);
              }
              const float wj = w[1][j], wd = wj * d[1][j];
              const float2 wj2 = make_float2(wj, wj);
              s01 = fma2(wj2, a01, s01);
              s2t2 = fma2(wj2, a2b2, s2t2);
              t01 = fma2(wj2, b01, t01);
              u01 = fma2(make_float2(wd, wd), a01, u01);
              u2 = fmaf(wd, a2b2.x, u2);
            }
            const float wi = w[0][i], wd = wi * d[0][i];
            const float2 wi2 = make_float2(wi, wi);
            v01 = fma2(wi2, s01, v01);
            v2z2 = fma2(wi2, s2t2, v2z2);
            z01 = fma2(wi2, t01, z01);
            x01 = fma2(make_float2(wd, wd), s01, x01);
            x2 = fmaf(wd, s2t2.x, x2);
            y01 = fma2(wi2, u01, y01);
            y2 = fmaf(wi, u2, y2);
          }
          vs[0] = v01.x;
          vs[1] = v01.y;
          vs[2] = v2z2.x;
          G[0] = x01.x;
          G[1] = x01.y;
          G[2] = x2;
          G[3] = y01.x;
          G[4] = y01.y;
          G[5] = y2;
          G[6] = z01.x;
          G[7] = z01.y;
          G[8] = v2z2.y;
        } else {
#pragma unroll
          for (int i = 0; i < 9; ++i) G[i] = 0.f;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            float si[3] = {0.f, 0.f, 0.f}, syi[3] = {0.f, 0.f, 0.f}, szi[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              float sj[3] = {0.f, 0.f, 0.f}, szj[3] = {0.f, 0.f, 0.f};
#pragma unroll
              for (int kk = 0; kk < 3; ++kk) {
                const float4 g = blk[i + 8 * j + 64 * kk];
                const float wk = w[2][kk];
                sj[0] += wk * g.x;
                sj[1] += wk * g.y;
                sj[2] += wk * g.z;
                const float wdk = wk * d[2][kk];
                szj[0] += wdk * g.x;
                szj[1] += wdk * g.y;
                szj[2] += wdk * g.z;
              }
              const float wj = w[1][j];
              const float wdj = wj * d[1][j];
#pragma unroll
              for (int r = 0; r < 3; ++r) {
                si[r] += wj * sj[r];
                syi[r] += wdj * sj[r];
                szi[r] += wj * szj[r];
              }
            }
            const float wi = w[0][i];
            const float wdi = wi * d[0][i];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
              vs[r] += wi * si[r];
              G[r] += wdi * si[r];      // column x
              G[3 + r] += wi * syi[r];  // column y
              G[6 + r] += wi * szi[r];  // column z
            }
          }
        }
      } else {
        float slot[12];
        gather_global(p.vel, sc, p.tile_slot, xp[0], xp[1], xp[2], slot);
#pragma unroll
        for (int r = 0; r < 3; ++r) vs[r] = slot[r];
#pragma unroll
        for (int r = 0; r < 9; ++r) G[r] = slot[3 + r];
      }
      const float four_inv_dx2 = 4.0f * sc.inv_dx * sc.inv_dx;
#pragma unroll
      for (int i = 0; i < 9; ++i) C[i] = four_inv_dx2 * G[i];
      v[0] = vs[0];
      v[1] = vs[1];
      v[2] = vs[2];
      refill.late();
      const MatDev& md = sc.mat[in.mat()];
      if (md.rheo == 2) {
        v[0] *= md.vfac;
        v[1] *= md.vfac;
        v[2] *= md.vfac;
#pragma unroll
        for (int i = 0; i < 9; ++i) C[i] *= md.afac;
      }
      x = in.f(0);
      y = in.f(1);
      z = in.f(2);
#pragma unroll
      for (int i = 0; i < 9; ++i) F[i] = in.f(3 + i);
      refill.early_read();
      float np[3] = {x + sc.dt * v[0], y + sc.dt * v[1], z + sc.dt * v[2]};
      // F <- (I + dt C) F
      float A[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) A[i] = sc.dt * C[i] + ((i % 4 == 0) ? 1.f : 0.f);
      float Fn[9];
      matmul(A, F, Fn);
      jp = in.f(kInJp);
      // One test for the reference's three (the inputs, the new x, v and C,
      // the new F; each of which leaves the particle as it was): a non-finite
      // position or velocity reaches np, a non-finite F or C reaches Fn.
      const float chk[16] = {np[0], np[1], np[2], jp,    xp[0], xp[1], xp[2], Fn[0],
                             Fn[1], Fn[2], Fn[3], Fn[4], Fn[5], Fn[6], Fn[7], Fn[8]};
      if (!all_finite(chk)) {
        atomicOr(ctx.status, kFaultNumerical);
        ok = false;
      }
      if (ok) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (np[a] < sc.lo[a] || np[a] > sc.hi[a]) v[a] = 0.f;
          np[a] = clampf(np[a], sc.lo[a], sc.hi[a]);
        }
        {
          x = np[0];
          y = np[1];
          z = np[2];
#pragma unroll
          for (int i = 0; i < 9; ++i) F[i] = Fn[i];
          // ---- plasticity (mpm.wgsl:1366-1479) on the updated F ----
          SR Fs[9];
#pragma unroll
          for (int i = 0; i < 9; ++i) Fs[i] = (SR)F[i];
          svd3<SR>(Fs, F, svd, stol, sweeps);
          float jp_new = jp;
          bool changed = true;
          const SR s_trial[3] = {svd.s[0], svd.s[1], svd.s[2]};
          if (plasticity_project<SR>(svd, md, jp_new, changed)) {
            // The FP32 form rebuilds F = U s V^T every substep (the reference).
            // The FP64 form keeps the trial F when the return mapping left
            // every singular value unchanged, and otherwise adds U diag(s -
            // s_trial) V^T to it: the same F in exact arithmetic (F = U s_trial
            // V^T), with the FP32 rounding of U and V scaled by the (small)
            // change in s instead of by F.  Finite: s lies in [0.05, 20] and F
            // = U s_trial V^T.
            if (changed || sizeof(SR) == 4) {
              float ds[3];
#pragma unroll
              for (int i = 0; i < 3; ++i) ds[i] = sizeof(SR) == 4 ? (float)svd.s[i] : (float)(svd.s[i] - s_trial[i]);
#pragma unroll
              for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int r = 0; r < 3; ++r)
                  F[3 * c + r] = (sizeof(SR) == 4 ? 0.0f : F[3 * c + r]) + (svd.u[r] * ds[0]) * svd.v[c] +
                                 (svd.u[3 + r] * ds[1]) * svd.v[3 + c] + (svd.u[6 + r] * ds[2]) * svd.v[6 + c];
            }
            jp = jp_new;
          } else {
            atomicOr(ctx.status, kFaultNumerical);
            ok = false;
          }
          // G2P results are published even when the return mapping
          // faults (the reference's g2p and plasticity are separate
          // dispatches); only the plasticity update is withheld.
          // v and C are read by nothing before the next call (the next
          // gather recomputes them from the grid; the scatter takes the
          // record), so a substep that writes a record skips them unless
          // the return mapping faulted: the last substep of a call
          // publishes them.
          plane(p, PX)[s] = x;
          plane(p, PY)[s] = y;
          plane(p, PZ)[s] = z;
          if (!kScatter || !ok || ctx.publish_vc) {
            plane(p, VX)[s] = v[0];
            plane(p, VY)[s] = v[1];
            plane(p, VZ)[s] = v[2];
#pragma unroll
            for (int i = 0; i < 9; ++i) plane(p, C0 + i)[s] = C[i];
          }
#pragma unroll
          for (int i = 0; i < 9; ++i) plane(p, F0 + i)[s] = F[i];
          plane(p, JP)[s] = jp;
        }
      }
    }
  } else {
    // P2G-only: read v and C and validate the whole state (the
    // reference's g2p checks, mpm.wgsl:1247-1255, moved to the first
    // launch of the call so that a non-finite upload latches before
    // anything moves).
    x = in.f(0);
    y = in.f(1);
    z = in.f(2);
#pragma unroll
    for (int i = 0; i < 9; ++i) F[i] = in.f(3 + i);
    refill.late();
    refill.early_read();
    v[0] = plane(p, VX)[s];
    v[1] = plane(p, VY)[s];
    v[2] = plane(p, VZ)[s];
#pragma unroll
    for (int i = 0; i < 9; ++i) C[i] = plane(p, C0 + i)[s];
    jp = in.f(kInJp);
    bool fin = finitef(x) && finitef(y) && finitef(z) && finitef(jp) && finitef(v[0]) && finitef(v[1]) &&
               finitef(v[2]) && finitef(lattice_pos(x, sc.ox, sc.inv_dx)) &&
               finitef(lattice_pos(y, sc.oy, sc.inv_dx)) && finitef(lattice_pos(z, sc.oz, sc.inv_dx));
#pragma unroll
    for (int i = 0; i < 9; ++i) fin = fin && finitef(F[i]) && finitef(C[i]);
    if (!fin) {
      atomicOr(ctx.status, kFaultNumerical);
      ok = false;
    }
  }
  const uint32_t mat = in.mat();
  const float mass = in.f(kInMass), vol = in.f(kInVol);
  refill.done();
  if constexpr (kScatter || WRITE_KEYS) {
    // lattice coordinates of the new position
    const float xq[3] = {lattice_pos(x, sc.ox, sc.inv_dx), lattice_pos(y, sc.oy, sc.inv_dx),
                         lattice_pos(z, sc.oz, sc.inv_dx)};
    const float bf[3] = {floorf(xq[0] - 0.5f), floorf(xq[1] - 0.5f), floorf(xq[2] - 0.5f)};
    if constexpr (kScatter) {
      // The record in its deposit form, so that no scatter thread repeats
      // per-particle arithmetic: Bd = B dx and, with fx = xp - base, the
      // momentum of node (0, 0, 0), q = m v - fx0 Bdx - fx1 Bdy - fx2 Bdz
      // (the reference's m v + B d with d = ((i, j, k) - fx) dx regrouped:
      // node (i, j, k) receives w (m, q + i Bdx + j Bdy + k Bdz)).  A particle
      // that faulted deposits nothing: mass 0, at a position off every grid.
      // FIXED: the fixed-order mode's own form (p2g_affine).
      float Bd[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) Bd[i] = 0.f;
      if (ok) {
        if constexpr (!kGather) {
          SR Fs[9];
#pragma unroll
          for (int i = 0; i < 9; ++i) Fs[i] = (SR)F[i];
          svd3<SR>(Fs, F, svd, stol, sweeps);
        }
        p2g_affine<FIXED, SR>(svd, sc.mat[mat], jp, mass, vol, C, sc.dt, sc.dx, sc.inv_dx, Bd);
      }
      const float mr = ok ? mass : 0.f;
      if constexpr (FIXED) {
        rec[0] = make_float4(x, y, z, mr);
        rec[1] = make_float4(ok ? mass * v[0] : 0.f, ok ? mass * v[1] : 0.f, ok ? mass * v[2] : 0.f, Bd[0]);
        rec[2] = make_float4(Bd[1], Bd[2], Bd[3], Bd[4]);
        rec[3] = make_float4(Bd[5], Bd[6], Bd[7], Bd[8]);
      } else {
        float q[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          q[r] = ok ? mass * v[r] : 0.f;
#pragma unroll
          for (int a = 0; a < 3; ++a) q[r] -= (ok ? xq[a] - bf[a] : 0.f) * Bd[3 * a + r];
      }
        rec[0] = make_float4(mr, q[0], q[1], q[2]);
        rec[1] = make_float4(Bd[0], Bd[1], Bd[2], Bd[3]);
        rec[2] = make_float4(Bd[4], Bd[5], Bd[6], Bd[7]);
        rec[3] = make_float4(Bd[8], mr != 0.f ? xq[0] : kOffGrid, xq[1], xq[2]);
      }
      // sparse storage: the tiles this record's deposit will touch
      if (SPARSE && sc.tile_cap && ok) {
        const int bx = (int)bf[0] - sc.winx, by = (int)bf[1] - sc.winy, bz = (int)bf[2] - sc.winz;
        const int lx = bx - ctx.rx, ly = by - ctx.ry, lz = bz - ctx.rz;
        if ((unsigned)lx <= 5u && (unsigned)ly <= 5u && (unsigned)lz <= 5u) {
          const uint32_t bits = block_tiles(lx, ly, lz);
          if (bits & ~ctx.tiles) atomicOr(&ctx.tiles, bits);
        } else {
          mark_far_tiles(sc, p.tile_mark, bx, by, bz);
        }
      }
    }
    if constexpr (WRITE_KEYS) {
      const int win[3] = {sc.winx, sc.winy, sc.winz};
      int nbase[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) nbase[a] = (xq[a] == xq[a]) ? (int)bf[a] - win[a] : 0;
      p.keys_by_id[p.orig[s]] = base_key(sc, nbase);
    }
  }
}

// A gather warp's shared memory: the velocity block, the particle inputs of
// its lanes' next round ([input][lane], the staged order), the scene record.
template <bool GATHER, bool SPARSE>
struct __align__(128) GatherWarp {
  float4 vel[GATHER ? kRegionNodes : 1];
  float in[kStagedInputs][32];
  SceneDev sc;
  GatherCtx ctx;
  uint32_t slots[SPARSE ? 27 : 1];  // sparse storage: slots of the tiles around the unit's, or kNoSlot
  uint32_t scene;   // scene whose record sc holds
  uint32_t parity;  // of the velocity block's next arrival
  uint64_t bar;
};

// MODE: kRecord (no gather: validate the state and compute the record from the
// SVD of F — the first substep of a call), kG2P (gather + return mapping, the
// last substep of a call), kG2PRecord (gather + return mapping + the record
// for the next scatter, with the return mapping's SVD reused).
//
// Every warp works alone: it takes units (a piece of a tile's particles) from
// the list, its first by its index and each later one from the counter, with
// the velocity block of the unit's tile fetched into its own shared memory by
// one TMA box, and shares no barrier with the other warps of its CTA.
// What bounds it: instruction issue (65% of the slots; 58 warp instructions a
// particle of mixed materials) and, behind that, the dependent chains of the
// SVD and instruction fetch (41 KB of code; it was 55, of which a second SVD
// for a case that never came was 13); 0.4 of the DRAM rate.  From a CTA per
// tile with a barrier per item, over all changes: 1.26 -> 1.13 ms at 16M
// particles (FP64 SVD, 256^3), 333 -> 279 us at 4M and 63 -> 52 us at 500k
// (FP32), with the records in deposit form.
// SPARSE: the group holds scenes on sparse storage (the tile lookups and marks
// cost the dense form up to 20% in registers and code: 278 -> 340 us at 4M).
template <int MODE, bool WRITE_KEYS, bool SPARSE, bool FIXED, class SR>
__global__ void __launch_bounds__(kGatherThreads, 5) k_g2p(PoolDev p, double tol, int sweeps,
                                                            int publish_all) {
  constexpr bool kGather = MODE != kRecord;
  constexpr bool kScatter = MODE != kG2P;
  constexpr uint32_t kWarps = kGatherThreads / 32;
  __shared__ GatherWarp<kGather, SPARSE> s_warp[kWarps];
  const uint32_t lane = threadIdx.x & 31u;
  GatherWarp<kGather, SPARSE>& w = s_warp[threadIdx.x >> 5];
  if (lane == 0) {
    w.scene = 0xffffffffu;
    w.ctx.tiles = 0;
    w.parity = 0;
    mbar_init(&w.bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  launch_next();
  wait_previous();
  // this SVD form's range of the list: units of FP32-SVD scenes, then FP64-SVD
  const uint32_t n32 = p.n_units[0];
  const uint32_t lo = sizeof(SR) == 8 ? n32 : 0u;
  const uint32_t hi = sizeof(SR) == 8 ? n32 + p.n_units[1] : n32;
  const SR stol = (SR)tol;
  // first units spread over the CTAs, so that a short list uses every SM
  for (uint32_t u = lo + (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < hi;) {
    const Item unit = p.units[unit_slot(p, n32, u)];
    uint32_t next = 0;  // this warp's next unit, taken now and read after this one's work
    if (lane == 0) next = lo + kWarps * gridDim.x + atomicAdd(p.work + (sizeof(SR) == 8 ? kWorkGather64 : kWorkGather32), 1u);
    // The inputs of a lane's next particle are copied to shared memory
    // (cp.async) from the moment this one's are consumed -- x and F before the
    // SVD, the rest before the stress -- and waited for apart: x and F as a
    // round begins, the rest after its G2P.  Those of a lane's first particle
    // are requested here, so that their loads overlap the velocity block's.
    auto fetch_early = [&](uint32_t k, uint32_t start, uint32_t count) {
      if (k < count) {
        // walk the planes with one pointer: PX..PZ, then F0..F8
        const size_t cap = p.cap;
        const float* src = p.planes + (start + k);
#pragma unroll
        for (int q = 0; q < 3; ++q, src += cap) cp_async4(&w.in[q][lane], src);
        src += (size_t)(F0 - 3) * cap;
#pragma unroll
        for (int q = 3; q < kInMass; ++q, src += cap) cp_async4(&w.in[q][lane], src);
      }
      cp_async_commit();
    };
    auto fetch_late = [&](uint32_t k, uint32_t start, uint32_t count) {
      if (k < count) {
        const size_t cap = p.cap;
        const float* src = p.planes + (size_t)MASS * cap + (start + k);
#pragma unroll
        for (int q = kInMass; q < kStagedInputs - 1; ++q, src += cap) cp_async4(&w.in[q][lane], src);
        cp_async4(&w.in[kStagedInputs - 1][lane], p.meta + (start + k));
      }
      cp_async_commit();
    };
    fetch_early(lane, unit.start, unit.count);
    fetch_late(lane, unit.start, unit.count);
    if (unit.scene != w.scene) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(p.scenes + unit.scene);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&w.sc);
      for (uint32_t k = lane; k < sizeof(SceneDev) / 4; k += 32) dst[k] = src[k];
      __syncwarp();
      if (lane == 0) {
        w.scene = unit.scene;
        // the scene's tensor map was written by a copy before this launch
        if (kGather) fence_tensormap(p.vel_maps + unit.scene);
      }
      __syncwarp();
    }
    const SceneDev& sc = w.sc;
    uint32_t* status = p.status + (size_t)sc.status * kStatusWords;
    // A latched fault, a spent substep budget or a retired scene: stand still.  A
    // vote, since another warp may latch a fault between two lanes' reads and
    // all lanes must go the same way around the warp barriers below.
    if (__all_sync(0xffffffffu, !scene_frozen(status) && sc.live)) {
      const uint32_t tw = sc.w;
      const uint32_t tx = unit.tile % tw, ty = (unit.tile / tw) % tw, tz = unit.tile / (tw * tw);
      const int rx = 4 * (int)tx - 1, ry = 4 * (int)ty - 1, rz = 4 * (int)tz - 1;
      if (lane == 0)
        w.ctx = GatherCtx{status, rx, ry, rz, (publish_all || budget_ends(status)) ? 1u : 0u, unit.start, unit.count, 0u};
      if constexpr (kGather) {
        // Stage the 8^3-node velocity block (out-of-grid nodes read as zero).
        if ((!SPARSE || sc.tile_cap == 0) && sc.n >= (uint32_t)kRegion) {
          if (lane == 0) {
            fence_proxy_async_smem();  // the lanes' reads of the block are done (__syncwarp below)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&w.bar)),
                         "r"((uint32_t)sizeof(w.vel))
                         : "memory");
            tma_load_box(w.vel, p.vel_maps + unit.scene, 4 * rx, ry, rz, &w.bar);
          }
          const uint32_t parity = w.parity;
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(&w.bar, parity))) {
            // The copy did not arrive: report it, wait once more (bounded)
            // for it and stop this warp.
            if (lane == 0) atomicOr(status, kFaultDeviceWait);
            mbar_wait_bounded(&w.bar, parity);
            cp_async_wait_all();
            return;
          }
          __syncwarp();
          if (lane == 0) w.parity = parity ^ 1u;
        } else if (SPARSE && sc.tile_cap) {
          // the slots of the 27 tiles around, then every node by cp.async
          if (lane < 27u) {
            const int ax = (int)tx + (int)(lane % 3u) - 1, ay = (int)ty + (int)((lane / 3u) % 3u) - 1,
                      az = (int)tz + (int)(lane / 9u) - 1;
            const bool in = (unsigned)ax < tw && (unsigned)ay < tw && (unsigned)az < tw;
            w.slots[lane] =
                in ? p.tile_slot[sc.key_off + (uint32_t)ax + tw * ((uint32_t)ay + tw * (uint32_t)az)] : kNoSlot;
          }
          __syncwarp();
#pragma unroll 4
          for (uint32_t r = lane; r < (uint32_t)kRegionNodes; r += 32) {
            // region coordinate l is node 4t - 1 + l: tile (l + 3) / 4 - 1, node (l + 3) % 4 in it
            const uint32_t lx = (r & 7u) + 3u, ly = ((r >> 3) & 7u) + 3u, lz = (r >> 6) + 3u;
            const uint32_t slot = w.slots[(lx >> 2) + 3u * (ly >> 2) + 9u * (lz >> 2)];
            const bool in = slot != kNoSlot && (unsigned)(rx + (int)lx - 3) < sc.n &&
                            (unsigned)(ry + (int)ly - 3) < sc.n && (unsigned)(rz + (int)lz - 3) < sc.n;
            if (in)
              cp_async16(&w.vel[r], p.vel + sc.grid_off + 64ull * slot + (lx & 3u) + 4u * (ly & 3u) + 16u * (lz & 3u));
            else
              w.vel[r] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
          cp_async_wait_all();
        } else {
          // a grid of fewer than 8 nodes an axis
          for (uint32_t r = lane; r < (uint32_t)kRegionNodes; r += 32) {
            const int64_t c =
                node_index(sc, p.tile_slot, rx + (int)(r & 7u), ry + (int)((r >> 3) & 7u), rz + (int)(r >> 6));
            w.vel[r] = c >= 0 ? p.vel[c] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      }
      __syncwarp();
      for (uint32_t k = lane; k < w.ctx.count; k += 32) {
        cp_async_wait<1>();
        const uint32_t s = w.ctx.start + k;
        auto early = [&] { fetch_early(k + 32u, w.ctx.start, w.ctx.count); };
        auto rest = [&] { fetch_late(k + 32u, w.ctx.start, w.ctx.count); };
        struct Refill {
          decltype(early)& e;
          decltype(rest)& l;
          __device__ __forceinline__ void late() const { cp_async_wait<0>(); }
          __device__ __forceinline__ void early_read() const { e(); }
          __device__ __forceinline__ void done() const { l(); }
        };
        float4 rec[4];
        particle_step<MODE, WRITE_KEYS, SPARSE, FIXED, SR>(
            p, sc, s, w.ctx, w.vel, stol, sweeps, StagedIn{&w.in[0][lane]}, Refill{early, rest},
            rec);
        if constexpr (kScatter) {
          float4* r4 = reinterpret_cast<float4*>(p.rec) + 4 * (size_t)s;
          r4[0] = rec[0];
          r4[1] = rec[1];
          r4[2] = rec[2];
          r4[3] = rec[3];
        }
      }
    }
    cp_async_wait_all();
    __syncwarp();
    if constexpr (kScatter && SPARSE) {
      // sparse storage: one store per tile the unit touched
      if (sc.tile_cap) {
        const uint32_t tw = sc.w;
        const uint32_t ax = (uint32_t)((w.ctx.rx + 1) >> 2) + lane % 3u - 1u,
                       ay = (uint32_t)((w.ctx.ry + 1) >> 2) + (lane / 3u) % 3u - 1u,
                       az = (uint32_t)((w.ctx.rz + 1) >> 2) + lane / 9u - 1u;
        if (lane < 27u && (w.ctx.tiles >> lane & 1u) && ax < tw && ay < tw && az < tw)
          p.tile_mark[sc.key_off + ax + tw * (ay + tw * az)] = 1;
        __syncwarp();
        if (lane == 0) w.ctx.tiles = 0;  // a frozen scene's unit marks none
      }
      __syncwarp();
    }
    u = __shfl_sync(0xffffffffu, next, 0);
  }
}

// Scatter of the next substep (mpm.wgsl:601-627): a particle with base =
// floor(xp - 0.5) deposits, at the node of offset (i,j,k), w (m, q + i Bdx +
// j Bdy + k Bdz) with w the quadratic B-spline weight of fx = xp - base; the
// gather writes its records in that form (particle_step).  Particles whose
// record mass is zero (numerical fault this substep) deposit nothing.
//
// Persistent CTAs over items (a tile's particles from the last regrouping,
// at most kStageMax), 224 threads.  Per item:
//  1. stage: the item's 64-byte records (contiguous slots) arrive in shared
//     memory as 2-D TMA tiles of 64 records (cp.async.bulk.tensor completing
//     on an mbarrier), issued while the previous item's block was flushed.
//     The tiles use the 64-byte swizzle: 16-byte chunk k of record j sits at
//     chunk k ^ ((j >> 1) & 3), which spreads the lanes' reads of one chunk
//     of different records over all shared-memory banks;
//  2. bin: every particle pushes itself onto the list of its current base
//     cell among the 6^3 cells whose stencils fit the tile's 8^3-node block,
//     so particles that moved since the regrouping are grouped with their new
//     cell-mates; one whose stencil leaves the block deposits straight to HBM;
//  3. deposit: a thread takes one x-slab i of the stencil and one cell: the
//     tile's own cells as the regrouping dealt them to warps (so that a
//     warp's flush atomics fall on distinct banks, count-ordered within the
//     warp), the three slabs of a cell in adjacent lanes, then the non-empty
//     margin cells particles moved into (listed by step 2).  It
//     adds the nine slab-i node contributions of its cell's particles in
//     registers and adds 9 x 4 sums to the shared block (add_node) for the
//     whole cell, not per particle; no two lanes of a warp add to the same
//     node in one step;
//  4. flush: every non-empty node of the 8^3 block goes to HBM with one
//     float4 atomic and is cleared for the next item.
// Every wait on the stage is bounded (about one second); a wait that gives
// up sets kFaultDeviceWait in the scene's status word and ends the CTA after
// a second bounded wait for its copy in flight.
//
// What bounds it: instruction issue and shared-memory latency, not bytes
// (17% of DRAM rate).  Lists instead of a counting sort, records written in
// deposit form by the gather instead of rewritten here, and the item's frame
// in shared memory took it from 0.832 to 0.773 ms on a 16M-particle scene
// (256^3), from 0.239 to 0.222 ms at 4M and from 43.3 to 40 us at 500k (the
// gather pays 0.03 ms for the form at 16M); swaps in flight together and a
// warp for the margin cells, to 0.715 and 0.204 ms.
__device__ __noinline__ void deposit_global(float4 c0, float4 c1, float4 c2, float4 c3, float4* acc,
                                            uint8_t* touched, const SceneDev* scp,
                                            const uint32_t* tile_slot) {
  const SceneDev& sc = *scp;
  const int win[3] = {sc.winx, sc.winy, sc.winz};
  const float Bd[9] = {c1.x, c1.y, c1.z, c1.w, c2.x, c2.y, c2.z, c2.w, c3.x};
  const float xp[3] = {c3.y, c3.z, c3.w};
  float wgt[3][3];
  int base[3];
  for (int a = 0; a < 3; ++a) {
    const float bf = floorf(xp[a] - 0.5f);
    base[a] = (int)bf - win[a];
    quad_weights(xp[a] - bf, wgt[a]);
  }
#pragma unroll 1
  for (int q = 0; q < 27; ++q) {
    const int i = q / 9, j = (q / 3) % 3, k = q % 3;
    const int64_t c = node_index(sc, tile_slot, base[0] + i, base[1] + j, base[2] + k);
    if (c < 0) continue;
    const float wt = wgt[0][i] * wgt[1][j] * wgt[2][k];
    const float fi = (float)i, fj = (float)j, fk = (float)k;
    const float4 v = make_float4(wt * c0.x, wt * (c0.y + Bd[0] * fi + Bd[3] * fj + Bd[6] * fk),
                                 wt * (c0.z + Bd[1] * fi + Bd[4] * fj + Bd[7] * fk),
                                 wt * (c0.w + Bd[2] * fi + Bd[5] * fj + Bd[8] * fk));
    atomicAdd(&acc[c], v);
    touch(touched, c);
  }
}

constexpr int kLocalCells = 216;  // 6^3 base cells whose stencils fit the 8^3 block
constexpr uint32_t kListEnd = 0xffffu;

// 16-byte chunk k of staged record j under the 64-byte swizzle.
__device__ __forceinline__ float4 stage_chunk(const float4* stage, uint32_t j, uint32_t k) {
  return stage[4 * j + (k ^ ((j >> 1) & 3u))];
}
__device__ __forceinline__ void stage_store(float4* stage, uint32_t j, const float4 (&rec)[4]) {
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) stage[4 * j + (k ^ ((j >> 1) & 3u))] = rec[k];
}

// Where an item's scatter lands, kept in shared memory so that it holds no
// registers: the scene's grid (the fields node_index reads), the 8^3-node
// block origin (rx, ry, rz) of its tile, and that origin with the lattice
// window added (a record's base cell is floor(xp - 0.5) - (bx, by, bz) in the
// block's 6^3 local cells).
struct ScatterItem {
  uint32_t n, w, key_off, tile_cap;
  uint64_t grid_off;
  int rx, ry, rz, bx, by, bz;
  uint32_t count, slot;
  uint32_t live;  // the scene takes deposits in this launch
  const SceneDev* sc;
  uint32_t* status;
};

__device__ __forceinline__ void scatter_item(ScatterItem& f, const PoolDev& p, const Item& item, uint32_t slot) {
  const SceneDev* sc = p.scenes + item.scene;
  const uint32_t w = sc->w;
  if (f.sc != sc) {
    f.sc = sc;
    f.n = sc->n;
    f.w = w;
    f.key_off = sc->key_off;
    f.tile_cap = sc->tile_cap;
    f.grid_off = sc->grid_off;
    f.status = p.status + (size_t)sc->status * kStatusWords;
    // A fault latched before this launch (or a spent substep budget, or a
    // retired scene) freezes the scene; one latched by this substep's gather
    // is handled per particle (m = 0 in its record).
    f.live = (scene_frozen(f.status) || !sc->live) ? 0u : 1u;
  }
  const uint32_t tx = item.tile % w, ty = (item.tile / w) % w, tz = item.tile / (w * w);
  f.rx = 4 * (int)tx - 1;
  f.ry = 4 * (int)ty - 1;
  f.rz = 4 * (int)tz - 1;
  f.bx = f.rx + sc->winx;
  f.by = f.ry + sc->winy;
  f.bz = f.rz + sc->winz;
  f.count = item.count;
  f.slot = slot;
}

// Shared-memory working set of one scatter item.
struct ScatterShared {
  float acc[4][kRegionFloats];  // the 8^3-node block: m, p.x, p.y, p.z
  uint32_t head[kLocalCells];   // first record of each local cell's list, or kListEnd
  uint16_t next[kStageMax];     // next record of the same cell
  uint8_t margin[kLocalCells];  // non-empty local cells outside the tile's own 4^3
  uint32_t n_margin;
};

// Scatter step 2 (bin) for a CTA of T threads: every staged record pushes
// itself (one shared-memory exchange) onto the list of its current base cell
// among the 6^3 local cells; the first record of a margin cell also lists the
// cell.  One whose stencil leaves the block deposits straight to HBM.  Lists
// take one pass and one barrier where a counting sort took a count, a scan by
// one warp and a ranked write with a barrier after each.  The caller
// synchronises after it.
template <int T>
__device__ __forceinline__ void bin_item(const float4* stage, const ScatterItem& f, const PoolDev& p, int acc_out,
                                         ScatterShared& ss) {
  const uint32_t count = f.count;
  const int bx = f.bx, by = f.by, bz = f.bz;
  for (uint32_t j = threadIdx.x; j < count; j += T) {
    const float4 c3 = stage_chunk(stage, j, 3);
    const int lx = (int)floorf(c3.y - 0.5f) - bx;
    const int ly = (int)floorf(c3.z - 0.5f) - by;
    const int lz = (int)floorf(c3.w - 0.5f) - bz;
    if ((unsigned)lx < 6u && (unsigned)ly < 6u && (unsigned)lz < 6u) {
      const uint32_t lc = (uint32_t)(lx + 6 * (ly + 6 * lz));
      const uint32_t old = atomicExch(&ss.head[lc], j);
      ss.next[j] = (uint16_t)old;
      if (old == kListEnd && ((unsigned)(lx - 1) >= 4u || (unsigned)(ly - 1) >= 4u || (unsigned)(lz - 1) >= 4u))
        ss.margin[atomicAdd(&ss.n_margin, 1u)] = (uint8_t)lc;
    } else {
      const float4 c0 = stage_chunk(stage, j, 0);
      if (c0.x != 0.f)
        deposit_global(c0, stage_chunk(stage, j, 1), stage_chunk(stage, j, 2), c3, p.acc[acc_out], p.touched[acc_out],
                       f.sc, p.tile_slot);
    }
  }
}

// The tile's own cell (local cell index) and x-slab that a core thread of the
// deposit takes, packed as lc | slab << 8: warp w holds slots 10w..10w+9 of
// the item's table, the three slab threads of a cell in adjacent lanes (a
// quarter-warp of a 16-byte record load then touches about three records
// instead of eight, and the lanes that read the same record are served by one
// broadcast); the two spare lanes of each warp (12 in all) take the 3 slabs of
// slots 60..63.
__device__ __forceinline__ uint32_t core_share(const uint8_t* order) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t q = warp * 2u + (lane - 30u);  // spare-lane index when lane >= 30
  const uint32_t slot = lane < 30u ? warp * 10u + lane / 3u : 60u + q / 3u;
  const uint32_t slab = lane < 30u ? lane % 3u : q % 3u;
  const uint32_t c = order[slot];
  return ((c & 3u) + 1u) + 6u * (((c >> 2) & 3u) + 1u + 6u * ((c >> 4) + 1u)) + (slab << 8);
}

// Adds a node's four sums to the shared block.  A float add in shared memory is
// a load, an add and a compare-and-swap, retried while other lanes win; the
// built-in runs the four one after the other, each waiting for the last.  Here
// the four loads, then the four swaps, are in flight together, and only a sum
// that met another writer takes the built-in (calls of 12..20 substeps: 1M
// particles 3.89 -> 3.81 ms, 4M 6.48 -> 6.31, 16M 40.2 -> 39.4; twelve in flight
// need the registers of the sums: 40.5).
__device__ __forceinline__ void add_node(ScatterShared& ss, int r, float2 xy, float2 zm) {
  const float add[4] = {zm.y, xy.x, xy.y, zm.x};
  uint32_t old[4], got[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) old[c] = *reinterpret_cast<volatile uint32_t*>(&ss.acc[c][r]);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    got[c] = atomicCAS(reinterpret_cast<uint32_t*>(&ss.acc[c][r]), old[c],
                       __float_as_uint(__uint_as_float(old[c]) + add[c]));
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (got[c] != old[c]) atomicAdd(&ss.acc[c][r], add[c]);
}

// Scatter step 3 (deposit) for a CTA of T >= 192 threads.  The first 192
// threads take the (cell, x-slab) pairs of the tile's own 64 cells (`share`,
// core_share): each warp holds 10 cells from the per-item table
// (k_item_order), which deals the cells so that a warp's 30 flush atomics of
// one node and channel fall on 30 different shared-memory banks, in
// particle-count order inside the warp (scatter -18% against a plain count
// order).  The (margin cell, slab) pairs of the non-empty cells particles moved
// into go to the warps beyond the core's from the start, then to all.  A thread adds the nine slab nodes of
// its cell's particles in registers and adds 9 x 4 sums to the shared block for
// the whole cell; no two lanes of a warp add to the same node in one step.
template <int T>
__device__ __forceinline__ void deposit_item(const float4* stage, uint32_t share, const ScatterItem& f,
                                             ScatterShared& ss) {
  static_assert(T >= 192, "the core cells take 6 warps of 10 cells x 3 slabs");
  // One loop (one copy of the code) over the core pairs, then the margin's.
#pragma unroll 1
  for (uint32_t u = threadIdx.x; u < 192u + 3u * ss.n_margin; u += T) {
    if (u >= 192u) share = ss.margin[(u - 192u) / 3u] + (((u - 192u) % 3u) << 8);
    uint32_t j = ss.head[share & 0xffu];
    if (j == kListEnd) continue;
    // Adds the particles of local cell lc in registers: node (slab, j, k) gets
    // w_slab(fx0) w_j(fx1) w_k(fx2) (m, q + slab Bdx + j Bdy + k Bdz), the sums
    // over j and k taken as running increments; per node of the slab (p.x, p.y)
    // and (p.z, m), accumulated in pairs.
    float2 axy[9], azm[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) axy[q] = azm[q] = make_float2(0.f, 0.f);
    const uint32_t lc = share & 0xffu;
    const float fslab = (float)(share >> 8);
    // xp - ox is the slab's argument t = fx0 - (1.5, 1, 0.5) of its weight
    // 0.5 (1.5 - fx)^2, 0.75 - (fx - 1)^2, 0.5 (fx - 0.5)^2; xp - oy, oz are fx1, fx2
    const float ox = (float)(f.bx + (int)(lc % 6u)) + (1.5f - 0.5f * fslab);
    const float oy = (float)(f.by + (int)((lc / 6u) % 6u));
    const float oz = (float)(f.bz + (int)(lc / 36u));
#pragma unroll 1
    do {
      const float4 c0 = stage_chunk(stage, j, 0), c1 = stage_chunk(stage, j, 1), c2 = stage_chunk(stage, j, 2),
                   c3 = stage_chunk(stage, j, 3);
      j = ss.next[j];
      const float ts = c3.y - ox;
      const float wi = fslab == 1.0f ? fmaf(-ts, ts, 0.75f) : 0.5f * ts * ts;
      float wy[3], wz[3];
      quad_weights(c3.z - oy, wy);
      quad_weights(c3.w - oz, wz);
      // momentum at node (slab, 0, 0), paired with the mass: (q.x, q.y), (q.z, m)
      float2 qxy = make_float2(fmaf(fslab, c1.x, c0.y), fmaf(fslab, c1.y, c0.z));
      float2 qzm = make_float2(fmaf(fslab, c1.z, c0.w), c0.x);
      const float2 dyxy = make_float2(c1.w, c2.x), dzxy = make_float2(c2.z, c2.w);
      const float dyz = c2.y, dzz = c3.x;
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) {
        if (jj) {
          qxy = add2(qxy, dyxy);
          qzm.x += dyz;
        }
        const float wij = wi * wy[jj];
        float2 cxy = qxy, czm = qzm;
#pragma unroll
        for (int kk = 0; kk < 3; ++kk) {
          if (kk) {
            cxy = add2(cxy, dzxy);
            czm.x += dzz;
          }
          const float wt = wij * wz[kk];
          const float2 w2 = make_float2(wt, wt);
          axy[3 * jj + kk] = fma2(w2, cxy, axy[3 * jj + kk]);
          azm[3 * jj + kk] = fma2(w2, czm, azm[3 * jj + kk]);
        }
      }
    } while (j != kListEnd);
    // ... and the slab's sums to the shared block.
    const uint32_t at = share & 0xffu;
    const int r0 = region_index((int)(at % 6u), (int)((at / 6u) % 6u), (int)(at / 36u)) + (int)(share >> 8);
#pragma unroll
    for (int jj = 0; jj < 3; ++jj)
#pragma unroll
      for (int kk = 0; kk < 3; ++kk) {
        const int r = r0 + kRsy * jj + kRsz * kk;
        add_node(ss, r, axy[3 * jj + kk], azm[3 * jj + kk]);
      }
  }
}

// Scatter step 4 (flush): every non-empty node of the 8^3 block goes to HBM
// with one float4 atomic and is cleared for the next item, as are the cell
// lists.  The caller synchronises before the block is reused.
template <int T>
__device__ __forceinline__ void flush_item(const ScatterItem& f, const PoolDev& p, int acc_out, ScatterShared& ss) {
  for (int r = threadIdx.x; r < kRegionNodes; r += T) {
    const int lx = r & 7, ly = (r >> 3) & 7, lz = r >> 6;
    const int q = region_index(lx, ly, lz);
    const float m = ss.acc[0][q], px = ss.acc[1][q], py = ss.acc[2][q], pz = ss.acc[3][q];
    if (m != 0.f || px != 0.f || py != 0.f || pz != 0.f) {
      ss.acc[0][q] = 0.f;
      ss.acc[1][q] = 0.f;
      ss.acc[2][q] = 0.f;
      ss.acc[3][q] = 0.f;
      const int64_t c = node_index(f, p.tile_slot, f.rx + lx, f.ry + ly, f.rz + lz);
      if (c >= 0) {
        atomicAdd(&p.acc[acc_out][c], make_float4(m, px, py, pz));
        touch(p.touched[acc_out], (uint64_t)c);
      }
    }
  }
  for (int r = threadIdx.x; r < kLocalCells; r += T) ss.head[r] = kListEnd;
  if (threadIdx.x == 0) ss.n_margin = 0;
}

__device__ __forceinline__ void clear_scatter_shared(ScatterShared& ss, int threads) {
  for (int r = threadIdx.x; r < 4 * kRegionFloats; r += threads) (&ss.acc[0][0])[r] = 0.f;
  for (int r = threadIdx.x; r < kLocalCells; r += threads) ss.head[r] = kListEnd;
  if (threadIdx.x == 0) ss.n_margin = 0;
}

__global__ void __launch_bounds__(kScatterThreads, 4) k_p2g(PoolDev p, const __grid_constant__ CUtensorMap rec_map,
                                                            int acc_out) {
  extern __shared__ __align__(128) unsigned char s_dyn[];
  // the swizzle pattern repeats every 512 bytes: align the stage to 1 KiB
  float4* s_stage =
      reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(s_dyn) + 1023u) & ~static_cast<uintptr_t>(1023u));
  __shared__ ScatterShared ss;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ __align__(16) Item s_desc;     // descriptor of the next item, copied ahead
  __shared__ ScatterItem s_item[2];         // this item's frame and the next one's
  __shared__ uint32_t s_next;
  launch_next();
  clear_scatter_shared(ss, kScatterThreads);
  wait_previous();
  const uint32_t n32 = p.n_items[0];
  const uint32_t n_items = n32 + p.n_items[1];
  if (blockIdx.x >= n_items) return;
  // Thread 0 stages an item (of 1..kStageMax particles) as ceil(count / 64)
  // tiles; rows past the item are loaded but not read.
  auto stage = [&](const Item& nx) {
    if (nx.count - 1u < (uint32_t)kStageMax) {
      const uint32_t boxes = (nx.count + kStageBoxRows - 1) / kStageBoxRows;
      fence_proxy_async_smem();
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&s_bar)),
                   "r"(boxes * kStageBoxRows * 64u)
                   : "memory");
      for (uint32_t b = 0; b < boxes; ++b)
        tma_load_rows(s_stage + (size_t)b * kStageBoxRows * 4, &rec_map, (int)(nx.start + b * kStageBoxRows), &s_bar);
    }
  };
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    fence_mbar_init();
    const uint32_t slot = item_slot(p, n32, blockIdx.x);
    const Item item = p.items[slot];
    stage(item);
    s_item[0].sc = s_item[1].sc = nullptr;
    scatter_item(s_item[0], p, item, slot);
  }
  __syncthreads();
  uint32_t parity = 0;
  for (uint32_t it = blockIdx.x; it < n_items; parity ^= 1u) {
    const ScatterItem& f = s_item[parity];
    // This CTA's next item, taken now; thread 0 copies its descriptor during
    // the deposit and stages its records after it, so that no thread waits
    // for the counter or the descriptor.
    uint32_t next = 0;
    if (threadIdx.x == 0) next = gridDim.x + atomicAdd(p.work + kWorkScatter, 1u);
    const uint32_t share = threadIdx.x < 192 ? core_share(p.item_order + (size_t)f.slot * 64) : 0u;
    const bool staged = f.count - 1u < (uint32_t)kStageMax;
    const bool ok = staged && mbar_wait_bounded(&s_bar, parity);
    const bool live = ok && f.live != 0u;
    if (live) bin_item<kScatterThreads>(s_stage, f, p, acc_out, ss);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (next < n_items) cp_async16(&s_desc, p.items + item_slot(p, n32, next));
      s_next = next;
    }
    if (live) deposit_item<kScatterThreads>(s_stage, share, f, ss);
    if (__syncthreads_or(!ok)) {
      // The stage did not arrive (or the item exceeds the stage): report it,
      // wait once more (bounded) for the copy in flight and stop this CTA.
      if (threadIdx.x == 0) {
        atomicOr(f.status, kFaultDeviceWait);
        cp_async_wait_all();
      }
      if (staged) mbar_wait_bounded(&s_bar, parity);
      return;
    }
    // Every thread is done with the stage: the next item's copy goes now.
    it = s_next;
    if (threadIdx.x == 0 && it < n_items) {
      cp_async_wait_all();
      const Item item = s_desc;
      stage(item);
      scatter_item(s_item[parity ^ 1u], p, item, item_slot(p, n32, it));
    }
    flush_item<kScatterThreads>(f, p, acc_out, ss);
    __syncthreads();
  }
}

// Fused gather + scatter of one substep (non-deterministic P2G): per item,
// the CTA runs the gather of every particle (G2P, F update, return mapping,
// B record) with the record kept in shared memory instead of HBM, then bins,
// deposits and flushes the item's records as k_p2g does.  Saves the record's
// 64-byte write and read per particle and one launch, and lets the gather
// (FP32/FP64/XU pipes) of one CTA overlap the deposit (shared-memory
// atomics) of the other CTA on the SM.  Items hold at most kStageMax
// particles (the regrouping cuts them), so the records fit the stage; an
// item that does not fit latches kFaultDeviceWait and is skipped.
//
// A fault latched when a CTA comes to a scene (its state is read with the
// scene's first item in that CTA) freezes the CTA's items of it (no gather, no
// deposit); a particle that faults during the gather deposits nothing (m = 0
// in its record).  The scene is frozen from the next substep on.
template <bool WRITE_KEYS, class SR>
__global__ void __launch_bounds__(kFusedThreads, 2) k_g2p2g(PoolDev p, double tol, int sweeps,
                                                              int acc_out) {
  extern __shared__ __align__(16) float4 s_stage[];  // kStageMax records, 64-byte swizzle
  __shared__ __align__(16) SceneDev s_sc;
  __shared__ __align__(16) float4 s_vel[kRegionNodes];
  __shared__ ScatterShared ss;
  __shared__ ScatterItem s_item;
  __shared__ GatherCtx s_ctx;
  const SR stol = (SR)tol;
  launch_next();
  clear_scatter_shared(ss, kFusedThreads);
  if (threadIdx.x == 0) s_item.sc = nullptr;
  wait_previous();
  // this SVD form's range of the work list: FP32-SVD items, then FP64-SVD items
  const uint32_t n32 = p.n_items[0];
  const uint32_t it_lo = sizeof(SR) == 8 ? n32 : 0u;
  const uint32_t it_hi = sizeof(SR) == 8 ? n32 + p.n_items[1] : n32;
  for (uint32_t it = it_lo + blockIdx.x; it < it_hi; it += gridDim.x) {
    const uint32_t slot = item_slot(p, n32, it);
    const Item item = p.items[slot];
    {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(p.scenes + item.scene);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&s_sc);
      for (int k = threadIdx.x; k < (int)(sizeof(SceneDev) / 4); k += kFusedThreads) dst[k] = src[k];
    }
    const bool fits = item.count <= (uint32_t)kStageMax;
    if (threadIdx.x == 0) {
      scatter_item(s_item, p, item, slot);
      if (!fits) {
        s_item.live = 0u;
        s_item.sc = nullptr;  // the flag is the item's, not the scene's
        atomicOr(s_item.status, kFaultDeviceWait);
      }
      s_ctx = GatherCtx{s_item.status, s_item.rx, s_item.ry, s_item.rz, budget_ends(s_item.status) ? 1u : 0u,
                        item.start, item.count, 0u};
    }
    __syncthreads();
    // Stage the 8^3-node velocity block (out-of-grid nodes read as zero).
    for (int r = threadIdx.x; r < kRegionNodes; r += kFusedThreads) {
      const int64_t c = node_index(s_sc, p.tile_slot, s_item.rx + (r & 7), s_item.ry + ((r >> 3) & 7),
                                   s_item.rz + (r >> 6));
      s_vel[r] = c >= 0 ? p.vel[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t share = threadIdx.x < 192 ? core_share(p.item_order + (size_t)slot * 64) : 0u;
    __syncthreads();
    const bool live = s_item.live != 0u;
    if (live) {
      for (uint32_t k = threadIdx.x; k < item.count; k += kFusedThreads) {
        const uint32_t s = item.start + k;
        float4 rec[4];
        particle_step<kG2PRecord, WRITE_KEYS, false, false, SR>(p, s_sc, s, s_ctx, s_vel, stol, sweeps, PoolIn{p, s}, NoRefill{},
                                                  rec);
        stage_store(s_stage, k, rec);
      }
      // a thread bins the records it wrote
      bin_item<kFusedThreads>(s_stage, s_item, p, acc_out, ss);
    }
    __syncthreads();
    if (live) deposit_item<kFusedThreads>(s_stage, share, s_item, ss);
    __syncthreads();
    flush_item<kFusedThreads>(s_item, p, acc_out, ss);
    __syncthreads();
  }
}

// Deterministic scatter (the fixed-order P2G of molla's
// mpm_deterministic_p2g.wgsl:85-150, restructured per tile).  Requires a
// regrouping after every gather, so that every particle of a tile item sits
// in its own base cell.  Thread (cell, slab) sums its cell's particles in slot
// order — (key, identity) order — in registers; the CTA then reduces the
// (cell, slab) partial sums of each of the tile's 6^3 footprint nodes in a
// fixed cell order and stores the block, without atomics.  A combine pass
// adds the blocks of the tiles covering each node, again in a fixed order.
// The result depends only on the scene's own particles and identities: it is
// bit-identical from run to run and whether or not other scenes share the
// launch.
__global__ void __launch_bounds__(kDetThreads, 2) k_p2g_det(PoolDev p, float4* __restrict__ blocks, int acc_out) {
  __shared__ uint32_t s_first[64], s_end[64];
  __shared__ float s_part[3 * 64 * 9 * 4];
  __shared__ uint32_t s_fault;
  launch_next();
  wait_previous();
  const float4* rec = reinterpret_cast<const float4*>(p.rec);
  const uint32_t n32 = p.n_items[0];
  const uint32_t n_items = n32 + p.n_items[1];
  const int cell = threadIdx.x & 63;
  const int slab = threadIdx.x >> 6;
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const uint32_t slot = item_slot(p, n32, it);
    const Item item = p.items[slot];
    const SceneDev* scp = p.scenes + item.scene;
    const uint32_t w = scp->w;
    const float ox = scp->ox, oy = scp->oy, oz = scp->oz, inv_dx = scp->inv_dx, dx = scp->dx;
    const int winx = scp->winx, winy = scp->winy, winz = scp->winz;
    uint32_t* status = p.status + (size_t)scp->status * kStatusWords;
    const uint32_t tx = item.tile % w, ty = (item.tile / w) % w, tz = item.tile / (w * w);
    if (threadIdx.x == 0) s_fault = (scene_frozen(status) || !scp->live) ? 1u : 0u;
    if (threadIdx.x < 64) {
      s_first[threadIdx.x] = 0;
      s_end[threadIdx.x] = 0;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < item.count; k += blockDim.x) {
      const uint32_t s = item.start + k;
      const uint32_t c = p.slot_key[s] & 63u;
      if (k == 0 || (p.slot_key[s - 1] & 63u) != c) s_first[c] = s;
      if (k + 1 == item.count || (p.slot_key[s + 1] & 63u) != c) s_end[c] = s + 1;
    }
    __syncthreads();
    float am[9], apx[9], apy[9], apz[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) am[q] = apx[q] = apy[q] = apz[q] = 0.f;
    if (s_fault == 0) {
      const int cx = cell & 3, cy = (cell >> 2) & 3, cz = cell >> 4;
      const int bx = 4 * (int)tx + cx, by = 4 * (int)ty + cy, bz = 4 * (int)tz + cz;  // this cell's base
      const int win[3] = {winx, winy, winz};
      const uint32_t end = s_end[cell];
      uint32_t s = s_first[cell];
      float4 n0, n1, n2, n3;  // the next record, loaded while this one is added
      auto load = [&](uint32_t at) {
        const float4* r = rec + 4 * (size_t)at;
        n0 = r[0];
        n1 = r[1];
        n2 = r[2];
        n3 = r[3];
      };
      if (s < end) load(s);
      for (; s < end; ++s) {
        const float4 r0 = n0, r1 = n1, r2 = n2, r3 = n3;
        if (s + 1 < end) load(s + 1);
        if (r0.w == 0.f) continue;
        const float mass = r0.w;
        const float B[9] = {r1.w, r2.x, r2.y, r2.z, r2.w, r3.x, r3.y, r3.z, r3.w};
        const float xp[3] = {lattice_pos(r0.x, ox, inv_dx), lattice_pos(r0.y, oy, inv_dx),
                             lattice_pos(r0.z, oz, inv_dx)};
        float wgt[3][3], fx[3];
        int base[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float bf = floorf(xp[a] - 0.5f);
          base[a] = (int)bf - win[a];
          fx[a] = xp[a] - bf;
          quad_weights(fx[a], wgt[a]);
        }
        const float wi = slab == 0 ? wgt[0][0] : (slab == 1 ? wgt[0][1] : wgt[0][2]);
        const float di = ((float)slab - fx[0]) * dx;
        const float qx[3] = {r1.x + B[0] * di, r1.y + B[1] * di, r1.z + B[2] * di};
        const bool own = base[0] == bx && base[1] == by && base[2] == bz;
        if (!own && slab == 0 && threadIdx.x < 64) atomicOr(status, kFaultNondeterministic);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float wij = wi * wgt[1][j];
          const float dj = ((float)j - fx[1]) * dx;
          const float qy[3] = {qx[0] + B[3] * dj, qx[1] + B[4] * dj, qx[2] + B[5] * dj};
#pragma unroll
          for (int kk = 0; kk < 3; ++kk) {
            const float wt = wij * wgt[2][kk];
            const float dk = ((float)kk - fx[2]) * dx;
            const float dm = wt * mass;
            const float px = wt * (qy[0] + B[6] * dk);
            const float py = wt * (qy[1] + B[7] * dk);
            const float pz = wt * (qy[2] + B[8] * dk);
            if (own) {
              am[3 * j + kk] += dm;
              apx[3 * j + kk] += px;
              apy[3 * j + kk] += py;
              apz[3 * j + kk] += pz;
            } else {
              // Not in its cell (positions set from outside the grid since
              // the last regrouping): deposited with an atomic that the
              // combine pass adds to, outside the fixed order; flagged in
              // the status word.
              const int64_t c = node_index(*scp, p.tile_slot, base[0] + slab, base[1] + j, base[2] + kk);
              if (c >= 0) {
                atomicAdd(&p.acc[acc_out][c], make_float4(dm, px, py, pz));
                touch(p.touched[acc_out], (uint64_t)c);
              }
            }
          }
        }
      }
    }
    {
      float* dst = s_part + ((slab * 64 + cell) * 9) * 4;
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        dst[4 * q] = am[q];
        dst[4 * q + 1] = apx[q];
        dst[4 * q + 2] = apy[q];
        dst[4 * q + 3] = apz[q];
      }
    }
    __syncthreads();
    // Node (nx, ny, nz) of the 6^3 footprint receives, from cell (cx, cy, cz)
    // with 0 <= n - c <= 2 per axis, the partial sum stored by thread
    // (cell, slab = nx - cx) at index 3 (ny - cy) + (nz - cz).
    float4* blk = blocks + (size_t)slot * kTileNodes;
    for (int q = threadIdx.x; q < kTileNodes; q += blockDim.x) {
      const int nx = q % 6, ny = (q / 6) % 6, nz = q / 36;
      float sm = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
      for (int cz = max(0, nz - 2); cz <= min(3, nz); ++cz)
        for (int cy = max(0, ny - 2); cy <= min(3, ny); ++cy)
          for (int cx = max(0, nx - 2); cx <= min(3, nx); ++cx) {
            const float* src = s_part + (((nx - cx) * 64 + (cx + 4 * cy + 16 * cz)) * 9 + 3 * (ny - cy) + (nz - cz)) * 4;
            sm += src[0];
            sx += src[1];
            sy += src[2];
            sz += src[3];
          }
      blk[q] = make_float4(sm, sx, sy, sz);
    }
    __syncthreads();
  }
}

// Combine pass of the deterministic scatter: node g of a scene receives the
// blocks of the (up to 8) occupied tiles whose footprint [4t, 4t+5] contains
// it, summed in (tz, ty, tx) order by the first such tile's thread.
__global__ void k_combine_det(PoolDev p, const float4* blocks, const uint32_t* tile_item,
                              int acc_out) {
  launch_next();
  wait_previous();
  const uint32_t n32 = p.n_items[0], total = n32 + p.n_items[1];
  for (uint32_t li = blockIdx.x; li < total; li += gridDim.x) {
    const uint32_t it = item_slot(p, n32, li);  // the item's slot, as tile_item holds it
    const Item item = p.items[it];
    const SceneDev* scp = p.scenes + item.scene;
    const int w = (int)scp->w, n = (int)scp->n;
    const uint32_t key_off = scp->key_off;
    const int tx = (int)(item.tile % (uint32_t)w), ty = (int)((item.tile / (uint32_t)w) % (uint32_t)w),
              tz = (int)(item.tile / (uint32_t)(w * w));
    for (int q = threadIdx.x; q < kTileNodes; q += blockDim.x) {
      const int g[3] = {4 * tx + q % 6, 4 * ty + (q / 6) % 6, 4 * tz + q / 36};
      if (g[0] >= n || g[1] >= n || g[2] >= n) continue;
      int lo[3], hi[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        hi[a] = g[a] / 4;
        lo[a] = max(0, (g[a] - 5 + 3) / 4);  // smallest t with 4t + 5 >= g
        hi[a] = min(hi[a], w - 1);
      }
      bool mine = false, found = false;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int cz = lo[2]; cz <= hi[2]; ++cz)
        for (int cy = lo[1]; cy <= hi[1]; ++cy)
          for (int cx = lo[0]; cx <= hi[0]; ++cx) {
            const uint32_t key = key_off + (uint32_t)(cx + w * (cy + w * cz));
            const uint32_t other = tile_item[key];
            if (other == 0xffffffffu) continue;
            if (!found) {
              found = true;
              mine = other == it;
              if (!mine) break;
            }
            const int l = (g[0] - 4 * cx) + 6 * ((g[1] - 4 * cy) + 6 * (g[2] - 4 * cz));
            const float4 b = blocks[(size_t)other * kTileNodes + l];
            sum.x += b.x;
            sum.y += b.y;
            sum.z += b.z;
            sum.w += b.w;
          }
      const int64_t c = mine ? node_index(*scp, p.tile_slot, g[0], g[1], g[2]) : -1;
      if (c >= 0) {
        // One writer per node; the cell holds zero or out-of-order deposits.
        float4& a = p.acc[acc_out][c];
        const float4 old = a;
        a = make_float4(old.x + sum.x, old.y + sum.y, old.z + sum.z, old.w + sum.w);
        touch(p.touched[acc_out], (uint64_t)c);
      }
    }
  }
}

// ---------------------------------------------------------------------------

template <int MODE, bool KEYS, bool SPARSE, bool FIXED, class SR>
static cudaError_t launch_gather_t(const PoolDev& p, double tol, int sweeps, int grid, cudaStream_t st,
                                   bool publish_all) {
  if (MODE == kRecord) {
    // opens a call, with no grid update before it
    const cudaError_t e = cudaMemsetAsync(p.work, 0, kWorkWords * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
  }
  return launch_dependent(k_g2p<MODE, KEYS, SPARSE, FIXED, SR>, grid, kGatherThreads, 0, st, p, tol, sweeps,
                          publish_all ? 1 : 0);
}

cudaError_t launch_gather(int mode, bool write_keys, bool sparse, bool fixed, bool svd_fp64, const PoolDev& p,
                          double tol, int sweeps, int grid, cudaStream_t st, bool publish_all) {
  auto pick = [&](auto m) {
    constexpr int M = decltype(m)::value;
    auto with = [&](auto keys, auto sp, auto fx) {
      constexpr bool K = decltype(keys)::value, S = decltype(sp)::value, X = decltype(fx)::value;
      return svd_fp64 ? launch_gather_t<M, K, S, X, double>(p, tol, sweeps, grid, st, publish_all)
                      : launch_gather_t<M, K, S, X, float>(p, tol, sweeps, grid, st, publish_all);
    };
    const std::true_type yes;
    const std::false_type no;
    // the fixed-order mode takes the sparse form, which serves dense scenes too
    if (fixed) return write_keys ? with(yes, yes, yes) : with(no, yes, yes);
    if (write_keys) return sparse ? with(yes, yes, no) : with(yes, no, no);
    return sparse ? with(no, yes, no) : with(no, no, no);
  };
  switch (mode) {
    case kRecord: return pick(std::integral_constant<int, kRecord>{});
    case kG2P: return pick(std::integral_constant<int, kG2P>{});
    case kG2PRecord: return pick(std::integral_constant<int, kG2PRecord>{});
    default: return cudaErrorInvalidValue;
  }
}

constexpr size_t kFusedStageBytes = (size_t)kStageMax * 64;

template <bool KEYS, class SR>
static cudaError_t launch_fused_t(const PoolDev& p, double tol, int sweeps, int acc_out, int grid,
                                  cudaStream_t st) {
  return launch_dependent(k_g2p2g<KEYS, SR>, grid, kFusedThreads, kFusedStageBytes, st, p, tol, sweeps, acc_out);
}

cudaError_t launch_fused(bool write_keys, bool svd_fp64, const PoolDev& p, double tol, int sweeps,
                         int acc_out, int grid, cudaStream_t st) {
  if (svd_fp64)
    return write_keys ? launch_fused_t<true, double>(p, tol, sweeps, acc_out, grid, st)
                      : launch_fused_t<false, double>(p, tol, sweeps, acc_out, grid, st);
  return write_keys ? launch_fused_t<true, float>(p, tol, sweeps, acc_out, grid, st)
                    : launch_fused_t<false, float>(p, tol, sweeps, acc_out, grid, st);
}

// stage tiles plus 1 KiB for the alignment of the swizzled stage
constexpr size_t kStageBytes = (size_t)kStageMax * 64 + 1024;
static_assert(kStageMax % kStageBoxRows == 0, "the stage holds whole TMA tiles");

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static bool encode_map(CUtensorMap* out, int rank, const float* base, const cuuint64_t* dims, const cuuint64_t* strides,
                       const cuuint32_t* box, CUtensorMapSwizzle swizzle, std::string* err) {
  static EncodeTiledFn encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      if (err) *err = "cuTensorMapEncodeTiled is not available from the driver";
      return false;
    }
    encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<float*>(base), dims,
                            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    if (err) *err = "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r);
    return false;
  }
  return true;
}

bool make_record_map(CUtensorMap* out, const float* rec, uint32_t cap, std::string* err) {
  // records: rows of 16 floats (64 bytes), cap rows; tiles of 64 rows
  const cuuint64_t dims[2] = {16, cap ? cap : 1};
  const cuuint64_t strides[1] = {64};
  const cuuint32_t box[2] = {16, (cuuint32_t)kStageBoxRows};
  return encode_map(out, 2, rec, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B, err);
}

bool make_velocity_map(CUtensorMap* out, const float4* vel, uint32_t n, std::string* err) {
  // n^3 nodes of four floats, x fastest; boxes of 8^3 nodes
  const cuuint64_t dims[3] = {4ull * n, n, n};
  const cuuint64_t strides[2] = {16ull * n, 16ull * n * n};
  const cuuint32_t box[3] = {4 * kRegion, kRegion, kRegion};
  return encode_map(out, 3, reinterpret_cast<const float*>(vel), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, err);
}

// Self-test of the scatter's bounded stage wait: one warp waits, through the
// same mbar_wait_bounded, on an mbarrier phase that nothing completes (one
// expected arrival, none made), then reports the way k_p2g does
// (kFaultDeviceWait in the status word) and records how long it waited.  No
// copy is in flight, so the CTA may end there.
__global__ void __launch_bounds__(32) k_selftest_wait(uint32_t* status, unsigned long long* waited_ns) {
  __shared__ __align__(8) uint64_t s_bar;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  const uint64_t t0 = global_ns();
  const bool ok = mbar_wait_bounded(&s_bar, 0u);
  if (__syncthreads_or(!ok) && threadIdx.x == 0) {
    atomicOr(status, kFaultDeviceWait);
    *waited_ns = global_ns() - t0;
  }
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(&s_bar)) : "memory");
}

cudaError_t launch_selftest_wait(uint32_t* status, unsigned long long* waited_ns, cudaStream_t st) {
  k_selftest_wait<<<1, 32, 0, st>>>(status, waited_ns);
  return cudaGetLastError();
}

cudaError_t launch_scatter(const PoolDev& p, const CUtensorMap& rec_map, int acc_out, int grid, cudaStream_t st) {
  return launch_dependent(k_p2g, grid, kScatterThreads, kStageBytes, st, p, rec_map, acc_out);
}

cudaError_t launch_scatter_det(const PoolDev& p, float4* blocks, int acc_out, int grid, cudaStream_t st) {
  return launch_dependent(k_p2g_det, grid, kDetThreads, 0, st, p, blocks, acc_out);
}

cudaError_t launch_combine_det(const PoolDev& p, const float4* blocks, const uint32_t* tile_item, uint32_t max_items,
                               int acc_out, cudaStream_t st) {
  if (!max_items) return cudaSuccess;
  return launch_dependent(k_combine_det, (int)std::min<uint32_t>(max_items, 148u * 16u), 128, 0, st, p, blocks, tile_item,
                          acc_out);
}

static int persistent(const void* fn, int threads, size_t dyn_smem = 0) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, dyn_smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  if (sms < 1) sms = 148;
  return sms * per_sm;
}

int gather_grid_size(bool svd_fp64) {
  return svd_fp64 ? persistent((const void*)k_g2p<kG2PRecord, false, false, false, double>, kGatherThreads)
                  : persistent((const void*)k_g2p<kG2PRecord, false, false, false, float>, kGatherThreads);
}

int fused_grid_size(bool svd_fp64) {
  // the record stage needs more than the default 48 KB of dynamic shared memory
  const void* fns[4] = {(const void*)k_g2p2g<false, double>, (const void*)k_g2p2g<true, double>,
                        (const void*)k_g2p2g<false, float>, (const void*)k_g2p2g<true, float>};
  for (const void* fn : fns)
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFusedStageBytes);
  return persistent(svd_fp64 ? fns[0] : fns[2], kFusedThreads, kFusedStageBytes);
}

int scatter_grid_size() {
  // the record stage needs more than the default 48 KB of dynamic shared memory
  cudaFuncSetAttribute((const void*)k_p2g, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageBytes);
  return persistent((const void*)k_p2g, kScatterThreads, kStageBytes);
}

}  // namespace mpm
