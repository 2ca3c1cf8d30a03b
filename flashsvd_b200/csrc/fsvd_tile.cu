// Decode for batches of 5..128 sequences (bf16): the factor products as tiled GEMMs on the 5th
// generation tensor cores.
//
// With more than 8 activation rows per factor row the 16 x 8 register tiles of the persistent
// interpreter (fsvd_kernel.cuh) no longer fit the batch; here a factor product is
//     D[128 factor rows, N batch columns] = W[128, K] . X[N, K]^T
// (N = batch rounded up to 16; from 65 sequences on two CTAs may take half of it each)
// issued as tcgen05.mma (cta_group::1, kind::f16, M = 128) by one thread per CTA, with both operands
// read from shared memory (128-byte swizzled, K-major, filled by TMA) and the fp32 accumulator in
// tensor memory.  The work is still bound by the factor stream from HBM (each factor byte is used
// for N <= 128 multiply-adds), so the kernel is organised around keeping TMA busy:
//   * one CTA = one tile of 128 factor rows x one K segment; the <= 8 segments of a tile are the CTAs
//     of a thread-block cluster: they exchange their partial sums through distributed shared memory
//     (each CTA finishes a slice of the batch columns, adding the segments in segment order), so
//     no partial sum goes through global memory and the result does not depend on timing;
//   * a ring of NS stages {W tile 16 KB, (second W tile), X tile(s)}: three threads issue the TMA copies
//     as slots free up, thread 32 issues the MMAs as slots fill and releases a slot with
//     tcgen05.commit, all eight warps read the accumulator back with tcgen05.ld for the epilogue;
//   * epilogues: store / residual / SwiGLU (two accumulators) / RoPE + q buffer / RoPE + key cache /
//     value cache, with the rounding points of the PyTorch low-rank path (every nn.Linear output
//     rounded to bf16), the same as the interpreter's.
// A decoder layer is 12 launches on the caller's stream (2 RMSNorm, 9 GEMM launches over its 13
// factors with the q / k / v lifts grouped, attention with the split merge inside the kernel); a
// model step is captured once into a CUDA graph.  Attention: batch_attn_kernel (1 or 2 query heads per
// kv head, shuffle-reduced dot products at the HBM rate), gqa_decode_attn_kernel (4 or 8: the heads as
// rows of a tensor-core tile).  The prompt pass (whole prompts as rows, fsvd_prompt_run) has its GEMM and
// attention kernels in fsvd_prompt.cuh.
// Tensor-parallel layer (fsvd_tile_tp_decode_layer): the o lift and the down lift end in the push
// epilogue (TE_PUSH: partial sums stored into every rank's exchange region over peer memory, one flag
// per CTA), exchange_reduce_rows_kernel sums them in rank order with the residual and applies the
// RMSNorm that follows; protocol in fsvd_exchange.h.
//
// Reference functions replaced: kernels/mlp/decode/dual_split_triton_pcat_s.py:39-120 (token-tiled
// SwiGLU MLP), kernels/attn/decode/densekv_reconstruct_triton.py:464-760 (q/k/v lift),
// runtime/attn/decode_registry.py:177-211 (rotary + append + attention), for batches > 8.
//
// Every wait in these kernels is bounded (clock64 budget); a wait that runs out sets the status word,
// the CTA frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <initializer_list>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/flashsvd_b200.h"
#include "fsvd_exchange.h"
#include "fsvd_stage.h"
#include "fsvd_tc.cuh"
#include "fsvd_tile.h"

namespace fsvd_tile {

constexpr int kThreads = 256;        // 8 warps: warp w reads accumulator lanes 32 (w % 4) .. + 31, every other 16 columns
constexpr int kWTileBytes = kTileM * kTileK * 2;   // 16 KB
constexpr int kMaxStages = 8;
constexpr int kMaxSegs = 8;           // K segments of a tile = CTAs of a cluster (portable size)

enum TileEpi : int {
  TE_STORE = 0,      // out[b, p] = rnd(acc)                        (bf16)
  TE_STORE_F32 = 1,  // out[b, p] = rnd(acc) kept in an fp32 container (logits)
  TE_RESID = 2,      // out[b, p] = rnd(resid[b, p] + rnd(acc))
  TE_SWIGLU = 3,     // out[b, p] = rnd(rnd(silu(rnd(accA))) * rnd(accB))      A = gate, B = up
  TE_ROPE_Q = 4,     // rotate the head's (j, j + Dh/2) pair at position seqlens[b], store to out[b, p]
  TE_ROPE_K = 5,     // same rotation, store into the key cache at position seqlens[b]
  TE_VCACHE = 6,     // store rnd(acc) into the value cache at position seqlens[b]
  TE_PUSH = 7,       // tensor-parallel partial sums: rnd(acc) into this rank's slot of every rank's exchange region
};

struct GemmArgs {
  int P, K, B, N;          // factor rows, reduction length, batch rows, batch columns of a tile (a multiple of 16)
  int tiles, segs, kbs;    // row tiles, K segments, k-blocks per segment
  int nh;                  // CTAs that share a row tile's batch columns (N each): 1 or 2
  int nkb;                 // k-blocks in all
  int nstages, two, epi;
  uint32_t tmem_cols;      // power of two >= 32
  int cpo;                 // batch columns finished by each CTA of a tile's cluster: ceil(N / segs) rounded up to 4
  uint32_t recv_off;       // byte offset of the partial sums this CTA receives; 0: they take the ring's place
  void* out;
  const void* resid;
  void* cache;             // TE_ROPE_K / TE_VCACHE: [rows, S_max, Hk, Dh]
  const void* cos_tab;
  const void* sin_tab;
  const int* seqlens;
  int Dh, HkDh, S_max, shared_cache;
  int* status;             // SyncState::status of the workspace
  long long wait_limit;
  unsigned long long* trace;   // debugging: %globaltimer marks, 16 per CTA (null = off)
  fsvd_exch::Geom ex;          // TE_PUSH: the exchange regions of all ranks (fsvd_exchange.h)
  const unsigned* ex_seq;      // TE_PUSH: this rank's exchange sequence number
};

__device__ __forceinline__ void tmark(const GemmArgs& a, int k) {
  if (a.trace && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    a.trace[((size_t)(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 16 + k] = t;
  }
}

// Up to three independent GEMMs in one launch (the q, k and v lifts of a layer): blockIdx.z picks
// the problem, CTAs outside a problem's (tiles, segs) range leave at once.
constexpr int kMaxGroup = 3;
struct GemmGroup {
  CUtensorMap maps[kMaxGroup][4];   // A, A2, X, X2
  GemmArgs args[kMaxGroup];
};

// ------------------------------------------------------------------------------- GEMM kernel
// grid = (tiles x nh, segs, problems).  Dynamic shared memory: [1 KB slack for alignment][NS stages][partial sums].
// What bounds it: the factor stream, then, launch by launch, the chain dependency -> activations ->
// multiply -> exchange -> epilogue.  Per launch after its dependency (7B shape, us, median of the CTAs
// past the epilogue): 128 columns 22 -> 12 (lifts with rotary 27 -> 12, gate / up 36 -> 12), 16 columns
// 4.4 -> 4.2; the step of 4 layers: 128 sequences 8.13 -> 6.50 ms, 32 sequences 5.32 -> 4.97 ms, 8 sequences of
// the 70B shape 2.95 -> 2.88 ms.
__global__ void __launch_bounds__(kThreads, 3) tile_gemm_kernel(const __grid_constant__ GemmGroup grp) {
  const GemmArgs& a = grp.args[blockIdx.z];
  if ((int)blockIdx.x >= a.tiles * a.nh || (int)blockIdx.y >= a.segs) return;
  const CUtensorMap& mapA = grp.maps[blockIdx.z][0];
  const CUtensorMap& mapA2 = grp.maps[blockIdx.z][1];
  const CUtensorMap& mapX = grp.maps[blockIdx.z][2];
  const CUtensorMap& mapX2 = grp.maps[blockIdx.z][3];
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * kMaxStages + 1];
  __shared__ uint32_t tmem_slot;
  __shared__ int giveup_sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = a.nh == 2 ? blockIdx.x >> 1 : blockIdx.x, seg = blockIdx.y;
  const int bcol = a.nh == 2 ? (int)(blockIdx.x & 1) * a.N : 0;   // first batch column
  tmark(a, 0);
  const int N = a.N, NS = a.nstages;
  const uint32_t xbytes = (uint32_t)N * 128u;
  const uint32_t stage_bytes = (uint32_t)kWTileBytes * (a.two ? 2u : 1u) + xbytes * (a.two ? 2u : 1u);
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kMaxStages]), accum = smem_u32(&bars[2 * kMaxStages]);
  volatile int* giveup = &giveup_sh;

  if (tid == 0) {
    giveup_sh = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    mbar_init(accum, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    __syncwarp();
    tc_alloc(smem_u32(&tmem_slot), a.tmem_cols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  tmark(a, 1);
  pdl_launch_dependents();
  if (a.recv_off) cluster_arrive();   // "this CTA runs": its receive buffer may be written from now on

  const int kb0 = seg * a.kbs, kb1 = min(a.nkb, kb0 + a.kbs);
  const int nit = kb1 - kb0;

  if (warp != 1 && warp < 4) {
    if (lane == 0) {
      // ---- producers: TMA copies of the stage operands.  One thread sustains about 24 GB/s of
      // copies (wait, arm, issue per box), so three threads (warps 0, 2, 3) share the stages.  A
      // ring slot always belongs to the same thread (slot % 3): a parity wait cannot tell phase k of
      // a slot's barrier from phase k + 2, and only a slot's single owner, which visits its rounds in
      // order, can never be two phases behind.
      // The factor tiles of the first NS stages do not depend on the kernel before this one and
      // are requested before pdl_wait().
      const int pj = warp == 0 ? 0 : warp - 1;
      constexpr int kProducers = 3;
      const int pre = min(nit, NS);
      for (int it = 0; it < pre; ++it) {
        if (it % kProducers != pj) continue;
        const uint32_t fb = full0 + 8 * it;
        const uint32_t dst = base + (uint32_t)it * stage_bytes;
        const int kcol = (kb0 + it) * kTileK;
        mbar_expect_tx(fb, stage_bytes);
        tma_box_2d(dst, &mapA, kcol, tile * kTileM, fb);
        if (a.two) tma_box_2d(dst + kWTileBytes, &mapA2, kcol, tile * kTileM, fb);
      }
      pdl_wait();
      for (int it = 0; it < nit; ++it) {
        const int s = it % NS, round = it / NS;
        if (s % kProducers != pj) continue;
        if (round > 0 && !wait_bar(empty0 + 8 * s, (uint32_t)(round - 1) & 1u, giveup, a.status, a.wait_limit, DS_COPY_TIMEOUT)) break;
        const uint32_t fb = full0 + 8 * s;
        uint32_t dst = base + (uint32_t)s * stage_bytes;
        const int kcol = (kb0 + it) * kTileK;
        if (it >= pre) {
          mbar_expect_tx(fb, stage_bytes);
          tma_box_2d(dst, &mapA, kcol, tile * kTileM, fb);
          if (a.two) tma_box_2d(dst + kWTileBytes, &mapA2, kcol, tile * kTileM, fb);
        }
        dst += (uint32_t)kWTileBytes * (a.two ? 2u : 1u);
        tma_box_2d(dst, &mapX, kcol, bcol, fb);
        if (a.two) tma_box_2d(dst + xbytes, &mapX2, kcol, bcol, fb);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issue: four 16-deep steps per k-block and accumulator.  The first activation tile
      // cannot arrive before the kernel in front has completed: the wait budget starts there.
      const uint32_t idesc = umma_idesc(N);
      bool ok = true;
      pdl_wait();
      for (int it = 0; it < nit && ok; ++it) {
        const int s = it % NS, round = it / NS;
        ok = wait_bar(full0 + 8 * s, (uint32_t)round & 1u, giveup, a.status, a.wait_limit, DS_COPY_TIMEOUT);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = base + (uint32_t)s * stage_bytes;
        const uint32_t sx = sa + (uint32_t)kWTileBytes * (a.two ? 2u : 1u);
        const uint64_t da = umma_desc(sa), dx = umma_desc(sx);
#pragma unroll
        for (int kk = 0; kk < kTileK / 16; ++kk)
          tc_mma(tmem, da + 2u * kk, dx + 2u * kk, idesc, (it > 0 || kk > 0) ? 1u : 0u);
        if (a.two) {
          const uint64_t da2 = umma_desc(sa + kWTileBytes), dx2 = umma_desc(sx + xbytes);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; ++kk)
            tc_mma(tmem + (uint32_t)N, da2 + 2u * kk, dx2 + 2u * kk, idesc, (it > 0 || kk > 0) ? 1u : 0u);
        }
        tc_commit(empty0 + 8 * s);   // the slot is free when these MMAs have read it
      }
      if (ok) tc_commit(accum);      // the accumulators are complete
    }
    __syncwarp();
  }

  // ---- everybody: wait for the kernel before this one (the epilogue reads what it wrote), then
  // for the accumulators
  pdl_wait();
  tmark(a, 2);
  const unsigned push_seq = a.epi == TE_PUSH ? *reinterpret_cast<const volatile unsigned*>(a.ex_seq) : 0u;

  // ---- this thread's share of the epilogue: row r of the tile, four batch columns at a time, every
  // ng-th group of four of the CTA's slice.  RoPE finishes rows j and j + Dh/2 of a head together, so
  // half as many rows are shared out over twice as many column groups.
  const int cpo = a.cpo;                     // batch columns finished by each CTA of the cluster
  const int half = a.Dh >> 1;
  const bool rope = a.epi == TE_ROPE_Q || a.epi == TE_ROPE_K;
  const int er = rope ? tid & (kTileM / 2 - 1) : tid & (kTileM - 1);
  const int j = rope ? er & (half - 1) : 0;  // (Dh is 64 or 128)
  const int r = rope ? 2 * (er - j) + j : er;
  const int p = tile * kTileM + r;           // factor row
  const int sl0 = 4 * (rope ? tid >> 6 : tid >> 7), sl_step = rope ? 16 : 8;
  const bool work = p < a.P;
  const int B = min(a.B, bcol + a.N);        // end of this CTA's columns (slices are rounded up: the last one may end past it)
  // Operands of four columns that do not depend on the accumulators: residual elements, or the
  // position and the rotary pair.  Those of the first four are requested before the accumulators are
  // complete, those of the next four before the arithmetic of the four at hand.
  auto operands = [&](int sl, uint32_t (&x)[4], int (&pos)[4]) {
    const int b0 = bcol + seg * cpo + sl;
    if (!work || sl >= cpo || b0 >= B) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = min(b0 + i, B - 1);
      if (a.epi == TE_RESID) {
        x[i] = reinterpret_cast<const unsigned short*>(a.resid)[(size_t)b * a.P + p];
      } else {
        pos[i] = a.seqlens[b];
        if (rope) {
          const size_t t = (size_t)min(pos[i], a.S_max - 1) * half + j;
          x[i] = reinterpret_cast<const unsigned short*>(a.cos_tab)[t] |
                 (uint32_t) reinterpret_cast<const unsigned short*>(a.sin_tab)[t] << 16;
        }
      }
    }
  };
  const int epi = a.epi, segs = a.segs, P = a.P;   // (indexed constant loads: once, not per column)
  const bool two = a.two != 0;
  void* const out = a.out;
  const bool has_operands = rope || a.epi == TE_RESID || a.epi == TE_VCACHE;
  uint32_t xn[4] = {0u, 0u, 0u, 0u};
  int posn[4] = {0, 0, 0, 0};
  if (has_operands) operands(sl0, xn, posn);

  bool have = nit > 0 ? wait_bar(accum, 0u, giveup, a.status, a.wait_limit, DS_BARRIER_TIMEOUT) : false;
  have = __all_sync(0xffffffffu, have);
  tc_fence_after();
  tmark(a, 3);

  // ---- the K segments of a tile are the CTAs of one cluster (rank = segment).  CTA j finishes the
  // batch columns [j cpo, (j + 1) cpo) (cpo a multiple of 4): every CTA sends its partial sums of
  // those columns to CTA j's shared memory, [accumulator][segment][group of four columns][row] x 16
  // bytes: the lanes of a warp hold consecutive rows, so a store (and the load below) covers 512
  // consecutive bytes.  (With the columns of a row next to each other instead, a warp's store hit
  // the same banks up to 32 times: 10 us of sending and 15 us of epilogue per launch at 128 columns.)
  // Where the buffer has its own place the CTAs of the cluster only have to be running before the
  // first store; where it reuses the ring every CTA must have its accumulators.  The sums are
  // complete after the second barrier.  Every CTA reaches both, whatever happened before.
  const float4* recv = reinterpret_cast<const float4*>(base_ptr + a.recv_off);
  const uint32_t recv_u32 = base + a.recv_off;
  const int nacc = a.two ? 2 : 1, cq = cpo >> 2;
  if (!a.recv_off) cluster_arrive();
  cluster_wait();
  tmark(a, 4);
  if (have) {
    const int arow = (warp & 3) * 32 + lane;   // accumulator lane = row of the tile
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    for (int acc = 0; acc < nacc; ++acc) {
      for (int c0 = (warp >> 2) * 16; c0 < N; c0 += 32) {
        float v[16];
        tc_ld16(trow + (uint32_t)(acc * N + c0), v);
        int owner = c0 / cpo, q = (c0 - owner * cpo) >> 2;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const uint32_t dst = recv_u32 + (uint32_t)((((acc * a.segs + seg) * cq + q) * kTileM + arow) * 16);
          if (owner < a.segs) st_cluster_v4(dst, (uint32_t)owner, v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
          if (++q == cq) {
            q = 0;
            ++owner;
          }
        }
      }
    }
  }
  tmark(a, 5);
  cluster_sync();
  tmark(a, 6);

  if (!*giveup && have && work) {
    for (int sl = sl0; sl < cpo; sl += sl_step) {
      const int b0 = bcol + seg * cpo + sl;
      if (b0 >= B) break;
      uint32_t x[4];
      int pos[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = xn[i], pos[i] = posn[i];
      if (has_operands) operands(sl + sl_step, xn, posn);
      // sums over the segments, in segment order, of four columns (and of the second accumulator,
      // or of the RoPE partner row)
      float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
      const float4* src = recv + (sl >> 2) * kTileM + r;
      for (int sg = 0; sg < segs; ++sg) {
        const float4 t = src[sg * cq * kTileM];
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
      if (two || rope) {
        src += two ? segs * cq * kTileM : half;
        for (int sg = 0; sg < segs; ++sg) {
          const float4 t = src[sg * cq * kTileM];
          u[0] += t.x; u[1] += t.y; u[2] += t.z; u[3] += t.w;
        }
      }
      // One compact code path per epilogue kind (this code often runs once per CTA, from a cold
      // instruction cache: the fewer lines it spans, the sooner it is through).
      const int nb = min(4, B - b0);
      const size_t o0 = (size_t)b0 * P + p;
      if (epi == TE_STORE) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < nb) stbf(out, o0 + (size_t)i * P, v[i]);
      } else if (epi == TE_RESID) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < nb) stbf(out, o0 + (size_t)i * P, __uint_as_float(x[i] << 16) + rnd(v[i]));
      } else if (epi == TE_PUSH) {
        // the same rounded partial sums into slot [parity][this rank] of every rank's region
        // (peer stores over NVLink; the rank's own region among them)
        for (int q = 0; q < a.ex.world; ++q) {
          unsigned char* dst = fsvd_exch::slot_ptr(a.ex, q, push_seq & 1u, a.ex.rank);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < nb) stbf(dst, o0 + (size_t)i * P, v[i]);
        }
      } else if (epi == TE_SWIGLU) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float g = rnd(v[i]), up = rnd(u[i]);
          const float sg = rnd(g / (1.0f + expf(-g)));
          if (i < nb) stbf(out, o0 + (size_t)i * P, sg * up);
        }
      } else if (epi == TE_STORE_F32) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < nb) reinterpret_cast<float*>(out)[o0 + (size_t)i * P] = rnd(v[i]);
      } else {
        // value cache / rotary epilogues
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b = b0 + i;
          if (i >= nb) continue;
          if (pos[i] >= a.S_max && epi != TE_ROPE_Q) {
            atomicCAS(a.status, (int)DS_OK, (int)DS_CACHE_FULL);
            continue;
          }
          const size_t oc = ((size_t)(a.shared_cache ? 0 : b) * a.S_max + pos[i]) * (size_t)a.HkDh + p;
          if (epi == TE_VCACHE) {
            stbf(a.cache, oc, v[i]);
          } else {
            const float cs = __uint_as_float(x[i] << 16), sn = __uint_as_float(x[i] & 0xffff0000u);
            const float x1 = rnd(v[i]), x2 = rnd(u[i]);
            const float o1 = rnd(rnd(x1 * cs) - rnd(x2 * sn));
            const float o2 = rnd(rnd(x2 * cs) + rnd(x1 * sn));
            if (epi == TE_ROPE_Q) {
              stbf(out, o0 + (size_t)i * P, o1);
              stbf(out, o0 + (size_t)i * P + half, o2);
            } else {
              stbf(a.cache, oc, o1);
              stbf(a.cache, oc + half, o2);
            }
          }
        }
      }
    }
  }

  // ---- release the tensor memory
  tmark(a, 7);
  tc_fence_before();
  __syncthreads();
  // TE_PUSH: every store of this CTA is ordered before the flags that thread q raises in rank q's
  // region: the CTA barrier above, then a store with release semantics at system scope (it orders the
  // writes the thread has observed through the barrier as well as its own)
  if (a.epi == TE_PUSH && tid < a.ex.world) {
    fsvd_exch::st_release_sys(fsvd_exch::flag_ptr(a.ex, tid, push_seq & 1u, a.ex.rank, tile * a.segs + seg), push_seq);
  }
  __syncwarp();
  if (*giveup)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);   // copies in flight towards this CTA land first
  if (warp == 0) tc_dealloc(tmem, a.tmem_cols);
  tmark(a, 8);
}

// ------------------------------------------------------------------------------- RMSNorm rows
// out[b, :] = rnd(w * rnd(x[r, :] * rsqrt(mean(x[r, :]^2) + eps))), r = b * row_mul + row_off, one CTA per
// row.  A thread's 16-byte pieces stay in registers between the two passes (rows up to 8192 wide).
// WIDE: x starts on a 16-byte boundary; a caller's hidden state that does not is read 2 bytes at a time
// (w and out always do: layer pointers are checked, out is the library's own).
template <bool WIDE>
__device__ __forceinline__ uint4 load_8bf(const __nv_bfloat16* p) {
  if (WIDE) return *reinterpret_cast<const uint4*>(p);
  const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
  return make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16, h[6] | (uint32_t)h[7] << 16);
}
template <bool WIDE>
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                           const __nv_bfloat16* __restrict__ w,
                                                           __nv_bfloat16* __restrict__ out, int d, float eps,
                                                           int row_mul, int row_off) {
  constexpr int U = 4;
  __shared__ float red[8];
  const int b = blockIdx.x, tid = threadIdx.x, n8 = d >> 3;
  pdl_launch_dependents();
  pdl_wait();
  const __nv_bfloat16* xr = x + (size_t)(b * row_mul + row_off) * d;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* orow = reinterpret_cast<uint4*>(out + (size_t)b * d);
  const bool fits = n8 <= 256 * U;
  uint4 v[U], wv[U];
  float ss = 0.0f;
  for (int i0 = tid; i0 < n8; i0 += 256 * U) {
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i0 + 256 * k < n8) {
        v[k] = load_8bf<WIDE>(xr + 8 * (i0 + 256 * k));
        wv[k] = wr[i0 + 256 * k];
      }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (i0 + 256 * k < n8) {
        const uint32_t u[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = __uint_as_float(u[j] << 16), hi = __uint_as_float(u[j] & 0xffff0000u);
          ss += lo * lo;
          ss += hi * hi;
        }
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)d + eps);
  auto finish = [&](int i, const uint4& xq, const uint4& wq) {
    const uint32_t xu[4] = {xq.x, xq.y, xq.z, xq.w}, wu[4] = {wq.x, wq.y, wq.z, wq.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o[j] = pack_bf16(__uint_as_float(wu[j] << 16) * rnd(__uint_as_float(xu[j] << 16) * inv),
                       __uint_as_float(wu[j] & 0xffff0000u) * rnd(__uint_as_float(xu[j] & 0xffff0000u) * inv));
    orow[i] = make_uint4(o[0], o[1], o[2], o[3]);
  };
  if (fits) {
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (tid + 256 * k < n8) finish(tid + 256 * k, v[k], wv[k]);
  } else {
    for (int i = tid; i < n8; i += 256) finish(i, load_8bf<WIDE>(xr + 8 * i), wr[i]);
  }
}

// ------------------------------------------------------------------------------- exchange + RMSNorm rows
// Second half of a tensor-parallel exchange (protocol: fsvd_exchange.h).  Row b is shared by the
// gridDim.y CTAs of a cluster, each with a slice of its columns:
//     wait until every rank's GEMM has posted exchange number seq in this rank's region,
//     h[b, :]  = rnd(resid[b, :] + rnd(sum over ranks, in rank order, of slot[rank][b, :]))
//     xn[b, :] = rnd(w * rnd(h[b, :] * rsqrt(mean(h[b, :]^2) + eps)))             (when xn != null)
// The slots are read past L1 (another GPU wrote them); the CTAs of a row exchange their sums of
// squares through distributed shared memory and add them in CTA order.  The last CTA of the grid to
// finish advances the rank's sequence number.  A wait that runs out records DS_PEER_TIMEOUT and the
// rank it waited for; the row is then computed from whatever the slots hold.
struct ReduceArgs {
  fsvd_exch::Geom ex;
  fsvd_exch::Ctrl* ctrl;
  int nflags;                    // CTAs of the pushing GEMM
  const __nv_bfloat16* resid;
  __nv_bfloat16* out;
  const __nv_bfloat16* norm_w;
  __nv_bfloat16* xn;
  int d;
  float eps;
  int* status;                   // SyncState::status, status_detail of the workspace
  long long wait_limit;
  unsigned long long* trace;     // optional: record [seq % trace_cap] = %globaltimer at {dependency met, all flags seen, done}
  unsigned trace_cap;            // (written by CTA (0, 0))
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, uint32_t rank, float v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

__global__ void __launch_bounds__(256) exchange_reduce_rows_kernel(const __grid_constant__ ReduceArgs a) {
  __shared__ float red[8];
  __shared__ float css[kMaxSegs];            // sums of squares of the row's column slices
  __shared__ int giveup_sh;
  const int b = blockIdx.x, tid = threadIdx.x;
  const int C = gridDim.y, c = blockIdx.y;    // C > 1: launched as clusters of C CTAs along y
  if (tid == 0) giveup_sh = 0;
  pdl_launch_dependents();
  pdl_wait();
  __syncthreads();
  volatile int* giveup = &giveup_sh;
  const unsigned seq = *reinterpret_cast<const volatile unsigned*>(&a.ctrl->seq);
  const unsigned par = seq & 1u;
  unsigned long long* rec = (a.trace && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) ? a.trace + (size_t)(seq % a.trace_cap) * 3 : nullptr;
  if (rec) rec[0] = global_ns();
  {
    const int total = a.ex.world * a.nflags;
    const long long c0 = clock64();
    for (int i = tid; i < total && !*giveup; i += 256) {
      const int src = i / a.nflags;
      const unsigned* f = fsvd_exch::flag_ptr(a.ex, a.ex.rank, par, src, i - src * a.nflags);
      unsigned spins = 0;
      while ((int)(fsvd_exch::ld_acquire_sys(f) - seq) < 0) {
        if ((++spins & 15u) == 0) {
          if (*giveup) break;
          if (clock64() - c0 > a.wait_limit) {
            if (atomicCAS(a.status, (int)DS_OK, (int)fsvd_exch::DS_PEER_TIMEOUT) == (int)DS_OK) a.status[1] = src;
            *giveup = 1;
            break;
          }
        }
      }
    }
  }
  __syncthreads();
  if (rec) rec[1] = global_ns();
  if (C > 1 && a.xn) cluster_sync();            // every CTA of the row runs before any writes into its shared memory

  const int cols = a.d / C, col0 = c * cols;    // the host makes cols a multiple of 8
  const size_t row = (size_t)b * a.d + col0;
  const unsigned char* slot0 = fsvd_exch::slot_ptr(a.ex, a.ex.rank, par, 0);
  float ss = 0.0f;
  for (int i = tid * 8; i < cols; i += 256 * 8) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
    for (int q = 0; q < a.ex.world; ++q) {
      const uint4 t = __ldcg(reinterpret_cast<const uint4*>(slot0 + (size_t)q * a.ex.slot_bytes + (row + i) * 2));
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&t);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f2 = __bfloat1622float2(h2[j]);
        acc[2 * j] += f2.x;
        acc[2 * j + 1] += f2.y;
      }
    }
    const uint4 rr = *reinterpret_cast<const uint4*>(a.resid + row + i);
    const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
    uint4 o;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f2 = __bfloat1622float2(r2[j]);
      const float h0 = rnd(f2.x + rnd(acc[2 * j])), h1 = rnd(f2.y + rnd(acc[2 * j + 1]));
      ss += h0 * h0 + h1 * h1;
      o2[j] = __floats2bfloat162_rn(h0, h1);
    }
    *reinterpret_cast<uint4*>(a.out + row + i) = o;
  }
  if (a.xn) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += red[i];
    if (C > 1) {
      if (tid < C) st_cluster_f32(smem_u32(&css[c]), (uint32_t)tid, tot);
      cluster_sync();
      tot = 0.0f;
      for (int j = 0; j < C; ++j) tot += css[j];
    }
    const float inv = rsqrtf(tot / (float)a.d + a.eps);
    for (int i = tid * 8; i < cols; i += 256 * 8) {
      // the thread reads back the eight values it stored above
      const uint4 hh = *reinterpret_cast<const uint4*>(a.out + row + i);
      const uint4 ww = *reinterpret_cast<const uint4*>(a.norm_w + col0 + i);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&hh);
      const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&ww);
      uint4 o;
      __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 hf = __bfloat1622float2(h2[j]), wf = __bfloat1622float2(w2[j]);
        o2[j] = __floats2bfloat162_rn(wf.x * rnd(hf.x * inv), wf.y * rnd(hf.y * inv));
      }
      *reinterpret_cast<uint4*>(a.xn + row + i) = o;
    }
  }
  // every CTA has read the sequence number before it arrives here: the last one moves it on
  __syncthreads();
  if (rec) rec[2] = global_ns();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&a.ctrl->done, 1u) == gridDim.x * gridDim.y - 1) {
      a.ctrl->done = 0u;
      *reinterpret_cast<volatile unsigned*>(&a.ctrl->seq) = seq + 1u;
    }
  }
}

// ------------------------------------------------------------------------------- attention
// Single-query attention of B sequences over their dense caches.  One CTA = (sequence, kv head,
// key split); its G = H / Hk query heads share the key and value rows it reads.  Each of the four
// warps walks its own groups of 8 keys with its own running softmax: a key (or value) row is one
// coalesced warp-wide load (lane t holds dims DPL t .. DPL t + DPL - 1), the 8 key rows and the 8
// value rows of a group are requested together, the 8 x G dot products are reduced with shuffles.
// The warps meet in shared memory; splits of a head are merged in split order by the CTA that
// arrives last.
constexpr int kAttnThreads = 128;
constexpr int kAttnWarps = 4;
constexpr int kKeyGroup = 8;
constexpr int kGqKeys = 32;      // keys per warp block of gqa_decode_attn_kernel
constexpr int kMaxSplit = 64;    // key splits of a sequence at most
constexpr int kPartPad = 4;      // a record of a split and head: DH sums, running maximum, running sum, padded to 16 bytes
// Fewest keys of a split: two groups (batch_attn_kernel), one block (gqa_decode_attn_kernel) for each warp.
constexpr int kBatchSplitKeys = 2 * kAttnWarps * kKeyGroup, kGqSplitKeys = kAttnWarps * kGqKeys;

struct AttnArgs {
  const __nv_bfloat16* q;        // [B, H, Dh], rotated
  const __nv_bfloat16* kcache;   // [rows, S_max, Hk, Dh]
  const __nv_bfloat16* vcache;
  const int* seqlens;
  __nv_bfloat16* out;            // [B, H, Dh]
  float* part;                   // [B, Hk, nsplit, G, Dh + kPartPad] (acc, m, l)
  int* counters;                 // [B, Hk]
  int B, H, Hk, Dh, S_max, nsplit, seqlen_add, shared_cache;
  float scale;
};

// FULL: the op on its own (fsvd_flash_decode) keeps softmax weights in 32 bits: expf, and on the tensor
// cores each weight as three bf16 numbers (split_bf16: all 24 bits; with two, 16 bits, 8
// sequences x 64 heads on 8 kv heads x 4096 keys took 43.2 us instead of 46.4).
// Inside a model step the weights are bf16 where they meet the tensor cores.
template <bool FULL>
__device__ __forceinline__ float weight(float x) { return FULL ? expf(x) : __expf(x); }

// The splits that a sequence of n positions is cut into: the launch has as many as a full cache takes, a short sequence
// in it uses fewer, and the CTAs of the others leave at once.  The op alone, caches of 4096 positions, us with all
// splits and with these: 1 sequence x 32 heads on 16 kv heads, 512 positions 18.4 and 11.1; 8 sequences x 64 heads
// on 8, 128 positions 15.9 and 11.1; a model step of 8 sequences, 4 layers, 8 positions 428 and 404.
__device__ __forceinline__ int splits_in_use(int n, int nsplit, int fewest) {
  return max(1, min(nsplit, (n + fewest - 1) / fewest));
}

// Merge of the splits of G heads, in split order, by the CTA that arrived last: the weight of every (split, head) once, in
// shared memory (sh: 2 nsplit G + 16 floats), then each thread sums four output dims over the splits with
// independent 16-byte loads.  out: [G, DH]
template <int DH, bool FULL>
__device__ __forceinline__ void merge_splits(const float* parts, int nsplit, int G, __nv_bfloat16* out, float* sh) {
  constexpr int rec = DH + kPartPad, U = 8;
  const int tid = threadIdx.x;
  float* wgt_s = sh;                       // [nsplit][G] maxima, then weights
  float* l_s = sh + nsplit * G;            // [nsplit][G] running sums of the splits
  float* den_s = l_s + nsplit * G;         // [G] sums, [8 + G] maxima
  for (int i = tid; i < nsplit * G; i += kAttnThreads) {
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(parts + (size_t)i * rec + DH));
    wgt_s[i] = ml.x;
    l_s[i] = ml.y;
  }
  __syncthreads();
  if (tid < G) {
    float mm = -INFINITY;
    for (int sp = 0; sp < nsplit; ++sp) mm = fmaxf(mm, wgt_s[sp * G + tid]);
    den_s[8 + tid] = mm;
  }
  __syncthreads();
  for (int i = tid; i < nsplit * G; i += kAttnThreads) {
    const float ms = wgt_s[i];
    wgt_s[i] = ms == -INFINITY ? 0.0f : weight<FULL>(ms - den_s[8 + i % G]);
  }
  __syncthreads();
  if (tid < G) {
    float den = 0.0f;
    for (int sp = 0; sp < nsplit; ++sp) den += wgt_s[sp * G + tid] * l_s[sp * G + tid];
    den_s[tid] = den;
  }
  __syncthreads();
  for (int i = tid; i < G * (DH / 4); i += kAttnThreads) {
    const int g = i / (DH / 4), d4 = (i - g * (DH / 4)) * 4;
    float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s0 = 0; s0 < nsplit; s0 += U) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)   // (past the last split: the last one again, so that U loads are always in flight)
        v[u] = __ldcg(reinterpret_cast<const float4*>(parts + ((size_t)min(s0 + u, nsplit - 1) * G + g) * rec + d4));
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (s0 + u < nsplit) {
          const float wg = wgt_s[(s0 + u) * G + g];
          num.x += wg * v[u].x; num.y += wg * v[u].y; num.z += wg * v[u].z; num.w += wg * v[u].w;
        }
    }
    const float den = den_s[g];
    uint2 o2 = make_uint2(0u, 0u);
    if (den > 0.0f) o2 = make_uint2(pack_bf16(num.x / den, num.y / den), pack_bf16(num.z / den, num.w / den));
    *reinterpret_cast<uint2*>(out + (size_t)g * DH + d4) = o2;
  }
}

template <int DPL>
__device__ __forceinline__ void ld_row(const __nv_bfloat16* row, int lane, float (&f)[DPL]);
template <>
__device__ __forceinline__ void ld_row<4>(const __nv_bfloat16* row, int lane, float (&f)[4]) {
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(row) + lane);
  f[0] = __uint_as_float(w.x << 16); f[1] = __uint_as_float(w.x & 0xffff0000u);
  f[2] = __uint_as_float(w.y << 16); f[3] = __uint_as_float(w.y & 0xffff0000u);
}
template <>
__device__ __forceinline__ void ld_row<2>(const __nv_bfloat16* row, int lane, float (&f)[2]) {
  const unsigned w = __ldg(reinterpret_cast<const unsigned*>(row) + lane);
  f[0] = __uint_as_float(w << 16); f[1] = __uint_as_float(w & 0xffff0000u);
}

// One query vector over the keys [k0, k0 + block) below `end`, k0 = begin, begin + stride, ..., by one warp in plain
// fp32; lane t gets dims DPL t .. DPL t + DPL - 1 of the sum over the values, the running maximum and the running sum.
// The tensor cores multiply every value row of a tile by every weight of it, the zeros of masked positions and of a
// weight's lower parts too, and 0 times an infinity is no number: the kernels take a row that came out as one
// again through here, where a position that a query does not see takes no part.  (Finite rows never do.)
template <int DH>
__device__ __noinline__ void attn_one_row(const __nv_bfloat16* q, const __nv_bfloat16* kbase, const __nv_bfloat16* vbase, size_t rowstride,
                                          int begin, int end, int block, int stride, float scale, float* acc, float* m, float* l) {
  constexpr int DPL = DH / 32;
  const int lane = threadIdx.x & 31;
  float qf[DPL], o[DPL], mm = -INFINITY, ll = 0.0f;
  ld_row<DPL>(q, lane, qf);
#pragma unroll
  for (int e = 0; e < DPL; ++e) o[e] = 0.0f;
  for (int k0 = begin; k0 < end; k0 += stride)
    for (int k = k0; k < min(k0 + block, end); ++k) {
      float kf[DPL], vf[DPL], s = 0.0f;
      ld_row<DPL>(kbase + (size_t)k * rowstride, lane, kf);
      ld_row<DPL>(vbase + (size_t)k * rowstride, lane, vf);
#pragma unroll
      for (int e = 0; e < DPL; ++e) s += qf[e] * kf[e];
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      s *= scale;
      const float mn = fmaxf(mm, s), corr = expf(mm - mn), p = expf(s - mn);
      mm = mn;
      ll = ll * corr + p;
#pragma unroll
      for (int e = 0; e < DPL; ++e) o[e] = o[e] * corr + p * vf[e];
    }
#pragma unroll
  for (int e = 0; e < DPL; ++e) acc[e] = o[e];
  *m = mm;
  *l = ll;
}

template <int DH, int G, bool FULL>
__global__ void __launch_bounds__(kAttnThreads) batch_attn_kernel(const AttnArgs a) {
  constexpr int DPL = DH / 32;
  __shared__ float wm[kAttnWarps][G], wl[kAttnWarps][G];
  __shared__ float wacc[kAttnWarps][G][DH];
  __shared__ int last_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch_dependents();
  pdl_wait();
  int idx = blockIdx.x;
  const int split = idx % a.nsplit;
  idx /= a.nsplit;
  const int hk = idx % a.Hk, b = idx / a.Hk;
  const int n = min(a.seqlens[b] + a.seqlen_add, a.S_max);
  const int nsplit = splits_in_use(n, a.nsplit, kBatchSplitKeys);
  if (split >= nsplit) return;
  const int per = (n + nsplit - 1) / nsplit;
  const int j0 = min(n, split * per), j1 = min(n, j0 + per);
  const size_t rowstride = (size_t)a.Hk * DH;
  const size_t cbase = ((size_t)b * a.S_max) * rowstride + (size_t)hk * DH;
  const __nv_bfloat16* kbase = a.kcache + cbase;
  const __nv_bfloat16* vbase = a.vcache + cbase;

  float q[G][DPL], acc[G][DPL], m[G], l[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    ld_row<DPL>(a.q + ((size_t)b * a.H + hk * G + g) * DH, lane, q[g]);
#pragma unroll
    for (int e = 0; e < DPL; ++e) {
      q[g][e] *= a.scale;
      acc[g][e] = 0.0f;
    }
    m[g] = -INFINITY;
    l[g] = 0.0f;
  }

  for (int c0 = j0 + warp * kKeyGroup; c0 < j1; c0 += kAttnWarps * kKeyGroup) {
    const int cn = min(kKeyGroup, j1 - c0);
    float kf[kKeyGroup][DPL], vf[kKeyGroup][DPL];
#pragma unroll
    for (int i = 0; i < kKeyGroup; ++i) {
      const int row = c0 + (i < cn ? i : cn - 1);   // past the end: the last row again, masked below
      ld_row<DPL>(kbase + (size_t)row * rowstride, lane, kf[i]);
      ld_row<DPL>(vbase + (size_t)row * rowstride, lane, vf[i]);
    }
    if (cn < kKeyGroup) {   // (the loads above stay unconditional: with a branch each the kernel took twice the time)
#pragma unroll
      for (int i = 0; i < kKeyGroup; ++i)
#pragma unroll
        for (int e = 0; e < DPL; ++e) vf[i][e] = i < cn ? vf[i][e] : 0.0f;   // its weight is 0, and 0 times an infinity is no number
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float s[kKeyGroup];
#pragma unroll
      for (int i = 0; i < kKeyGroup; ++i) {
        float d = 0.0f;
#pragma unroll
        for (int e = 0; e < DPL; ++e) d += kf[i][e] * q[g][e];
        s[i] = d;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; i < kKeyGroup; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
      }
      float cm = -INFINITY;
#pragma unroll
      for (int i = 0; i < kKeyGroup; ++i) {
        if (i >= cn) s[i] = -INFINITY;                          // past the split
        cm = fmaxf(cm, s[i]);
      }
      const float mn = fmaxf(m[g], cm);
      const float corr = weight<FULL>(m[g] - mn);                 // 0 when m is still -inf
      m[g] = mn;
      float ps = 0.0f;
#pragma unroll
      for (int e = 0; e < DPL; ++e) acc[g][e] *= corr;
#pragma unroll
      for (int i = 0; i < kKeyGroup; ++i) {
        const float pr = weight<FULL>(s[i] - mn);               // 0 for the masked rows
        ps += pr;
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[g][e] += pr * vf[i][e];
      }
      l[g] = l[g] * corr + ps;
    }
  }
  // ---- the warps meet
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) {
      wm[warp][g] = m[g];
      wl[warp][g] = l[g];
    }
#pragma unroll
    for (int e = 0; e < DPL; ++e) wacc[warp][g][lane * DPL + e] = acc[g][e];
  }
  __syncthreads();
  constexpr int rec = DH + kPartPad;
  float* const parts = a.part + (((size_t)b * a.Hk + hk) * a.nsplit) * G * rec;
  float* mine = parts + (size_t)split * G * rec;
  for (int i = tid; i < G * DH; i += kAttnThreads) {
    const int g = i / DH, dd = i - g * DH;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, wm[w][g]);
    float num = 0.0f, den = 0.0f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float wgt = wm[w][g] == -INFINITY ? 0.0f : weight<FULL>(wm[w][g] - mm);
      num += wgt * wacc[w][g][dd];
      den += wgt * wl[w][g];
    }
    if (nsplit == 1) {
      a.out[((size_t)b * a.H + hk * G + g) * DH + dd] = __float2bfloat16_rn(den > 0.0f ? num / den : 0.0f);
    } else {
      mine[(size_t)g * rec + dd] = num;
      if (dd == 0) {
        mine[(size_t)g * rec + DH] = mm;
        mine[(size_t)g * rec + DH + 1] = den;
      }
    }
  }
  if (nsplit == 1) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int old = atomicAdd(&a.counters[b * a.Hk + hk], 1);
    last_sh = old == nsplit - 1;
    if (old == nsplit - 1) a.counters[b * a.Hk + hk] = 0;
  }
  __syncthreads();
  if (!last_sh) return;
  __threadfence();
  static_assert(kAttnWarps * G * DH >= 2 * kMaxSplit * G + 16);
  merge_splits<DH, FULL>(parts, nsplit, G, a.out + ((size_t)b * a.H + hk * G) * DH, &wacc[0][0][0]);
}

// ------------------------------------------------------------------------------- grouped-query decode attention
// Single-query attention for H / Hk = 4 or 8 query heads per kv head on the tensor cores: the G
// heads that share a kv head are the rows of one m16n8k16 tile (rows G .. 15 are zero), so a key /
// value row is read once per sequence and multiplied for all its heads at once, instead of one
// shuffle-reduced dot product per head and key (which ran at 0.9 TB/s for 8 heads per kv head).
// One CTA = (sequence, kv head, key split) as in batch_attn_kernel; each of its 4 warps walks its own blocks of 32 keys: cp.async of the 32 key
// rows and 32 value rows into the warp's own shared-memory stage, S = Q K^T, running softmax,
// O += P V with ldmatrix.trans value fragments (the fragment code of prompt_attn_kernel).  The warps
// merge in shared memory, the splits of a head in split order by the CTA that arrives last.

template <int DH, bool FULL>
__global__ void __launch_bounds__(kAttnThreads, 3) gqa_decode_attn_kernel(const AttnArgs a) {
  constexpr int STRIDE = DH * 2 + 16;
  constexpr int KS = DH / 16, NT = kGqKeys / 8, DT = DH / 8;
  constexpr int PIECES = DH / 8;                       // 16-byte pieces of a row
  extern __shared__ __align__(16) unsigned char gq_smem[];
  __shared__ int last_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  pdl_launch_dependents();
  pdl_wait();
  const int G = a.H / a.Hk;
  int idx = blockIdx.x;
  const int split = idx % a.nsplit;
  idx /= a.nsplit;
  const int hk = idx % a.Hk, b = idx / a.Hk;
  const int n = min(a.seqlens[b] + a.seqlen_add, a.S_max);
  const int nsplit = splits_in_use(n, a.nsplit, kGqSplitKeys);
  if (split >= nsplit) return;
  const int per = ((n + nsplit - 1) / nsplit + kGqKeys - 1) / kGqKeys * kGqKeys;   // whole blocks per split
  const int j0 = min(n, split * per), j1 = min(n, j0 + per);
  const size_t rowstride = (size_t)a.Hk * DH;
  const size_t cbase = ((size_t)b * a.S_max) * rowstride + (size_t)hk * DH;
  const __nv_bfloat16* kbase = a.kcache + cbase;
  const __nv_bfloat16* vbase = a.vcache + cbase;
  unsigned char* ks_s = gq_smem + (size_t)warp * (2 * kGqKeys * STRIDE);
  unsigned char* vs_s = ks_s + kGqKeys * STRIDE;

  // Q fragments: row g of the tile = head hk G + g (zero for g >= G), rows 8 .. 15 zero
  uint32_t qa[KS][2];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    qa[ks][0] = qa[ks][1] = 0u;
    if (g < G) {
      const __nv_bfloat16* qp = a.q + ((size_t)b * a.H + hk * G + g) * DH + ks * 16 + 2 * t;
      qa[ks][0] = *reinterpret_cast<const uint32_t*>(qp);
      qa[ks][1] = *reinterpret_cast<const uint32_t*>(qp + 8);
    }
  }
  float o[DT][2];
#pragma unroll
  for (int d = 0; d < DT; ++d) o[d][0] = o[d][1] = 0.0f;
  float mrow = -INFINITY, lrow = 0.0f;

  for (int k0 = j0 + warp * kGqKeys; k0 < j1; k0 += kAttnWarps * kGqKeys) {
    // ---- stage this warp's 32 key rows and 32 value rows (rows past the split repeat its last row;
    // their scores are masked)
    __syncwarp();
    for (int i = lane; i < kGqKeys * PIECES; i += 32) {
      const int r = i / PIECES, c = i - r * PIECES;
      const size_t src = (size_t)min(k0 + r, j1 - 1) * rowstride + (size_t)c * 8;
      const uint32_t dk = smem_u32(ks_s + r * STRIDE + c * 16), dv = smem_u32(vs_s + r * STRIDE + c * 16);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dk), "l"(kbase + src) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dv), "l"(vbase + src) : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // ---- S = Q K^T: 16 (G used) query heads x 32 keys
    float sc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.0f;
      const unsigned char* kr = ks_s + (nt * 8 + g) * STRIDE + 4 * t;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(kr + ks * 32);
        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(kr + ks * 32 + 16);
        mma_bf16_16816(sc[nt], qa[ks][0], 0u, qa[ks][1], 0u, b0, b1);
      }
    }
    // ---- scale, mask, running softmax of row g (its 32 scores sit in the 4 lanes of the group)
    float mx = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int kj = k0 + nt * 8 + 2 * t + e;
        const float v = kj < j1 ? sc[nt][e] * a.scale : -INFINITY;
        sc[nt][e] = v;
        mx = fmaxf(mx, v);
      }
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(mrow, mx);           // finite: key k0 is inside the split
    const float corr = weight<FULL>(mrow - mn);
    mrow = mn;
    float ps = 0.0f;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float pr = weight<FULL>(sc[nt][e] - mn);
        sc[nt][e] = pr;
        ps += pr;
      }
    }
    ps += __shfl_xor_sync(0xffffffffu, ps, 1);
    ps += __shfl_xor_sync(0xffffffffu, ps, 2);
    lrow = lrow * corr + ps;
#pragma unroll
    for (int d = 0; d < DT; ++d) {
      o[d][0] *= corr;
      o[d][1] *= corr;
    }
    // ---- O += P V, 16 keys per step (rows 8 .. 15 of P are zero)
#pragma unroll
    for (int kk = 0; kk < kGqKeys / 16; ++kk) {
      constexpr int W = FULL ? 3 : 1;           // bf16 numbers of a weight
      uint32_t p[3][2];
      if (FULL) {
        split_bf16(sc[2 * kk][0], sc[2 * kk][1], p[0][0], p[1][0], p[2][0]);
        split_bf16(sc[2 * kk + 1][0], sc[2 * kk + 1][1], p[0][1], p[1][1], p[2][1]);
      } else {
        p[0][0] = pack_bf16(sc[2 * kk][0], sc[2 * kk][1]);
        p[0][1] = pack_bf16(sc[2 * kk + 1][0], sc[2 * kk + 1][1]);
      }
      const int lr = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
      const unsigned char* vr = vs_s + lr * STRIDE + ((lane >> 4) & 1) * 16;
#pragma unroll
      for (int j = 0; j < DT / 2; ++j) {
        uint32_t b0, b1, b2, b3;
        const uint32_t addr = (uint32_t)__cvta_generic_to_shared(vr + j * 32);
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(addr));
        float c0[4] = {o[2 * j][0], o[2 * j][1], 0.0f, 0.0f}, c1[4] = {o[2 * j + 1][0], o[2 * j + 1][1], 0.0f, 0.0f};
#pragma unroll
        for (int w = W - 1; w >= 0; --w) {
          mma_bf16_16816(c0, p[w][0], 0u, p[w][1], 0u, b0, b1);
          mma_bf16_16816(c1, p[w][0], 0u, p[w][1], 0u, b2, b3);
        }
        o[2 * j][0] = c0[0]; o[2 * j][1] = c0[1];
        o[2 * j + 1][0] = c1[0]; o[2 * j + 1][1] = c1[1];
      }
    }
  }

  // ---- the four warps meet in shared memory (the stages are free): [warp][head] records
  constexpr int rec = DH + kPartPad;
  __syncthreads();
  float* wpart = reinterpret_cast<float*>(gq_smem);
  if (g < G) {
    float* mine = wpart + ((size_t)warp * G + g) * rec;
#pragma unroll
    for (int d = 0; d < DT; ++d) {
      mine[d * 8 + 2 * t] = o[d][0];
      mine[d * 8 + 2 * t + 1] = o[d][1];
    }
    if (t == 0) {
      mine[DH] = mrow;
      mine[DH + 1] = lrow;
    }
  }
  if (FULL) {
    bool none = false;   // "no number" among this thread's sums
#pragma unroll
    for (int d = 0; d < DT; ++d) none |= o[d][0] != o[d][0] || o[d][1] != o[d][1];
    unsigned again = __ballot_sync(0xffffffffu, g < G && none);
    for (int gg = 0; again; ++gg, again >>= 4)
      if (again & 15u) {
        float acc[DH / 32], mm, ll;
        attn_one_row<DH>(a.q + ((size_t)b * a.H + hk * G + gg) * DH, kbase, vbase, rowstride, j0 + warp * kGqKeys, j1, kGqKeys,
                         kAttnWarps * kGqKeys, a.scale, acc, &mm, &ll);
        float* mine = wpart + ((size_t)warp * G + gg) * rec;
#pragma unroll
        for (int e = 0; e < DH / 32; ++e) mine[lane * (DH / 32) + e] = acc[e];
        if (lane == 0) {
          mine[DH] = mm;
          mine[DH + 1] = ll;
        }
      }
  }
  __syncthreads();
  float* const parts = a.part + (((size_t)b * a.Hk + hk) * a.nsplit) * G * rec;
  float* gpart = parts + (size_t)split * G * rec;
  for (int i = tid; i < G * DH; i += kAttnThreads) {
    const int gg = i / DH, dd = i - gg * DH;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, wpart[((size_t)w * G + gg) * rec + DH]);
    float num = 0.0f, den = 0.0f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float* pr = wpart + ((size_t)w * G + gg) * rec;
      const float wgt = pr[DH] == -INFINITY ? 0.0f : weight<FULL>(pr[DH] - mm);
      num += wgt * pr[dd];
      den += wgt * pr[DH + 1];
    }
    if (nsplit == 1) {
      a.out[((size_t)b * a.H + hk * G + gg) * DH + dd] = __float2bfloat16_rn(den > 0.0f ? num / den : 0.0f);
    } else {
      gpart[(size_t)gg * rec + dd] = num;
      if (dd == 0) {
        gpart[(size_t)gg * rec + DH] = mm;
        gpart[(size_t)gg * rec + DH + 1] = den;
      }
    }
  }
  if (nsplit == 1) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int old = atomicAdd(&a.counters[b * a.Hk + hk], 1);
    last_sh = old == nsplit - 1;
    if (old == nsplit - 1) a.counters[b * a.Hk + hk] = 0;
  }
  __syncthreads();
  if (!last_sh) return;
  __threadfence();
  merge_splits<DH, FULL>(parts, nsplit, G, a.out + ((size_t)b * a.H + hk * G) * DH, wpart);
}

}  // namespace fsvd_tile
#include "fsvd_prompt.cuh"
namespace fsvd_tile {

// ------------------------------------------------------------------------------- step head / tail
__device__ __forceinline__ void copy_row(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int d) {
  for (int i = threadIdx.x; i < (d >> 3); i += blockDim.x) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
}
__global__ void embed_rows_kernel(const __nv_bfloat16* __restrict__ table, const int* __restrict__ tokens,
                                  __nv_bfloat16* __restrict__ out, int d, int vocab) {
  const int b = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const int tok = min(max(tokens[b], 0), vocab - 1);
  copy_row(table + (size_t)tok * d, out + (size_t)b * d, d);
}
// First kernel of a prompt pass: row r = b n + t takes token prompt[b, off + t] at position
// seqlens[b] + t of sequence b.
__global__ void prompt_begin_kernel(const __nv_bfloat16* __restrict__ table, const int* __restrict__ prompt, int ld, int off, int n,
                                    const int* __restrict__ seqlens, int* rowpos, int* rowseq, __nv_bfloat16* __restrict__ out,
                                    int d, int vocab) {
  const int r = blockIdx.x, b = r / n, t = r - b * n;
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    rowpos[r] = seqlens[b] + t;
    rowseq[r] = b;
  }
  const int tok = min(max(prompt[(size_t)b * ld + off + t], 0), vocab - 1);
  copy_row(table + (size_t)tok * d, out + (size_t)r * d, d);
}
// Last kernel of a prompt pass that is not the prompt's last.
__global__ void advance_kernel(int* seqlens, int nseq, int n) {
  pdl_launch_dependents();
  pdl_wait();
  if ((int)threadIdx.x < nseq) seqlens[threadIdx.x] += n;
}

// token[b] = argmax_v logits[b, v] (lowest index among equal maxima); logs it; CTA 0 of the last
// row... every row advances its own sequence length, row 0 the step counter.
__global__ void __launch_bounds__(256) argmax_rows_kernel(const float* __restrict__ logits, int vocab, int* tokens,
                                                          int* token_log, int* step_counter, int* seqlens,
                                                          int max_steps, int B, int advance) {
  __shared__ float bv[8];
  __shared__ int bi[8];
  const int b = blockIdx.x, tid = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const float* row = logits + (size_t)b * vocab;
  float best = -INFINITY;
  int besti = 0x7fffffff;
  for (int i = tid; i < vocab; i += 256) {
    const float v = row[i];
    if (v > best || (v == best && i < besti)) {
      best = v;
      besti = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
    if (ov > best || (ov == best && oi < besti)) {
      best = ov;
      besti = oi;
    }
  }
  if ((tid & 31) == 0) {
    bv[tid >> 5] = best;
    bi[tid >> 5] = besti;
  }
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < 8; ++i)
      if (bv[i] > best || (bv[i] == best && bi[i] < besti)) {
        best = bv[i];
        besti = bi[i];
      }
    if (besti == 0x7fffffff) besti = 0;
    tokens[b] = besti;
    const int step = *step_counter;
    if (token_log && step < max_steps) token_log[(size_t)step * B + b] = besti;
    seqlens[b] += advance;
  }
}
__global__ void bump_step_kernel(int* step_counter) {
  pdl_launch_dependents();
  pdl_wait();
  *step_counter += 1;
}

// ------------------------------------------------------------------------------- host side
static thread_local char g_err[512];
static int fail(int code, const char* msg) {
  snprintf(g_err, sizeof(g_err), "%s", msg);
  fsvd_tile_set_error(code, g_err);
  return code;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// bf16 [rows, cols] row-major with row stride ld elements, boxes of box_rows x 64 columns, 128-byte swizzle
static int encode_sw128(CUtensorMap* tm, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(FSVD_ERR_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16) return fail(FSVD_ERR_ALIGN, "operand rows must start on 16-byte boundaries");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)kTileK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  const CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FSVD_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return 0;
}

static size_t al256(size_t x) { return (x + 255) / 256 * 256; }
static int round16(int b) { return b <= 16 ? 16 : (b + 15) / 16 * 16; }

struct GemmPlan {
  CUtensorMap mapA, mapA2, mapX, mapX2;
  GemmArgs a;
  dim3 grid;
  size_t smem;
};

static int g_sms = 0, g_smem_optin = 0;
static int device_limits() {
  if (g_sms) return 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(FSVD_ERR_CUDA, "cudaGetDevice failed");
  cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&g_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (g_sms < 1 || g_smem_optin < 64 * 1024) return fail(FSVD_ERR_CUDA, "device limits unavailable");
  return 0;
}

// Segments of the K range: about one CTA per SM, at least 4 k-blocks (64 KB of factor) per CTA
// where the matrix has them, at most kMaxSegs segments, none empty.
static int ctas_per_sm_wanted() {
  static int v = [] {
    const char* e = getenv("FSVD_TILE_CTAS_PER_SM");
    const int x = e ? atoi(e) : 1;
    return x >= 1 && x <= 4 ? x : 1;
  }();
  return v;
}
static void split_k(int tiles, int nkb, int sms, int& segs, int& kbs) {
  int want = (ctas_per_sm_wanted() * sms + tiles / 2) / tiles;
  if (want > kMaxSegs) want = kMaxSegs;
  if (want > nkb / 4) want = nkb / 4;
  if (want < 1) want = 1;
  kbs = (nkb + want - 1) / want;
  segs = (nkb + kbs - 1) / kbs;
}

static unsigned long long* g_tile_trace = nullptr;
static int g_tile_trace_epi = -1;
struct Scratch {
  int* status;
  long long wait_limit;
};

// y[B, P] = epilogue(W[P, K] . x[B, K]^T); W2 / x2: the second accumulator of TE_SWIGLU.
static int plan_gemm(GemmPlan& g, const void* W, const void* W2, int P, int K, int ldw, const void* x, const void* x2,
                     int ldx, int B, int epi, const Scratch& sc, int force_segs = 0) {
  if (int e = device_limits()) return e;
  memset(&g, 0, sizeof(g));
  GemmArgs& a = g.a;
  a.tiles = (P + kTileM - 1) / kTileM;
  // Wide batches: two CTAs take half of the columns each where the row tiles alone leave SMs idle (8 K
  // segments do not make up for it), or where two accumulators of all columns take the whole shared
  // memory of an SM and with it the K split.  The second CTA finds the factor tile in L2.
  a.nh = B > 64 && (epi == TE_SWIGLU || (epi == TE_STORE && a.tiles * kMaxSegs < g_sms)) ? 2 : 1;
  const int N = round16((B + a.nh - 1) / a.nh);
  a.P = P; a.K = K; a.B = B; a.N = N;
  a.nkb = (K + kTileK - 1) / kTileK;
  a.two = W2 ? 1 : 0;
  a.epi = epi;
  const int nacc = a.two ? 2 : 1;
  uint32_t cols = 32;
  while (cols < (uint32_t)(nacc * N)) cols <<= 1;
  a.tmem_cols = cols;
  const size_t stage = (size_t)kWTileBytes * nacc + (size_t)N * 128 * nacc;
  size_t smem = 0;
  int cap = kMaxSegs;
  for (int attempt = 0; attempt < 2; ++attempt) {
    split_k(a.tiles * a.nh, a.nkb, g_sms, a.segs, a.kbs);
    if (force_segs > 0) {   // the caller wants this many segments (problems of one grouped launch)
      const int want = force_segs < a.nkb ? force_segs : a.nkb;
      a.kbs = (a.nkb + want - 1) / want;
      a.segs = (a.nkb + a.kbs - 1) / a.kbs;
    }
    if (a.segs > cap) {   // second attempt: fewer, longer segments
      a.kbs = (a.nkb + cap - 1) / cap;
      a.segs = (a.nkb + a.kbs - 1) / a.kbs;
    }
    a.cpo = ((N + a.segs - 1) / a.segs + 3) / 4 * 4;   // a multiple of 4: partial sums travel four columns per store
    int ns = (int)((size_t)(g_smem_optin - 2048) / stage);
    if (ns > kMaxStages) ns = kMaxStages;
    if (ns > a.kbs) ns = a.kbs;
    // keep the ring small enough for two CTAs per SM: the clusters of a launch then fit the GPCs in
    // one wave (with one CTA per SM, 24 clusters of 6 do not fit 8 GPCs of 16-20 SMs)
    if (ns > 2 && (size_t)ns * stage > 110 * 1024) {
      ns = (int)((size_t)(110 * 1024) / stage);
      if (ns < 2) ns = 2;
    }
    if (ns < 1) return fail(FSVD_ERR_UNSUPPORTED, "shared memory too small for one stage");
    a.nstages = ns;
    smem = 1024 + (size_t)ns * stage;
    // the partial sums the cluster's CTAs send each other: in a place of their own (then a CTA may send
    // before its peers have finished) where that leaves two CTAs per SM and the launch, the three lifts
    // of a layer together, resident at once; else in the ring's
    const size_t recv = (size_t)nacc * a.segs * a.cpo * kTileM * 4;
    const bool lift = epi == TE_ROPE_Q || epi == TE_ROPE_K || epi == TE_VCACHE;
    const int per_sm = (int)((size_t)(228 * 1024) / (smem + recv + 1280));
    if (smem + recv <= 112 * 1024 && (!lift || per_sm * g_sms >= 3 * a.tiles * a.segs)) {
      a.recv_off = (uint32_t)(ns * stage);
      smem += recv;
    } else {
      a.recv_off = 0;
      if (smem < 1024 + recv) smem = 1024 + recv;
    }
    // co-resident CTAs must not ask for more than the 512 tensor-memory columns of an SM
    const size_t floor_smem = (size_t)232448 / (512 / cols + 1) + 1024;
    if (smem < floor_smem) smem = floor_smem;
    // one CTA per SM and more CTAs than SMs would run in two waves: take fewer segments instead
    if (attempt == 0 && smem > 113 * 1024 && a.tiles * a.nh * a.segs > g_sms && a.segs > 1) {
      cap = g_sms / (a.tiles * a.nh) > 0 ? g_sms / (a.tiles * a.nh) : 1;
      continue;
    }
    break;
  }
  if (smem > (size_t)g_smem_optin - 1024) return fail(FSVD_ERR_UNSUPPORTED, "shared memory plan exceeds the device limit");
  g.smem = smem;
  g.grid = dim3((unsigned)(a.tiles * a.nh), (unsigned)a.segs);
  a.status = sc.status;
  a.wait_limit = sc.wait_limit;
  a.trace = (g_tile_trace_epi < 0 || g_tile_trace_epi == epi) ? g_tile_trace : nullptr;
  if (int e = encode_sw128(&g.mapA, W, P, K, ldw, kTileM)) return e;
  if (int e = encode_sw128(&g.mapX, x, B, K, ldx, N)) return e;
  if (W2) {
    if (int e = encode_sw128(&g.mapA2, W2, P, K, ldw, kTileM)) return e;
    if (int e = encode_sw128(&g.mapX2, x2, B, K, ldx, N)) return e;
  } else {
    g.mapA2 = g.mapA;
    g.mapX2 = g.mapX;
  }
  return 0;
}

// Launch with the programmatic-stream-serialization attribute (see pdl_wait above).
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, unsigned cluster_y,
                                      cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cluster_y > 0) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = cluster_y;
    at[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  return launch_pdl_cluster(kern, grid, block, smem, 0u, st, std::forward<Args>(args)...);
}

// A kernel's dynamic shared-memory limit belongs to a device: raised on the current one, once.
class SmemLimit {
  std::atomic<unsigned long long> raised{0};   // a bit per device
 public:
  template <typename K>
  cudaError_t raise(K* kern, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev < 64 && (raised.load(std::memory_order_relaxed) >> dev & 1))) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) raised.fetch_or(1ull << dev);
    return e;
  }
};

// (takes the error off the thread, so that no later check of the caller's reports it again)
static int launch_failed(const char* what) {
  cudaGetLastError();
  return fail(FSVD_ERR_CUDA, what);
}

static int launch_group(const GemmPlan* const* plans, int n, cudaStream_t st);
static int launch_gemm(const GemmPlan& g, cudaStream_t st) {
  const GemmPlan* one[1] = {&g};
  return launch_group(one, 1, st);
}
static int launch_group(const GemmPlan* const* plans, int n, cudaStream_t st) {
  static SmemLimit limit;
  if (limit.raise(tile_gemm_kernel, g_smem_optin - 1024) != cudaSuccess)
    return launch_failed("cudaFuncSetAttribute failed for the tile kernel");
  GemmGroup grp;
  memset(&grp, 0, sizeof(grp));
  dim3 grid(1, 1, (unsigned)n);
  size_t smem = 0;
  for (int i = 0; i < n; ++i) {
    const GemmPlan& g = *plans[i];
    grp.maps[i][0] = g.mapA; grp.maps[i][1] = g.mapA2; grp.maps[i][2] = g.mapX; grp.maps[i][3] = g.mapX2;
    grp.args[i] = g.a;
    if (g.grid.x > grid.x) grid.x = g.grid.x;
    if (g.grid.y > grid.y) grid.y = g.grid.y;
    if (g.smem > smem) smem = g.smem;
  }
  // grid.y = K segments = CTAs of a cluster (the problems of a group have the same number)
  if (launch_pdl_cluster(tile_gemm_kernel, grid, dim3(kThreads), smem, grid.y, st, grp) != cudaSuccess)
    return launch_failed("tile kernel launch failed");
  fsvd_tile_count_launch();
  return 0;
}

// ---- workspace of the tile path (fsvd_dims with B > 8)
struct TileWs {
  size_t sync, counters, xn, pbuf, qbuf, attn, mid, hact, apart, total;
  int nsplit;
};
// Key splits of a sequence.  pairs = sequences x kv heads, positions = longest sequence the cache holds.
static int attn_splits(int pairs, int G, int positions, int sms, int most) {
  if (G >= 4) {
    // grouped-query kernel: 3 CTAs per SM, at least one block of 32 keys for each of a CTA's 4 warps
    most = std::min(most, (positions + kGqSplitKeys - 1) / kGqSplitKeys);
    return std::max(1, std::min((3 * sms + pairs - 1) / pairs, most));
  }
  // Three waves of the 8 CTAs of 4 warps that an SM holds, so that the SMs even out: not more than 8 splits
  // for that, the merge grows with them, but as many as one wave takes.  Measured, 4 layers, 4 steps (us):
  // 8 sequences x 32 heads x 2048 keys 5 splits 2659, 8 2588, 16 2636; 32 sequences 2 splits 4999, 4 4862, 8
  // 4872; 128 sequences x 640 keys 1 split 6494, 2 6658.  A split gets two groups of keys per warp: attention
  // half with 2 heads per kv head, 8 sequences, 300 keys 78 us with one, 74 with two.
  most = std::max(1, std::min(most, (positions + kBatchSplitKeys - 1) / kBatchSplitKeys));
  const int wave = (8 * sms + pairs - 1) / pairs;
  return std::min(most, std::min((24 * sms + pairs - 1) / pairs, std::max(8, wave)));
}
static int attn_nsplit(const fsvd_dims& D, int sms) {
  if (D.rows_are_positions || D.Hk < 1) return 1;   // prompt pass: row blocks share the cache rows instead
  const int G = D.H / D.Hk;
  return attn_splits(D.B * D.Hk, G, D.S_max, sms, G >= 4 ? kMaxSplit : 16);
}
static int imax(int a, int b) { return a > b ? a : b; }
static TileWs tile_layout(const fsvd_dims& D, int sms) {
  TileWs L;
  const int B = D.B;
  const int HD = D.H * D.Dh;
  const int Rqkv = D.Rq + D.Rk + D.Rv;
  size_t o = 0;
  L.sync = o;      o += al256(sizeof(SyncState));
  L.counters = o;  o += al256((size_t)B * D.Hk * 4);   // attention: arrivals of the splits of a head
  L.xn = o;        o += al256((size_t)B * imax(D.d, 8) * 2);
  L.pbuf = o;      o += al256((size_t)B * imax(imax(Rqkv, D.Ru + D.Rg), imax(D.Ro, D.Rd)) * 2);
  L.qbuf = o;      o += al256((size_t)B * HD * 2);
  L.attn = o;      o += al256((size_t)B * HD * 2);
  L.mid = o;       o += al256((size_t)B * D.d * 2);
  L.hact = o;      o += al256((size_t)B * D.I * 2);
  L.nsplit = attn_nsplit(D, sms);
  L.apart = o;     o += al256((size_t)B * D.Hk * L.nsplit * (D.H / imax(D.Hk, 1)) * (D.Dh + kPartPad) * 4);
  L.total = o;
  return L;
}

static int check_tile_dims(const fsvd_dims& D) {
  if (D.dtype != FSVD_DTYPE_BF16) return fail(FSVD_ERR_UNSUPPORTED, "batches above 8 need bf16 factors (dtype 0)");
  if (D.B < 1 || D.B > 128) return fail(FSVD_ERR_UNSUPPORTED, "batch outside 1..128");
  if (D.Dh != 64 && D.Dh != 128) return fail(FSVD_ERR_UNSUPPORTED, "head_dim must be 64 or 128");
  {
    const int G = D.Hk > 0 && D.H % D.Hk == 0 ? D.H / D.Hk : 0;
    if (G != 1 && G != 2 && G != 4 && G != 8) return fail(FSVD_ERR_UNSUPPORTED, "H / Hk must be 1, 2, 4 or 8");
  }
  if (D.Rg != D.Ru) return fail(FSVD_ERR_UNSUPPORTED, "gate and up ranks must be equal for batches above 8");
  const int m8[] = {D.d, D.I, D.Rq, D.Rk, D.Rv, D.Ro, D.Rg, D.Ru, D.Rd};
  for (int v : m8)
    if (v <= 0 || v % 8) return fail(FSVD_ERR_ALIGN, "sizes and ranks must be positive multiples of 8");
  if ((D.H * D.Dh + kTileM - 1) / kTileM > 1024 || (D.Hk * D.Dh + kTileM - 1) / kTileM > 1024)
    return fail(FSVD_ERR_UNSUPPORTED, "more than 1024 row tiles in a q / k / v lift");
  if ((D.d + kTileM - 1) / kTileM > 4096 || (D.I + kTileM - 1) / kTileM > 4096 || (D.vocab + kTileM - 1) / kTileM > 4096)
    return fail(FSVD_ERR_UNSUPPORTED, "more than 4096 row tiles");
  if (D.S_max < 1) return fail(FSVD_ERR_ARG, "S_max");
  return 0;
}

struct LayerPlan {
  GemmPlan g[9];
  AttnArgs at;
};

// The largest segment count, from the largest of the three planned counts (at most the smallest
// number of k-blocks) down to 2, that cuts all three K ranges into exactly that many non-empty
// segments; 0 when there is none.
static int common_segments(int nkb_q, int nkb_k, int nkb_v, int segs_q, int segs_k, int segs_v) {
  auto segs_for = [](int nkb, int want) { const int kbs = (nkb + want - 1) / want; return (nkb + kbs - 1) / kbs; };
  const int nkb_min = std::min(nkb_q, std::min(nkb_k, nkb_v));
  for (int S = std::min(std::max(segs_q, std::max(segs_k, segs_v)), nkb_min); S >= 2; --S)
    if (segs_for(nkb_q, S) == S && segs_for(nkb_k, S) == S && segs_for(nkb_v, S) == S) return S;
  return 0;
}

static int plan_layer(LayerPlan& lp, const fsvd_dims& D, const fsvd_layer& Lw, const void* cos_tab, const void* sin_tab,
                      const int* seqlens, const void* x_in, void* x_out, char* ws, const TileWs& L, long long wait_limit,
                      const void* xn_in = nullptr) {
  const int B = D.B, HD = D.H * D.Dh, KD = D.Hk * D.Dh, Rqkv = D.Rq + D.Rk + D.Rv;
  Scratch sc = {&reinterpret_cast<SyncState*>(ws + L.sync)->status, wait_limit};
  __nv_bfloat16* xn = reinterpret_cast<__nv_bfloat16*>(ws + L.xn);
  __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(ws + L.pbuf);
  __nv_bfloat16* qb = reinterpret_cast<__nv_bfloat16*>(ws + L.qbuf);
  __nv_bfloat16* attn = reinterpret_cast<__nv_bfloat16*>(ws + L.attn);
  __nv_bfloat16* mid = reinterpret_cast<__nv_bfloat16*>(ws + L.mid);
  __nv_bfloat16* hact = reinterpret_cast<__nv_bfloat16*>(ws + L.hact);
  auto rope = [&](GemmArgs& a, void* cache) {
    a.cache = cache; a.cos_tab = cos_tab; a.sin_tab = sin_tab; a.seqlens = seqlens;
    a.Dh = D.Dh; a.HkDh = KD; a.S_max = D.S_max; a.shared_cache = D.rows_are_positions ? 1 : 0;
  };
  int e;
  // 0: [p_q | p_k | p_v] = rms(x) . qkv_v^T
  // xn_in: the caller already holds rms(x) . ln1 (the kernel before this layer wrote it)
  if ((e = plan_gemm(lp.g[0], Lw.qkv_v, nullptr, Rqkv, D.d, D.d, xn_in ? xn_in : xn, nullptr, D.d, B, TE_STORE, sc))) return e;
  lp.g[0].a.out = pb;
  // 1-3: lifts with rotary / cache append
  if ((e = plan_gemm(lp.g[1], Lw.q_u, nullptr, HD, D.Rq, D.Rq, pb, nullptr, Rqkv, B, TE_ROPE_Q, sc))) return e;
  lp.g[1].a.out = qb;
  rope(lp.g[1].a, nullptr);
  if ((e = plan_gemm(lp.g[2], Lw.k_u, nullptr, KD, D.Rk, D.Rk, pb + D.Rq, nullptr, Rqkv, B, TE_ROPE_K, sc))) return e;
  rope(lp.g[2].a, Lw.k_cache);
  if ((e = plan_gemm(lp.g[3], Lw.v_u, nullptr, KD, D.Rv, D.Rv, pb + D.Rq + D.Rk, nullptr, Rqkv, B, TE_VCACHE, sc))) return e;
  rope(lp.g[3].a, Lw.v_cache);
  if (lp.g[1].a.segs != lp.g[2].a.segs || lp.g[1].a.segs != lp.g[3].a.segs) {
    // the three lifts go out as one launch when they cut K into the same number of segments: look for
    // a count (>= 2) that all three can take
    const int S = common_segments(lp.g[1].a.nkb, lp.g[2].a.nkb, lp.g[3].a.nkb, lp.g[1].a.segs, lp.g[2].a.segs, lp.g[3].a.segs);
    if (S >= 2) {
      LayerPlan t = lp;
      const bool planned = !plan_gemm(t.g[1], Lw.q_u, nullptr, HD, D.Rq, D.Rq, pb, nullptr, Rqkv, B, TE_ROPE_Q, sc, S) &&
                           !plan_gemm(t.g[2], Lw.k_u, nullptr, KD, D.Rk, D.Rk, pb + D.Rq, nullptr, Rqkv, B, TE_ROPE_K, sc, S) &&
                           !plan_gemm(t.g[3], Lw.v_u, nullptr, KD, D.Rv, D.Rv, pb + D.Rq + D.Rk, nullptr, Rqkv, B, TE_VCACHE, sc, S);
      // (the shared-memory plan may still have changed a count: then the separate plans stay)
      if (planned && t.g[1].a.segs == S && t.g[2].a.segs == S && t.g[3].a.segs == S) {
        t.g[1].a.out = qb;
        rope(t.g[1].a, nullptr);
        rope(t.g[2].a, Lw.k_cache);
        rope(t.g[3].a, Lw.v_cache);
        for (int i = 1; i < 4; ++i) lp.g[i] = t.g[i];
      }
    }
  }
  // attention
  AttnArgs& at = lp.at;
  memset(&at, 0, sizeof(at));
  at.q = qb; at.kcache = reinterpret_cast<const __nv_bfloat16*>(Lw.k_cache);
  at.vcache = reinterpret_cast<const __nv_bfloat16*>(Lw.v_cache);
  at.seqlens = seqlens; at.out = attn;
  at.part = reinterpret_cast<float*>(ws + L.apart);
  at.counters = reinterpret_cast<int*>(ws + L.counters);
  at.B = B; at.H = D.H; at.Hk = D.Hk; at.Dh = D.Dh; at.S_max = D.S_max; at.nsplit = L.nsplit; at.seqlen_add = 1;
  at.shared_cache = D.rows_are_positions ? 1 : 0;
  at.scale = 1.0f / sqrtf((float)D.Dh);
  // 4-5: o projection + residual
  if ((e = plan_gemm(lp.g[4], Lw.o_v, nullptr, D.Ro, HD, HD, attn, nullptr, HD, B, TE_STORE, sc))) return e;
  lp.g[4].a.out = pb;
  if ((e = plan_gemm(lp.g[5], Lw.o_u, nullptr, D.d, D.Ro, D.Ro, pb, nullptr, D.Ro, B, TE_RESID, sc))) return e;
  lp.g[5].a.out = mid;
  lp.g[5].a.resid = x_in;
  // 6-8: MLP
  if ((e = plan_gemm(lp.g[6], Lw.upgate_v, nullptr, D.Ru + D.Rg, D.d, D.d, xn, nullptr, D.d, B, TE_STORE, sc))) return e;
  lp.g[6].a.out = pb;
  if ((e = plan_gemm(lp.g[7], Lw.gate_u, Lw.up_u, D.I, D.Rg, D.Rg, pb + D.Ru, pb, D.Ru + D.Rg, B, TE_SWIGLU, sc))) return e;
  lp.g[7].a.out = hact;
  if ((e = plan_gemm(lp.g[8], Lw.down_v, nullptr, D.Rd, D.I, D.I, hact, nullptr, D.I, B, TE_STORE, sc))) return e;
  lp.g[8].a.out = pb;
  (void)mid;
  return 0;
}

template <int DH, bool FULL>
static cudaError_t launch_prompt_attn(const PaArgs& pa, int nseq, cudaStream_t st) {
  constexpr int smem = 4 * kPaKeys * (DH * 2 + 16);
  static_assert(kPaWarps * kPaTailSlots * (DH + kPartPad) * 4 <= smem && kPaWarps * 2 * kPaTailKeys * (DH * 2 + 16) <= smem);
  static SmemLimit limit;
  const cudaError_t e = limit.raise(prompt_attn_kernel<DH, FULL>, smem);
  if (e != cudaSuccess) return e;
  const int G = pa.H / pa.Hk, rpb = kPaSlots / G, tpos = kPaTailSlots / G;
  const int ctas = (pa.full_from + rpb - 1) / rpb + (FULL ? 0 : (pa.L - pa.full_from + tpos - 1) / tpos);
  return launch_pdl(prompt_attn_kernel<DH, FULL>, dim3((unsigned)ctas, (unsigned)pa.Hk, (unsigned)nseq), dim3(kPaWarps * 32), (size_t)smem,
                    st, pa);
}
// rows of nseq sequences, L consecutive positions each
static int launch_prompt_attn(PaArgs pa, int Dh, int nseq, cudaStream_t st) {
  const bool full = nseq > 1 && (nseq <= 4 || pa.H / pa.Hk < 4);
  pa.full_from = nseq > 1 ? pa.L : std::max(0, pa.L - kFullRows);
  const cudaError_t e = Dh == 128 ? (full ? launch_prompt_attn<128, true>(pa, nseq, st) : launch_prompt_attn<128, false>(pa, nseq, st))
                                  : (full ? launch_prompt_attn<64, true>(pa, nseq, st) : launch_prompt_attn<64, false>(pa, nseq, st));
  if (e != cudaSuccess) return launch_failed("attention kernel launch failed");
  fsvd_tile_count_launch();
  return 0;
}

template <int DH, bool FULL>
static cudaError_t launch_attn_g(const AttnArgs& at, cudaStream_t st) {
  const dim3 grid((unsigned)(at.B * at.Hk * at.nsplit)), threads(kAttnThreads);
  switch (at.H / at.Hk) {
    case 1: return launch_pdl(batch_attn_kernel<DH, 1, FULL>, grid, threads, 0, st, at);
    case 2: return launch_pdl(batch_attn_kernel<DH, 2, FULL>, grid, threads, 0, st, at);
    default: {
      // 4 or 8 heads per kv head: the heads as rows of a tensor-core tile
      constexpr int smem = kAttnWarps * 2 * kGqKeys * (DH * 2 + 16);
      static SmemLimit limit;
      const cudaError_t e = limit.raise(gqa_decode_attn_kernel<DH, FULL>, smem);
      return e != cudaSuccess ? e : launch_pdl(gqa_decode_attn_kernel<DH, FULL>, grid, threads, (size_t)smem, st, at);
    }
  }
}
static PaArgs prompt_args(const AttnArgs& at) {
  PaArgs pa;   // (a row sees the keys up to its own position: seqlen_add is 1 on this route)
  pa.q = at.q; pa.kcache = at.kcache; pa.vcache = at.vcache; pa.rowpos = at.seqlens; pa.rowseq = nullptr; pa.out = at.out;
  pa.L = at.B; pa.H = at.H; pa.Hk = at.Hk; pa.S_max = at.S_max;
  pa.scale_log2 = at.scale * 1.4426950408889634f;
  return pa;
}
static int launch_attn(const AttnArgs& at, cudaStream_t st, bool full = false) {
  if (at.shared_cache) return launch_prompt_attn(prompt_args(at), at.Dh, 1, st);   // the rows are consecutive positions of one sequence
  const cudaError_t e = at.Dh == 128 ? (full ? launch_attn_g<128, true>(at, st) : launch_attn_g<128, false>(at, st))
                                     : (full ? launch_attn_g<64, true>(at, st) : launch_attn_g<64, false>(at, st));
  if (e != cudaSuccess) return launch_failed("attention kernel launch failed");
  fsvd_tile_count_launch();
  return 0;
}

// The last GEMM of a layer (down lift + residual) is planned per call site: its output buffer
// differs between the per-layer entry point and the model.
static int launch_reduce(const ReduceArgs& r, int rows, cudaStream_t st) {
  // wide rows are cut into four column slices (a cluster of four CTAs per row)
  const unsigned C = (r.d >= 2048 && r.d % 32 == 0) ? 4u : 1u;
  if (launch_pdl_cluster(exchange_reduce_rows_kernel, dim3((unsigned)rows, C), dim3(256), 0, C > 1 ? C : 0u, st, r) != cudaSuccess)
    return launch_failed("exchange kernel launch failed");
  fsvd_tile_count_launch();
  return 0;
}

// r1 / r2 (tensor-parallel layer): the o lift and the down lift push their partial sums to every
// rank; r1 replaces the second RMSNorm (sum + residual + norm), r2 finishes the layer output.
static int run_layer(const LayerPlan& lp, const GemmPlan& down_lift, const fsvd_dims& D, const fsvd_layer& Lw,
                     const void* x_in, char* ws, const TileWs& L, cudaStream_t st, const ReduceArgs* r1 = nullptr,
                     const ReduceArgs* r2 = nullptr, bool have_xn = false) {
  __nv_bfloat16* xn = reinterpret_cast<__nv_bfloat16*>(ws + L.xn);
  const __nv_bfloat16* mid = reinterpret_cast<const __nv_bfloat16*>(ws + L.mid);
  int e;
  if (!have_xn) {
    launch_pdl(reinterpret_cast<uintptr_t>(x_in) % 16 ? rmsnorm_rows_kernel<false> : rmsnorm_rows_kernel<true>, dim3(D.B), dim3(256), 0,
               st, reinterpret_cast<const __nv_bfloat16*>(x_in), reinterpret_cast<const __nv_bfloat16*>(Lw.ln1_w), xn, D.d, D.eps, 1, 0);
    fsvd_tile_count_launch();
  }
  if ((e = launch_gemm(lp.g[0], st))) return e;
  if (lp.g[1].a.segs == lp.g[2].a.segs && lp.g[1].a.segs == lp.g[3].a.segs) {
    // the q, k and v lifts read the same rank vector and write disjoint outputs: one launch
    // (possible when they cut K into the same number of segments = cluster size)
    const GemmPlan* qkv[3] = {&lp.g[1], &lp.g[2], &lp.g[3]};
    if ((e = launch_group(qkv, 3, st))) return e;
  } else {
    for (int i = 1; i < 4; ++i)
      if ((e = launch_gemm(lp.g[i], st))) return e;
  }
  if ((e = launch_attn(lp.at, st))) return e;
  if ((e = launch_gemm(lp.g[4], st))) return e;
  if ((e = launch_gemm(lp.g[5], st))) return e;
  if (r1) {
    if ((e = launch_reduce(*r1, D.B, st))) return e;
  } else {
    launch_pdl(rmsnorm_rows_kernel<true>, dim3(D.B), dim3(256), 0, st, mid, reinterpret_cast<const __nv_bfloat16*>(Lw.ln2_w), xn,
               D.d, D.eps, 1, 0);
    fsvd_tile_count_launch();
  }
  for (int i = 6; i < 9; ++i)
    if ((e = launch_gemm(lp.g[i], st))) return e;
  if ((e = launch_gemm(down_lift, st))) return e;
  if (r2 && (e = launch_reduce(*r2, D.B, st))) return e;
  if (cudaGetLastError() != cudaSuccess) return fail(FSVD_ERR_CUDA, "kernel launch failed");
  return 0;
}

static int plan_down_lift(GemmPlan& g, const fsvd_dims& D, const fsvd_layer& Lw, void* x_out, char* ws, const TileWs& L,
                          long long wait_limit) {
  Scratch sc = {&reinterpret_cast<SyncState*>(ws + L.sync)->status, wait_limit};
  if (int e = plan_gemm(g, Lw.down_u, nullptr, D.d, D.Rd, D.Rd, ws + L.pbuf, nullptr, D.Rd, D.B, TE_RESID, sc)) return e;
  g.a.out = x_out;
  g.a.resid = ws + L.mid;
  return 0;
}

// Tensor-parallel layer: the plans of the single-GPU layer on the rank's shards, with the two
// residual lifts turned into pushes and the reductions that complete them.
struct TpPlan {
  LayerPlan lp;
  GemmPlan dl;
  ReduceArgs r1, r2;
};
static int plan_tp_layer(TpPlan& tp, const fsvd_dims& D, const fsvd_layer& Lw, const void* cos_tab, const void* sin_tab,
                         const int* seqlens, const void* x_in, const void* xn_in, void* x_out, const void* next_norm_w,
                         void* xn_out, const fsvd_exchange& ex, char* ws, const TileWs& L, long long wait_limit) {
  if (int e = plan_layer(tp.lp, D, Lw, cos_tab, sin_tab, seqlens, x_in, x_out, ws, L, wait_limit, xn_in)) return e;
  if (int e = plan_down_lift(tp.dl, D, Lw, x_out, ws, L, wait_limit)) return e;
  fsvd_exch::Ctrl* ctrl = reinterpret_cast<fsvd_exch::Ctrl*>(ex.geom.region[ex.geom.rank]);
  int* status = &reinterpret_cast<SyncState*>(ws + L.sync)->status;
  auto to_push = [&](GemmPlan& g, ReduceArgs& r, const void* resid, void* out, const void* norm_w, void* xn) -> int {
    if ((unsigned)(g.a.tiles * g.a.segs) > ex.geom.flag_cap) return fail(FSVD_ERR_UNSUPPORTED, "more CTAs in a lift than exchange flags");
    g.a.epi = TE_PUSH;
    g.a.out = nullptr;
    g.a.resid = nullptr;
    g.a.ex = ex.geom;
    g.a.ex_seq = &ctrl->seq;
    memset(&r, 0, sizeof(r));
    r.ex = ex.geom;
    r.ctrl = ctrl;
    r.nflags = g.a.tiles * g.a.segs;
    r.resid = reinterpret_cast<const __nv_bfloat16*>(resid);
    r.out = reinterpret_cast<__nv_bfloat16*>(out);
    r.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w);
    r.xn = reinterpret_cast<__nv_bfloat16*>(xn);
    r.d = D.d;
    r.eps = D.eps;
    r.status = status;
    r.wait_limit = wait_limit;
    r.trace = ex.trace_cap ? ex.trace : nullptr;
    r.trace_cap = ex.trace_cap;
    return 0;
  };
  if (int e = to_push(tp.lp.g[5], tp.r1, x_in, ws + L.mid, Lw.ln2_w, ws + L.xn)) return e;
  return to_push(tp.dl, tp.r2, ws + L.mid, x_out, next_norm_w, next_norm_w ? xn_out : nullptr);
}

}  // namespace fsvd_tile

// ------------------------------------------------------------------------------- entry points
using namespace fsvd_tile;

int fsvd_tile_flash_decode(const void* q, const void* k_cache, const void* v_cache, const int* cache_seqlens, int seqlen_add,
                           void* out, int B, int H, int Hk, int Dh, int S_max, float scale, float* part, size_t part_floats,
                           int* counters, void* stream) {
  if (int e = device_limits()) return e;
  AttnArgs at;
  memset(&at, 0, sizeof(at));
  at.q = reinterpret_cast<const __nv_bfloat16*>(q);
  at.kcache = reinterpret_cast<const __nv_bfloat16*>(k_cache);
  at.vcache = reinterpret_cast<const __nv_bfloat16*>(v_cache);
  at.seqlens = cache_seqlens; at.out = reinterpret_cast<__nv_bfloat16*>(out);
  at.part = part; at.counters = counters;
  at.B = B; at.H = H; at.Hk = Hk; at.Dh = Dh; at.S_max = S_max; at.seqlen_add = seqlen_add; at.scale = scale;
  const int fits = (int)std::min<size_t>(part_floats / ((size_t)B * H * (Dh + kPartPad)), kMaxSplit);
  at.nsplit = attn_splits(B * Hk, H / Hk, S_max, g_sms, std::max(1, fits));
  return launch_attn(at, (cudaStream_t)stream, true);
}

size_t fsvd_tile_workspace_bytes(const fsvd_dims* dims) {
  if (!dims || device_limits()) return 0;
  if (check_tile_dims(*dims)) return 0;
  return tile_layout(*dims, g_sms).total;
}

int fsvd_tile_decode_layer(const fsvd_dims* dims, const fsvd_layer* layer, const void* cos_tab, const void* sin_tab,
                           const int* cache_seqlens, const void* x_in, void* x_out, void* ws, size_t ws_bytes,
                           long long wait_limit, void* stream) {
  const fsvd_dims& D = *dims;
  if (int e = device_limits()) return e;
  if (int e = check_tile_dims(D)) return e;
  const TileWs L = tile_layout(D, g_sms);
  if (!ws || ws_bytes < L.total) return fail(FSVD_ERR_WORKSPACE, "workspace too small for this batch");
  if (x_in == x_out) return fail(FSVD_ERR_ARG, "x_in and x_out must differ");
  // the plans of the last call are kept: a decode loop calls with the same arguments every token
  struct Cached {
    fsvd_dims D;
    fsvd_layer Lw;
    const void *cos_tab, *sin_tab, *x_in;
    const int* seqlens;
    void *x_out, *ws;
    long long wait_limit;
    LayerPlan lp;
    GemmPlan dl;
    bool valid = false;
  };
  static std::mutex mu;
  static std::vector<Cached*> cache;
  std::lock_guard<std::mutex> lock(mu);
  Cached* c = nullptr;
  for (Cached* k : cache)
    if (k->valid && !memcmp(&k->D, &D, sizeof(D)) && !memcmp(&k->Lw, layer, sizeof(*layer)) && k->cos_tab == cos_tab &&
        k->sin_tab == sin_tab && k->x_in == x_in && k->seqlens == cache_seqlens && k->x_out == x_out && k->ws == ws &&
        k->wait_limit == wait_limit)
      c = k;
  if (!c) {
    if (cache.size() >= 128) {
      for (Cached* k : cache) delete k;
      cache.clear();
    }
    c = new Cached();
    c->D = D; c->Lw = *layer; c->cos_tab = cos_tab; c->sin_tab = sin_tab; c->x_in = x_in; c->seqlens = cache_seqlens;
    c->x_out = x_out; c->ws = ws; c->wait_limit = wait_limit;
    int e = plan_layer(c->lp, D, *layer, cos_tab, sin_tab, cache_seqlens, x_in, x_out, reinterpret_cast<char*>(ws), L, wait_limit);
    if (!e) e = plan_down_lift(c->dl, D, *layer, x_out, reinterpret_cast<char*>(ws), L, wait_limit);
    if (e) {
      delete c;
      return e;
    }
    c->valid = true;
    cache.push_back(c);
  }
  return run_layer(c->lp, c->dl, D, *layer, x_in, reinterpret_cast<char*>(ws), L, (cudaStream_t)stream);
}

int fsvd_tile_tp_decode_layer(const fsvd_dims* dims, const fsvd_layer* layer, const void* cos_tab, const void* sin_tab,
                              const int* cache_seqlens, const void* x_in, const void* x_norm_in, void* x_out,
                              const void* next_norm_w, void* x_norm_out, fsvd_exchange* ex, void* ws, size_t ws_bytes,
                              long long wait_limit, void* stream) {
  const fsvd_dims& D = *dims;
  if (int e = device_limits()) return e;
  if (int e = check_tile_dims(D)) return e;
  if (D.rows_are_positions) return fail(FSVD_ERR_UNSUPPORTED, "the tensor-parallel layer takes one row per sequence");
  if (D.d != ex->d || D.B > ex->max_rows) return fail(FSVD_ERR_ARG, "the exchange was created for another width or fewer rows");
  const TileWs L = tile_layout(D, g_sms);
  if (!ws || ws_bytes < L.total) return fail(FSVD_ERR_WORKSPACE, "workspace too small for this batch");
  if (x_in == x_out) return fail(FSVD_ERR_ARG, "x_in and x_out must differ");
  if ((reinterpret_cast<uintptr_t>(x_in) | reinterpret_cast<uintptr_t>(x_out) | reinterpret_cast<uintptr_t>(layer->ln2_w)) & 15)
    return fail(FSVD_ERR_ALIGN, "x_in, x_out and the norm weights must be 16-byte aligned");
  if ((reinterpret_cast<uintptr_t>(x_norm_in) | reinterpret_cast<uintptr_t>(next_norm_w) | reinterpret_cast<uintptr_t>(x_norm_out)) & 15)
    return fail(FSVD_ERR_ALIGN, "x_norm_in, next_norm_w and x_norm_out must be 16-byte aligned");
  if (next_norm_w && !x_norm_out) return fail(FSVD_ERR_ARG, "next_norm_w needs x_norm_out");
  struct Cached {
    fsvd_dims D;
    fsvd_layer Lw;
    const void *cos_tab, *sin_tab, *x_in, *xn_in, *next_w, *xn_out;
    const int* seqlens;
    void *x_out, *ws;
    const fsvd_exchange* ex;
    unsigned long long ex_id;
    long long wait_limit;
    TpPlan tp;
  };
  static std::mutex mu;
  static std::vector<Cached*> cache;
  std::lock_guard<std::mutex> lock(mu);
  Cached* c = nullptr;
  for (Cached* k : cache)
    if (!memcmp(&k->D, &D, sizeof(D)) && !memcmp(&k->Lw, layer, sizeof(*layer)) && k->cos_tab == cos_tab &&
        k->sin_tab == sin_tab && k->x_in == x_in && k->seqlens == cache_seqlens && k->x_out == x_out && k->ws == ws &&
        k->ex == ex && k->ex_id == ex->id && k->wait_limit == wait_limit && k->xn_in == x_norm_in && k->next_w == next_norm_w &&
        k->xn_out == x_norm_out)
      c = k;
  if (!c) {
    if (cache.size() >= 256) {
      for (Cached* k : cache) delete k;
      cache.clear();
    }
    c = new Cached();
    c->D = D; c->Lw = *layer; c->cos_tab = cos_tab; c->sin_tab = sin_tab; c->x_in = x_in; c->seqlens = cache_seqlens;
    c->x_out = x_out; c->ws = ws; c->ex = ex; c->ex_id = ex->id; c->wait_limit = wait_limit;
    c->xn_in = x_norm_in; c->next_w = next_norm_w; c->xn_out = x_norm_out;
    if (int e = plan_tp_layer(c->tp, D, *layer, cos_tab, sin_tab, cache_seqlens, x_in, x_norm_in, x_out, next_norm_w, x_norm_out,
                              *ex, reinterpret_cast<char*>(ws), L, wait_limit)) {
      delete c;
      return e;
    }
    cache.push_back(c);
  }
  return run_layer(c->tp.lp, c->tp.dl, D, *layer, x_in, reinterpret_cast<char*>(ws), L, (cudaStream_t)stream, &c->tp.r1, &c->tp.r2,
                   x_norm_in != nullptr);
}

// ---- whole-model decode for batches above 8: the launches of a step captured once in a CUDA graph
struct fsvd_tile_model {
  fsvd_dims D;
  TileWs L;
  char* ws = nullptr;
  char* extra = nullptr;
  __nv_bfloat16* xbuf[2] = {nullptr, nullptr};
  int *tokens = nullptr, *seqlens = nullptr, *step_counter = nullptr, *token_log = nullptr;
  float* logits = nullptr;
  int max_steps = 0;
  std::vector<LayerPlan> layers;
  std::vector<GemmPlan> down;
  std::vector<fsvd_layer> lw;
  GemmPlan head;
  const void *embed = nullptr, *final_norm = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  long long launches_per_step = 0;
};

static int tile_model_record(fsvd_tile_model* m, cudaStream_t st) {
  const fsvd_dims& D = m->D;
  int e;
  launch_pdl(embed_rows_kernel, dim3(D.B), dim3(256), 0, st, reinterpret_cast<const __nv_bfloat16*>(m->embed),
             (const int*)m->tokens, m->xbuf[0], D.d, D.vocab);
  fsvd_tile_count_launch();
  for (int l = 0; l < D.n_layers; ++l)
    if ((e = run_layer(m->layers[l], m->down[l], D, m->lw[l], m->xbuf[l & 1], m->ws, m->L, st))) return e;
  __nv_bfloat16* xn = reinterpret_cast<__nv_bfloat16*>(m->ws + m->L.xn);
  launch_pdl(rmsnorm_rows_kernel<true>, dim3(D.B), dim3(256), 0, st, (const __nv_bfloat16*)m->xbuf[D.n_layers & 1],
             reinterpret_cast<const __nv_bfloat16*>(m->final_norm), xn, D.d, D.eps, 1, 0);
  fsvd_tile_count_launch();
  if ((e = launch_gemm(m->head, st))) return e;
  launch_pdl(argmax_rows_kernel, dim3(D.B), dim3(256), 0, st, (const float*)m->logits, D.vocab, m->tokens, m->token_log,
             m->step_counter, m->seqlens, m->max_steps, D.B, 1);
  launch_pdl(bump_step_kernel, dim3(1), dim3(1), 0, st, m->step_counter);
  fsvd_tile_count_launch();
  fsvd_tile_count_launch();
  if (cudaGetLastError() != cudaSuccess) return fail(FSVD_ERR_CUDA, "kernel launch failed");
  return 0;
}

int fsvd_tile_model_destroy(fsvd_tile_model* m) {
  if (!m) return 0;
  if (m->exec) cudaGraphExecDestroy(m->exec);
  if (m->graph) cudaGraphDestroy(m->graph);
  cudaFree(m->ws);
  cudaFree(m->extra);
  cudaFree(m->xbuf[0]);
  cudaFree(m->xbuf[1]);
  delete m;
  return 0;
}

// A stream on which fresh device memory is zeroed before any other stream can use it.  (cudaMemset goes to the
// default stream and returns at once: a launch on a non-blocking stream would not wait for it.  A stream of
// its own does not wait for what the default stream has queued.)
struct SideStream {
  cudaStream_t st = nullptr;
  cudaError_t clear(void* p, size_t bytes) {
    cudaError_t ce = st ? cudaSuccess : cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    return ce != cudaSuccess ? ce : cudaMemsetAsync(p, 0, bytes, st);
  }
  cudaError_t wait() { return cudaStreamSynchronize(st); }
  ~SideStream() {
    if (st) cudaStreamDestroy(st);
  }
};

int fsvd_tile_model_create(const fsvd_dims* dims, const fsvd_layer* layers, const void* embed, const void* final_norm_w,
                           const void* lm_head, const void* cos_tab, const void* sin_tab, int max_steps, long long wait_limit,
                           fsvd_tile_model** out) {
  const fsvd_dims& D = *dims;
  if (int e = device_limits()) return e;
  if (int e = check_tile_dims(D)) return e;
  if (D.n_layers < 1 || D.vocab < 1) return fail(FSVD_ERR_ARG, "n_layers / vocab");
  if (max_steps < 1) max_steps = 1;
  fsvd_tile_model* m = new fsvd_tile_model();
  m->D = D;
  m->L = tile_layout(D, g_sms);
  m->max_steps = max_steps;
  m->embed = embed;
  m->final_norm = final_norm_w;
  const size_t extra = al256((size_t)D.B * 4) * 2 + al256(4) + al256((size_t)max_steps * D.B * 4) + al256((size_t)D.B * D.vocab * 4);
  cudaError_t ce = cudaMalloc(&m->ws, m->L.total);
  if (ce == cudaSuccess) ce = cudaMalloc(&m->extra, extra);
  if (ce == cudaSuccess) ce = cudaMalloc(&m->xbuf[0], al256((size_t)D.B * D.d * 2));
  if (ce == cudaSuccess) ce = cudaMalloc(&m->xbuf[1], al256((size_t)D.B * D.d * 2));
  SideStream side;   // the clears run while the plans are made
  if (ce == cudaSuccess) ce = side.clear(m->ws, m->L.total);
  if (ce == cudaSuccess) ce = side.clear(m->extra, extra);
  if (ce != cudaSuccess) {
    fsvd_tile_model_destroy(m);
    return fail(FSVD_ERR_CUDA, "allocating model scratch failed");
  }
  size_t o = 0;
  m->tokens = reinterpret_cast<int*>(m->extra + o);        o += al256((size_t)D.B * 4);
  m->seqlens = reinterpret_cast<int*>(m->extra + o);       o += al256((size_t)D.B * 4);
  m->step_counter = reinterpret_cast<int*>(m->extra + o);  o += al256(4);
  m->token_log = reinterpret_cast<int*>(m->extra + o);     o += al256((size_t)max_steps * D.B * 4);
  m->logits = reinterpret_cast<float*>(m->extra + o);
  m->layers.resize(D.n_layers);
  m->down.resize(D.n_layers);
  m->lw.assign(layers, layers + D.n_layers);
  int e = 0;
  for (int l = 0; l < D.n_layers && !e; ++l) {
    e = plan_layer(m->layers[l], D, layers[l], cos_tab, sin_tab, m->seqlens, m->xbuf[l & 1], m->xbuf[(l + 1) & 1], m->ws, m->L, wait_limit);
    if (!e) e = plan_down_lift(m->down[l], D, layers[l], m->xbuf[(l + 1) & 1], m->ws, m->L, wait_limit);
  }
  if (!e) {
    Scratch sc = {&reinterpret_cast<SyncState*>(m->ws + m->L.sync)->status, wait_limit};
    e = plan_gemm(m->head, lm_head, nullptr, D.vocab, D.d, D.d, m->ws + m->L.xn, nullptr, D.d, D.B, TE_STORE_F32, sc);
    m->head.a.out = m->logits;
  }
  if (e) {
    fsvd_tile_model_destroy(m);
    return e;
  }
  // capture the launches of one step (nothing runs here; the shared-memory attribute of the GEMM
  // kernel is raised to the device limit first, outside the capture)
  if (cudaFuncSetAttribute(tile_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, g_smem_optin - 1024) != cudaSuccess) {
    fsvd_tile_model_destroy(m);
    return launch_failed("cudaFuncSetAttribute failed for the tile kernel");
  }
  const cudaStream_t cs = side.st;
  if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) e = fail(FSVD_ERR_CUDA, "stream capture failed");
  if (!e) {
    const long long before = fsvd_tile_launches();
    e = tile_model_record(m, cs);
    m->launches_per_step = fsvd_tile_launches() - before;
    fsvd_tile_count_launches(-m->launches_per_step);   // recorded, not run
    cudaGraph_t g = nullptr;
    if (cudaStreamEndCapture(cs, &g) != cudaSuccess || !g) e = e ? e : fail(FSVD_ERR_CUDA, "stream capture failed");
    m->graph = g;
  }
  if (!e && cudaGraphInstantiate(&m->exec, m->graph, 0) != cudaSuccess) e = fail(FSVD_ERR_CUDA, "cudaGraphInstantiate failed");
  if (!e && side.wait() != cudaSuccess) e = fail(FSVD_ERR_CUDA, "clearing model scratch failed");
  if (e) {
    fsvd_tile_model_destroy(m);
    return e;
  }
  *out = m;
  return 0;
}

int fsvd_tile_model_step(fsvd_tile_model* m, int n_steps, void* stream) {
  for (int i = 0; i < n_steps; ++i) {
    if (cudaGraphLaunch(m->exec, (cudaStream_t)stream) != cudaSuccess) return fail(FSVD_ERR_CUDA, "cudaGraphLaunch failed");
    fsvd_tile_count_launches(m->launches_per_step);
  }
  return 0;
}

void fsvd_tile_model_buffers(fsvd_tile_model* m, int** tokens, int** seqlens, int** token_log, int** step_counter,
                             float** logits, float** hidden) {
  if (tokens) *tokens = m->tokens;
  if (seqlens) *seqlens = m->seqlens;
  if (token_log) *token_log = m->token_log;
  if (step_counter) *step_counter = m->step_counter;
  if (logits) *logits = m->logits;
  if (hidden) *hidden = reinterpret_cast<float*>(m->xbuf[m->D.n_layers & 1]);
}
void* fsvd_tile_model_ws(fsvd_tile_model* m) { return m->ws; }
int fsvd_tile_model_launches_per_step(fsvd_tile_model* m) { return (int)m->launches_per_step; }
int fsvd_tile_model_reset(fsvd_tile_model* m, void* stream) {
  if (cudaMemsetAsync(m->ws + m->L.sync, 0, m->L.xn - m->L.sync, (cudaStream_t)stream) != cudaSuccess)
    return fail(FSVD_ERR_CUDA, "cudaMemsetAsync failed");
  return 0;
}

// ---- prompt pass (kernels in fsvd_prompt.cuh)
// Rows of a pass at most.  What a pass keeps per row is allocated with the program, for the longest pass its
// caches can take: a run allocates and frees nothing, and a graph that has captured one keeps valid addresses.
constexpr int kPromptRows = 2048;
static int prompt_pass_positions(const fsvd_dims& D) { return std::min(D.S_max, std::max(1, kPromptRows / D.B)); }
enum PromptW { PW_QKV, PW_QU, PW_KU, PW_VU, PW_OV, PW_OU, PW_UG, PW_GU, PW_UU, PW_DV, PW_DU, PW_COUNT };
enum PromptX { PX_XN, PX_PQ, PX_PK, PX_PV, PX_ATTN, PX_PO, PX_PUP, PX_PGATE, PX_HACT, PX_PD, PX_COUNT };

struct fsvd_tile_prompt {
  fsvd_dims D;                       // D.B = sequences
  std::vector<fsvd_layer> lw;
  std::vector<CUtensorMap> wmaps;    // [layer][PW_COUNT]
  CUtensorMap xmaps[PX_COUNT];
  const void *embed = nullptr, *final_norm = nullptr, *cos_tab = nullptr, *sin_tab = nullptr;
  // the decode model's buffers: positions are read and advanced, the last position's token and logits go there
  int *tokens = nullptr, *seqlens = nullptr, *step_counter = nullptr, *token_log = nullptr;
  float* logits = nullptr;
  int max_steps = 0;
  long long wait_limit = 0;
  SyncState* sync = nullptr;         // the decode model's
  __nv_bfloat16* last = nullptr;     // normalised last rows
  char* ws = nullptr;                // rows of everything below
  int *rowpos = nullptr, *rowseq = nullptr;
  __nv_bfloat16 *x = nullptr, *mid = nullptr, *xn = nullptr, *pbuf = nullptr, *qbuf = nullptr, *attn = nullptr, *hact = nullptr;
  GemmPlan head;
};

int fsvd_tile_prompt_destroy(fsvd_tile_prompt* p) {
  if (!p) return 0;
  cudaFree(p->last);
  cudaFree(p->ws);
  delete p;
  return 0;
}

// Scratch for the rows of the longest pass.
static int prompt_scratch(fsvd_tile_prompt* p) {
  const fsvd_dims& D = p->D;
  // whole tiles: with 2045 rows, the last tile partly outside the tensor maps, 2041 positions through 4 layers of the 7B
  // shape took 3.07 ms, with 2048 rows 2.92
  const int rows = (prompt_pass_positions(D) * D.B + kTileM - 1) / kTileM * kTileM;
  const int HD = D.H * D.Dh, Rqkv = D.Rq + D.Rk + D.Rv, Rmlp = D.Ru + D.Rg;
  const int pw = imax(imax(Rqkv, Rmlp), imax(D.Ro, D.Rd));
  const size_t n = (size_t)rows;
  const size_t bytes[] = {n * 4, n * 4, n * D.d * 2, n * D.d * 2, n * D.d * 2, n * pw * 2, n * HD * 2, n * HD * 2, n * D.I * 2};
  size_t total = 0, off[9];
  for (int i = 0; i < 9; ++i) {
    off[i] = total;
    total += al256(bytes[i]);
  }
  // (not cleared: the rows past a pass's last one, multiplied too, reach only accumulator rows that are never stored)
  if (cudaMalloc(&p->ws, total) != cudaSuccess) return launch_failed("allocating prompt scratch failed");
  p->rowpos = reinterpret_cast<int*>(p->ws + off[0]);
  p->rowseq = reinterpret_cast<int*>(p->ws + off[1]);
  __nv_bfloat16** t[] = {&p->x, &p->mid, &p->xn, &p->pbuf, &p->qbuf, &p->attn, &p->hact};
  for (int i = 0; i < 7; ++i) *t[i] = reinterpret_cast<__nv_bfloat16*>(p->ws + off[2 + i]);
  const struct { const __nv_bfloat16* base; int K, ld; } f[PX_COUNT] = {
      {p->xn, D.d, D.d}, {p->pbuf, D.Rq, Rqkv}, {p->pbuf + D.Rq, D.Rk, Rqkv}, {p->pbuf + D.Rq + D.Rk, D.Rv, Rqkv}, {p->attn, HD, HD},
      {p->pbuf, D.Ro, D.Ro}, {p->pbuf, D.Ru, Rmlp}, {p->pbuf + D.Ru, D.Rg, Rmlp}, {p->hact, D.I, D.I}, {p->pbuf, D.Rd, D.Rd}};
  for (int i = 0; i < PX_COUNT; ++i)
    if (int e = encode_sw128(&p->xmaps[i], f[i].base, rows, f[i].K, f[i].ld, kTileM)) return e;
  return 0;
}

int fsvd_tile_prompt_create(const fsvd_dims* dims, const fsvd_layer* layers, const void* embed, const void* final_norm_w,
                            const void* lm_head, const void* cos_tab, const void* sin_tab, const fsvd_tile_decode_state* st,
                            long long wait_limit, fsvd_tile_prompt** out) {
  const fsvd_dims& D = *dims;
  if (int e = device_limits()) return e;
  if (int e = check_tile_dims(D)) return e;
  if (D.n_layers < 1 || D.vocab < 1) return fail(FSVD_ERR_ARG, "n_layers / vocab");
  fsvd_tile_prompt* p = new fsvd_tile_prompt();
  p->D = D;
  p->lw.assign(layers, layers + D.n_layers);
  p->embed = embed;
  p->final_norm = final_norm_w;
  p->cos_tab = cos_tab;
  p->sin_tab = sin_tab;
  p->tokens = st->tokens; p->seqlens = st->seqlens; p->step_counter = st->step_counter; p->token_log = st->token_log;
  p->logits = st->logits;
  p->max_steps = st->max_steps;
  p->wait_limit = wait_limit;
  p->sync = reinterpret_cast<SyncState*>(st->ws);
  int e = cudaMalloc(&p->last, (size_t)D.B * D.d * 2) == cudaSuccess ? prompt_scratch(p) : launch_failed("allocating prompt scratch failed");
  const int HD = D.H * D.Dh, KD = D.Hk * D.Dh;
  p->wmaps.resize((size_t)D.n_layers * PW_COUNT);
  for (int l = 0; l < D.n_layers && !e; ++l) {
    const fsvd_layer& w = layers[l];
    CUtensorMap* m = &p->wmaps[(size_t)l * PW_COUNT];
    const struct { const void* base; int rows, K; } f[PW_COUNT] = {
        {w.qkv_v, D.Rq + D.Rk + D.Rv, D.d}, {w.q_u, HD, D.Rq}, {w.k_u, KD, D.Rk}, {w.v_u, KD, D.Rv}, {w.o_v, D.Ro, HD}, {w.o_u, D.d, D.Ro},
        {w.upgate_v, D.Ru + D.Rg, D.d}, {w.gate_u, D.I, D.Rg}, {w.up_u, D.I, D.Ru}, {w.down_v, D.Rd, D.I}, {w.down_u, D.d, D.Rd}};
    for (int i = 0; i < PW_COUNT && !e; ++i) e = encode_sw128(&m[i], f[i].base, f[i].rows, f[i].K, f[i].K, kPgBoxRows);
  }
  if (!e) {
    Scratch sc = {&p->sync->status, wait_limit};
    e = plan_gemm(p->head, lm_head, nullptr, D.vocab, D.d, D.d, p->last, nullptr, D.d, D.B, TE_STORE_F32, sc);
    p->head.a.out = p->logits;
  }
  if (e) {
    fsvd_tile_prompt_destroy(p);
    return e;
  }
  *out = p;
  return 0;
}

struct PgSpec {   // one problem of a launch
  int w, w2, x, x2, P, K, epi;
  void* out;
  const void* resid;
  void* cache;
};
// N of a tile: the value with the shortest estimate of waves x k-blocks x (fetch of a k-block at 64
// bytes per clock and SM, or its multiply-adds at 4096 per clock, whichever is longer).
static int pg_tile_n(const PgSpec* sp, int n, int tiles_m, int quantum, bool two) {
  long long best = -1;
  int nt = quantum;
  for (int c = kPgBoxRows; c <= (two ? kPgBufCols / 2 : kPgBufCols); c += kPgBoxRows) {
    if (c % quantum) continue;
    long long tiles = 0;
    int nkb = 0;
    for (int i = 0; i < n; ++i) {
      tiles += (long long)tiles_m * ((sp[i].P + c - 1) / c);
      nkb = imax(nkb, (sp[i].K + kTileK - 1) / kTileK);
    }
    const long long kb = imax((kTileM + c) * 128 / 64, 2 * c) * (two ? 2 : 1);
    const long long cost = (tiles + g_sms - 1) / g_sms * (nkb * kb + 600);
    if (best < 0 || cost < best) {
      best = cost;
      nt = c;
    }
  }
  return nt;
}
static int launch_prompt_gemm(fsvd_tile_prompt* p, int layer, const PgSpec* sp, int n, int rows, cudaStream_t st) {
  PgArgs a;
  memset(&a, 0, sizeof(a));
  const fsvd_dims& D = p->D;
  a.nprob = n;
  a.rows = rows;
  a.tiles_m = (rows + kTileM - 1) / kTileM;
  a.rowpos = p->rowpos; a.rowseq = p->rowseq; a.cos_tab = p->cos_tab; a.sin_tab = p->sin_tab;
  a.Dh = D.Dh; a.HkDh = D.Hk * D.Dh; a.S_max = D.S_max;
  a.status = &p->sync->status;
  a.wait_limit = p->wait_limit;
  const bool two = sp[0].w2 >= 0;
  const bool rope = sp[0].epi == TE_ROPE_Q;
  const int nt = pg_tile_n(sp, n, a.tiles_m, rope ? D.Dh : kPgBoxRows, two);
  const CUtensorMap* wm = &p->wmaps[(size_t)layer * PW_COUNT];
  for (int i = 0; i < n; ++i) {
    PgProblem& q = a.pr[i];
    q.W = wm[sp[i].w];
    q.X = p->xmaps[sp[i].x];
    if (two) {
      q.W2 = wm[sp[i].w2];
      q.X2 = p->xmaps[sp[i].x2];
    }
    q.P = sp[i].P;
    q.nkb = (sp[i].K + kTileK - 1) / kTileK;
    q.nt = nt;
    q.tile0 = a.total;
    q.epi = sp[i].epi;
    q.two = two ? 1 : 0;
    q.out = sp[i].out; q.resid = sp[i].resid; q.cache = sp[i].cache;
    a.total += a.tiles_m * ((q.P + nt - 1) / nt);
  }
  a.stage_bytes = (kTileM + nt) * 128 * (two ? 2 : 1);
  a.nstages = (g_smem_optin - 4096) / a.stage_bytes;
  if (a.nstages > kPgMaxStages) a.nstages = kPgMaxStages;
  const int grid = a.total < g_sms ? a.total : g_sms;
  static SmemLimit limit;
  if (limit.raise(prompt_gemm_kernel, g_smem_optin - 2048) != cudaSuccess)
    return launch_failed("cudaFuncSetAttribute failed for the prompt kernel");
  if (launch_pdl(prompt_gemm_kernel, dim3((unsigned)grid), dim3(kPgThreads), (size_t)1024 + (size_t)a.nstages * a.stage_bytes, st, a) != cudaSuccess)
    return launch_failed("prompt kernel launch failed");
  fsvd_tile_count_launch();
  return 0;
}

// prompt: device int32 [D.B, >= L] with row stride ld.
int fsvd_tile_prompt_run(fsvd_tile_prompt* p, const int* prompt, int ld, int L, void* stream) {
  const fsvd_dims& D = p->D;
  cudaStream_t st = (cudaStream_t)stream;
  const int most = prompt_pass_positions(D);
  const int passes = (L + most - 1) / most, len = (L + passes - 1) / passes;
  const int HD = D.H * D.Dh, KD = D.Hk * D.Dh, Rqkv = D.Rq + D.Rk + D.Rv;
  int e = 0;   // after a launch that failed nothing more is launched: no layer over stale rows, no position moved
  auto launched = [&](cudaError_t ce) {
    if (ce != cudaSuccess) e = launch_failed("prompt kernel launch failed");
    else fsvd_tile_count_launch();
  };
  auto norm = [&](const __nv_bfloat16* x, const void* w, __nv_bfloat16* out, int rows, int mul, int off) {
    if (!e)
      launched(launch_pdl(rmsnorm_rows_kernel<true>, dim3((unsigned)rows), dim3(256), 0, st, x, reinterpret_cast<const __nv_bfloat16*>(w),
                          out, D.d, D.eps, mul, off));
  };
  for (int off = 0; off < L; off += len) {
    const int n = L - off < len ? L - off : len, rows = n * D.B;
    launched(launch_pdl(prompt_begin_kernel, dim3((unsigned)rows), dim3(128), 0, st, reinterpret_cast<const __nv_bfloat16*>(p->embed),
                        prompt, ld, off, n, (const int*)p->seqlens, p->rowpos, p->rowseq, p->x, D.d, D.vocab));
    PaArgs pa;
    pa.q = p->qbuf; pa.rowpos = p->rowpos; pa.rowseq = p->rowseq; pa.out = p->attn;
    pa.L = n; pa.H = D.H; pa.Hk = D.Hk; pa.S_max = D.S_max;
    pa.scale_log2 = 1.4426950408889634f / sqrtf((float)D.Dh);
    for (int l = 0; l < D.n_layers; ++l) {
      const fsvd_layer& w = p->lw[l];
      auto gemm = [&](std::initializer_list<PgSpec> sp) {
        if (!e) e = launch_prompt_gemm(p, l, sp.begin(), (int)sp.size(), rows, st);
      };
      norm(p->x, w.ln1_w, p->xn, rows, 1, 0);
      gemm({{PW_QKV, -1, PX_XN, -1, Rqkv, D.d, TE_STORE, p->pbuf, nullptr, nullptr}});
      gemm({{PW_QU, -1, PX_PQ, -1, HD, D.Rq, TE_ROPE_Q, p->qbuf, nullptr, nullptr},
            {PW_KU, -1, PX_PK, -1, KD, D.Rk, TE_ROPE_K, nullptr, nullptr, w.k_cache},
            {PW_VU, -1, PX_PV, -1, KD, D.Rv, TE_VCACHE, nullptr, nullptr, w.v_cache}});
      pa.kcache = reinterpret_cast<const __nv_bfloat16*>(w.k_cache);
      pa.vcache = reinterpret_cast<const __nv_bfloat16*>(w.v_cache);
      if (!e) e = launch_prompt_attn(pa, D.Dh, D.B, st);
      gemm({{PW_OV, -1, PX_ATTN, -1, D.Ro, HD, TE_STORE, p->pbuf, nullptr, nullptr}});
      gemm({{PW_OU, -1, PX_PO, -1, D.d, D.Ro, TE_RESID, p->mid, p->x, nullptr}});
      norm(p->mid, w.ln2_w, p->xn, rows, 1, 0);
      gemm({{PW_UG, -1, PX_XN, -1, D.Ru + D.Rg, D.d, TE_STORE, p->pbuf, nullptr, nullptr}});
      gemm({{PW_GU, PW_UU, PX_PGATE, PX_PUP, D.I, D.Rg, TE_SWIGLU, p->hact, nullptr, nullptr}});
      gemm({{PW_DV, -1, PX_HACT, -1, D.Rd, D.I, TE_STORE, p->pbuf, nullptr, nullptr}});
      gemm({{PW_DU, -1, PX_PD, -1, D.d, D.Rd, TE_RESID, p->x, p->mid, nullptr}});
      if (e) return e;
    }
    if (off + n < L) {
      launched(launch_pdl(advance_kernel, dim3(1), dim3(128), 0, st, p->seqlens, D.B, n));
      if (e) return e;
      continue;
    }
    // the last position of every sequence: final norm, head, argmax
    norm(p->x, p->final_norm, p->last, D.B, n, n - 1);
    if (!e) e = launch_gemm(p->head, st);
    if (!e)
      launched(launch_pdl(argmax_rows_kernel, dim3(D.B), dim3(256), 0, st, (const float*)p->logits, D.vocab, p->tokens, p->token_log,
                          p->step_counter, p->seqlens, p->max_steps, D.B, n));
    if (!e) launched(launch_pdl(bump_step_kernel, dim3(1), dim3(1), 0, st, p->step_counter));
  }
  return e;
}
void* fsvd_tile_prompt_ws(fsvd_tile_prompt* p) { return p->sync; }

// Debugging aid: while a device buffer is set, every GEMM CTA planned afterwards records nine
// %globaltimer marks (entry, set-up done, dependency met, accumulators done, cluster barrier 1,
// partial sums sent, cluster barrier 2, epilogue done, exit) at [cta][16]; later launches overwrite
// earlier ones.  Not part of the public header.
// Host arithmetic of the planner, callable without a device (unit tests): the K split of a GEMM of
// `tiles` row tiles and `nkb` k-blocks on `sms` SMs, and the segment count the three q / k / v lifts
// can share (0 = none: they go out as separate launches).
extern "C" void fsvd_tile_debug_split_k(int tiles, int nkb, int sms, int* segs, int* kbs) {
  split_k(tiles, nkb, sms, *segs, *kbs);
}
extern "C" int fsvd_tile_debug_common_segments(int nkb_q, int nkb_k, int nkb_v, int segs_q, int segs_k, int segs_v) {
  return common_segments(nkb_q, nkb_k, nkb_v, segs_q, segs_k, segs_v);
}

extern "C" void fsvd_tile_debug_trace(void* dev_ptr) { g_tile_trace = reinterpret_cast<unsigned long long*>(dev_ptr); }
extern "C" void fsvd_tile_debug_trace_epilogue(int epi) { g_tile_trace_epi = epi; }   // -1: every GEMM
