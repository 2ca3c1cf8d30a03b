// Prompt pass: the factor products of many prompt positions at once, and their causal attention.
//
// A pass takes up to kPromptRows rows = (sequence, position) pairs through all layers.  With hundreds
// of rows a factor product is a dense contraction, bound by the tensor cores and by what the SMs can
// fetch from L2:
//     D[128 rows, N factor rows] = X[128 rows, K] . W[N factor rows, K]^T,   N = 64, 128, 192 or 256
// with the activations as the M side, so that a thread of the epilogue holds consecutive outputs of
// one row and stores 16 bytes at a time.  One persistent CTA per SM walks the tiles of the launch (row
// tile fastest: the CTAs that run together read one factor tile from L2): three producer threads keep a
// ring of {X tile, W tile} k-blocks filled by TMA (a k-block is up to five boxes, and one thread that waits,
// arms and issues them all was what the ring waited for: 2041 positions through 4 layers of the 7B shape 3.39 ms
// with one, 3.12 ms with three; 6 prompts of 190 1.70 and 1.56 ms), another thread issues the tcgen05.mma,
// four warps run the epilogue of the tile before out of the other half of tensor memory.
//
// Included by fsvd_tile.cu (shares its launch helpers).
#pragma once
#include "fsvd_tc.cuh"

namespace fsvd_tile {

constexpr int kPgThreads = 256;      // warp 1 MMA, warps 2..5 epilogue, warps 0, 6, 7 producers
constexpr int kPgProducers = 3;      // a ring slot always belongs to the same one: slot % kPgProducers
constexpr int kPgMaxStages = 8;
constexpr int kPgBufCols = 256;      // tensor-memory columns of an accumulator buffer (two buffers)
constexpr int kPgBoxRows = 64;       // factor rows of a TMA box
constexpr int kPgMaxProblems = 3;

struct PgProblem {
  CUtensorMap X, X2, W, W2;          // X2 / W2: second accumulator (TE_SWIGLU)
  int P, nkb, nt, tile0;             // factor rows, k-blocks, N of a tile, first tile of the problem
  int epi, two;
  void* out;                         // bf16 [rows, P] (TE_STORE, TE_RESID, TE_SWIGLU, TE_ROPE_Q)
  const void* resid;
  void* cache;                       // TE_ROPE_K / TE_VCACHE
};
struct PgArgs {
  PgProblem pr[kPgMaxProblems];
  int nprob, rows, tiles_m, total, nstages, stage_bytes;
  const int *rowpos, *rowseq;        // position and cache row of every row
  const void *cos_tab, *sin_tab;
  int Dh, HkDh, S_max;
  int* status;
  long long wait_limit;
};

// 32 consecutive accumulator columns of this thread's lane
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 outputs of one row, 8 at a time; `n` of them (a multiple of 8) exist
__device__ __forceinline__ void store32(__nv_bfloat16* dst, const float (&v)[32], int n) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (8 * q < n)
      reinterpret_cast<uint4*>(dst)[q] = make_uint4(pack_bf16(v[8 * q], v[8 * q + 1]), pack_bf16(v[8 * q + 2], v[8 * q + 3]),
                                                    pack_bf16(v[8 * q + 4], v[8 * q + 5]), pack_bf16(v[8 * q + 6], v[8 * q + 7]));
}
__device__ __forceinline__ void load32(const __nv_bfloat16* src, float (&v)[32], int n) {
  uint4 t[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = 8 * q < n ? reinterpret_cast<const uint4*>(src)[q] : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t w[4] = {t[q].x, t[q].y, t[q].z, t[q].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[8 * q + 2 * i] = __uint_as_float(w[i] << 16);
      v[8 * q + 2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
}
__device__ __forceinline__ void mbar_arrive_local(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct PgTile {
  int p, m, n;   // problem, row tile, factor tile
};
__device__ __forceinline__ PgTile pg_tile(const PgArgs& a, int tile) {
  PgTile t;
  t.p = 0;
#pragma unroll
  for (int i = 1; i < kPgMaxProblems; ++i)
    if (i < a.nprob && tile >= a.pr[i].tile0) t.p = i;
  const int l = tile - a.pr[t.p].tile0;
  t.n = l / a.tiles_m;
  t.m = l - t.n * a.tiles_m;
  return t;
}

__global__ void __launch_bounds__(kPgThreads, 1) prompt_gemm_kernel(const __grid_constant__ PgArgs a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * kPgMaxStages + 4];
  __shared__ uint32_t tmem_slot;
  __shared__ int giveup_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NS = a.nstages;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kPgMaxStages]);
  const uint32_t afull0 = smem_u32(&bars[2 * kPgMaxStages]), aempty0 = smem_u32(&bars[2 * kPgMaxStages + 2]);
  volatile int* giveup = &giveup_sh;
  if (tid == 0) {
    giveup_sh = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(afull0 + 8 * i, 1);
      mbar_init(aempty0 + 8 * i, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    __syncwarp();
    tc_alloc(smem_u32(&tmem_slot), 2 * kPgBufCols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0 || warp >= 6) {
    if (lane == 0) {
      const int pj = warp == 0 ? 0 : warp - 5;
      int s = 0, round = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < a.total && ok; tile += gridDim.x) {
        const PgTile t = pg_tile(a, tile);
        const PgProblem& pr = a.pr[t.p];
        const uint32_t wbytes = (uint32_t)pr.nt * 128u;
        const uint32_t bytes = (kTileM * 128u + wbytes) * (pr.two ? 2u : 1u);
        for (int kb = 0; kb < pr.nkb; ++kb) {
          if (s % kPgProducers != pj) {   // another producer's slot
            if (++s == NS) {
              s = 0;
              ++round;
            }
            continue;
          }
          if (round > 0 && !(ok = wait_bar(empty0 + 8 * s, (uint32_t)(round - 1) & 1u, giveup, a.status, a.wait_limit, DS_COPY_TIMEOUT))) break;
          const uint32_t fb = full0 + 8 * s;
          uint32_t dst = base + (uint32_t)s * (uint32_t)a.stage_bytes;
          const int kcol = kb * kTileK;
          mbar_expect_tx(fb, bytes);
          tma_box_2d(dst, &pr.X, kcol, t.m * kTileM, fb);
          dst += kTileM * 128u;
          for (int r = 0; r < pr.nt; r += kPgBoxRows) tma_box_2d(dst + (uint32_t)r * 128u, &pr.W, kcol, t.n * pr.nt + r, fb);
          dst += wbytes;
          if (pr.two) {
            tma_box_2d(dst, &pr.X2, kcol, t.m * kTileM, fb);
            dst += kTileM * 128u;
            for (int r = 0; r < pr.nt; r += kPgBoxRows) tma_box_2d(dst + (uint32_t)r * 128u, &pr.W2, kcol, t.n * pr.nt + r, fb);
          }
          if (++s == NS) {
            s = 0;
            ++round;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0, round = 0, cnt = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < a.total && ok; tile += gridDim.x, ++cnt) {
        const PgTile t = pg_tile(a, tile);
        const PgProblem& pr = a.pr[t.p];
        const uint32_t idesc = umma_idesc(pr.nt), wbytes = (uint32_t)pr.nt * 128u;
        const int buf = cnt & 1, use = cnt >> 1;
        if (use > 0 && !(ok = wait_bar(aempty0 + 8 * buf, (uint32_t)(use - 1) & 1u, giveup, a.status, a.wait_limit, DS_BARRIER_TIMEOUT))) break;
        tc_fence_after();
        const uint32_t d0 = tmem + (uint32_t)(buf * kPgBufCols);
        for (int kb = 0; kb < pr.nkb; ++kb) {
          if (!(ok = wait_bar(full0 + 8 * s, (uint32_t)round & 1u, giveup, a.status, a.wait_limit, DS_COPY_TIMEOUT))) break;
          tc_fence_after();
          const uint32_t sx = base + (uint32_t)s * (uint32_t)a.stage_bytes, sw = sx + kTileM * 128u;
          const uint64_t dx = umma_desc(sx), dw = umma_desc(sw);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; ++kk)
            tc_mma(d0, dx + 2u * kk, dw + 2u * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          if (pr.two) {
            const uint64_t dx2 = umma_desc(sw + wbytes), dw2 = umma_desc(sw + wbytes + kTileM * 128u);
#pragma unroll
            for (int kk = 0; kk < kTileK / 16; ++kk)
              tc_mma(d0 + (uint32_t)(kPgBufCols / 2), dx2 + 2u * kk, dw2 + 2u * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit(empty0 + 8 * s);
          if (++s == NS) {
            s = 0;
            ++round;
          }
        }
        if (ok) tc_commit(afull0 + 8 * buf);
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue: warp w reads accumulator lanes 32 (w % 4) .. + 31; thread = one row of the tile
    const int ew = warp & 3;
    const uint32_t tlane = (uint32_t)(ew * 32) << 16;
    int cnt = 0;
    for (int tile = blockIdx.x; tile < a.total; tile += gridDim.x, ++cnt) {
      const PgTile t = pg_tile(a, tile);
      const PgProblem& pr = a.pr[t.p];
      const int buf = cnt & 1, use = cnt >> 1;
      bool ok = wait_bar(afull0 + 8 * buf, (uint32_t)use & 1u, giveup, a.status, a.wait_limit, DS_BARRIER_TIMEOUT);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint32_t d0 = tmem + tlane + (uint32_t)(buf * kPgBufCols);
      const int row = t.m * kTileM + ew * 32 + lane;
      const bool in = row < a.rows;
      const int p0 = t.n * pr.nt;
      float v[32], u[32];
      if (pr.epi == TE_STORE) {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(pr.out) + (size_t)row * pr.P;
        for (int c = 0; c < pr.nt; c += 32) {
          if (p0 + c >= pr.P) break;
          tc_ld32(d0 + c, v);
          if (in) store32(o + p0 + c, v, pr.P - p0 - c);
        }
      } else if (pr.epi == TE_RESID) {
        const __nv_bfloat16* rs = reinterpret_cast<const __nv_bfloat16*>(pr.resid) + (size_t)row * pr.P;
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(pr.out) + (size_t)row * pr.P;
        for (int c = 0; c < pr.nt; c += 32) {
          if (p0 + c >= pr.P) break;
          load32(rs + p0 + c, u, in ? pr.P - p0 - c : 0);
          tc_ld32(d0 + c, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = u[i] + rnd(v[i]);
          if (in) store32(o + p0 + c, v, pr.P - p0 - c);
        }
      } else if (pr.epi == TE_SWIGLU) {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(pr.out) + (size_t)row * pr.P;
        for (int c = 0; c < pr.nt; c += 32) {
          if (p0 + c >= pr.P) break;
          tc_ld32(d0 + c, v);
          tc_ld32(d0 + kPgBufCols / 2 + c, u);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float g = rnd(v[i]);
            v[i] = rnd(g / (1.0f + expf(-g))) * rnd(u[i]);
          }
          if (in) store32(o + p0 + c, v, pr.P - p0 - c);
        }
      } else {
        const int pos = in ? a.rowpos[row] : 0, half = a.Dh >> 1;
        const bool store = in && (pos < a.S_max || pr.epi == TE_ROPE_Q);
        if (in && pos >= a.S_max) atomicCAS(a.status, (int)DS_OK, (int)DS_CACHE_FULL);
        __nv_bfloat16* o = pr.epi == TE_ROPE_Q
                               ? reinterpret_cast<__nv_bfloat16*>(pr.out) + (size_t)row * pr.P
                               : reinterpret_cast<__nv_bfloat16*>(pr.cache) + ((size_t)(in ? a.rowseq[row] : 0) * a.S_max + pos) * a.HkDh;
        if (pr.epi == TE_VCACHE) {
          for (int c = 0; c < pr.nt; c += 32) {
            if (p0 + c >= pr.P) break;
            tc_ld32(d0 + c, v);
            if (store) store32(o + p0 + c, v, pr.P - p0 - c);
          }
        } else {
          // whole heads (nt is a multiple of Dh): column j of a head rotates with column j + Dh/2
          const size_t tab = (size_t)min(pos, a.S_max - 1) * half;
          const __nv_bfloat16* ct = reinterpret_cast<const __nv_bfloat16*>(a.cos_tab) + tab;
          const __nv_bfloat16* st = reinterpret_cast<const __nv_bfloat16*>(a.sin_tab) + tab;
          for (int h = 0; h < pr.nt; h += a.Dh) {
            if (p0 + h >= pr.P) break;
            for (int j = 0; j < half; j += 32) {
              tc_ld32(d0 + h + j, v);
              tc_ld32(d0 + h + half + j, u);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 cw = reinterpret_cast<const uint4*>(ct + j)[q], sw4 = reinterpret_cast<const uint4*>(st + j)[q];
                const uint32_t cc[4] = {cw.x, cw.y, cw.z, cw.w}, ss[4] = {sw4.x, sw4.y, sw4.z, sw4.w};
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const float cs = __uint_as_float((e & 1) ? (cc[e >> 1] & 0xffff0000u) : (cc[e >> 1] << 16));
                  const float sn = __uint_as_float((e & 1) ? (ss[e >> 1] & 0xffff0000u) : (ss[e >> 1] << 16));
                  const float x1 = rnd(v[8 * q + e]), x2 = rnd(u[8 * q + e]);
                  v[8 * q + e] = rnd(x1 * cs) - rnd(x2 * sn);
                  u[8 * q + e] = rnd(x2 * cs) + rnd(x1 * sn);
                }
              }
              if (store) {
                store32(o + p0 + h + j, v, 32);
                store32(o + p0 + h + half + j, u, 32);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_local(aempty0 + 8 * buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*giveup)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);   // copies in flight towards this CTA land first
  if (warp == 0) tc_dealloc(tmem, 2 * kPgBufCols);
}

// ------------------------------------------------------------------------------- causal attention
// Attention of the rows of a pass over their sequences' caches, which already hold the rows' own keys
// and values.  A CTA takes 64 query vectors of one sequence and kv head (64 / G consecutive positions x
// the G query heads that share the head), 16 per warp; key / value blocks of 64 positions are staged by
// cp.async one block ahead and serve all of them.  S = Q K^T and O += P V on mma.sync m16n8k16 (bf16,
// fp32 accumulation) with fragments taken by ldmatrix; running softmax in base 2; only blocks that reach
// past a query's own position are masked.  Query blocks with the longest range start first.
//
// Softmax weights meet the value rows rounded to bf16, or with all their 24 bits as three bf16 numbers (FULL), so that
// a prompt has no fewer bits than a feed token by token, whose kernels have fp32 weights up to 4 sequences or with 1 or
// 2 heads per kv head.  All rows of several such sequences are FULL.  A single sequence has its last kFullRows positions FULL
// (they decide the first token), by CTAs of their own in front of the others: 16 query vectors, the key blocks dealt
// out to the four warps, which are through long before a block of 64 with as many keys.  The earlier rows are bound
// by mma.sync: 2041 positions through 4 layers of 32 heads of 128 take 2.80 ms with no FULL row, 2.77 like this, 2.90 with
// the last block of 64 rows FULL and 3.12 with all of them; 4 prompts of 180 (all FULL) 1.39 and 1.40 ms.
constexpr int kPaWarps = 4;
constexpr int kPaSlots = 16 * kPaWarps;
constexpr int kPaKeys = 64;
constexpr int kFullRows = 16;
constexpr int kPaTailSlots = 16, kPaTailKeys = 32;   // query vectors of a CTA, keys of a warp's block

struct PaArgs {
  const __nv_bfloat16* q;        // [rows, H, Dh], rotated
  const __nv_bfloat16* kcache;   // [*, S_max, Hk, Dh]
  const __nv_bfloat16* vcache;
  const int* rowpos;             // [rows]: positions of a sequence's rows are consecutive
  const int* rowseq;             // [rows] cache row, or null: cache row 0
  __nv_bfloat16* out;            // [rows, H, Dh]
  int L, H, Hk, S_max;           // rows per sequence
  int full_from;                 // rows of a sequence from here on go to the CTAs of 16 query vectors (L: none)
  float scale_log2;              // softmax scale x log2(e)
};

// Rows r0 .. rlast of the sequence whose first row is seq0.
template <int DH, bool FULL>
__device__ __forceinline__ void prompt_attn_rows(const PaArgs& a, unsigned char* pa_smem, int seq0, int r0, int rlast) {
  constexpr int STRIDE = DH * 2 + 16;                 // bytes of a staged row (padded: no bank conflicts)
  constexpr int KS = DH / 16, NT = kPaKeys / 8, DT = DH / 8, PIECES = DH / 8;
  constexpr int STAGE = 2 * kPaKeys * STRIDE;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int G = a.H / a.Hk, hk = blockIdx.y;
  const int nmax = min(a.rowpos[seq0 + rlast] + 1, a.S_max);   // keys the CTA's last row sees
  const int nfirst = a.rowpos[seq0 + r0] + 1;                  // ... and its first row
  const int m0 = warp * 16 + g;
  int rowq[2], headq[2], nl[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + 8 * i;
    const int r = r0 + m / G;
    rowq[i] = seq0 + min(r, rlast);
    headq[i] = hk * G + m % G;
    nl[i] = r <= rlast ? min(nfirst + m / G, a.S_max) : 0;
  }
  uint32_t qa[KS][4];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const __nv_bfloat16* qp = a.q + ((size_t)rowq[i] * a.H + headq[i]) * DH + ks * 16 + 2 * t;
      qa[ks][i] = *reinterpret_cast<const uint32_t*>(qp);
      qa[ks][2 + i] = *reinterpret_cast<const uint32_t*>(qp + 8);
    }
  }
  float o[DT][4];
#pragma unroll
  for (int d = 0; d < DT; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.0f;
  float mrow[2] = {-INFINITY, -INFINITY}, lrow[2] = {0.0f, 0.0f};
  const size_t rowstride = (size_t)a.Hk * DH;
  const size_t cbase = (size_t)(a.rowseq ? a.rowseq[seq0] : 0) * a.S_max * rowstride + (size_t)hk * DH;
  const __nv_bfloat16* kbase = a.kcache + cbase;
  const __nv_bfloat16* vbase = a.vcache + cbase;
  const uint32_t sm0 = smem_u32(pa_smem);

  auto stage = [&](int k0, int st) {
    const uint32_t dk = sm0 + (uint32_t)(st * STAGE), dv = dk + kPaKeys * STRIDE;
#pragma unroll
    for (int i = tid; i < kPaKeys * PIECES; i += kPaWarps * 32) {
      const int r = i / PIECES, c = i - r * PIECES;
      const size_t src = (size_t)min(k0 + r, nmax - 1) * rowstride + (size_t)c * 8;   // past the end: masked below
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dk + r * STRIDE + c * 16), "l"(kbase + src) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dv + r * STRIDE + c * 16), "l"(vbase + src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0, 0);
  int st = 0;
  for (int k0 = 0; k0 < nmax; k0 += kPaKeys, st ^= 1) {
    if (k0 + kPaKeys < nmax) {
      stage(k0 + kPaKeys, st ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const uint32_t ks_s = sm0 + (uint32_t)(st * STAGE), vs_s = ks_s + kPaKeys * STRIDE;
    // ---- S = Q K^T: 16 query vectors x 64 keys per warp; ldmatrix.x4 of the key rows gives the two
    // k-halves of key tiles 2 j and 2 j + 1
    float sc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.0f;
    const uint32_t kaddr = ks_s + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * STRIDE + ((lane >> 3) & 1) * 16);
#pragma unroll
    for (int j = 0; j < NT / 2; ++j) {
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t b0, b1, b2, b3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(kaddr + (uint32_t)(j * 16 * STRIDE + ks * 32)));
        mma_bf16_16816(sc[2 * j], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
        mma_bf16_16816(sc[2 * j + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
      }
    }
    if (k0 + kPaKeys > nfirst) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (k0 + nt * 8 + 2 * t + (e & 1) >= nl[e >> 1]) sc[nt][e] = -INFINITY;
    }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      mx[0] = fmaxf(mx[0], fmaxf(sc[nt][0], sc[nt][1]));
      mx[1] = fmaxf(mx[1], fmaxf(sc[nt][2], sc[nt][3]));
    }
    float corr[2], mref[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      const float mn = fmaxf(mrow[i], mx[i]);
      mref[i] = mn == -INFINITY ? 0.0f : mn * a.scale_log2;   // nothing visible yet: every weight is 0
      corr[i] = exp2f(mrow[i] * a.scale_log2 - mref[i]);
      mrow[i] = mn;
    }
    float ps[2] = {0.0f, 0.0f};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pr = exp2f(fmaf(sc[nt][e], a.scale_log2, -mref[e >> 1]));
        sc[nt][e] = pr;
        ps[e >> 1] += pr;
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) lrow[i] = lrow[i] * corr[i] + ps[i];   // summed over the row's four lanes at the end
#pragma unroll
    for (int d = 0; d < DT; ++d) {
      o[d][0] *= corr[0]; o[d][1] *= corr[0];
      o[d][2] *= corr[1]; o[d][3] *= corr[1];
    }
#pragma unroll
    for (int kk = 0; kk < kPaKeys / 16; ++kk) {
      constexpr int W = FULL ? 3 : 1;   // bf16 numbers of a weight
      uint32_t p[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float x = sc[2 * kk + (i >> 1)][2 * (i & 1)], y = sc[2 * kk + (i >> 1)][2 * (i & 1) + 1];
        if (FULL) split_bf16(x, y, p[0][i], p[1][i], p[2][i]);
        else p[0][i] = pack_bf16(x, y);
      }
      const uint32_t vaddr = vs_s + (uint32_t)((kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * STRIDE + ((lane >> 4) & 1) * 16);
#pragma unroll
      for (int j = 0; j < DT / 2; ++j) {
        uint32_t b0, b1, b2, b3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(vaddr + j * 32));
#pragma unroll
        for (int w = W - 1; w >= 0; --w) {
          mma_bf16_16816(o[2 * j], p[w][0], p[w][1], p[w][2], p[w][3], b0, b1);
          mma_bf16_16816(o[2 * j + 1], p[w][0], p[w][1], p[w][2], p[w][3], b2, b3);
        }
      }
    }
    __syncthreads();   // the stage is overwritten by the block after the next
  }
  unsigned again[2];   // rows (four lanes each) that met the infinite value of a position they do not see, or of one with a short weight
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 1);
    lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 2);
    bool none = false;   // "no number" among this thread's sums
#pragma unroll
    for (int d = 0; d < DT; ++d) none |= o[d][2 * i] != o[d][2 * i] || o[d][2 * i + 1] != o[d][2 * i + 1];
    again[i] = __ballot_sync(0xffffffffu, nl[i] > 0 && none);
    if (nl[i] == 0 || (again[i] >> (lane & 28) & 15u)) continue;
    const float inv = lrow[i] > 0.0f ? 1.0f / lrow[i] : 0.0f;
    __nv_bfloat16* op = a.out + ((size_t)rowq[i] * a.H + headq[i]) * DH + 2 * t;
#pragma unroll
    for (int d = 0; d < DT; ++d) *reinterpret_cast<uint32_t*>(op + d * 8) = pack_bf16(o[d][2 * i] * inv, o[d][2 * i + 1] * inv);
  }
#pragma unroll 1
  for (int m = 0; m < 16 && (again[0] | again[1]); ++m)   // rows 0 .. 7 and 8 .. 15 of the warp
    if ((m < 8 ? again[0] : again[1]) >> (4 * (m & 7)) & 15u) {
      const int r = r0 + (warp * 16 + m) / G, n = min(nfirst + r - r0, a.S_max);
      const size_t at = ((size_t)(seq0 + r) * a.H + hk * G + (warp * 16 + m) % G) * DH;
      float acc[DH / 32], mm, ll;
      attn_one_row<DH>(a.q + at, kbase, vbase, rowstride, 0, n, n, n, a.scale_log2 * 0.6931471805599453f, acc, &mm, &ll);
#pragma unroll
      for (int e = 0; e < DH / 32; ++e) a.out[at + lane * (DH / 32) + e] = __float2bfloat16_rn(acc[e] / ll);
    }
}

// Rows r0 .. rlast (at most 16 / G of them), the keys in blocks of 32 dealt out to the warps, which merge at the end.
template <int DH>
__device__ __forceinline__ void prompt_attn_tail(const PaArgs& a, unsigned char* pa_smem, int seq0, int r0, int rlast) {
  constexpr int STRIDE = DH * 2 + 16, KS = DH / 16, NT = kPaTailKeys / 8, DT = DH / 8, PIECES = DH / 8;
  constexpr int rec = DH + kPartPad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int G = a.H / a.Hk, hk = blockIdx.y;
  const int nfirst = a.rowpos[seq0 + r0] + 1, nmax = min(a.rowpos[seq0 + rlast] + 1, a.S_max);
  int nl[2];
  uint32_t qa[KS][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = g + 8 * i, r = r0 + m / G;
    nl[i] = r <= rlast ? min(nfirst + m / G, a.S_max) : 0;
    const __nv_bfloat16* qp = a.q + ((size_t)(seq0 + min(r, rlast)) * a.H + hk * G + m % G) * DH + 2 * t;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      qa[ks][i] = *reinterpret_cast<const uint32_t*>(qp + ks * 16);
      qa[ks][2 + i] = *reinterpret_cast<const uint32_t*>(qp + ks * 16 + 8);
    }
  }
  float o[DT][4], mrow[2] = {-INFINITY, -INFINITY}, lrow[2] = {0.0f, 0.0f};   // maxima in units of log2
#pragma unroll
  for (int d = 0; d < DT; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.0f;
  const size_t rowstride = (size_t)a.Hk * DH;
  const size_t cbase = (size_t)(a.rowseq ? a.rowseq[seq0] : 0) * a.S_max * rowstride + (size_t)hk * DH;
  const __nv_bfloat16* kbase = a.kcache + cbase;
  const __nv_bfloat16* vbase = a.vcache + cbase;
  const uint32_t ks_s = smem_u32(pa_smem) + (uint32_t)(warp * 2 * kPaTailKeys * STRIDE), vs_s = ks_s + kPaTailKeys * STRIDE;

  for (int k0 = warp * kPaTailKeys; k0 < nmax; k0 += kPaWarps * kPaTailKeys) {
    __syncwarp();
    for (int i = lane; i < kPaTailKeys * PIECES; i += 32) {
      const int r = i / PIECES, c = i - r * PIECES;
      const size_t src = (size_t)min(k0 + r, nmax - 1) * rowstride + (size_t)c * 8;   // past the end: masked below
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ks_s + r * STRIDE + c * 16), "l"(kbase + src) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vs_s + r * STRIDE + c * 16), "l"(vbase + src) : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    float sc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.0f;
    const uint32_t kaddr = ks_s + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * STRIDE + ((lane >> 3) & 1) * 16);
#pragma unroll
    for (int j = 0; j < NT / 2; ++j) {
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t b0, b1, b2, b3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(kaddr + (uint32_t)(j * 16 * STRIDE + ks * 32)));
        mma_bf16_16816(sc[2 * j], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
        mma_bf16_16816(sc[2 * j + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
      }
    }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sc[nt][e] = k0 + nt * 8 + 2 * t + (e & 1) < nl[e >> 1] ? sc[nt][e] * a.scale_log2 : -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], sc[nt][e]);
      }
    float ps[2] = {0.0f, 0.0f}, mref[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      const float mn = fmaxf(mrow[i], mx[i]);
      mref[i] = mn == -INFINITY ? 0.0f : mn;   // nothing visible yet: every weight is 0
      const float corr = exp2f(mrow[i] - mref[i]);
      mrow[i] = mn;
      lrow[i] *= corr;
#pragma unroll
      for (int d = 0; d < DT; ++d) {
        o[d][2 * i] *= corr;
        o[d][2 * i + 1] *= corr;
      }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sc[nt][e] = exp2f(sc[nt][e] - mref[e >> 1]);
        ps[e >> 1] += sc[nt][e];
      }
    lrow[0] += ps[0];   // (summed over the row's four lanes at the end)
    lrow[1] += ps[1];
#pragma unroll
    for (int kk = 0; kk < kPaTailKeys / 16; ++kk) {
      uint32_t p[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        split_bf16(sc[2 * kk + (i >> 1)][2 * (i & 1)], sc[2 * kk + (i >> 1)][2 * (i & 1) + 1], p[0][i], p[1][i], p[2][i]);
      const uint32_t vaddr = vs_s + (uint32_t)((kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * STRIDE + ((lane >> 4) & 1) * 16);
#pragma unroll
      for (int j = 0; j < DT / 2; ++j) {
        uint32_t b0, b1, b2, b3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(vaddr + j * 32));
#pragma unroll
        for (int w = 2; w >= 0; --w) {
          mma_bf16_16816(o[2 * j], p[w][0], p[w][1], p[w][2], p[w][3], b0, b1);
          mma_bf16_16816(o[2 * j + 1], p[w][0], p[w][1], p[w][2], p[w][3], b2, b3);
        }
      }
    }
  }
  // ---- the warps meet in shared memory (the stages are free): [warp][query vector] records
  __syncthreads();
  float* const recs = reinterpret_cast<float*>(pa_smem);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 1);
    lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 2);
    float* mine = recs + (warp * kPaTailSlots + g + 8 * i) * rec;
    bool none = false;   // "no number" among this thread's sums
#pragma unroll
    for (int d = 0; d < DT; ++d) {
      mine[d * 8 + 2 * t] = o[d][2 * i];
      mine[d * 8 + 2 * t + 1] = o[d][2 * i + 1];
      none |= o[d][2 * i] != o[d][2 * i] || o[d][2 * i + 1] != o[d][2 * i + 1];
    }
    if (t == 0) {
      mine[DH] = mrow[i];
      mine[DH + 1] = lrow[i];
    }
    unsigned again = __ballot_sync(0xffffffffu, nl[i] > 0 && none);
    __syncwarp();
#pragma unroll 1
    for (int m = 8 * i; again; ++m, again >>= 4)
      if (again & 15u) {
        const int r = r0 + m / G;
        float acc[DH / 32], mm, ll;
        attn_one_row<DH>(a.q + ((size_t)(seq0 + r) * a.H + hk * G + m % G) * DH, kbase, vbase, rowstride, warp * kPaTailKeys,
                         min(nfirst + r - r0, a.S_max), kPaTailKeys, kPaWarps * kPaTailKeys, a.scale_log2 * 0.6931471805599453f, acc,
                         &mm, &ll);
        float* to = recs + (warp * kPaTailSlots + m) * rec;
#pragma unroll
        for (int e = 0; e < DH / 32; ++e) to[lane * (DH / 32) + e] = acc[e];
        if (lane == 0) {
          to[DH] = mm * 1.4426950408889634f;
          to[DH + 1] = ll;
        }
      }
  }
  __syncthreads();
  for (int i = tid; i < (rlast - r0 + 1) * G * (DH / 2); i += kPaWarps * 32) {
    const int m = i / (DH / 2), d = 2 * (i - m * (DH / 2));
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kPaWarps; ++w) mm = fmaxf(mm, recs[(w * kPaTailSlots + m) * rec + DH]);
    float x = 0.0f, y = 0.0f, den = 0.0f;
#pragma unroll
    for (int w = 0; w < kPaWarps; ++w) {
      const float* pr = recs + (w * kPaTailSlots + m) * rec;
      const float wgt = pr[DH] == -INFINITY ? 0.0f : exp2f(pr[DH] - mm);
      x += wgt * pr[d];
      y += wgt * pr[d + 1];
      den += wgt * pr[DH + 1];
    }
    const float inv = den > 0.0f ? 1.0f / den : 0.0f;
    *reinterpret_cast<uint32_t*>(a.out + ((size_t)(seq0 + r0 + m / G) * a.H + hk * G + m % G) * DH + d) = pack_bf16(x * inv, y * inv);
  }
}

// (FULL: a CTA less per SM and no spills in the loop; 2 prompts of 100 positions, 4 layers of 32 heads of 128 1183 -> 1161 us, as
// without full weights)
template <int DH, bool FULL>
__global__ void __launch_bounds__(kPaWarps * 32, (DH == 64 ? 4 : 3) - (FULL ? 1 : 0)) prompt_attn_kernel(const PaArgs a) {
  extern __shared__ __align__(16) unsigned char pa_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int G = a.H / a.Hk, seq0 = blockIdx.z * a.L;
  const int tpos = kPaTailSlots / G, ntail = FULL ? 0 : (a.L - a.full_from + tpos - 1) / tpos;
  if ((int)blockIdx.x < ntail) {
    const int r0 = a.full_from + (ntail - 1 - (int)blockIdx.x) * tpos;
    prompt_attn_tail<DH>(a, pa_smem, seq0, r0, min(r0 + tpos, a.L) - 1);
    return;
  }
  const int rpb = kPaSlots / G;                                   // positions per CTA
  const int r0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * rpb;    // first row of the CTA, inside the sequence
  prompt_attn_rows<DH, FULL>(a, pa_smem, seq0, r0, min(r0 + rpb, a.full_from) - 1);
}

}  // namespace fsvd_tile
