// Batched mode: thousands of independent transpositions in one persistent launch.
//
// Every problem keeps the schedule of its own plan (tile shape, access widths, loop order). The work is
// cut into segments when the batch is made: a run of up to kSegTiles complete tiles, of ragged tiles, or
// of row units (one per warp) of one problem. A CTA takes two segments round robin and then claims them
// from a counter, so long and short problems balance across the GPU. Nothing waits on another CTA.
#pragma once
#include "../../include/ttcb200.h"
#include "kernels.cuh"

namespace ttcb {

enum { kSegFull = 1, kSegRows = 2, kSegRagged = 3 };
constexpr int kSegTiles = 128;  // decoded at once, a thread each

// A segment, and what its problem's complete tiles need of the plan's descriptor (the rest is read
// through desc): a CTA brings the next segment's record while it works on this one.
struct BatchSeg {
  const void* A;
  void* B;
  const unsigned char* desc;  // TileDesc or RowDesc, followed by its tables (device memory)
  int32_t kind;               // kSegFull, kSegRows, kSegRagged
  int32_t va, vb;             // access widths for this problem (1 = scalar)
  int32_t nt;                 // tiles (complete or ragged) or groups of 8 row units
  uint32_t t0;                // the first
  int32_t rag_vec;            // ragged tiles: by vectors (see kRagVec)
  int32_t P, LA, LB, padA;
  int32_t stages;             // ring stages that fit the batch's ring (1 .. kMaxStages)
  int32_t a_bytes, stage_bytes;
  int32_t off_segA, off_segB, off_gtab;
  int32_t reg;                // every thread's offsets fit the register path
  int32_t ng;
  FastDiv divLA, divLB, divSigma;
  struct Grid {
    FastDiv div;  // complete-tile count of the dimension
    int64_t sA, sB;
  } g[TTCB_MAXR];
};
static_assert(sizeof(BatchSeg) % 16 == 0, "records are copied by 16 bytes");

// Batch status codes written by the device (0 = ok): a TTCB_ERR_* code.
enum { kBatchBadSegment = TTCB_ERR_INVALID_ARG };

// Whether a segment's record is one that batch_kernel knows, within `smem` bytes of dynamic shared memory.
__device__ __forceinline__ bool segment_ok(const BatchSeg& s, uint32_t smem) {
  if (s.nt < 1) return false;
  if (s.kind == kSegFull)
    return s.nt <= kSegTiles && s.stages >= 1 && s.stages <= kMaxStages && s.stage_bytes > 0 &&
           (uint64_t)s.stages * (uint32_t)s.stage_bytes <= smem;
  return s.kind == kSegRows || (s.kind == kSegRagged && s.stage_bytes > 0 && (uint32_t)s.stage_bytes <= smem);
}

// CTAs per SM that the register budget is sized for: 4 (64 registers), or 3 when B is read back too, as
// the staged kernel's. What bounds a batch is latency: a segment starts with its tables and its first copies
// (about 4 us under load), and other CTAs have to cover that. 1024 fp32 problems of 105 Ki elements on
// average: 357 us with two CTAs and a problem search per claim, 326 with three, 284 with four.
constexpr int batch_min_blocks(bool beta) { return beta ? 3 : 4; }

// The complete tiles of a segment, through a ring of s.stages stages of which stages - 2 are in flight
// (none in a ring of one or two) and one CTA barrier per tile, as in the staged kernel. Each thread
// computes its tile-relative offsets once per segment, from the tables in global memory, when they fit
// registers (s.reg: at most kRegVec vectors per thread and side), else per vector. info: the segment's tiles
// (A and B base), decoded before the call's barrier; `next`: started with the first copies.
template <typename TA, typename TB, int VA, int VB, bool BETA, bool STREAM, typename Next>
__device__ __forceinline__ void batch_tiles(const BatchSeg& s, const int64_t (*info)[2], TA alpha, TB beta,
                                            unsigned char* smem, const Next& next) {
  const int tid = threadIdx.x;
  const TA* __restrict__ A = static_cast<const TA*>(s.A);
  TB* __restrict__ B = static_cast<TB*>(s.B);
  const int P = s.P, nvA = P / VA, nvB = P / VB;
  const bool reg = s.reg;
  const int64_t* segA = reinterpret_cast<const int64_t*>(s.desc + s.off_segA);
  const int64_t* segB = reinterpret_cast<const int64_t*>(s.desc + s.off_segB);
  const uint16_t* gtab = reinterpret_cast<const uint16_t*>(s.desc + s.off_gtab);
  // register path: A source offsets, staged byte offsets (two per register), B offsets, gather byte
  // offsets (two per register) of the thread's vectors u = tid + k * kThreads
  int32_t rA[kRegVec], rB[kRegVec];
  uint32_t dA[kRegVec / 2];
  constexpr int kGp = (kRegVec * VB + 1) / 2;
  uint32_t gp[kGp];
#pragma unroll
  for (int e = 0; e < kGp; ++e) gp[e] = 0;
#pragma unroll
  for (int u = 0; u < kRegVec; ++u) {
    rA[u] = rB[u] = 0;
    if (!(u & 1)) dA[u >> 1] = 0;
    const int i = tid + u * kThreads;
    if (reg && i < nvA) {
      const int p = i * VA, sg = (int)fdiv((uint32_t)p, s.divLA);
      rA[u] = (int32_t)__ldg(segA + sg) + (p - sg * s.LA);
      dA[u >> 1] |= ((uint32_t)(p + (int)fdiv((uint32_t)p, s.divSigma) * s.padA) * (uint32_t)sizeof(TA)) << ((u & 1) * 16);
    }
    if (reg && i < nvB) {
      const int q = i * VB, sg = (int)fdiv((uint32_t)q, s.divLB);
      rB[u] = (int32_t)__ldg(segB + sg) + (q - sg * s.LB);
      uint16_t pos[VB];
      ld_u16s<TA, VB>(gtab + q, pos);
#pragma unroll
      for (int j = 0; j < VB; ++j) {
        const int e = u * VB + j;
        gp[e >> 1] |= ((uint32_t)pos[j] * (uint32_t)sizeof(TA)) << ((e & 1) * 16);
      }
    }
  }
  const uint32_t stage0 = smem_u32(smem);
  auto issue = [&](int k, int stage) {
    const TA* At = A + info[k][0];
    const TB* Bt = B + info[k][1];
    const uint32_t sb = stage0 + (uint32_t)(stage * s.stage_bytes), sbB = sb + (uint32_t)s.a_bytes;
    if (reg) {
#pragma unroll
      for (int u = 0; u < kRegVec; ++u) {
        if (tid + u * kThreads < nvA)
          cp_async<VA * sizeof(TA)>(sb + ((dA[u >> 1] >> ((u & 1) * 16)) & 0xffffu), At + rA[u]);
        if (BETA && tid + u * kThreads < nvB)
          cp_async<VB * sizeof(TB)>(sbB + (uint32_t)((tid + u * kThreads) * VB * (int)sizeof(TB)), Bt + rB[u]);
      }
    } else {
      for (int i = tid; i < nvA; i += kThreads) {
        const int p = i * VA, sg = (int)fdiv((uint32_t)p, s.divLA);
        cp_async<VA * sizeof(TA)>(sb + (uint32_t)((p + (int)fdiv((uint32_t)p, s.divSigma) * s.padA) * (int)sizeof(TA)),
                                  At + (__ldg(segA + sg) + (p - sg * s.LA)));
      }
      if (BETA) {
        for (int i = tid; i < nvB; i += kThreads) {
          const int q = i * VB, sg = (int)fdiv((uint32_t)q, s.divLB);
          cp_async<VB * sizeof(TB)>(sbB + (uint32_t)(q * (int)sizeof(TB)), Bt + (__ldg(segB + sg) + (q - sg * s.LB)));
        }
      }
    }
  };
  // one B vector: gather VB staged elements (byte offsets from the stage base), scale, combine, store
  auto out_vec = [&](const unsigned char* st, int q, const uint32_t* off, TB* dst) {
    Vec<TB, VB> out, bv;
    if (BETA) bv = *reinterpret_cast<const Vec<TB, VB>*>(st + s.a_bytes + q * (int)sizeof(TB));
#pragma unroll
    for (int j = 0; j < VB; ++j) {
      const TA tj = scale_a(alpha, *reinterpret_cast<const TA*>(st + off[j]));
      if (BETA)
        out.v[j] = combine<TA, TB>(tj, bv.v[j], beta);
      else
        out.v[j] = finish<TA, TB>(tj);
    }
    st_vec<TB, VB>(dst, out, STREAM);
  };
  const int S = s.stages, D = S > 2 ? S - 2 : 0, nt = s.nt;
  __syncthreads();  // the decoded tiles
  next();
  for (int j = 0; j < D; ++j) {
    if (j < nt) issue(j, j);
    cp_async_commit();
  }
  int cur = 0, nxt = D;  // stages of tiles k and k + D
  for (int k = 0; k < nt; ++k) {
    if (k + D < nt) issue(k + D, nxt);
    cp_async_commit();
    switch (D) {  // tile k's copies are complete once at most D groups are pending
      case 0: cp_async_wait<0>(); break;
      case 1: cp_async_wait<1>(); break;
      case 2: cp_async_wait<2>(); break;
      case 3: cp_async_wait<3>(); break;
      case 4: cp_async_wait<4>(); break;
      default: cp_async_wait<5>(); break;
    }
    __syncthreads();
    const unsigned char* st = smem + cur * s.stage_bytes;
    TB* Bt = B + info[k][1];
    if (reg) {
#pragma unroll
      for (int u = 0; u < kRegVec; ++u) {
        if (tid + u * kThreads < nvB) {
          uint32_t off[VB];
#pragma unroll
          for (int j = 0; j < VB; ++j) {
            const int e = u * VB + j;
            off[j] = (e & 1) ? (gp[e >> 1] >> 16) : (gp[e >> 1] & 0xffffu);
          }
          out_vec(st, (tid + u * kThreads) * VB, off, Bt + rB[u]);
        }
      }
    } else {
      for (int i = tid; i < nvB; i += kThreads) {
        const int q = i * VB, sg = (int)fdiv((uint32_t)q, s.divLB);
        uint16_t pos[VB];
        ld_u16s<TA, VB>(gtab + q, pos);
        uint32_t off[VB];
#pragma unroll
        for (int j = 0; j < VB; ++j) off[j] = (uint32_t)pos[j] * (uint32_t)sizeof(TA);
        out_vec(st, q, off, Bt + (__ldg(segB + sg) + (q - sg * s.LB)));
      }
    }
    if (S == 1) __syncthreads();  // the next tile is copied into the same stage
    cur = cur + 1 >= S ? 0 : cur + 1;
    nxt = nxt + 1 >= S ? 0 : nxt + 1;
  }
}

// The ragged tiles of a segment: descriptor header and tables in shared memory (one stage, run tables,
// gather table).
template <typename TA, typename TB, bool BETA, bool STREAM>
__device__ __noinline__ void batch_ragged(const BatchSeg& s, TA alpha, TB beta, TileDesc& d, TileInfo* info,
                                          unsigned char* smem) {
  constexpr int MA = 16 / sizeof(TA), MB = 16 / sizeof(TB);
  for (int i = threadIdx.x; i < (int)(sizeof(TileDesc) / 4); i += kThreads)
    reinterpret_cast<uint32_t*>(&d)[i] = reinterpret_cast<const uint32_t*>(s.desc)[i];
  __syncthreads();
  int64_t* segA = reinterpret_cast<int64_t*>(smem + s.stage_bytes);
  uint16_t* gtab = reinterpret_cast<uint16_t*>(segA + d.nsegA + d.nsegB);
  const TA* A = static_cast<const TA*>(s.A);
  TB* B = static_cast<TB*>(s.B);
  if (s.rag_vec && s.va == MA && s.vb == MB)
    ragged_pass<TA, TB, MA, MB, BETA, STREAM>(d, s.desc, A, B, alpha, beta, smem, s.a_bytes, s.stage_bytes, segA, gtab,
                                              info, 0, 1, s.t0, s.t0 + (uint32_t)s.nt, 1);
  else
    ragged_pass<TA, TB, 1, 1, BETA, STREAM>(d, s.desc, A, B, alpha, beta, smem, s.a_bytes, s.stage_bytes, segA, gtab,
                                            info, 0, 1, s.t0, s.t0 + (uint32_t)s.nt, 1);
}

template <typename TA, typename TB, bool BETA, bool STREAM>
__device__ __noinline__ void batch_rows(const BatchSeg& s, TA alpha, TB beta) {
  const RowDesc& d = *reinterpret_cast<const RowDesc*>(s.desc);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int MA = 16 / sizeof(TA);
  constexpr int MB = 16 / sizeof(TB);
  constexpr int MR = MA < MB ? MA : MB;
  const TA* A = static_cast<const TA*>(s.A);
  TB* B = static_cast<TB*>(s.B);
  for (int k = 0; k < s.nt; ++k) {
    const uint32_t u = (s.t0 + (uint32_t)k) * (kThreads / 32) + warp;
    if (u >= (uint32_t)d.nunits) break;
    if (s.va == MR && s.vb == MR)
      row_unit<TA, TB, MR, BETA, STREAM>(d, u, A, B, alpha, beta, lane);
    else
      row_unit<TA, TB, 1, BETA, STREAM>(d, u, A, B, alpha, beta, lane);
  }
}

// counter[0]: segments claimed, counter[1]: finished CTAs; the last one sets both back to zero.
// counter[2]: the first error; a segment whose record is not a sound one is left out. CTA b
// takes segments b and b + gridDim.x first; each further claim is issued two segments ahead and each record
// copied one ahead, so neither is waited for.
template <typename TA, typename TB, bool BETA, bool STREAM>
__global__ void __launch_bounds__(kThreads, batch_min_blocks(BETA))
    batch_kernel(const BatchSeg* __restrict__ segs, unsigned int nseg, unsigned int* __restrict__ counter, TA alpha,
                 TB beta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) BatchSeg rec[2];
  __shared__ int64_t tiles[kSegTiles][2];
  __shared__ TileDesc d;      // ragged tiles
  __shared__ TileInfo rag[1];
  __shared__ unsigned int s_next;
  constexpr int MA = 16 / sizeof(TA);
  constexpr int MB = 16 / sizeof(TB);
  constexpr int HA = MA >= 2 ? MA / 2 : 1;  // the half-width vectors (8 bytes) where they differ
  constexpr int HB = MB >= 2 ? MB / 2 : 1;
  constexpr int kRec16 = (int)(sizeof(BatchSeg) / 16);
  const int tid = threadIdx.x;
  const unsigned int G = gridDim.x;
  unsigned int next = blockIdx.x + G, pending = nseg;  // thread 0: the next segment and the one after it
  const bool claiming = 2 * G < nseg;
  if (blockIdx.x < nseg && tid < kRec16)
    cp_async<16>(smem_u32(&rec[0]) + tid * 16, reinterpret_cast<const unsigned char*>(segs + blockIdx.x) + tid * 16);
  if (claiming && tid == 0) pending = 2 * G + atomicAdd(&counter[0], 1u);
  for (int cur = 0; blockIdx.x < nseg; cur ^= 1) {
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();  // the record is there, and every thread is done with the segment before
    const BatchSeg& s = rec[cur];
    if (tid == 0) {
      s_next = next;
      next = pending;
      if (claiming) pending = 2 * G + atomicAdd(&counter[0], 1u);
    }
    auto prefetch = [&]() {
      const unsigned int n = s_next;
      if (n < nseg && tid < kRec16)
        cp_async<16>(smem_u32(&rec[cur ^ 1]) + tid * 16, reinterpret_cast<const unsigned char*>(segs + n) + tid * 16);
    };
    uint32_t smem;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(smem));
    const bool ok = segment_ok(s, smem);
    if (ok && s.kind == kSegFull) {
      if (tid < s.nt) {
        uint32_t t = s.t0 + (uint32_t)tid;
        int64_t bA = 0, bB = 0;
        for (int g = 0; g < s.ng; ++g) {
          const uint32_t q = fdiv(t, s.g[g].div), blk = t - q * s.g[g].div.d;
          t = q;
          bA += (int64_t)blk * s.g[g].sA;
          bB += (int64_t)blk * s.g[g].sB;
        }
        tiles[tid][0] = bA;
        tiles[tid][1] = bB;
      }
      const int va = s.va >= MA ? MA : (s.va >= HA ? HA : 1);
      const int vb = s.vb >= MB ? MB : (s.vb >= HB ? HB : 1);
#define TTCB_BATCH_TILES(VA_, VB_) batch_tiles<TA, TB, VA_, VB_, BETA, STREAM>(s, tiles, alpha, beta, smem_raw, prefetch)
      if (va == MA) {
        if (vb == MB) TTCB_BATCH_TILES(MA, MB);
        else if (vb == HB) TTCB_BATCH_TILES(MA, HB);
        else TTCB_BATCH_TILES(MA, 1);
      } else if (va == HA) {
        if (vb == MB) TTCB_BATCH_TILES(HA, MB);
        else if (vb == HB) TTCB_BATCH_TILES(HA, HB);
        else TTCB_BATCH_TILES(HA, 1);
      } else {
        if (vb == MB) TTCB_BATCH_TILES(1, MB);
        else if (vb == HB) TTCB_BATCH_TILES(1, HB);
        else TTCB_BATCH_TILES(1, 1);
      }
#undef TTCB_BATCH_TILES
    } else {
      __syncthreads();
      prefetch();
      if (!ok) {
        if (tid == 0) atomicCAS(&counter[2], 0u, (unsigned int)kBatchBadSegment);
      } else if (s.kind == kSegRows)
        batch_rows<TA, TB, BETA, STREAM>(s, alpha, beta);
      else
        batch_ragged<TA, TB, BETA, STREAM>(s, alpha, beta, d, rag, smem_raw);
    }
    if (s_next >= nseg) break;
  }
  if (claiming && tid == 0) {
    __threadfence();
    if (atomicAdd(&counter[1], 1u) == G - 1) {
      atomicExch(&counter[0], 0u);
      atomicExch(&counter[1], 0u);
      __threadfence();
    }
  }
}

}  // namespace ttcb
