// C ABI of batched mode: one persistent launch (optionally replayed from a captured CUDA graph)
// for many independent transpositions, each with the schedule of its own plan.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <memory>
#include <vector>

#include "../../include/ttcb200.h"
#include "batch_kernels.cuh"
#include "launch.h"
#include "plan.h"

namespace ttcb {
BatchKernelRef pick_batch_ss(int);
BatchKernelRef pick_batch_dd(int);
BatchKernelRef pick_batch_cc(int);
BatchKernelRef pick_batch_zz(int);
BatchKernelRef pick_batch_sd(int);
BatchKernelRef pick_batch_ds(int);
BatchKernelRef pick_batch_cz(int);
BatchKernelRef pick_batch_zc(int);

BatchKernelRef pick_batch_kernel(ttcb_dtype ta, ttcb_dtype tb, int variant) {
  if (ta == TTCB_S && tb == TTCB_S) return pick_batch_ss(variant);
  if (ta == TTCB_D && tb == TTCB_D) return pick_batch_dd(variant);
  if (ta == TTCB_C && tb == TTCB_C) return pick_batch_cc(variant);
  if (ta == TTCB_Z && tb == TTCB_Z) return pick_batch_zz(variant);
  if (ta == TTCB_S && tb == TTCB_D) return pick_batch_sd(variant);
  if (ta == TTCB_D && tb == TTCB_S) return pick_batch_ds(variant);
  if (ta == TTCB_C && tb == TTCB_Z) return pick_batch_cz(variant);
  if (ta == TTCB_Z && tb == TTCB_C) return pick_batch_zc(variant);
  return BatchKernelRef();
}
}  // namespace ttcb

struct ttcb_batch {
  int count = 0;
  ttcb_dtype ta = TTCB_S, tb = TTCB_S;
  int beta_nonzero = 0;
  bool streaming = false;
  int device = 0;
  unsigned char alpha[16] = {0};
  unsigned char beta[16] = {0};
  int64_t bytes = 0;
  unsigned int nseg = 0;
  int blocks = 0;
  int smem = 0;                       // the ring (or a ragged tile's stage and tables)
  void* d_segs = nullptr;             // ttcb::BatchSeg[nseg]
  unsigned char* d_desc = nullptr;    // the problems' descriptors
  unsigned int* d_counter = nullptr;  // segments claimed, CTAs finished, status
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  cudaStream_t capture_stream = nullptr;
};

// The thread-local last-error message lives in abi.cu.
extern "C" void ttcb_internal_set_error(const char* msg);
static ttcb_status bfail(ttcb_status s, const std::string& msg) {
  ttcb_internal_set_error(msg.c_str());
  return s;
}
static ttcb_status bcuda(cudaError_t e, const char* what) {
  return bfail(TTCB_ERR_CUDA, std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

static void batch_free(ttcb_batch* b) {
  if (!b) return;
  if (b->graph_exec) cudaGraphExecDestroy(b->graph_exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->capture_stream) cudaStreamDestroy(b->capture_stream);
  if (b->d_segs) cudaFree(b->d_segs);
  if (b->d_desc) cudaFree(b->d_desc);
  if (b->d_counter) cudaFree(b->d_counter);
  delete b;
}

static int batch_variant(const ttcb_batch* b) { return b->beta_nonzero ? 2 : (b->streaming ? 1 : 0); }

extern "C" {

ttcb_status ttcb_batch_create(ttcb_batch** out, int count, const ttcb_plan* const* plans, const void* const* A,
                              void* const* B, const void* alpha, const void* beta, int blocks) {
  if (!out) return bfail(TTCB_ERR_INVALID_ARG, "batch output pointer is NULL");
  *out = nullptr;
  if (count < 1 || !plans || !A || !B || !alpha) return bfail(TTCB_ERR_INVALID_ARG, "empty batch or NULL argument");
  const ttcb_plan* p0 = plans[0];
  if (!p0) return bfail(TTCB_ERR_INVALID_ARG, "plan 0 is NULL");
  if (p0->beta_nonzero && !beta) return bfail(TTCB_ERR_BETA, "plans were created for beta != 0 but beta is NULL");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return bcuda(e, "cudaGetDevice");
  const int EA = dtype_bytes(p0->ta), EB = dtype_bytes(p0->tb);

  ttcb_batch* b = new (std::nothrow) ttcb_batch();
  if (!b) return bfail(TTCB_ERR_ALLOC, "host allocation of the batch failed");
  b->count = count;
  b->ta = p0->ta;
  b->tb = p0->tb;
  b->beta_nonzero = p0->beta_nonzero;
  b->streaming = p0->streaming;
  b->device = dev;
  std::memcpy(b->alpha, alpha, EA);
  if (p0->beta_nonzero) std::memcpy(b->beta, beta, EB);

  // Problems of the batch: every plan, and for a plan whose ragged tiles its edge plans move, those
  // edge plans as problems of their own (offset into the plan's A and B).
  struct Entry {
    const ttcb_plan* p;
    const void* A;
    void* B;
    int edges;      // its ragged tiles are problems of their own (the edge plans that follow it)
    int own;        // 1: the caller's plan itself (0: one of its edge plans)
  };
  std::vector<Entry> ent;
  ent.reserve(count);
  for (int i = 0; i < count; ++i) {
    const ttcb_plan* p = plans[i];
    if (!p) {
      batch_free(b);
      return bfail(TTCB_ERR_INVALID_ARG, "plan " + std::to_string(i) + " is NULL");
    }
    if (p->ta != b->ta || p->tb != b->tb || p->beta_nonzero != b->beta_nonzero) {
      batch_free(b);
      return bfail(TTCB_ERR_INVALID_ARG, "all plans of a batch need the same types and beta flag");
    }
    if (p->device != dev && !p->empty) {
      batch_free(b);
      return bfail(TTCB_ERR_INVALID_ARG, "plan " + std::to_string(i) + " belongs to another device");
    }
    if (!p->empty && (!A[i] || !B[i])) {
      batch_free(b);
      return bfail(TTCB_ERR_INVALID_ARG, "A or B of problem " + std::to_string(i) + " is NULL");
    }
    const bool edges = !p->empty && p->kernel == TTCB_KERNEL_TILE && p->nedge > 0;
    ent.push_back({p, A[i], B[i], edges ? 1 : 0, 1});
    for (int k = 0; edges && k < p->nedge; ++k) {
      const ttcb_plan* q = p->edge[k];
      ent.push_back({q, static_cast<const char*>(A[i]) + q->base_offA * EA,
                     static_cast<char*>(B[i]) + q->base_offB * EB, 0, 0});
    }
  }
  // The batched kernel stages A in the plain layout (element p at p + (p / sigmaA) * padA); a plan
  // with shifted A runs takes part through a host copy of itself planned without them.
  std::vector<std::unique_ptr<ttcb_plan>> unshifted;
  for (Entry& e : ent) {
    const ttcb_plan* p = e.p;
    if (p->empty || p->kernel != TTCB_KERNEL_TILE) continue;
    if (!reinterpret_cast<const TileDesc*>(p->host_desc.data())->shiftA) continue;
    std::unique_ptr<ttcb_plan> q(new (std::nothrow) ttcb_plan());
    if (!q) {
      batch_free(b);
      return bfail(TTCB_ERR_ALLOC, "host allocation of a batch problem failed");
    }
    q->rank = p->rank;
    for (int i = 0; i < p->rank; ++i) {
      q->perm[i] = p->perm[i];
      q->size[i] = p->size[i];
      q->lda[i] = p->lda[i];
      q->ldb[i] = p->ldb[i];
    }
    q->ta = p->ta;
    q->tb = p->tb;
    q->beta_nonzero = p->beta_nonzero;
    q->tuning = p->tuning;
    q->tuning.shifted_runs = -1;
    q->depth = p->depth;
    q->base_offA = p->base_offA;
    q->base_offB = p->base_offB;
    q->device = p->device;
    std::string err;
    if (plan_build_host(q.get(), err) != TTCB_OK || q->kernel != TTCB_KERNEL_TILE ||
        q->host_desc.size() < sizeof(TileDesc)) {
      batch_free(b);
      return bfail(TTCB_ERR_UNSUPPORTED, "a batch problem could not be planned for the batched kernel: " + err);
    }
    // the batch moves the complete tiles of the same grid: the tile must not change
    const TileDesc* a = reinterpret_cast<const TileDesc*>(p->host_desc.data());
    const TileDesc* c = reinterpret_cast<const TileDesc*>(q->host_desc.data());
    if (a->P != c->P || a->ntiles != c->ntiles || a->nfull != c->nfull) {
      batch_free(b);
      return bfail(TTCB_ERR_UNSUPPORTED, "a batch problem planned without shifted runs changed its tiles");
    }
    e.p = q.get();
    unshifted.push_back(std::move(q));
  }
  const int n = (int)ent.size();
  b->count = n;

  // descriptors back to back, 16-byte aligned
  std::vector<int64_t> desc_off(n, -1);
  int64_t desc_bytes = 0;
  for (int i = 0; i < n; ++i) {
    if (!ent[i].p->empty) {
      desc_off[i] = desc_bytes;
      desc_bytes += (ent[i].p->host_desc.size() + 15) & ~size_t(15);
    }
  }
  std::vector<unsigned char> hdesc(std::max<int64_t>(desc_bytes, 16), 0);
  const bool beta_nz = b->beta_nonzero != 0;
  // One record per problem, then its segments: runs of at most kSegTiles tiles of about target bytes
  // (set below, once the grid is known).
  std::vector<ttcb::BatchSeg> prob(n);
  int max_stage = 0, max_ragged = 0;
  for (int i = 0; i < n; ++i) {
    const ttcb_plan* p = ent[i].p;
    ttcb::BatchSeg& q = prob[i];
    std::memset(&q, 0, sizeof(q));
    if (p->empty) continue;
    std::memcpy(hdesc.data() + desc_off[i], p->host_desc.data(), p->host_desc.size());
    q.A = ent[i].A;
    q.B = ent[i].B;
    q.desc = reinterpret_cast<const unsigned char*>((uintptr_t)desc_off[i]);  // its offset, until the upload
    q.va = p->vecA;
    q.vb = p->vecB;
    while (q.va > 1 && (uintptr_t)q.A % (q.va * EA)) q.va /= 2;
    while (q.vb > 1 && (uintptr_t)q.B % (q.vb * EB)) q.vb /= 2;
    if (ent[i].own) b->bytes += ttcb_plan_bytes(p);  // an edge plan's bytes are its parent's
    if (p->kernel == TTCB_KERNEL_ROW) {
      q.kind = ttcb::kSegRows;
      q.va = q.vb = std::min(q.va, q.vb);
      continue;
    }
    const TileDesc* td = reinterpret_cast<const TileDesc*>(p->host_desc.data());
    q.kind = ttcb::kSegFull;
    q.rag_vec = p->rag_inline == ttcb::kRagVec;
    q.P = td->P;
    q.LA = td->LA;
    q.LB = td->LB;
    q.padA = td->padA;
    q.a_bytes = (int)ttcb::al16((size_t)td->stage_elems * EA);
    q.stage_bytes = (int)ttcb::async_stage_bytes(td->stage_elems, td->P, EA, EB, beta_nz);
    q.off_segA = td->off_segA;
    q.off_segB = td->off_segB;
    q.off_gtab = td->off_gtab;
    // (the access widths actually used: half or scalar widths where the kernel has no third)
    const int wa = q.va * EA == 16 ? q.va : q.va * EA == 8 && EA < 8 ? q.va : 1;
    const int wb = q.vb * EB == 16 ? q.vb : q.vb * EB == 8 && EB < 8 ? q.vb : 1;
    q.reg = td->reg_ok && td->P / wa <= 4 * ttcb::kThreads && td->P / wb <= 4 * ttcb::kThreads;
    q.ng = td->ngrid;
    q.divLA = td->divLA;
    q.divLB = td->divLB;
    q.divSigma = td->divSigmaA;
    for (int g = 0; g < td->ngrid; ++g) {
      q.g[g].div = td->g[g].divf;
      q.g[g].sA = td->g[g].strideA;
      q.g[g].sB = td->g[g].strideB;
    }
    max_stage = std::max(max_stage, q.stage_bytes);
    if (!ent[i].edges && td->nrag0 + td->nrag1 > 0)
      max_ragged = std::max(max_ragged, q.stage_bytes + 8 * (td->nsegA + td->nsegB) + 4 * ((td->P + 1) / 2));
  }
  // The ring: what lets batch_min_blocks CTAs share an SM (228 KB less 1 KB and about 4 KB of static shared
  // memory per CTA), more where a tile needs it. At 1024 fp32 problems it holds three stages or more of
  // nine tiles in ten.
  b->smem = std::max({beta_nz ? 72 * 1024 : 52 * 1024, (max_stage + 15) & ~15, (max_ragged + 15) & ~15});
  ttcb::BatchKernelRef k = ttcb::pick_batch_kernel(b->ta, b->tb, batch_variant(b));
  if (!k.func) {
    batch_free(b);
    return bfail(TTCB_ERR_DTYPE, "no batched kernel for this type pair");
  }
  ttcb::allow_large_smem(k.func);
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.func, ttcb::kThreads, b->smem);
  if (e != cudaSuccess || per_sm < 1) {
    batch_free(b);
    return e != cudaSuccess ? bcuda(e, "occupancy query") : bfail(TTCB_ERR_UNSUPPORTED, "batch tile too large");
  }
  const int64_t most = blocks > 0 ? blocks : (int64_t)per_sm * sms;
  // About twelve segments per CTA, at most 128 KB: fewer and longer ones leave the CTAs on more problems at
  // once, far apart in memory, and a longer tail (1024 problems of 105 Ki elements: 284 us with twelve,
  // 296 with eight, 334 with four; 303 with 24)
  const int64_t target = std::min<int64_t>(std::max<int64_t>(b->bytes / (12 * most), 16 * 1024), 128 * 1024);
  std::vector<ttcb::BatchSeg> segs;
  std::vector<std::pair<int64_t, uint32_t>> order;  // (key, segment): largest first
  const int64_t elem = EA + EB * (beta_nz ? 2 : 1);
  auto cut = [&](const ttcb::BatchSeg& q, int kind, int64_t items, int64_t item_bytes, int limit) {
    const int64_t per = std::min<int64_t>(std::max<int64_t>(target / std::max<int64_t>(item_bytes, 1), 1), limit);
    const int64_t pieces = (items + per - 1) / per;
    for (int64_t j = 0, t = 0; j < pieces; ++j) {
      const int64_t m = (items - t + (pieces - j) - 1) / (pieces - j);
      ttcb::BatchSeg s = q;
      s.kind = kind;
      s.t0 = (uint32_t)t;
      s.nt = (int32_t)m;
      const int64_t weight = m * item_bytes + 8192;  // (a segment's start costs about as much as 8 KB)
      const int64_t bucket = (int64_t)(2.0 * std::log2((double)weight));
      order.push_back({-(bucket * 1024 + kind * 256 + q.va * 16 + q.vb), (uint32_t)segs.size()});
      segs.push_back(s);
      t += m;
    }
  };
  for (int i = 0; i < n; ++i) {
    const ttcb_plan* p = ent[i].p;
    if (p->empty) continue;
    ttcb::BatchSeg& q = prob[i];
    if (q.kind == ttcb::kSegRows) {
      const RowDesc* rd = reinterpret_cast<const RowDesc*>(p->host_desc.data());
      cut(q, ttcb::kSegRows, (rd->nunits + 7) / 8, 8 * (int64_t)rd->chunk * elem, 1 << 20);
      continue;
    }
    const TileDesc* td = reinterpret_cast<const TileDesc*>(p->host_desc.data());
    q.stages = std::min(b->smem / q.stage_bytes, ttcb::kMaxStages);
    cut(q, ttcb::kSegFull, td->nfull, td->P * elem, ttcb::kSegTiles);
    if (!ent[i].edges) cut(q, ttcb::kSegRagged, (int64_t)td->nrag0 + td->nrag1, 4 * td->P * elem, 1 << 20);
  }
  if (segs.size() >= (size_t)1 << 30) {
    batch_free(b);
    return bfail(TTCB_ERR_UNSUPPORTED, "batch too large");
  }
  // The largest segments first, so that the last ones claimed are small; among segments of a size those
  // of one access width together (CTAs of an SM then share their instructions).
  std::stable_sort(order.begin(), order.end(), [](const auto& x, const auto& y) { return x.first < y.first; });
  {
    std::vector<ttcb::BatchSeg> sorted;
    sorted.reserve(segs.size());
    for (const auto& o : order) sorted.push_back(segs[o.second]);
    segs.swap(sorted);
  }
  b->nseg = (unsigned int)segs.size();
  b->blocks = (int)std::max<int64_t>(std::min<int64_t>(most, b->nseg), 1);

  // device copies
  if ((e = cudaMalloc(&b->d_desc, hdesc.size())) != cudaSuccess ||
      (e = cudaMalloc(&b->d_segs, sizeof(ttcb::BatchSeg) * std::max<size_t>(segs.size(), 1))) != cudaSuccess ||
      (e = cudaMalloc(&b->d_counter, 4 * sizeof(unsigned int))) != cudaSuccess) {
    cudaGetLastError();
    batch_free(b);
    return bfail(TTCB_ERR_ALLOC, std::string("cudaMalloc for the batch failed: ") + cudaGetErrorString(e));
  }
  for (ttcb::BatchSeg& s : segs) s.desc = b->d_desc + reinterpret_cast<uintptr_t>(s.desc);
  if ((e = cudaMemcpy(b->d_desc, hdesc.data(), hdesc.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (!segs.empty() && (e = cudaMemcpy(b->d_segs, segs.data(), sizeof(ttcb::BatchSeg) * segs.size(),
                                        cudaMemcpyHostToDevice)) != cudaSuccess) ||
      (e = cudaMemset(b->d_counter, 0, 4 * sizeof(unsigned int))) != cudaSuccess) {
    batch_free(b);
    return bcuda(e, "batch descriptor upload");
  }
  *out = b;
  return TTCB_OK;
}

static ttcb_status batch_enqueue(ttcb_batch* b, cudaStream_t s) {
  if (b->nseg == 0) return TTCB_OK;
  ttcb::BatchKernelRef k = ttcb::pick_batch_kernel(b->ta, b->tb, batch_variant(b));
  cudaError_t e = k.fn(b->d_segs, b->nseg, b->d_counter, b->alpha, b->beta, b->blocks, b->smem, s);
  if (e != cudaSuccess) return bcuda(e, "batched kernel launch");
  return TTCB_OK;
}

ttcb_status ttcb_batch_launch(ttcb_batch* b, ttcb_stream_t stream) {
  if (!b) return bfail(TTCB_ERR_INVALID_ARG, "batch is NULL");
  return batch_enqueue(b, reinterpret_cast<cudaStream_t>(stream));
}

ttcb_status ttcb_batch_graph_launch(ttcb_batch* b, ttcb_stream_t stream) {
  if (!b) return bfail(TTCB_ERR_INVALID_ARG, "batch is NULL");
  if (b->nseg == 0) return TTCB_OK;
  cudaError_t e;
  if (!b->graph_exec) {
    // capture once on a private stream (the legacy default stream cannot be captured)
    if ((e = cudaStreamCreateWithFlags(&b->capture_stream, cudaStreamNonBlocking)) != cudaSuccess)
      return bcuda(e, "cudaStreamCreate");
    if ((e = cudaStreamBeginCapture(b->capture_stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
      return bcuda(e, "cudaStreamBeginCapture");
    ttcb_status st = batch_enqueue(b, b->capture_stream);
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(b->capture_stream, &g);
    if (st != TTCB_OK) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    if (e != cudaSuccess) return bcuda(e, "cudaStreamEndCapture");
    b->graph = g;
    if ((e = cudaGraphInstantiate(&b->graph_exec, g, 0)) != cudaSuccess) {
      b->graph_exec = nullptr;
      return bcuda(e, "cudaGraphInstantiate");
    }
  }
  if ((e = cudaGraphLaunch(b->graph_exec, reinterpret_cast<cudaStream_t>(stream))) != cudaSuccess)
    return bcuda(e, "cudaGraphLaunch");
  return TTCB_OK;
}

ttcb_status ttcb_batch_status(ttcb_batch* b, ttcb_stream_t stream) {
  if (!b) return bfail(TTCB_ERR_INVALID_ARG, "batch is NULL");
  int st = 0;
  cudaError_t e = cudaMemcpyAsync(&st, b->d_counter + 2, sizeof(int), cudaMemcpyDeviceToHost,
                                  reinterpret_cast<cudaStream_t>(stream));
  if (e == cudaSuccess) e = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return bcuda(e, "batch status read");
  if (st != 0) return bfail(TTCB_ERR_INVALID_ARG, "batched kernel reported status " + std::to_string(st));
  return TTCB_OK;
}

int ttcb_test_batch_segment(ttcb_batch* b, unsigned int k, int kind, int nt, int stages) {
  if (!b || k >= b->nseg) return -1;
  ttcb::BatchSeg s;
  unsigned char* at = static_cast<unsigned char*>(b->d_segs) + sizeof(s) * k;
  if (cudaMemcpy(&s, at, sizeof(s), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  const int was = s.kind;
  if (kind >= 0) s.kind = kind;
  if (nt >= 0) s.nt = nt;
  if (stages >= 0) s.stages = stages;
  if (cudaMemcpy(at, &s, sizeof(s), cudaMemcpyHostToDevice) != cudaSuccess) return -1;
  return was;
}

int64_t ttcb_batch_bytes(const ttcb_batch* b) { return b ? b->bytes : 0; }

void ttcb_batch_destroy(ttcb_batch* b) { batch_free(b); }

}  // extern "C"
