// kvt_p2d_attn: the fused P->D paged-KV transfer kernel for sm_100a.
//
// One launch walks the block tables of every request scheduled in a step (the job of the
// reference's CPU ParseBlock generators, kvtransfer/src/parse_block_flash.cpp:10-130,
// parse_block_flashinfer.cpp:15-72, parse_block_ragged.cpp:29-217), converts between cache
// layouts (FlashAttention NHD, FlashInfer HND, ragged, MLA single-tensor), re-shards heads for
// TP-mismatched prefill/decode ranks (group_off placement of parse_block_common.cpp:81-129),
// optionally quantises bf16 -> block-scaled e4m3 (the reference only has an unscaled cast,
// kvtransfer/src/copy_kernels.cu:287-481) and stores straight into the destination cache,
// which may be local memory, a peer GPU's memory mapped over NVLink, or mapped pinned host
// memory.  No staging buffer and no library copy is involved.
//
// Work unit ("tile"): tile_tokens consecutive token slots of one request for one of K / V in
// one layer, all transferred heads.  Copies move with TMA: one elected thread issues a
// cp.async.bulk.tensor load of the {head_bytes, heads, tokens} box into shared memory and a
// cp.async.bulk.tensor store of the same box through a destination map whose strides encode
// the destination layout, so the NHD<->HND permutation is done by the copy engine and the SM
// issues two instructions per 8-32 KiB.  A ragged edge (a chunk that starts or ends inside a
// block) is loaded as a whole tile and leaves as one untiled bulk store per contiguous run of
// its own slots.  fp8 pages inside one GPU are expanded by a kernel of their own, fed by untiled bulk copies; the quantiser,
// other expansions and layouts TMA cannot describe run on a vector SIMT path.  TMA loads never use cluster multicast.
//
// Every wait is bounded; on a bad block id or a timeout the kernel records a status word and
// skips the access instead of faulting.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "kvt_kernels.h"
#include "smem_grant.h"

namespace {

constexpr int kMaxStages = 8;
constexpr int kMaxDevices = 64;
constexpr uint32_t kSmemBudget = 200 * 1024;     // bytes of dynamic shared memory we ask for at most
constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 2 GHz: bound of an mbarrier wait
constexpr uint32_t kStagePayload = 4096;         // quantiser staging per warp: e4m3 payload of a tile ...
constexpr uint32_t kStageScales = 256;           // ... and its scale bytes
constexpr uint32_t kStagePerWarp = kStagePayload + kStageScales;

struct TileInfo {
  uint32_t req;        // request index
  uint32_t tok_lo;     // first absolute token slot of the tile
  uint32_t copy_lo;    // [copy_lo, copy_hi) are copied
  uint32_t copy_hi;
  uint32_t zero_hi;    // [copy_hi', zero_hi) are zero-filled on the destination (tail pad)
  uint32_t sblk, dblk; // physical block ids
  uint32_t s_slot0, d_slot0;
  bool ok;
};

__device__ __forceinline__ void set_status(uint32_t* status, uint32_t code, uint32_t detail) {
  if (status != nullptr) {
    if (atomicCAS(status, 0u, code) == 0u) status[1] = detail;
  }
}

// Where the plan is.  A short one travels in the launch's parameters (IN_LAUNCH): its upload would be a copy in front of the
// kernel and, from Python, a pinned buffer and a device tensor.  us a pass with an uploaded plan / this way, packing included: one
// layer of 333 tokens 33.1 / 8.2, fp8 -> bf16 of 32 layers of 4003 tokens 147 / 137, 24 blocks to host memory 1034 / 999.
// The lanes read it by generic addresses, coalesced as from memory: an index into the parameter space would be served lane by lane.
template <bool IN_LAUNCH>
struct PlanParam {};
template <>
struct PlanParam<true> {
  uint32_t words[KVT_PLAN_IN_LAUNCH / 4u];
};
template <bool IN_LAUNCH>
struct PlanView {
  const KvtReqDesc* reqs;
  const uint32_t* block_ids;
  __device__ __forceinline__ PlanView(const KvtAttnLaunch& p, const PlanParam<IN_LAUNCH>& param) {
    if constexpr (IN_LAUNCH) {
      uint64_t at = reinterpret_cast<uint64_t>(&param.words[0]);
      asm volatile("" : "+l"(at));
      reqs = reinterpret_cast<const KvtReqDesc*>(at);
      block_ids = reinterpret_cast<const uint32_t*>(at + (uint64_t)p.n_reqs * sizeof(KvtReqDesc));
    } else {
      reqs = p.reqs;
      block_ids = p.block_ids;
    }
  }
  __device__ __forceinline__ uint32_t load(const uint32_t* w) const {
    if constexpr (IN_LAUNCH) return *w;
    else return __ldg(w);
  }
};

// Largest r with reqs[r].first_tile <= t.
template <bool IN_LAUNCH>
__device__ __forceinline__ uint32_t find_req(const PlanView<IN_LAUNCH>& plan, uint32_t n, uint32_t t) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (plan.load(&plan.reqs[mid].first_tile) <= t) lo = mid; else hi = mid;
  }
  return lo;
}

template <bool IN_LAUNCH>
__device__ __forceinline__ TileInfo decode_tile(const KvtAttnLaunch& p, const PlanView<IN_LAUNCH>& plan, uint32_t tile) {
  TileInfo ti;
  const uint32_t r = find_req(plan, p.n_reqs, tile);
  const KvtReqDesc rd = plan.reqs[r];
  const uint32_t tt = p.tile_tokens;
  const uint32_t local = tile - rd.first_tile;
  const uint32_t tok_lo = (rd.seen_tokens / tt + local) * tt;
  const uint32_t tok_hi = tok_lo + tt;
  const uint32_t end_tok = rd.seen_tokens + rd.new_tokens;
  uint32_t end_pad = end_tok;
  if (rd.flags & KVT_REQ_PAD_TAIL) {
    end_pad = (end_tok + p.dst.ntpb - 1) / p.dst.ntpb * p.dst.ntpb;
  }
  ti.req = r;
  ti.tok_lo = tok_lo;
  ti.copy_lo = max(rd.seen_tokens, tok_lo);
  ti.copy_hi = max(ti.copy_lo, min(end_tok, tok_hi));
  ti.zero_hi = max(ti.copy_hi, min(end_pad, tok_hi));
  const uint32_t sbi = tok_lo / p.src.ntpb;
  const uint32_t dbi = tok_lo / p.dst.ntpb;
  ti.s_slot0 = tok_lo - sbi * p.src.ntpb;
  ti.d_slot0 = tok_lo - dbi * p.dst.ntpb;
  ti.ok = true;
  ti.sblk = 0;
  ti.dblk = 0;
  const bool need_src = ti.copy_hi > ti.copy_lo;
  if (need_src) {
    if (sbi >= rd.n_src_blocks) {
      ti.ok = false;
    } else {
      ti.sblk = plan.load(&plan.block_ids[rd.src_blk_off + sbi]);
      if (ti.sblk >= p.src.num_blocks) ti.ok = false;
    }
  }
  if (dbi >= rd.n_dst_blocks) {
    ti.ok = false;
  } else {
    ti.dblk = plan.load(&plan.block_ids[rd.dst_blk_off + dbi]);
    if (ti.dblk >= p.dst.num_blocks) ti.ok = false;
  }
  return ti;
}

// Work item w of a launch -> layer, K or V, tile of the layer.
__device__ __forceinline__ void split_work(const KvtAttnLaunch& p, uint64_t w, uint64_t total, uint32_t per_layer,
                                           uint32_t& layer, uint32_t& kv, uint32_t& tile) {
  uint32_t rem;
  if ((total >> 32) == 0u) {   // a 32-bit division costs a fraction of a 64-bit one
    layer = (uint32_t)w / per_layer;
    rem = (uint32_t)w - layer * per_layer;
  } else {
    layer = (uint32_t)(w / per_layer);
    rem = (uint32_t)(w - (uint64_t)layer * per_layer);
  }
  kv = rem / p.total_tiles;
  tile = rem - kv * p.total_tiles;
}

// What is left to do of a tile once it has been decoded: ntok token slots to copy, then nzero to zero on the destination.
struct TileMove {
  uint32_t sblk, dblk, s_slot, d_slot, ntok, nzero, layer, kv;
  __device__ __forceinline__ bool set(const TileInfo& ti) {   // true: something is left
    sblk = ti.sblk;
    dblk = ti.dblk;
    s_slot = ti.s_slot0 + (ti.copy_lo - ti.tok_lo);
    d_slot = ti.d_slot0 + (ti.copy_lo - ti.tok_lo);
    ntok = ti.copy_hi - ti.copy_lo;
    nzero = ti.zero_hi - ti.copy_hi;
    return (ntok | nzero) != 0u;
  }
};
// The move that lane j holds, in every lane of the warp.
__device__ __forceinline__ TileMove move_of_lane(const TileMove& mine, int j) {
  TileMove m;
  m.sblk = __shfl_sync(0xffffffffu, mine.sblk, j);
  m.dblk = __shfl_sync(0xffffffffu, mine.dblk, j);
  m.s_slot = __shfl_sync(0xffffffffu, mine.s_slot, j);
  m.d_slot = __shfl_sync(0xffffffffu, mine.d_slot, j);
  m.ntok = __shfl_sync(0xffffffffu, mine.ntok, j);
  m.nzero = __shfl_sync(0xffffffffu, mine.nzero, j);
  m.layer = __shfl_sync(0xffffffffu, mine.layer, j);
  m.kv = __shfl_sync(0xffffffffu, mine.kv, j);
  return m;
}

// ---- PTX wrappers -----------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* ptr) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(ptr));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ void tma_load_5d(uint32_t smem_dst, const void* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_5d(const void* map, uint32_t smem_src, int c0, int c1, int c2, int c3,
                                             int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.global.shared::cta.bulk_group"
      " [%0, {%2, %3, %4, %5, %6}], [%1];"
      ::"l"(map), "r"(smem_src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void bulk_store_flat(void* gdst, uint32_t smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void tma_load_5d_hint(uint32_t smem_dst, const void* map, uint32_t bar, int c0, int c1,
                                                 int c2, int c3, int c4, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7], %8;"
      ::"r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar), "l"(pol)
      : "memory");
}
__device__ __forceinline__ void tma_store_5d_hint(const void* map, uint32_t smem_src, int c0, int c1, int c2, int c3,
                                                  int c4, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.5d.global.shared::cta.bulk_group.L2::cache_hint"
      " [%0, {%2, %3, %4, %5, %6}], [%1], %7;"
      ::"l"(map), "r"(smem_src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "l"(pol)
      : "memory");
}
__device__ __forceinline__ void bulk_store_flat_hint(void* gdst, uint32_t smem_src, uint32_t bytes, uint64_t pol) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(gdst),
               "r"(smem_src), "r"(bytes), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void bulk_store_run(char* gdst, uint32_t smem_src, uint32_t bytes, bool hinted, uint64_t pol) {
  if (hinted) bulk_store_flat_hint(gdst, smem_src, bytes, pol); else bulk_store_flat(gdst, smem_src, bytes);
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ int4 ld_nc_16(const void* p) {
  int4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st_16(void* p, int4 v) {
  asm volatile("st.global.v4.s32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

__device__ __forceinline__ uint32_t ld_nc_u8(const void* p) {   // volatile: issued here, beside the row's other loads
  uint32_t v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// 32 bytes per thread in one access where the address allows it (sm_100 has 256-bit loads and stores), else two of 16.
__device__ __forceinline__ void ld_nc_32(const void* p, bool aligned32, uint32_t w[8]) {
  if (aligned32) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
  } else {
    const int4 a = ld_nc_16(p), b = ld_nc_16(static_cast<const char*>(p) + 16);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  }
}
__device__ __forceinline__ void st_32(void* p, bool aligned32, const uint32_t w[8]) {
  if (aligned32) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    st_16(p, make_int4(w[0], w[1], w[2], w[3]));
    st_16(static_cast<char*>(p) + 16, make_int4(w[4], w[5], w[6], w[7]));
  }
}

// ---- block-scaled fp8 helpers -----------------------------------------------------------
// Scale of a 32-value group: the smallest power of two s with amax / s <= 448 (e4m3 max), stored
// as a biased UE8M0 exponent byte.  amax == 0 maps to exponent 127 (scale 1).
__device__ __forceinline__ uint32_t ue8m0_from_amax(float amax) {
  if (!(amax > 0.f)) return 127u;
  const float ratio = amax * (1.0f / 448.0f);
  const uint32_t bits = __float_as_uint(ratio);
  int e = static_cast<int>((bits >> 23) & 0xffu);
  const uint32_t mant = bits & 0x7fffffu;
  if (e == 0) {  // subnormal ratio: the smallest normal power of two is already large enough
    return 1u;
  }
  if (mant != 0u) e += 1;  // round the scale up so the largest value does not saturate
  if (e > 254) e = 254;
  if (e < 1) e = 1;
  return static_cast<uint32_t>(e);
}
__device__ __forceinline__ float scale_from_ue8m0(uint32_t e) { return __uint_as_float(e << 23); }

__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Largest magnitude of 16 bf16 values, in packed arithmetic: |x| and max are exact, and a NaN loses against a number
// as it does in fmaxf.
__device__ __forceinline__ float amax_bf16x16(const uint32_t w[8]) {
  __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
  for (int k = 1; k < 8; ++k) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[k])));
  return fmaxf(fmaxf(0.f, __low2float(m)), __high2float(m));
}

__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}

// ---- SIMT tile movers ---------------------------------------------------------------------
// Rows are enumerated in destination order so that consecutive threads write consecutive
// destination addresses (NVLink and PCIe like long contiguous write runs).
//
// Division of chunk numbers of a tile by one divisor: n * ceil(2^32 / d) >> 32 is floor(n / d) as long as n * d < 2^32,
// so for tiles of at most 2^16 chunks.  m == 0: d is 1, or the tile is larger than that and takes the plain division.
struct TileDiv {
  uint32_t d, m;
  __device__ __forceinline__ TileDiv(uint32_t d_, uint32_t chunks)
      : d(d_), m(d_ > 1u && chunks <= 65536u ? 0xffffffffu / d_ + 1u : 0u) {}
  __device__ __forceinline__ uint32_t quot(uint32_t n) const {
    if (m != 0u) return __umulhi(n, m);
    return d == 1u ? n : n / d;
  }
};
// The chunks (16 or 32 bytes) of tiles of one launch: divisors that are the same for every full tile are made once.
struct TileRows {
  uint32_t cpr;          // chunks per row
  bool token_inner;
  TileDiv row_div, full_div;
  __device__ __forceinline__ TileRows(const KvtAttnLaunch& p, uint32_t cpr_)
      : cpr(cpr_), token_inner(p.dst.token_stride < p.dst.head_stride),
        row_div(cpr_, p.tile_tokens * p.n_heads * cpr_),
        full_div(token_inner ? p.tile_tokens : p.n_heads, p.tile_tokens * p.n_heads * cpr_) {}
};
struct RowIter {
  const TileRows& r;
  uint32_t ntok, chunks;
  TileDiv inner_div;
  __device__ __forceinline__ RowIter(const KvtAttnLaunch& p, const TileRows& r_, uint32_t ntok_)
      : r(r_), ntok(ntok_), chunks(ntok_ * p.n_heads * r_.cpr), inner_div(r_.full_div) {
    if (r.token_inner && ntok_ != p.tile_tokens) inner_div = TileDiv(ntok_, chunks);
  }
  // chunk i, counted in destination order -> token, head and chunk of the row
  __device__ __forceinline__ void decode(uint32_t i, uint32_t& t, uint32_t& h, uint32_t& c) const {
    const uint32_t row = r.row_div.quot(i);
    c = i - row * r.cpr;
    const uint32_t q = inner_div.quot(row);
    const uint32_t rest = row - q * inner_div.d;
    t = r.token_inner ? rest : q;
    h = r.token_inner ? q : rest;
  }
};

__device__ __forceinline__ void simt_copy_tile(const KvtAttnLaunch& p, const TileRows& rows, const TileMove& ti,
                                       const char* __restrict__ src, char* __restrict__ dst, uint32_t tid,
                                       uint32_t nthr) {
  const RowIter it(p, rows, ti.ntok);
  const uint32_t chunks = it.chunks;
  const int64_t s_base = (int64_t)ti.sblk * p.src.block_stride + (int64_t)ti.kv * p.src.kv_stride +
                         (int64_t)ti.s_slot * p.src.token_stride +
                         (int64_t)p.src_head0 * p.src.head_stride;
  const int64_t d_base = (int64_t)ti.dblk * p.dst.block_stride + (int64_t)ti.kv * p.dst.kv_stride +
                         (int64_t)ti.d_slot * p.dst.token_stride +
                         (int64_t)p.dst_head0 * p.dst.head_stride;
  constexpr int U = 4;
  for (uint32_t base = tid; base < chunks; base += nthr * U) {
    int4 v[U];
    int64_t doff[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * nthr;
      doff[u] = -1;
      if (i < chunks) {
        uint32_t t, h, c;
        it.decode(i, t, h, c);
        v[u] = ld_nc_16(src + s_base + (int64_t)t * p.src.token_stride + (int64_t)h * p.src.head_stride + (c << 4));
        doff[u] = d_base + (int64_t)t * p.dst.token_stride + (int64_t)h * p.dst.head_stride + (c << 4);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (doff[u] >= 0) st_16(dst + doff[u], v[u]);
    }
  }
}

// Chunk i of a tile (16 bf16 values of a row, in w) -> 16 e4m3 codes at their place behind `rows` and the group's scale
// byte behind `scales` (both the address of the tile's first slot and head).  The lanes of a warp hold consecutive chunks
// and all take part in the shuffles.  With `stage` the tile goes to shared memory instead (see simt_quant_tile).
__device__ __forceinline__ void quant_chunk(const KvtAttnLaunch& p, const RowIter& it, const uint32_t w[8], uint32_t i, bool active,
                                            char* rows, char* scales, bool wide_scales, unsigned char* stage) {
  float amax = amax_bf16x16(w);
  // the partner lane holds the other half of the 32-value group
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  const uint32_t e = ue8m0_from_amax(amax);
  const float inv = __uint_as_float((254u - e) << 23);  // 1 / 2^(e-127)
  uint32_t t, h, c;   // decoded again: cheaper than registers held across the loads
  it.decode(i, t, h, c);
  if (active) {
    int4 q;
    q.x = pack_e4m3x4(bf16lo(w[0]) * inv, bf16hi(w[0]) * inv, bf16lo(w[1]) * inv, bf16hi(w[1]) * inv);
    q.y = pack_e4m3x4(bf16lo(w[2]) * inv, bf16hi(w[2]) * inv, bf16lo(w[3]) * inv, bf16hi(w[3]) * inv);
    q.z = pack_e4m3x4(bf16lo(w[4]) * inv, bf16hi(w[4]) * inv, bf16lo(w[5]) * inv, bf16hi(w[5]) * inv);
    q.w = pack_e4m3x4(bf16lo(w[6]) * inv, bf16hi(w[6]) * inv, bf16lo(w[7]) * inv, bf16hi(w[7]) * inv);
    // staged: chunk i of the tile in destination order sits at byte 16 i of the buffer, rows of a head are adjacent
    if (stage != nullptr) *reinterpret_cast<int4*>(stage + (i << 4)) = q;
    else st_16(rows + (int64_t)t * p.dst.token_stride + (int64_t)h * p.dst.head_stride + (c << 4), q);
  }
  char* sc = scales + (int64_t)t * p.dst.scale_token_stride + (int64_t)h * p.dst.scale_head_stride + (c >> 1);
  if (wide_scales) {
    // eight neighbouring lanes hold 128 values of one row = four scales: one 4-byte store instead of
    // four 1-byte stores (over NVLink every store is a packet of its own, whatever its size)
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t e1 = __shfl_sync(0xffffffffu, e, (lane & ~7u) + 2u);
    const uint32_t e2 = __shfl_sync(0xffffffffu, e, (lane & ~7u) + 4u);
    const uint32_t e3 = __shfl_sync(0xffffffffu, e, (lane & ~7u) + 6u);
    if (active && (lane & 7u) == 0u) {
      const uint32_t packed = e | (e1 << 8) | (e2 << 16) | (e3 << 24);
      // staged: chunk i owns scale byte i / 2; lanes with lane % 8 == 0 hold a multiple of eight, so the word is 4-byte
      // aligned whatever the row length
      if (stage != nullptr) *reinterpret_cast<uint32_t*>(stage + kStagePayload + (i >> 1)) = packed;
      else *reinterpret_cast<uint32_t*>(sc) = packed;
    }
  } else if (active && (c & 1u) == 0u) {
    *sc = static_cast<char>(e);
  }
}

// Scale rows of a multiple of four bytes at 4-byte aligned addresses leave as 32-bit words.
__device__ __forceinline__ bool scales_as_words(const KvtAttnLaunch& p, uint32_t cpr, const char* scales) {
  return (cpr & 7u) == 0u && ((reinterpret_cast<uint64_t>(scales) | (uint64_t)p.dst.scale_token_stride |
                               (uint64_t)p.dst.scale_head_stride) & 3u) == 0u;
}

// bf16 source rows -> e4m3 rows + UE8M0 scales.  One thread converts 16 values (32 B in,
// 16 B out); two neighbouring lanes form one 32-value scale group.
// With `stage` (a warp's own shared-memory buffer, warp-per-tile mode) a full tile bound for an HND
// destination is quantised into shared memory and leaves as one bulk copy per head (payload) plus one
// per head (scales): the async-copy engine writes NVLink packets of 256 bytes where the warp's own
// 16-byte stores leave as 128-byte ones (measured 615 GB/s of link for those against 705 for bulk stores).
__device__ __forceinline__ void simt_quant_tile(const KvtAttnLaunch& p, const TileRows& rows, const TileMove& ti,
                                       const char* __restrict__ src, char* __restrict__ dst, uint32_t tid,
                                       uint32_t nthr, unsigned char* stage) {
  const uint32_t cpr = rows.cpr;  // 32-byte source chunks per row (even: head_dim % 32 == 0)
  const RowIter it(p, rows, ti.ntok);
  const uint32_t chunks = it.chunks;
  const int64_t s_base = (int64_t)ti.sblk * p.src.block_stride + (int64_t)ti.kv * p.src.kv_stride +
                         (int64_t)ti.s_slot * p.src.token_stride + (int64_t)p.src_head0 * p.src.head_stride;
  const int64_t d_blk = (int64_t)ti.dblk * p.dst.block_stride;
  const int64_t d_base = d_blk + (int64_t)ti.kv * p.dst.kv_stride + (int64_t)ti.d_slot * p.dst.token_stride +
                         (int64_t)p.dst_head0 * p.dst.head_stride;
  const int64_t sc_base = d_blk + p.dst.scale_base + (int64_t)ti.kv * p.dst.scale_kv_stride +
                          (int64_t)ti.d_slot * p.dst.scale_token_stride +
                          (int64_t)p.dst_head0 * p.dst.scale_head_stride;
  const bool wide_scales = scales_as_words(p, cpr, dst + sc_base);
  const uint32_t run_bytes = it.ntok * p.dst.head_bytes;          // one head's rows of the tile, contiguous in HND
  const uint32_t sc_run = it.ntok * (cpr >> 1);
  const bool wide_rows = ((reinterpret_cast<uint64_t>(src + s_base) | (uint64_t)p.src.token_stride |
                           (uint64_t)p.src.head_stride) & 31u) == 0u;
  const bool staged = stage != nullptr && wide_scales && rows.token_inner && nthr == 32u &&
                      p.dst.token_stride == (int64_t)p.dst.head_bytes && p.dst.scale_token_stride == (int64_t)(cpr >> 1) &&
                      chunks * 16u <= kStagePayload && (chunks >> 1) <= kStageScales &&
                      ((run_bytes | sc_run | (uint32_t)p.dst.head_stride | (uint32_t)p.dst.scale_head_stride) & 15u) == 0u &&
                      ((reinterpret_cast<uintptr_t>(dst + d_base) | reinterpret_cast<uintptr_t>(dst + sc_base)) & 15u) == 0u;
  if (staged) {
    // the bulk stores of this warp's previous tile must have read the buffer before it is refilled
    if (tid == 0) bulk_wait_read<0>();
    __syncwarp();
  }
  // Two rounds in flight per thread: the loads of both are issued before either is converted.
  const uint32_t rounds = (chunks + nthr - 1) / nthr;
  for (uint32_t rnd = 0; rnd < rounds; rnd += 2) {
    uint32_t w[2][8];
    bool active[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t i = (rnd + u) * nthr + tid;
      active[u] = (rnd + u) < rounds && i < chunks;
#pragma unroll
      for (int k = 0; k < 8; ++k) w[u][k] = 0;
      if (active[u]) {
        uint32_t t, h, c;
        it.decode(i, t, h, c);
        ld_nc_32(src + s_base + (int64_t)t * p.src.token_stride + (int64_t)h * p.src.head_stride + (c << 5), wide_rows, w[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      quant_chunk(p, it, w[u], (rnd + u) * nthr + tid, active[u], dst + d_base, dst + sc_base, wide_scales,
                  staged ? stage : nullptr);
  }
  if (staged) {
    __syncwarp();
    fence_proxy_async();          // the buffer was written through the generic proxy, the copies read it through the async one
    if (tid == 0) {
      for (uint32_t h = 0; h < p.n_heads; ++h) {
        bulk_store_flat(dst + d_base + (int64_t)h * p.dst.head_stride, smem_u32(stage + h * run_bytes), run_bytes);
        bulk_store_flat(dst + sc_base + (int64_t)h * p.dst.scale_head_stride, smem_u32(stage + kStagePayload + h * sc_run),
                        sc_run);
      }
      bulk_commit();
    }
    __syncwarp();
  }
}

// 16 e4m3 codes and their group's scale exponent -> 16 bf16 values.
__device__ __forceinline__ void expand_chunk(const int4& q, uint32_t e, uint32_t o[8]) {
  const float s = scale_from_ue8m0(e);
  const uint32_t qw[4] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z, (uint32_t)q.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(qw[k] & 0xffffu), __NV_E4M3);
    const __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(qw[k] >> 16), __NV_E4M3);
    const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&h01));
    const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&h23));
    const __nv_bfloat162 b01 = __floats2bfloat162_rn(f01.x * s, f01.y * s);
    const __nv_bfloat162 b23 = __floats2bfloat162_rn(f23.x * s, f23.y * s);
    o[2 * k] = *reinterpret_cast<const uint32_t*>(&b01);
    o[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&b23);
  }
}

// e4m3 rows + UE8M0 scales -> bf16 rows.  One thread expands 16 values (16 B in, 32 B out), with four chunks and their
// scale bytes in flight.
__device__ __forceinline__ void simt_dequant_tile(const KvtAttnLaunch& p, const TileRows& rows, const TileMove& ti,
                                       const char* __restrict__ src, char* __restrict__ dst, uint32_t tid,
                                       uint32_t nthr) {
  const RowIter it(p, rows, ti.ntok);
  const uint32_t chunks = it.chunks;
  const int64_t s_blk = (int64_t)ti.sblk * p.src.block_stride;
  const int64_t s_base = s_blk + (int64_t)ti.kv * p.src.kv_stride + (int64_t)ti.s_slot * p.src.token_stride +
                         (int64_t)p.src_head0 * p.src.head_stride;
  const int64_t sc_base = s_blk + p.src.scale_base + (int64_t)ti.kv * p.src.scale_kv_stride +
                          (int64_t)ti.s_slot * p.src.scale_token_stride +
                          (int64_t)p.src_head0 * p.src.scale_head_stride;
  const int64_t d_base = (int64_t)ti.dblk * p.dst.block_stride + (int64_t)ti.kv * p.dst.kv_stride +
                         (int64_t)ti.d_slot * p.dst.token_stride + (int64_t)p.dst_head0 * p.dst.head_stride;
  const bool wide_rows = ((reinterpret_cast<uint64_t>(dst + d_base) | (uint64_t)p.dst.token_stride |
                           (uint64_t)p.dst.head_stride) & 31u) == 0u;
  constexpr int U = 4;
  for (uint32_t base = tid; base < chunks; base += nthr * U) {
    int4 q[U];
    uint32_t e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * nthr;
      if (i < chunks) {
        uint32_t t, h, c;
        it.decode(i, t, h, c);
        q[u] = ld_nc_16(src + s_base + (int64_t)t * p.src.token_stride + (int64_t)h * p.src.head_stride + (c << 4));
        e[u] = ld_nc_u8(src + sc_base + (int64_t)t * p.src.scale_token_stride + (int64_t)h * p.src.scale_head_stride + (c >> 1));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * nthr;
      if (i >= chunks) break;
      uint32_t o[8];
      expand_chunk(q[u], e[u], o);
      uint32_t t, h, c;   // decoded again: cheaper than registers held across the loads
      it.decode(i, t, h, c);
      st_32(dst + d_base + (int64_t)t * p.dst.token_stride + (int64_t)h * p.dst.head_stride + (c << 5), wide_rows, o);
    }
  }
}

// Zero destination slots [copy_hi, zero_hi) of a tile (tail pad of the last block).
__device__ __forceinline__ void simt_zero_tail(const KvtAttnLaunch& p, const TileMove& ti,
                                               char* __restrict__ dst, uint32_t tid, uint32_t nthr) {
  const TileRows rows(p, p.dst.head_bytes >> 4);
  const RowIter it(p, rows, ti.nzero);
  const uint32_t chunks = it.chunks;
  const int64_t d_base = (int64_t)ti.dblk * p.dst.block_stride + (int64_t)ti.kv * p.dst.kv_stride +
                         (int64_t)(ti.d_slot + ti.ntok) * p.dst.token_stride +
                         (int64_t)p.dst_head0 * p.dst.head_stride;
  for (uint32_t i = tid; i < chunks; i += nthr) {
    uint32_t t, h, c;
    it.decode(i, t, h, c);
    st_16(dst + d_base + (int64_t)t * p.dst.token_stride + (int64_t)h * p.dst.head_stride + (c << 4),
          make_int4(0, 0, 0, 0));
  }
}

// Who owns a tile.  GROUP = 1: a warp (many tiles in flight per SM, nobody waits at tile boundaries).
// GROUP = 4: four warps share a tile, so that more of it is in flight at once, which tiles of 16 KiB
// and more of the local quantiser gain by, in launches of any length (the figures are in launch_impl).
// GROUP = 0: the whole CTA (longer contiguous write runs, which is what a PCIe destination prefers).
// The owners of a CTA take consecutive tiles and the launcher
// sizes the grid to the tiles, so that every resident CTA is full of busy warps: a CTA keeps its
// registers until its last warp exits, and half-empty CTAs of one launch would keep the CTAs of
// launches on other streams off the SM.
template <int MODE, bool USE_TMA, int GROUP, bool IN_LAUNCH>
__device__ __forceinline__ void simt_pass(const KvtAttnLaunch& p, const PlanView<IN_LAUNCH>& plan, uint64_t total, uint32_t per_layer,
                                          unsigned char* stage_base) {
  constexpr uint32_t kGroupThreads = GROUP > 0 ? 32u * GROUP : 0u;
  const uint32_t tid = GROUP > 0 ? (threadIdx.x % kGroupThreads) : threadIdx.x;
  const uint32_t nthr = GROUP > 0 ? kGroupThreads : blockDim.x;
  const uint32_t owners = GROUP > 0 ? (blockDim.x / kGroupThreads) : 1u;
  const uint32_t me = GROUP > 0 ? (threadIdx.x / kGroupThreads) : 0u;
  if (me >= owners) return;   // a block size that is not a multiple of the group: the odd warps sit out
  unsigned char* stage = (GROUP == 1 && MODE == KVT_MODE_BF16_TO_MXFP8 && stage_base != nullptr)
                             ? stage_base + (size_t)me * kStagePerWarp : nullptr;
  const TileRows rows(p, MODE == KVT_MODE_BF16_TO_MXFP8 ? p.src.head_bytes >> 5 : p.src.head_bytes >> 4);
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t step = (uint64_t)gridDim.x * owners;
  // The walk from a tile number to its block ids is a chain of dependent loads: the lanes walk the owner's next 32 tiles
  // at once, then the tiles are moved one after the other.
  for (uint64_t first = (uint64_t)blockIdx.x * owners + me; first < total; first += 32u * step) {
    const uint64_t w = first + lane * step;
    TileMove mine = {};
    bool work = false;
    if (w < total) {
      uint32_t tile;
      split_work(p, w, total, per_layer, mine.layer, mine.kv, tile);
      const TileInfo ti = decode_tile(p, plan, tile);
      if (!ti.ok) {
        if (tid < 32u) set_status(p.status, KVT_ERR_BLOCK_RANGE, tile);
      } else {
        work = mine.set(ti);
        if (USE_TMA) work = mine.nzero != 0u;   // the TMA pass copies
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, work); todo != 0u; todo &= todo - 1u) {
      const TileMove ti = move_of_lane(mine, __ffs(todo) - 1);
      const char* src = reinterpret_cast<const char*>(p.src_layers[p.layer_begin + ti.layer]);
      char* dst = reinterpret_cast<char*>(p.dst_layers[p.layer_begin + ti.layer]);
      if (ti.ntok != 0u && !USE_TMA) {
        if constexpr (MODE == KVT_MODE_COPY) {
          simt_copy_tile(p, rows, ti, src, dst, tid, nthr);
        } else if constexpr (MODE == KVT_MODE_BF16_TO_MXFP8) {
          simt_quant_tile(p, rows, ti, src, dst, tid, nthr, stage);
        } else {
          simt_dequant_tile(p, rows, ti, src, dst, tid, nthr);
        }
      }
      if (ti.nzero != 0u) simt_zero_tail(p, ti, dst, tid, nthr);
    }
  }
  if (stage != nullptr) {
    // the bulk stores of the last tile must be complete before this CTA reports the launch done
    if (tid == 0) bulk_wait_all();
    __syncwarp();
    fence_proxy_async();
  }
}

// Token slots [lo, lo + n) of a tile in shared memory leave as untiled bulk stores, one per run that both sides hold
// contiguously: per head for an HND page, per token (or one in all) for an NHD page.  `dst` is the address of slot lo,
// first moved head.
__device__ __forceinline__ void bulk_store_slots(const KvtAttnLaunch& p, char* dst, uint32_t tile_smem, uint32_t lo, uint32_t n,
                                                 bool hinted, uint64_t pol) {
  const bool token_inner = p.tile_order != 0u;
  const uint32_t hb = p.dst.head_bytes;
  const uint32_t s_outer = (token_inner ? p.tile_tokens : p.n_heads) * hb;
  const int64_t d_outer = token_inner ? p.dst.head_stride : p.dst.token_stride;
  const int64_t d_inner = token_inner ? p.dst.token_stride : p.dst.head_stride;
  uint32_t n_outer = token_inner ? p.n_heads : n, n_inner = token_inner ? n : p.n_heads, run = hb;
  if (d_inner == (int64_t)hb) {
    run = n_inner * hb;
    n_inner = 1;
    if (s_outer == run && d_outer == (int64_t)run) {
      run *= n_outer;
      n_outer = 1;
    }
  }
  const uint32_t sm = tile_smem + lo * (token_inner ? hb : s_outer);
  for (uint32_t o = 0; o < n_outer; ++o)
    for (uint32_t i = 0; i < n_inner; ++i)
      bulk_store_run(dst + (int64_t)o * d_outer + (int64_t)i * d_inner, sm + o * s_outer + i * hb, run, hinted, pol);
}

// The last CTA to finish publishes the flag after a system-scope fence, so a reader on the destination GPU or on the host
// that sees the flag also sees the data.
__device__ __forceinline__ void publish_completion(const KvtAttnLaunch& p) {
  if (p.flag == nullptr || p.done_counter == nullptr) return;
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t prev = atomicAdd(p.done_counter, 1u);
    if (prev == gridDim.x - 1) {
      *p.done_counter = 0;  // re-arm for the next launch on this stream
      __threadfence_system();
      asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p.flag), "l"(p.flag_value) : "memory");
    }
  }
}

// ---- the kernel ---------------------------------------------------------------------------
template <int MODE, bool USE_TMA, bool IN_LAUNCH>
__global__ void __launch_bounds__(512, 2) kvt_p2d_attn_kernel(const __grid_constant__ KvtAttnLaunch p,
                                                            const uint32_t n_stages, const uint32_t tile_bytes,
                                                            const uint32_t warp_tiles,
                                                            const __grid_constant__ PlanParam<IN_LAUNCH> plan_param) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const PlanView<IN_LAUNCH> plan(p, plan_param);
  const uint32_t n_layers = p.layer_end - p.layer_begin;
  const uint32_t per_layer = p.total_tiles * p.src.kv_count;
  const uint64_t total = (uint64_t)n_layers * per_layer;

  // Work index w -> (layer, kv, tile).  Consecutive CTAs take consecutive tiles of one layer.
  if constexpr (USE_TMA) {
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)n_stages * tile_bytes);
    if (threadIdx.x == 0) {
      for (uint32_t s = 0; s < n_stages; ++s) mbar_init(smem_u32(&bars[s]), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      fence_proxy_async();
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // Producer warp.  All 32 lanes decode tiles in parallel (the block-table walk is a chain
      // of dependent loads, so doing it on one thread would serialise ~1 us per tile); lane 0
      // runs the software pipeline: at most n_stages-1 loads in flight, one store behind.
      const uint32_t lane = threadIdx.x;
      // dmap == nullptr: the tile (or the n slots from lo that the request has in it) is stored by untiled bulk copies
      // from `flat` on.  A partly filled tile is LOADED whole: its other slots are cache memory of the same block, read
      // and dropped.
      struct Slot { const void* dmap; char* flat; int c1, c2, c3, c4; uint32_t lo, n; };
      Slot slots[kMaxStages];
      uint32_t issued = 0, stored = 0;
      bool failed = false;
      const bool token_inner = p.tile_order != 0u;
      const bool flat_store = p.store_form != 0u;
      const bool hinted = p.cache_hint != 0u;
      const uint64_t pol = hinted ? policy_evict_first() : 0ull;
      auto consume_one = [&]() {
        const uint32_t s = stored % n_stages;
        const uint32_t bar = smem_u32(&bars[s]);
        const uint32_t parity = (stored / n_stages) & 1u;
        const long long t0 = clock64();
        while (!mbar_try_wait(bar, parity)) {
          if (clock64() - t0 > kWaitCycles) {
            failed = true;
            break;
          }
        }
        if (failed) {
          set_status(p.status, KVT_ERR_TMA_TIMEOUT, stored);
          return;
        }
        const uint32_t sm = smem_u32(smem + (size_t)s * tile_bytes);
        if (slots[s].n != p.tile_tokens) {
          bulk_store_slots(p, slots[s].flat, sm, slots[s].lo, slots[s].n, hinted, pol);
        } else if (slots[s].dmap == nullptr) {
          bulk_store_run(slots[s].flat, sm, tile_bytes, hinted, pol);
        } else if (hinted) {
          tma_store_5d_hint(slots[s].dmap, sm, 0, slots[s].c1, slots[s].c2, slots[s].c3, slots[s].c4, pol);
        } else {
          tma_store_5d(slots[s].dmap, sm, 0, slots[s].c1, slots[s].c2, slots[s].c3, slots[s].c4);
        }
        bulk_commit();
        ++stored;
      };
      for (uint64_t batch = 0;; batch += 32) {
        const uint64_t w = blockIdx.x + (batch + lane) * (uint64_t)gridDim.x;
        bool mine = false;
        TileInfo ti;
        ti.sblk = ti.dblk = ti.s_slot0 = ti.d_slot0 = ti.tok_lo = ti.copy_lo = ti.copy_hi = 0;
        uint32_t layer = 0, kv = 0;
        if (w < total) {
          uint32_t tile;
          split_work(p, w, total, per_layer, layer, kv, tile);
          ti = decode_tile(p, plan, tile);
          mine = ti.ok && ti.copy_hi > ti.copy_lo;  // bad tiles are reported by the SIMT pass
        }
        const unsigned any = __ballot_sync(0xffffffffu, w < total);
        unsigned todo = __ballot_sync(0xffffffffu, mine);
        if (any == 0u) break;
        while (todo != 0u) {
          const int j = __ffs(todo) - 1;
          todo &= todo - 1u;
          const uint32_t j_sblk = __shfl_sync(0xffffffffu, ti.sblk, j);
          const uint32_t j_dblk = __shfl_sync(0xffffffffu, ti.dblk, j);
          const uint32_t j_ss = __shfl_sync(0xffffffffu, ti.s_slot0, j);
          const uint32_t j_ds = __shfl_sync(0xffffffffu, ti.d_slot0, j);
          const uint32_t j_layer = __shfl_sync(0xffffffffu, layer, j);
          const uint32_t j_kv = __shfl_sync(0xffffffffu, kv, j);
          const uint32_t j_lo = __shfl_sync(0xffffffffu, ti.copy_lo - ti.tok_lo, j);
          const uint32_t j_n = __shfl_sync(0xffffffffu, ti.copy_hi - ti.copy_lo, j);
          if (lane == 0 && !failed) {
            if (n_stages == 1) {
              if (issued > stored) consume_one();
              if (!failed) bulk_wait_read<0>();
            } else if (issued - stored == n_stages - 1) {
              consume_one();
              // the stage refilled below was last read by the store issued one step earlier
              if (!failed) bulk_wait_read<1>();
            }
            if (!failed) {
              const uint32_t s = issued % n_stages;
              const uint32_t bar = smem_u32(&bars[s]);
              const CUtensorMap* smap = reinterpret_cast<const CUtensorMap*>(p.src_maps) + (p.layer_begin + j_layer);
              const CUtensorMap* dmap = reinterpret_cast<const CUtensorMap*>(p.dst_maps) + (p.layer_begin + j_layer);
              mbar_expect_tx(bar, tile_bytes);
              // coordinate order of the maps: {row, head, slot, block, kv}, or {row, slot, head, block, kv} when the
              // tile is kept token-inner (heads outermost in shared memory, the order of an HND destination)
              const int s1 = token_inner ? (int)j_ss : (int)p.src_head0;
              const int s2 = token_inner ? (int)p.src_head0 : (int)j_ss;
              if (hinted) {
                tma_load_5d_hint(smem_u32(smem + (size_t)s * tile_bytes), smap, bar, 0, s1, s2, (int)j_sblk, (int)j_kv, pol);
              } else {
                tma_load_5d(smem_u32(smem + (size_t)s * tile_bytes), smap, bar, 0, s1, s2, (int)j_sblk, (int)j_kv);
              }
              slots[s].dmap = flat_store ? nullptr : dmap;
              slots[s].flat = reinterpret_cast<char*>(p.dst_layers[p.layer_begin + j_layer]) +
                              (int64_t)j_dblk * p.dst.block_stride + (int64_t)j_kv * p.dst.kv_stride +
                              (int64_t)(j_ds + j_lo) * p.dst.token_stride + (int64_t)p.dst_head0 * p.dst.head_stride;
              slots[s].c1 = token_inner ? (int)j_ds : (int)p.dst_head0;
              slots[s].c2 = token_inner ? (int)p.dst_head0 : (int)j_ds;
              slots[s].c3 = (int)j_dblk;
              slots[s].c4 = (int)j_kv;
              slots[s].lo = j_lo;
              slots[s].n = j_n;
              ++issued;
            }
          }
        }
      }
      if (lane == 0) {
        while (!failed && stored < issued) consume_one();
        bulk_wait_all();
        fence_proxy_async();
      }
      __syncwarp();
    }
  }

  // SIMT pass: everything the TMA pass does not take (with TMA: tail zeros and the report of bad tiles).
  // without TMA tiles a non-zero tile_bytes says that every warp owns a staging buffer of that size
  unsigned char* stage_base = (!USE_TMA && tile_bytes == kStagePerWarp) ? smem : nullptr;
  if (warp_tiles == 1u) {
    simt_pass<MODE, USE_TMA, 1>(p, plan, total, per_layer, stage_base);
  } else if (warp_tiles == 4u) {
    simt_pass<MODE, USE_TMA, 4>(p, plan, total, per_layer, nullptr);
  } else {
    simt_pass<MODE, USE_TMA, 0>(p, plan, total, per_layer, nullptr);
  }

  publish_completion(p);
}

// ---- expansion fed by the bulk-copy engine --------------------------------------------------
// Block-scaled fp8 -> bf16 inside one GPU is bound by HBM, and by how the tiles are read: a warp that walks a tile with
// its own loads has 2 KiB of it in flight and comes back to the same DRAM pages many times.  Here warp 0 of a CTA walks the
// block tables and brings each tile's rows and scale bytes into shared memory with untiled bulk copies, one per run that
// the source holds contiguously; the other warps convert from shared memory and store straight into the destination.  Tiles
// pass through a ring of as many stages as fit the CTA's share of an SM's shared memory, four at most, with a full and an empty
// mbarrier each: tiles of up to 24 KiB of codes have one or more brought ahead of the one being converted.  Larger ones have a
// stage alone, and the SM's other CTAs cover the wait for it: 16 heads (32 KiB), 16 layers of 2 x 3000 tokens, 596 MB, 106 us
// against 174 with a warp per tile and 146 with four; one layer of 300 tokens 12, 60 and 22.  Measured (HND fp8 -> NHD bf16,
// 8 heads, 32 layers of 3 x ~1334 tokens, 795 MB read and written): 197 us with a warp per tile, 178 with four, 170 with
// eight, 135 this way (5.9 TB/s); one layer of 300 tokens 34 -> 11 us.  Staging the converted rows too, so that the bulk engine
// stores them, loses (174 to 206 us at 2 to 4 KiB a warp).  The other direction does not gain (the quantiser's
// arithmetic fills the same warps: 174 against 158 us at 2 heads, 304 against 283 at 8) and stays with its own loads.
//
// WARPS convert in each of CTAS CTAs per SM: 32 warps a SM either way, which is what keeps HBM busy, in few CTAs with deep stages for
// large tiles and in many for small ones, whose hand-over the others then hide.  us a launch with 4 warps in 6 CTAs for all / with
// these: 8 heads, 32 layers of 4003 tokens 138 / 135 (5.9 TB/s), 4 heads 82 / 74, 2 heads of 8000 tokens 86 / 78, 16 heads, 16 layers
// 140 / 135, 20 heads (40 KiB, too large for a sixth of an SM) 66 / 22.  The other shape: 2 heads 104, 3 heads (6 KiB) 70 against 63.
// More warps a CTA (10 in 4, 12 in 3, 16 in 2) are slower at every size.
struct ConvLarge { static constexpr uint32_t WARPS = 8, CTAS = 4; };
struct ConvSmall { static constexpr uint32_t WARPS = 4, CTAS = 8; };
constexpr uint32_t kConvLargeTile = 8192;                 // bytes of codes from which a tile is large
constexpr int kConvStages = 4;
constexpr uint32_t kConvEnd = 0xffffffffu;                // layer of the slot behind the last tile

struct ConvSlot {
  TileMove move;
  uint32_t scales_here;      // the tile's scale bytes are in the stage, behind its rows
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The calling lane's wait.  Lanes read their own clocks, so at the limit some may give up where others were served.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > kWaitCycles) return false;
  return true;
}
// The wait of a whole warp, with one outcome for all of its lanes: they go on, or leave, together.
__device__ __forceinline__ bool warp_wait_bounded(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity)) != 0;
}
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst),
               "l"(gsrc), "r"(bytes), "r"(bar)
               : "memory");
}

// How a tile's source rows lie in a stage: row (token t, head h) at t * s_t + h * s_h, the order in which the source holds
// them, so that a run of them is one copy.
struct ConvRows {
  bool by_token;             // heads of a token adjacent in the source (NHD); else the rows of a head (HND), or single rows
  uint32_t s_t, s_h;
  __device__ __forceinline__ explicit ConvRows(const KvtAttnLaunch& p) {
    const uint32_t hb = p.src.head_bytes;
    const bool by_head = p.src.head_stride != (int64_t)hb && p.src.token_stride == (int64_t)hb;
    by_token = p.src.head_stride == (int64_t)hb;
    s_t = by_head ? hb : p.n_heads * hb;
    s_h = by_head ? p.tile_tokens * hb : hb;
  }
};

template <typename SHAPE, bool IN_LAUNCH>
__global__ void __launch_bounds__(32u * (1u + SHAPE::WARPS), SHAPE::CTAS)
    kvt_p2d_expand_kernel(const __grid_constant__ KvtAttnLaunch p, const uint32_t n_stages, const uint32_t tile_bytes,
                          const uint32_t stage_bytes, const __grid_constant__ PlanParam<IN_LAUNCH> plan_param) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr uint32_t kConvWarps = SHAPE::WARPS;
  const PlanView<IN_LAUNCH> plan(p, plan_param);
  __shared__ uint64_t full[kConvStages], empty[kConvStages];
  __shared__ ConvSlot slots[kConvStages];
  const uint32_t per_layer = p.total_tiles * p.src.kv_count;
  const uint64_t total = (uint64_t)(p.layer_end - p.layer_begin) * per_layer;
  const uint32_t lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < n_stages; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), kConvWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  __syncthreads();
  const uint32_t hb = p.src.head_bytes;
  const uint32_t sb = hb >> 5;               // scale bytes of a row
  const ConvRows lay(p);
  if (threadIdx.x < 32u) {
    uint32_t issued = 0;
    bool failed = false;
    // the next stage, free again (its converting warps are bounded in their own waits)
    auto acquire = [&]() {
      const uint32_t s = issued % n_stages;
      if (issued >= n_stages && !warp_wait_bounded(smem_u32(&empty[s]), (issued / n_stages - 1u) & 1u)) {
        if (lane == 0) set_status(p.status, KVT_ERR_TMA_TIMEOUT, issued);
        failed = true;
      }
      ++issued;
      return s;
    };
    for (uint64_t first = blockIdx.x; first < total && !failed; first += 32u * (uint64_t)gridDim.x) {
      const uint64_t w = first + lane * (uint64_t)gridDim.x;
      TileMove mine = {};
      bool work = false;
      if (w < total) {
        uint32_t tile;
        split_work(p, w, total, per_layer, mine.layer, mine.kv, tile);
        const TileInfo ti = decode_tile(p, plan, tile);
        if (ti.ok) work = mine.set(ti); else set_status(p.status, KVT_ERR_BLOCK_RANGE, tile);
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, work); todo != 0u; todo &= todo - 1u) {
        const TileMove m = move_of_lane(mine, __ffs(todo) - 1);
        const uint32_t s = acquire();
        if (failed) break;
        const uint32_t bar = smem_u32(&full[s]), stage = smem_u32(smem + (size_t)s * stage_bytes);
        const char* blk = reinterpret_cast<const char*>(p.src_layers[p.layer_begin + m.layer]) +
                          (int64_t)m.sblk * p.src.block_stride;
        const char* rows = blk + (int64_t)m.kv * p.src.kv_stride + (int64_t)m.s_slot * p.src.token_stride +
                           (int64_t)p.src_head0 * p.src.head_stride;
        // runs of the rows: n of `run` bytes, g_step apart in the source and s_step in the stage
        uint32_t n, run, s_step;
        int64_t g_step;
        if (lay.by_token) {
          n = m.ntok; run = p.n_heads * hb; s_step = lay.s_t; g_step = p.src.token_stride;
        } else if (lay.s_t == hb && lay.s_h != hb) {
          n = p.n_heads; run = m.ntok * hb; s_step = lay.s_h; g_step = p.src.head_stride;
        } else {
          n = m.ntok * p.n_heads; run = hb; s_step = hb; g_step = 0;    // single rows
        }
        const bool singles = g_step == 0 && n > 1u;
        if (!singles && n > 1u && g_step == (int64_t)run && s_step == run) {
          run *= n;
          n = 1;
        }
        // the scale bytes of the whole tile (its other slots belong to the same block)
        const uint32_t sc_run = p.tile_tokens * sb;
        const char* scales = nullptr;
        uint32_t sc_n = 0, sc_len = sc_run;
        if (m.ntok != 0u) {
          scales = blk + p.src.scale_base + (int64_t)m.kv * p.src.scale_kv_stride +
                   (int64_t)(m.s_slot / p.tile_tokens * p.tile_tokens) * p.src.scale_token_stride +
                   (int64_t)p.src_head0 * p.src.scale_head_stride;
          const bool dense = p.n_heads == 1u || p.src.scale_head_stride == (int64_t)sc_run;
          if (p.src.scale_token_stride == (int64_t)sb &&
              ((reinterpret_cast<uint64_t>(scales) | sc_run | (p.n_heads > 1u ? (uint64_t)p.src.scale_head_stride : 0u)) & 15u) == 0u) {
            sc_n = dense ? 1u : p.n_heads;
            if (dense) sc_len = p.n_heads * sc_run;
          }
        }
        if (lane == 0) {
          slots[s].move = m;
          slots[s].scales_here = sc_n;
          mbar_expect_tx(bar, m.ntok * p.n_heads * hb + sc_n * sc_len);
        }
        __syncwarp();
        if (m.ntok != 0u) {
          for (uint32_t r = lane; r < n; r += 32u) {
            int64_t g = (int64_t)r * g_step;
            if (singles) g = (int64_t)(r / p.n_heads) * p.src.token_stride + (int64_t)(r % p.n_heads) * p.src.head_stride;
            bulk_load(stage + r * s_step, rows + g, run, bar);
          }
          for (uint32_t r = lane; r < sc_n; r += 32u)
            bulk_load(stage + tile_bytes + r * sc_len, scales + (int64_t)r * p.src.scale_head_stride, sc_len, bar);
        }
      }
    }
    if (!failed) {
      const uint32_t s = acquire();
      if (!failed && lane == 0) {
        slots[s].move.layer = kConvEnd;
        mbar_expect_tx(smem_u32(&full[s]), 0);
      }
    }
    __syncwarp();
  } else {
    const uint32_t tid = threadIdx.x - 32u;
    const TileRows rows(p, hb >> 4);
    for (uint32_t k = 0;; ++k) {
      const uint32_t s = k % n_stages;
      const uint32_t bar = smem_u32(&full[s]), parity = (k / n_stages) & 1u;
      if (!warp_wait_bounded(bar, parity)) {
        if (lane == 0) set_status(p.status, KVT_ERR_TMA_TIMEOUT, k);
        warp_wait_bounded(bar, parity);      // copies may still be on their way into this CTA's shared memory
        break;
      }
      const TileMove m = slots[s].move;
      if (m.layer == kConvEnd) break;
      const unsigned char* tile = smem + (size_t)s * stage_bytes;
      char* dst = reinterpret_cast<char*>(p.dst_layers[p.layer_begin + m.layer]);
      char* d_blk = dst + (int64_t)m.dblk * p.dst.block_stride;
      char* d_rows = d_blk + (int64_t)m.kv * p.dst.kv_stride + (int64_t)m.d_slot * p.dst.token_stride +
                     (int64_t)p.dst_head0 * p.dst.head_stride;
      if (m.ntok != 0u) {
        const RowIter it(p, rows, m.ntok);
        const bool wide_rows = ((reinterpret_cast<uint64_t>(d_rows) | (uint64_t)p.dst.token_stride |
                                 (uint64_t)p.dst.head_stride) & 31u) == 0u;
        const unsigned char* sc_tile = tile + tile_bytes + (m.s_slot % p.tile_tokens) * sb;
        const char* sc_far = reinterpret_cast<const char*>(p.src_layers[p.layer_begin + m.layer]) +
                             (int64_t)m.sblk * p.src.block_stride + p.src.scale_base + (int64_t)m.kv * p.src.scale_kv_stride +
                             (int64_t)m.s_slot * p.src.scale_token_stride + (int64_t)p.src_head0 * p.src.scale_head_stride;
        const bool here = slots[s].scales_here != 0u;
#pragma unroll 2
        for (uint32_t i = tid; i < it.chunks; i += 32u * kConvWarps) {
          uint32_t t, h, c;
          it.decode(i, t, h, c);
          const int4 q = *reinterpret_cast<const int4*>(tile + t * lay.s_t + h * lay.s_h + (c << 4));
          const uint32_t e = here ? sc_tile[(h * p.tile_tokens + t) * sb + (c >> 1)]
                                  : ld_nc_u8(sc_far + (int64_t)t * p.src.scale_token_stride +
                                             (int64_t)h * p.src.scale_head_stride + (c >> 1));
          uint32_t o[8];
          expand_chunk(q, e, o);
          st_32(d_rows + (int64_t)t * p.dst.token_stride + (int64_t)h * p.dst.head_stride + (c << 5), wide_rows, o);
        }
      }
      if (m.nzero != 0u) simt_zero_tail(p, m, dst, tid, 32u * kConvWarps);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty[s]));
    }
  }
  publish_completion(p);
}

struct DriverApi {
  CUresult (*encode_tiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                           const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                           CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) = nullptr;
  bool tried = false;
};
DriverApi g_driver;

bool load_driver_api() {
  if (g_driver.tried) return g_driver.encode_tiled != nullptr;
  g_driver.tried = true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
      qres == cudaDriverEntryPointSuccess) {
    g_driver.encode_tiled = reinterpret_cast<decltype(g_driver.encode_tiled)>(fn);
  }
  return g_driver.encode_tiled != nullptr;
}

// BLLM_KVTRANS_SIMT_TILE overrides KvtAttnLaunch::simt_tile: 1 = a warp per tile, 4 = four warps per
// tile (lower latency of a lone short launch, lower throughput of overlapped ones), 2 = a CTA per tile.
int simt_choice(const KvtAttnLaunch& a) {
  static const int env_simt = [] {
    const char* v = getenv("BLLM_KVTRANS_SIMT_TILE");
    return v != nullptr ? atoi(v) : 0;
  }();
  return env_simt != 0 ? env_simt : (int)a.simt_tile;
}

// BLLM_KVTRANS_QUANT_STAGE: 0 = direct 16-byte stores always, 1 = staged bulk stores always; unset =
// staged for a remote destination (668 against 614 GB/s of link), direct for a local one (2842
// against 2494 GB/s of source).
bool quant_staged(const KvtAttnLaunch& a) {
  static const int stage_env = [] {
    const char* v = getenv("BLLM_KVTRANS_QUANT_STAGE");
    return v == nullptr ? -1 : atoi(v);
  }();
  return stage_env > 0 || (stage_env < 0 && a.dst_remote != 0);
}

// More than 48 KiB of shared memory, the kernel's own arrays (at most 1 KiB) included, take an opt-in.
template <typename KERNEL>
cudaError_t opt_in(KERNEL kern, size_t smem, SmemGrant& grant) {
  if (smem <= 47 * 1024) return cudaSuccess;
  int dev = 0;
  cudaGetDevice(&dev);
  return (cudaError_t)grant.ask(dev, smem, [kern](size_t bytes) {
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  });
}

// The plan as a parameter of the launch.
template <bool IN_LAUNCH>
PlanParam<IN_LAUNCH> plan_param(const KvtAttnLaunch& a) {
  PlanParam<IN_LAUNCH> out;
  if constexpr (IN_LAUNCH) memcpy(out.words, a.plan, a.plan_bytes);
  return out;
}

// The expansion kernel serves what leaves the way of reading open (simt_tile 0, no threads asked for: its CTAs have one size),
// in tiles of at least 4 KiB of codes (with 2 KiB, one head, the hand-over of a tile costs more than its reading: 32 layers of
// 6000 tokens 51 us against 43) of which its CTAs fit an SM; for the rest it says cudaErrorNotSupported and the SIMT kernel
// serves it.
template <typename SHAPE>
cudaError_t launch_expand_as(const KvtAttnLaunch& a, int grid_ctas, int sms, uint64_t total, uint64_t tile_bytes, uint64_t stage_bytes,
                             cudaStream_t stream) {
  const uint64_t budget = kSmemBudget / SHAPE::CTAS;
  if (stage_bytes > budget) return cudaErrorNotSupported;
  uint64_t stages = budget / stage_bytes;
  if (stages > (uint64_t)kConvStages) stages = kConvStages;
  uint64_t grid = (uint64_t)grid_ctas;
  if (grid_ctas <= 0) {
    const uint64_t tiles = tile_bytes < (128u << 10) ? (128u << 10) / tile_bytes : 1u;
    grid = std::max<uint64_t>((uint64_t)SHAPE::CTAS * sms, std::min<uint64_t>((total + tiles - 1) / tiles, 1u << 30));
  }
  if (grid > total) grid = total;
  const size_t smem = stages * stage_bytes;
  const auto go = [&](auto in_launch) {
    constexpr bool kIn = decltype(in_launch)::value;
    static SmemGrant grant;
    const cudaError_t e = opt_in(kvt_p2d_expand_kernel<SHAPE, kIn>, smem, grant);
    if (e != cudaSuccess) return e;
    kvt_p2d_expand_kernel<SHAPE, kIn><<<(int)grid, 32u * (1u + SHAPE::WARPS), smem, stream>>>(
        a, (uint32_t)stages, (uint32_t)tile_bytes, (uint32_t)stage_bytes, plan_param<kIn>(a));
    return cudaGetLastError();
  };
  return a.plan != nullptr ? go(std::true_type{}) : go(std::false_type{});
}

cudaError_t launch_expand(const KvtAttnLaunch& a, int grid_ctas, int threads_asked, int sms, uint64_t total, cudaStream_t stream) {
  const uint64_t rows = (uint64_t)a.n_heads * a.tile_tokens;
  const uint64_t tile_bytes = (rows * a.src.head_bytes + 127u) & ~127ull;
  const uint64_t stage_bytes = tile_bytes + ((rows * (a.src.head_bytes >> 5) + 127u) & ~127ull);
  if (threads_asked > 0 || simt_choice(a) != 0 || a.dst_remote != 0 || tile_bytes < 4096u) return cudaErrorNotSupported;
  return tile_bytes >= kConvLargeTile ? launch_expand_as<ConvLarge>(a, grid_ctas, sms, total, tile_bytes, stage_bytes, stream)
                                      : launch_expand_as<ConvSmall>(a, grid_ctas, sms, total, tile_bytes, stage_bytes, stream);
}

template <int MODE, bool USE_TMA, bool IN_LAUNCH>
cudaError_t launch_as(const KvtAttnLaunch& a, int grid, int threads, uint32_t stages, uint32_t tile_bytes, size_t smem,
                      uint32_t warp_tiles, cudaStream_t stream) {
  auto kern = kvt_p2d_attn_kernel<MODE, USE_TMA, IN_LAUNCH>;
  static SmemGrant grant;
  const cudaError_t e = opt_in(kern, smem, grant);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, stream>>>(a, stages, tile_bytes, warp_tiles, plan_param<IN_LAUNCH>(a));
  return cudaGetLastError();
}

template <int MODE, bool USE_TMA>
cudaError_t launch_impl(const KvtAttnLaunch& a, int grid, int threads, uint32_t stages, uint32_t tile_bytes,
                        size_t smem, cudaStream_t stream) {
  const int choice = simt_choice(a);
  uint32_t warp_tiles;
  const uint64_t total = (uint64_t)(a.layer_end - a.layer_begin) * a.total_tiles * a.src.kv_count;
  const uint32_t warps = (uint32_t)(threads / 32);
  if (choice == 2) {
    warp_tiles = 0u;
  } else if (choice == 1 || (choice == 4 && threads % 128 == 0)) {
    warp_tiles = (uint32_t)choice;
  } else {
    // Four warps share a tile of 16 KiB or more of the local quantiser, so that more of it is in flight at once: 32 layers
    // of 500 tiles of 8 heads 283 us against 307 with a warp per tile (5.6 TB/s), 2 heads (8 KiB) 158 against 159, one head
    // 57 against 45.  The staged form (remote destinations) and the host-side copies keep a tile with one warp.
    const uint64_t tile = (uint64_t)a.n_heads * a.tile_tokens * a.src.head_bytes;
    warp_tiles = MODE == KVT_MODE_BF16_TO_MXFP8 && threads % 128 == 0 && tile >= 16384u && !quant_staged(a) ? 4u : 1u;
  }
  if (!USE_TMA && warp_tiles != 0u) {
    const uint64_t owners = warps / warp_tiles;
    const uint64_t need = (total + owners - 1) / owners;
    if ((uint64_t)grid > need) grid = (int)need;
  }
  if (MODE == KVT_MODE_BF16_TO_MXFP8 && !USE_TMA && warp_tiles == 1u) {
    if (quant_staged(a)) {
      tile_bytes = kStagePerWarp;
      smem = (size_t)warps * kStagePerWarp;
    }
  }
  return a.plan != nullptr ? launch_as<MODE, USE_TMA, true>(a, grid, threads, stages, tile_bytes, smem, warp_tiles, stream)
                           : launch_as<MODE, USE_TMA, false>(a, grid, threads, stages, tile_bytes, smem, warp_tiles, stream);
}

}  // namespace

extern "C" uint32_t kvt_req_tiles(uint32_t seen, uint32_t new_tokens, uint32_t tile_tokens, uint32_t flags,
                                  uint32_t dst_ntpb) {
  if (tile_tokens == 0) return 0;
  uint64_t end_tok = (uint64_t)seen + new_tokens;
  if ((flags & KVT_REQ_PAD_TAIL) && dst_ntpb > 0) end_tok = (end_tok + dst_ntpb - 1) / dst_ntpb * dst_ntpb;
  if (end_tok <= seen && new_tokens == 0) return 0;
  const uint64_t first = seen / tile_tokens;
  const uint64_t last = (end_tok + tile_tokens - 1) / tile_tokens;
  return (uint32_t)(last - first);
}

extern "C" int kvt_encode_tensor_map(void* out, uint64_t base, const KvtLayout* l, uint32_t box_heads,
                                     uint32_t box_tokens) {
  return kvt_encode_tensor_map_ordered(out, base, l, box_heads, box_tokens, 0);
}

extern "C" int kvt_tile_is_flat(const KvtLayout* l, uint32_t n_heads, uint32_t tile_tokens, uint32_t token_inner) {
  const int64_t hb = l->head_bytes;
  if (token_inner) {
    // heads outermost: rows of a head adjacent, heads adjacent (HND pages)
    return l->token_stride == hb && (n_heads == 1 || l->head_stride == (int64_t)tile_tokens * hb) ? 1 : 0;
  }
  // tokens outermost: heads of a token adjacent, tokens adjacent (NHD pages, all heads moved)
  return l->head_stride == hb && (tile_tokens == 1 || l->token_stride == (int64_t)n_heads * hb) ? 1 : 0;
}

extern "C" int kvt_encode_tensor_map_ordered(void* out, uint64_t base, const KvtLayout* l, uint32_t box_heads,
                                             uint32_t box_tokens, uint32_t token_inner) {
  if (!load_driver_api()) return -1;
  if (l->head_bytes % 16 != 0 || (base & 15) != 0) return -2;
  if (l->head_bytes / 4 > 256 || box_heads > 256 || box_tokens > 256) return -3;
  if (box_heads == 0 || box_tokens == 0 || box_heads > l->num_heads || box_tokens > l->ntpb) return -3;
  const int64_t strides[4] = {l->head_stride, l->token_stride, l->block_stride,
                              l->kv_count > 1 ? l->kv_stride : l->block_stride * (int64_t)l->num_blocks};
  for (int i = 0; i < 4; ++i) {
    if (strides[i] <= 0 || (strides[i] % 16) != 0 || strides[i] >= (1ll << 40)) return -4;
  }
  cuuint64_t gdim[5] = {l->head_bytes / 4, l->num_heads, l->ntpb, l->num_blocks, l->kv_count ? l->kv_count : 1};
  cuuint64_t gstr[4] = {(cuuint64_t)strides[0], (cuuint64_t)strides[1], (cuuint64_t)strides[2],
                        (cuuint64_t)strides[3]};
  cuuint32_t box[5] = {l->head_bytes / 4, box_heads, box_tokens, 1, 1};
  if (token_inner) {   // the slot dimension before the head dimension: a tile lands as [head][slot][row]
    gdim[1] = l->ntpb;
    gdim[2] = l->num_heads;
    gstr[0] = (cuuint64_t)strides[1];
    gstr[1] = (cuuint64_t)strides[0];
    box[1] = box_tokens;
    box[2] = box_heads;
  }
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = g_driver.encode_tiled(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_UINT32, 5,
                                     reinterpret_cast<void*>(base), gdim, gstr, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (int)r;
}

extern "C" int kvt_launch_p2d_attn(const KvtAttnLaunch* args, int grid_ctas, int threads, int use_tma,
                                   void* stream_) {
  const KvtAttnLaunch& a = *args;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (a.n_reqs == 0 || a.total_tiles == 0 || a.layer_end <= a.layer_begin) return (int)cudaSuccess;
  if (a.plan != nullptr && (a.plan_bytes > KVT_PLAN_IN_LAUNCH || a.plan_bytes < (uint64_t)a.n_reqs * sizeof(KvtReqDesc)))
    return (int)cudaErrorInvalidValue;
  if (a.tile_tokens == 0 || a.src.ntpb % a.tile_tokens != 0 || a.dst.ntpb % a.tile_tokens != 0)
    return (int)cudaErrorInvalidValue;
  if (a.src.kv_count != a.dst.kv_count || a.n_heads == 0) return (int)cudaErrorInvalidValue;
  if (a.src_head0 + a.n_heads > a.src.num_heads || a.dst_head0 + a.n_heads > a.dst.num_heads)
    return (int)cudaErrorInvalidValue;
  if (a.mode == KVT_MODE_COPY) {
    if (a.src.head_bytes != a.dst.head_bytes || a.src.head_bytes % 16 != 0) return (int)cudaErrorInvalidValue;
  } else if (a.mode == KVT_MODE_BF16_TO_MXFP8) {
    if (a.src.head_bytes != 2 * a.dst.head_bytes || a.src.head_bytes % 64 != 0) return (int)cudaErrorInvalidValue;
  } else if (a.mode == KVT_MODE_MXFP8_TO_BF16) {
    if (2 * a.src.head_bytes != a.dst.head_bytes || a.dst.head_bytes % 64 != 0) return (int)cudaErrorInvalidValue;
  } else {
    return (int)cudaErrorInvalidValue;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  static std::atomic<int> sm_cache[kMaxDevices];
  int sms = dev >= 0 && dev < kMaxDevices ? sm_cache[dev].load(std::memory_order_relaxed) : 0;
  if (sms == 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < kMaxDevices) sm_cache[dev].store(sms, std::memory_order_relaxed);
  }
  const int threads_asked = threads;
  // Default: four CTAs per SM.  Many small CTAs, each with one tile in flight, measured faster
  // than one deep software pipeline per SM, and they let launches on different streams share SMs.
  int grid = grid_ctas > 0 ? grid_ctas : 4 * sms;
  const uint64_t total = (uint64_t)(a.layer_end - a.layer_begin) * a.total_tiles * a.src.kv_count;
  const bool tma = use_tma && a.mode == KVT_MODE_COPY && a.src_maps != nullptr && a.dst_maps != nullptr;
  const uint32_t tile_bytes = tma ? a.src.head_bytes * a.n_heads * a.tile_tokens : 0u;
  int resident = grid;   // CTAs that are on the GPU together
  if (tma && grid_ctas <= 0 && a.dst_remote == 0 && tile_bytes != 0) {
    // Inside one GPU: as many CTAs per SM as have two tiles each in 200 KiB, 4 to 12.  One thread drives a CTA's tiles, so
    // small ones want more CTAs: 4 KiB tiles (1 head), 1024 a layer, 32 layers 64 us with 12 a SM, 85 with 6, 99 with 4; 8 KiB
    // tiles, 16384 in all, 59 / 65 / 78.  Tiles of 32 KiB have one stage each at 4 to 6 a SM, so nothing but the other CTAs of
    // the SM covers a CTA's wait.  They keep 4: one launch of 2048 or 5120 tiles takes 33.8 and 65.5 us with 4, 31.8 and 65.5
    // with 6, but one-layer launches of 1024 tiles overlapping on 8 streams move 3172 and 2966 GB/s.
    const int per_sm = (int)std::min(12u, std::max(4u, kSmemBudget / 2u / tile_bytes));
    grid = resident = per_sm * sms;
    // A long launch: CTAs of 128 KiB of tiles, handed to the SMs as they become free.  With a fixed share for each the slowest
    // one ends the launch: 32 layers of 8192 tokens and 8 heads (32768 tiles, 1 GiB) take 339 us dealt out and 369 to 375 with
    // a fixed share at 6 or 4 a SM, 12288 tiles 140 and 150.  Long means one and a half times the CTAs that run together (6 a SM
    // at least): below that a mostly empty second wave costs more than it evens out.  us dealt out / fixed share: 4096 tiles
    // (1.15 waves) 60 / 56, 5120 (1.44) 66 / 66, 5500 (1.55) 70 / 72, 6656 (1.87) 79 / 84; 16 KiB tiles (4 heads) 7168 (1.01) 57 /
    // 49, 9216 (1.30) 64 / 60, 11000 (1.55) 70 / 70, 13312 (1.87) 81 / 83.  Over NVLink the link bounds either.
    const uint64_t tiles = tile_bytes < (128u << 10) ? (128u << 10) / tile_bytes : 1u;
    const uint64_t want = (total + tiles - 1) / tiles;
    const int together = std::max(grid, 6 * sms);
    if (want > (uint64_t)together + (uint64_t)together / 2u) {
      grid = (int)(want < (1u << 30) ? want : (1u << 30));
      resident = together;
    }
    if (threads <= 0) threads = 64;      // the second warp zeroes tails; 12 CTAs of 128 threads would not fit the registers
  }
  if ((uint64_t)grid > total) grid = (int)total;
  if (threads <= 0) threads = use_tma ? 128 : 512;
  if (threads > 512) threads = 512;
  threads = (threads + 31) / 32 * 32;
  if (tma) {
    if (tile_bytes % 128 != 0 || tile_bytes > kSmemBudget) return (int)cudaErrorInvalidValue;
    // the shared-memory budget of an SM is split among the CTAs meant to live on it together
    const uint32_t ctas_per_sm = sms > 0 ? (uint32_t)((std::min(grid, resident) + sms - 1) / sms) : 1u;
    uint32_t stages = kSmemBudget / (ctas_per_sm > 0 ? ctas_per_sm : 1u) / tile_bytes;
    if (stages > (uint32_t)kMaxStages) stages = kMaxStages;
    if (stages < 1) stages = 1;
    // BLLM_KVTRANS_TMA_STAGES caps the pipeline depth: fewer stages = less shared memory per
    // CTA, so that CTAs of launches on different streams can share an SM.
    static const int env_stages = [] {
      const char* v = getenv("BLLM_KVTRANS_TMA_STAGES");
      return v != nullptr ? atoi(v) : 0;
    }();
    if (env_stages > 0 && stages > (uint32_t)env_stages) stages = (uint32_t)env_stages;
    if (a.tma_stages > 0 && stages > a.tma_stages) stages = a.tma_stages;
    if (a.store_form != 0u && !kvt_tile_is_flat(&a.dst, a.n_heads, a.tile_tokens, a.tile_order)) return (int)cudaErrorInvalidValue;
    const uint64_t per_cta = (total + grid - 1) / grid;
    if (stages > per_cta + 1) stages = (uint32_t)per_cta + 1;
    if (stages < 1) stages = 1;
    const size_t smem = (size_t)stages * tile_bytes + kMaxStages * sizeof(uint64_t);
    return (int)launch_impl<KVT_MODE_COPY, true>(a, grid, threads, stages, tile_bytes, smem, stream);
  }
  cudaError_t expand;
  switch (a.mode) {
    case KVT_MODE_COPY:
      return (int)launch_impl<KVT_MODE_COPY, false>(a, grid, threads, 0, 0, 0, stream);
    case KVT_MODE_BF16_TO_MXFP8:
      return (int)launch_impl<KVT_MODE_BF16_TO_MXFP8, false>(a, grid, threads, 0, 0, 0, stream);
    default:
      if ((expand = launch_expand(a, grid_ctas, threads_asked, sms, total, stream)) != cudaErrorNotSupported) return (int)expand;
      return (int)launch_impl<KVT_MODE_MXFP8_TO_BF16, false>(a, grid, threads, 0, 0, 0, stream);
  }
}
