// Block-sparse flash-attention forward for sm_100a: TMA-fed tcgen05.mma with S/P and O
// accumulators in tensor memory.
//
// Replaces, for this framework, the forward of the flash-attention fork that the reference calls
// at orchestrated_attn/orchestrated_attn_impl.py:326-337 (one call per scheduled tile) and the
// running-state Triton kernel at easy_context/dist_flash_attn/lightseq_async_attn.py:110-215.
// Differences by design: one launch walks a whole list of key/value segments per query block
// (carrying the running max / sum / O in registers and TMEM, so no merge kernel between tiles),
// segments may live in different buffers (own K/V, a staging ring, a peer GPU's memory reached
// through a unicast TMA tensor map), and the epilogue can either overwrite (O, lse) or merge into
// an existing partial (O, lse) — possibly a mailbox in a peer GPU's memory.
//
// CTA: warps 0-3 softmax / correction / epilogue of sub-tile 0 (one thread per query
// row, 128 score columns each), warps 4-7 the same for sub-tile 1, then one TMA producer warp and
// the tcgen05.mma issuer warps (one elected thread each; the first owns the TMEM allocation). The two
// sub-tiles run ping-pong, so that the tensor core works on one while the softmax warps work on
// the other:
//   FEW = false: 256 query rows, 128 per sub-tile; both sub-tiles visit every key tile
//   FEW = true:  up to 128 query rows, the same ones in both sub-tiles, which take the key tiles in
//                turn (decoding: a handful of rows behind a long cache)
// TMEM (512 columns):
//   FEW = false: S 128 | P0 64 | P1 64 | O0 128 | O1 128. The score tile is shared: a softmax thread has its row's
//                128 scores in registers 300 clocks after they are there, and from then on the other sub-tile's
//                next scores may be computed. Q K^T and P V then have an issuing warp each.
//   FEW = true:  S0 | S1 | O0 | O1, P (bf16) overwrites the first 64 columns of its S; one issuing warp.
// P is consumed from TMEM as the A operand of the PV product.
//
// Two kinds of launches use the kernel. Table launches (ua_attn_fwd) read rows, segments and tiles
// from device tables. Dense launches (ua_attn_fwd_dense: all queries against all keys, causal or
// not) carry their one row and segment in the kernel parameters, so that nothing is uploaded, and
//   * pack the query heads of a key/value head: row r of a tile is query token r / G, head r % G
//     (G heads of a group, a power of two), so that a decoding step reads its cache once per
//     key/value head and not once per query head;
//   * split the keys over several CTAs when the rows alone leave SMs idle: every part writes its
//     normalised fp32 O and lse, and combine_kernel merges them (see plan_dense).
#include "arg_blocks.h"
#include "attn_common.cuh"
#include "host_common.cuh"
#include "ptx.cuh"

namespace ua {

constexpr int FWD_SOFTMAX_WARPS = 8;
constexpr int FWD_TMA_WARP = 8;
constexpr int FWD_QK_WARP = 9;         // issues S = Q K^T; owns the TMEM allocation
constexpr int FWD_PV_WARP = 10;        // issues O += P V
// three warpgroups (the last one: TMA, MMA and an idle warp), so that the register file can be
// re-balanced by warpgroup: a softmax thread holds its row's 128 scores besides everything else (the assembler
// allocates for the new number behind setmaxnreg); 2 x 216 + 72 <= 3 x 168. (FEW: 8 bytes of spills, 36 of reloads, by -Xptxas -v.)
constexpr int FWD_THREADS = 384;
constexpr int FWD_REGS_LAUNCH = 168, FWD_REGS_LOAD = 72, FWD_REGS_SOFTMAX = 216;
static_assert(2 * FWD_REGS_SOFTMAX + FWD_REGS_LOAD <= 3 * FWD_REGS_LAUNCH, "setmaxnreg may only redistribute the launch-time pool");
// What a pair of 128 x 128 tiles (one of each sub-tile) takes. The tensor core needs 2048 clocks for its 32 products,
// the special-function units the same for the exponentials. Before, one thread issued all products and P overwrote S:
// 3320 clocks a pair. With the softmax left out (P handed on as it came) the same products took 2980, because the
// tensor core accepts an instruction only when the one before has started, so that every wait (70 clocks even if
// the phase is complete) and commit (30) of the issuing thread leaves it idle, ten of them a pair: two issuing
// warps 2210. And a sub-tile's cycle was its softmax plus its own products; with a shared score tile Q K^T of the next
// tile no longer waits for P V. What is left of it follows the score tile: loaded into registers (290 clocks), seen by the
// issuing warp (230), Q K^T (512 - 630), seen by the softmax warps (290), twice a pair: 2850.
// The instructions of all roles are kept few and close together (one vote for all that is rare, errors reported by a call,
// loops over segments not unrolled, 32-bit divisions, operand descriptors by addition): the instruction cache missed 99
// times a pair before, 22 now, and every miss stops all four warps of a sub-tile; builds that differ in nothing but that
// (15 and 53 misses a pair) took 918 and 968 us for 16384 tokens, 8 heads. B200, us, before -> now: 8192 causal tokens, 32 heads
// 510 -> 432; 16384 tokens, 8 heads 990 -> 847, 32 heads 3450 -> 3050 (1275 -> 1440 TFLOP/s); 512 queries behind 32768 keys, 32 / 8
// heads 260 -> 222; 1000 causal tokens, 32 / 8 heads 26.6 -> 22.5 (19 with early launches and the shorter
// start of an item). Part of the exponentials as a polynomial of degree 5 on the FMA
// pipe (1/8, 1/4, 3/8 of them, at the 914 us of the time): 924, 956, 1048 us. P handed over in two parts (96 + 32 keys): 2 %
// slower in this form.
constexpr int FWD_TILE_BYTES = ATTN_TILE * ATTN_D * 2;  // 32 KB: [2 d-halves][128 rows][128 B]

struct FwdRow {
  int q_src;      // slot in tmQ
  int q_start;    // first query token inside that source
  int q_len;      // query tokens in this block row
  int seg_begin;  // [seg_begin, seg_end) into segs
  int seg_end;
  int o_slot;     // slot in the output tables
  int o_start;    // first output row inside that slot
  int accumulate; // 1: merge with the (O, lse) already stored there
  int q_wait_flag;   // staging flag of the query block (0: in place), see AttnSeg::wait_flag
  int q_wait_count;
};

struct FwdParams {
  CUtensorMap tmQ[ATTN_MAX_SRC];
  CUtensorMap tmK[ATTN_MAX_SRC];
  CUtensorMap tmV[ATTN_MAX_SRC];
  __nv_bfloat16* o_ptr[ATTN_MAX_SRC];
  float* lse_ptr[ATTN_MAX_SRC];
  long o_row_stride[ATTN_MAX_SRC];   // elements between consecutive tokens (Nh * D)
  long o_batch_stride[ATTN_MAX_SRC];
  long lse_head_stride[ATTN_MAX_SRC];
  long lse_batch_stride[ATTN_MAX_SRC];
  const FwdRow* rows;
  const AttnSeg* segs;
  const int2* tiles;   // (row index, 256-row tile index inside the row), heaviest first
  int n_tiles;
  int n_heads;
  int kv_group;        // query heads per key/value head
  float scale_log2;    // softmax scale * log2(e)
  int* status;
  // dense launches (rows == nullptr)
  FwdRow dense_row;
  AttnSeg dense_seg;
  int pack_shift;      // log2 of the query heads packed into the rows of a tile (0 in table launches)
  int n_split;         // CTAs that share the keys of a tile
  float* part_o;       // not null: fp32 partial results [batch, parts, tokens, heads, 128] ...
  float* part_lse;     // ... and [batch, parts, tokens, heads]; parts = n_split
  int n_parts;
  int tail_heads;      // see item_index
  int persist;         // CTAs take over further items (0: one item per CTA)
  StageParams stage;   // optional in-kernel staging of remote K/V (and Q) blocks
  KernelTrace trace;   // optional per-CTA time stamps
};

// One work item of a launch: what a CTA of a grid without cancellation would have been.
struct FwdItem {
  FwdRow row;
  int row_idx;
  int batch, split;
  int q_head, kv_head;       // query head of packed row 0, key/value head
  int r0, rows_here;         // first (packed) row inside the block row, valid rows
  int tok0, tok_last;        // their query tokens
  int linear;                // index in the grid (time stamps)
  int exists;                // 0: there is no further item
};
// What the producer hands to the other roles: the item, the key tiles it visits and its first segments, which would
// otherwise be a global-memory latency at the beginning of every item and segment of every role.
constexpr int FWD_SEG_CACHE = 4;
struct FwdWork : FwdItem {
  int total;
  AttnSeg seg[FWD_SEG_CACHE];
};

// Where results go, copied into shared memory at the start: kernel parameters that are indexed by a
// run-time slot, or have not been touched for a while, come through the constant cache with several
// hundred clocks a miss.
struct FwdOut {
  __nv_bfloat16* o;
  float* lse;
  long o_row_stride, o_batch_stride, lse_head_stride, lse_batch_stride;
};
template <bool FEW>
struct FwdHot {
  FwdOut out[FEW ? 1 : ATTN_MAX_SRC];      // (FEW launches are dense: one slot)
  float* part_o;         // as in FwdParams
  float* part_lse;
  int n_parts, n_heads, pack_shift;
};

template <bool FEW>
struct __align__(1024) FwdSmem {
  static constexpr int STAGES = FEW ? 3 : 2;      // (the second Q tile's room goes to the rings)
  uint8_t q[FEW ? 1 : 2][FWD_TILE_BYTES];
  uint8_t k[STAGES][FWD_TILE_BYTES];
  uint8_t v[STAGES][FWD_TILE_BYTES];
  uint8_t o_stage[FEW ? 1 : FWD_SOFTMAX_WARPS][FEW ? 16 : 4096];   // see fwd_epilogue
  uint64_t q_full[2];
  uint64_t k_full[STAGES];
  uint64_t k_empty[STAGES];
  uint64_t v_full[STAGES];
  uint64_t v_empty[STAGES];
  uint64_t s_full[2];
  uint64_t p_full[2];
  uint64_t q_empty;
  uint64_t s_free;       // the scores have been read into registers
  uint64_t pv_done[2];   // O += P V of a tile is complete: P may be overwritten, O read
  uint4 clc;             // response of a cancellation request
  uint64_t clc_full;
  FwdWork item[2];       // item number n in slot n & 1
  uint64_t item_full[2];
  uint64_t item_empty[2];
  FwdHot<FEW> hot;
  float2 stat[FEW ? ATTN_TILE : 1];     // sub-tile 1's reference maximum and sum per row, for sub-tile 0
  uint64_t stat_full;    // ... and its O is complete
  uint64_t merged;       // sub-tile 0 has read both
  uint32_t tmem_base;
  int abort_flag;
  int stage_slot;
};
static_assert(sizeof(FwdSmem<false>) + 1024 <= 232448, "FwdSmem exceeds the 227 KB a CTA may use");
static_assert(sizeof(FwdSmem<true>) + 1024 <= 232448, "FwdSmem exceeds the 227 KB a CTA may use");

// 128-key tiles [first, end) of a segment that the query tokens [t0, t_last] have to visit (tiles
// above the upper or below the lower bound of all of them are skipped).
struct TileRange { int first, end; };
__host__ __device__ __forceinline__ TileRange seg_tiles(const AttnSeg& sg, int t0, int t_last) {
  TileRange tr{0, (sg.len + ATTN_TILE - 1) / ATTN_TILE};
  if (sg.causal & SEG_UPPER) {
    const int last = t_last + sg.diag;  // largest allowed key index
    const int nc = last < 0 ? 0 : last / ATTN_TILE + 1;
    tr.end = nc < tr.end ? nc : tr.end;
  }
  if (sg.causal & SEG_LOWER) {
    const int lo = t0 + sg.lo < 0 ? 0 : (t0 + sg.lo) / ATTN_TILE;
    tr.first = lo < tr.end ? lo : tr.end;
  }
  return tr;
}

// Optional pipeline trace (compile with -DUA_FWD_PROF): CTA (0, 0) records clock64() at the
// hand-over points of one key tile of every role into g_fwd_prof; ua_fwd_prof_read copies it out.
#ifdef UA_FWD_PROF
__device__ long long g_fwd_prof[64];
#define FWD_PROF(cond, slot) do { if ((cond) && blockIdx.x == 0 && blockIdx.y == 0) g_fwd_prof[slot] = clock64(); } while (0)
#else
#define FWD_PROF(cond, slot) do { } while (0)
#endif
constexpr int FWD_PROF_TILE = 8;
constexpr int FWD_PROF_SPAN = 32;      // tiles between the stamps 0 and 5 of the MMA warp


template <bool FEW>
__device__ __forceinline__ FwdItem fwd_item(const FwdParams& p, int bx, int by) {
  FwdItem it;
  constexpr int CTA_ROWS = FEW ? ATTN_TILE : 2 * ATTN_TILE;
  const bool dense = p.rows == nullptr;
  // (packed launches: `head` is the key/value head and stands for all its query heads)
  const ItemIndex ix = item_index(bx, p.n_tiles, gridDim.x / p.n_tiles, p.tail_heads);
  const int head = ix.head, i = ix.tile;
  // dense tiles run from the last rows to the first: under a causal mask the heaviest ones come first
  const int2 tl = dense ? make_int2(0, (p.n_tiles - 1 - i) / p.n_split) : p.tiles[i];
  it.split = dense ? (p.n_tiles - 1 - i) % p.n_split : 0;
  it.batch = by;
  it.row = dense ? p.dense_row : p.rows[tl.x];
  it.row_idx = tl.x;
  it.q_head = head << p.pack_shift;
  it.kv_head = it.q_head / p.kv_group;
  it.r0 = tl.y * CTA_ROWS;
  it.rows_here = min(CTA_ROWS, (it.row.q_len << p.pack_shift) - it.r0);
  it.tok0 = it.r0 >> p.pack_shift;
  it.tok_last = (it.r0 + it.rows_here - 1) >> p.pack_shift;
  it.linear = by * gridDim.x + bx;
  it.exists = 1;
  return it;
}
__device__ __forceinline__ AttnSeg fwd_seg(const FwdParams& p, int e) {
  return p.rows == nullptr ? p.dense_seg : p.segs[e];
}
// key tiles of a segment that the item visits: all of them, or its share of a split launch
__device__ __forceinline__ TileRange fwd_tiles(const FwdParams& p, const FwdItem& it, const AttnSeg& sg) {
  TileRange tr = seg_tiles(sg, it.tok0, it.tok_last);
  if (p.n_split > 1) {
    const int n = tr.end - tr.first, base = tr.first;
    // (in 32 bits: a 64-bit division is a hundred instructions. q and r are n's quotient and remainder by n_split <= 2^16, so that
    // no product here exceeds max(n, n_split^2 - n_split).)
    const unsigned q = static_cast<unsigned>(n) / p.n_split, r = static_cast<unsigned>(n) % p.n_split;
    tr.first = base + static_cast<int>(q * it.split + r * it.split / p.n_split);
    tr.end = base + static_cast<int>(q * (it.split + 1) + r * (it.split + 1) / p.n_split);
  }
  return tr;
}
__device__ __forceinline__ void fwd_publish(const FwdParams& p, const FwdItem& it, FwdWork& dst) {
  static_cast<FwdItem&>(dst) = it;
  int n = 0;
#pragma unroll 1
  for (int e = it.row.seg_begin; e < it.row.seg_end; ++e) {
    const AttnSeg sg = fwd_seg(p, e);
    const TileRange tr = fwd_tiles(p, it, sg);
    n += tr.end - tr.first;
    if (e - it.row.seg_begin < FWD_SEG_CACHE) dst.seg[e - it.row.seg_begin] = sg;
  }
  dst.total = n;
}

// The output of one item: this thread's row (l: row sum, m_use: reference maximum, `any`: its sub-tile has
// seen a key tile) normalised, merged with what is there (row.accumulate) or written as a fp32 part
// of a split launch.
// `ready` waits until the last product is complete; what does not depend on it comes first.
template <typename Ready>
__device__ __forceinline__ void fwd_epilogue(FwdSmem<false>& s, uint32_t slot, uint32_t tO, float l, float m_use, bool any, Ready ready) {
  const FwdItem& it = s.item[slot];
  const float NEG_INF = -INFINITY;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = warp >> 2, quad = warp & 3;
  const int psh = s.hot.pack_shift;
  const int r_cta = w * ATTN_TILE + quad * 32 + lane;
  const int rows_here = it.rows_here;
  const bool valid_row = r_cta < rows_here;
  const int r_blk = (it.r0 + r_cta) >> psh;
  const int hmask = (1 << psh) - 1;
  const int qh = it.q_head + (r_cta & hmask);                      // query head of this row
  const FwdOut& od = s.hot.out[it.row.o_slot];
  const long orow = static_cast<long>(it.row.o_start + r_blk);
  float* lptr = od.lse + it.batch * od.lse_batch_stride + qh * od.lse_head_stride + orow;
  float lse = NEG_INF;
  float inv = 0.f;
  // (a row whose keys were all masked has m_use = -inf and l = 0)
  if (any && l > 0.f && m_use > NEG_INF) {
    lse = (m_use + log2f(l)) * 0.6931471805599453f;
    inv = 1.0f / l;
  }
  float w_old = 0.f, w_new = 1.f;
  if (it.row.accumulate && valid_row) {
    const float lse_old = *lptr;
    const float mx = fmaxf(lse_old, lse);
    if (mx == NEG_INF) {
      w_old = 0.f; w_new = 0.f;
    } else {
      const float eo = __expf(lse_old - mx), en = __expf(lse - mx);
      const float tot = eo + en;
      w_old = eo / tot; w_new = en / tot;
      lse = mx + __logf(tot);
    }
  }
  const float fnew = inv * w_new;
  // fp32 part of a split launch: rows of 128 floats, [batch, parts, tokens, heads]
  const bool f32 = s.hot.part_o != nullptr;
  const long part0 = f32 ? (static_cast<long>(it.batch) * s.hot.n_parts + it.split) * it.row.q_len : 0;
  if (f32) {
    lptr = s.hot.part_lse + (part0 + r_blk) * s.hot.n_heads + qh;
    if (any && l != l) lse = l;          // a NaN score makes the whole row one without keys (combine_kernel), not this part
  }
  if (valid_row) *lptr = lse;
  if (!it.row.accumulate) {
    // A thread owns a row, so storing from registers would scatter 16 bytes to each of 32 rows per
    // instruction. The warps turn their blocks of 32 rows x 128 bytes around in shared memory instead
    // (16-byte chunks swizzled by row: no bank conflicts either way) and store four whole rows of a block
    // at a time. From the end of an item's products to its last store 8800 clocks before, 3900 now (with the
    // destinations in shared memory); forward (us): 512 queries behind 32768 keys 288 -> 281, 4 x 2000
    // tokens 168 -> 165, causal 8k tokens, 32 heads 508 -> 501.
    // (Without a key tile, `any` false, fnew is 0 and what tensor memory holds is not used.)
    uint8_t* blk = s.o_stage[warp];
    const int sub = lane >> 3, ch = lane & 7;                      // row of four, 16-byte chunk
    const long row_bytes = f32 ? static_cast<long>(s.hot.n_heads) * ATTN_D * 4 : od.o_row_stride * 2;
    const int head_bytes = f32 ? ATTN_D * 4 : ATTN_D * 2;
    const int rc0 = w * ATTN_TILE + quad * 32 + sub;               // this lane's first row inside the CTA's tile
    // row 0 of the CTA's tile
    uint8_t* base = f32 ? reinterpret_cast<uint8_t*>(s.hot.part_o + ((part0 + it.tok0) * s.hot.n_heads + it.q_head) * ATTN_D)
                        : reinterpret_cast<uint8_t*>(od.o + it.batch * od.o_batch_stride +
                                                     (it.row.o_start + static_cast<long>(it.tok0)) * od.o_row_stride +
                                                     static_cast<long>(it.q_head) * ATTN_D);
    base += ch * 16;
    uint8_t* dst[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i] = base + ((rc0 + i * 4) >> psh) * row_bytes + ((rc0 + i * 4) & hmask) * head_bytes;
    ready();
#pragma unroll 1
    for (int c = 0; c * 128 < head_bytes; ++c) {
      if (f32) {
        uint32_t ov[32];
        tmem_ld_x32(tO + c * 32, ov);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float f[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) f[i] = (fnew == 0.f) ? 0.f : __uint_as_float(ov[q * 4 + i]) * fnew;
          *reinterpret_cast<float4*>(blk + sw128_offset(lane, q)) = make_float4(f[0], f[1], f[2], f[3]);
        }
      } else {
        uint32_t ov[2][32];
        tmem_ld_x32(tO + c * 64, ov[0]);
        tmem_ld_x32(tO + c * 64 + 32, ov[1]);
        tmem_wait_ld();
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = (fnew == 0.f) ? 0.f : __uint_as_float(ov[hf][q * 8 + i]) * fnew;
            *reinterpret_cast<uint4*>(blk + sw128_offset(lane, hf * 4 + q)) =
                make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
        }
      }
      __syncwarp();
      uint4 val[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) val[i] = *reinterpret_cast<const uint4*>(blk + sw128_offset(i * 4 + sub, ch));
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (rc0 + i * 4 < rows_here) *reinterpret_cast<uint4*>(dst[i]) = val[i];
        dst[i] += 128;
      }
      __syncwarp();
    }
    return;
  }
  // a merge with what is there: straight from registers
  ready();
  __nv_bfloat16* optr = od.o + it.batch * od.o_batch_stride + orow * od.o_row_stride + static_cast<long>(qh) * ATTN_D;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    uint32_t ov[32];
    if (any) {
      tmem_ld_x32(tO + c * 32, ov);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) ov[i] = 0u;
    }
    if (valid_row) {
      uint4* d4 = reinterpret_cast<uint4*>(optr + c * 32);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = (fnew == 0.f) ? 0.f : __uint_as_float(ov[q * 8 + i]) * fnew;
        const uint4 old = d4[q];
        const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float lo = __uint_as_float(ow[i] << 16);
          const float hi = __uint_as_float(ow[i] & 0xFFFF0000u);
          f[2 * i] += w_old * lo;
          f[2 * i + 1] += w_old * hi;
        }
        uint4 o;
        o.x = pack_bf16x2(f[0], f[1]);
        o.y = pack_bf16x2(f[2], f[3]);
        o.z = pack_bf16x2(f[4], f[5]);
        o.w = pack_bf16x2(f[6], f[7]);
        d4[q] = o;
      }
    }
  }
}

// One step of a transpose of 16-byte pieces over lanes: of the pair (a, b), a lane with `odd` gives a for its partner's b.
template <int XOR>
__device__ __forceinline__ void swap_pieces(uint4& a, uint4& b, int odd) {
  uint4 x = odd ? a : b;
  x.x = __shfl_xor_sync(0xFFFFFFFFu, x.x, XOR);
  x.y = __shfl_xor_sync(0xFFFFFFFFu, x.y, XOR);
  x.z = __shfl_xor_sync(0xFFFFFFFFu, x.z, XOR);
  x.w = __shfl_xor_sync(0xFFFFFFFFu, x.w, XOR);
  if (odd) a = x;
  else b = x;
}

// FEW: the output of one item of up to 128 rows, of whose key tiles each sub-tile has seen half. The rows are the same, and so are their
// lanes in tensor memory: sub-tile 0's warps take both sub-tiles' O from there, and sub-tile 1's maximum and sum
// from shared memory, and write one result. Two fp32 parts per CTA and a launch that merged them -> this (B200, us, cold L2): 16
// sequences of 8123 keys, one query, 32 / 8 heads 105.5 -> 103.4; 6 of 2449 keys, 16 heads 39.9 -> 36; 36 queries behind
// 1913 keys, 8 heads 21.5 -> 19.5.
__device__ __forceinline__ void few_epilogue(FwdSmem<true>& s, uint32_t slot, uint32_t tO, float l0, float m0) {
  const FwdWork& it = s.item[slot];
  const float NEG_INF = -INFINITY;
  const int r = threadIdx.x;                                       // row = thread: warps 0-3
  const float2 other = s.stat[r];
  const float m = fmaxf(m0, other.x);
  const float a0 = fast_exp2(m0 - m), a1 = fast_exp2(other.x - m);
  const float l = (m0 > NEG_INF || l0 != l0 ? a0 * l0 : 0.f) + (other.x > NEG_INF || other.y != other.y ? a1 * other.y : 0.f);
  const bool live = l > 0.f && m > NEG_INF, use0 = live && m0 > NEG_INF, use1 = live && other.x > NEG_INF;
  const float lse0 = live ? (m + log2f(l)) * 0.6931471805599453f : NEG_INF;
  const float f0 = a0 / l, f1 = a1 / l;
  const int psh = s.hot.pack_shift;
  const bool valid_row = r < it.rows_here, f32 = s.hot.part_o != nullptr;
  const int tok = (it.r0 + r) >> psh, qh = it.q_head + (r & ((1 << psh) - 1));
  const FwdOut& od = s.hot.out[0];
  const long part = (static_cast<long>(it.batch) * s.hot.n_parts + it.split) * it.row.q_len + tok;
  float* lptr = f32 ? s.hot.part_lse + part * s.hot.n_heads + qh : od.lse + it.batch * od.lse_batch_stride + qh * od.lse_head_stride + tok;
  // (in a part, a NaN score is handed on: it makes the whole row one without keys, see combine_kernel)
  if (valid_row) *lptr = f32 && l != l ? l : lse0;
  __nv_bfloat16* obase = od.o + it.batch * od.o_batch_stride;
  __nv_bfloat16* optr = obase + tok * od.o_row_stride + static_cast<long>(qh) * ATTN_D;
  float* pptr = s.hot.part_o + (part * s.hot.n_heads + qh) * ATTN_D;
  // (what tensor memory holds of a sub-tile without a key tile, or with all of its keys masked, is not used)
  const auto columns = [&](int c, float (&f)[32]) {
    uint32_t u[32], v[32];
    tmem_ld_x32(tO + c * 32, u);
    tmem_ld_x32(tO + 128 + c * 32, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i)
      f[i] = (use0 ? __uint_as_float(u[i]) * f0 : 0.f) + (use1 ? __uint_as_float(v[i]) * f1 : 0.f);
  };
  // Many rows: four lanes exchange their rows' 16-byte pieces, so that a store covers 64 bytes of each of eight rows (8 of
  // each of 32 otherwise, a quarter of a sector). Causal 1000 tokens, 8 heads 16.0 -> 15.2 us; with the 4 rows of a decode
  // step it cost 0.3 to 1.4 us instead (2 x 600 keys 11.6 -> 12.3).
  if (!f32 && it.rows_here > 32 && ((reinterpret_cast<uintptr_t>(obase) | (od.o_row_stride * 2)) & 15) == 0) {
    const int lane4 = r & 3;
    __nv_bfloat16* dst[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int rr = r - lane4 + k;
      dst[k] = rr < it.rows_here ? obase + static_cast<long>((it.r0 + rr) >> psh) * od.o_row_stride +
                                       static_cast<long>(it.q_head + (rr & ((1 << psh) - 1))) * ATTN_D + lane4 * 8
                                 : nullptr;
    }
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      float f[32];
      columns(c, f);
      uint4 u4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        u4[q] = make_uint4(pack_bf16x2(f[q * 8], f[q * 8 + 1]), pack_bf16x2(f[q * 8 + 2], f[q * 8 + 3]), pack_bf16x2(f[q * 8 + 4], f[q * 8 + 5]),
                           pack_bf16x2(f[q * 8 + 6], f[q * 8 + 7]));
      swap_pieces<1>(u4[0], u4[1], lane4 & 1);
      swap_pieces<1>(u4[2], u4[3], lane4 & 1);
      swap_pieces<2>(u4[0], u4[2], lane4 >> 1);
      swap_pieces<2>(u4[1], u4[3], lane4 >> 1);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (dst[k] != nullptr) *reinterpret_cast<uint4*>(dst[k] + c * 32) = u4[k];
    }
    return;
  }
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    float f[32];
    columns(c, f);
    if (!valid_row) continue;
    if (f32) {
#pragma unroll
      for (int q = 0; q < 8; ++q)
        reinterpret_cast<float4*>(pptr + c * 32)[q] = make_float4(f[q * 4], f[q * 4 + 1], f[q * 4 + 2], f[q * 4 + 3]);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q)        // (8 bytes, as combine_kernel)
        reinterpret_cast<uint2*>(optr + c * 32)[q] = make_uint2(pack_bf16x2(f[q * 4], f[q * 4 + 1]), pack_bf16x2(f[q * 4 + 2], f[q * 4 + 3]));
    }
  }
}

// The columns of a segment that query r sees are [seg_first_of, seg_end_of); both grow with r.
__device__ __forceinline__ int seg_end_of(const AttnSeg& sg, int r) {
  return (sg.causal & SEG_UPPER) ? min(sg.len, r + sg.diag + 1) : sg.len;
}
__device__ __forceinline__ int seg_first_of(const AttnSeg& sg, int r) {
  return (sg.causal & SEG_LOWER) ? max(0, r + sg.lo) : 0;
}
// A branch that is never taken (a CTA's 2^32nd score tile), meant to keep the arrival on s_free, which the other sub-tile's
// scores wait for, in front of the arithmetic behind it. What the compiler makes of it was not looked at; measured (nvcc
// 12.9.86, 16k tokens, 8 heads): 1038 us without it, 917 with it. Another compiler may need it elsewhere, or not at all.
#define PIN if (__builtin_expect(cnt == 0xFFFFFFFFu, 0)) break;

// Persistent CTAs: the grid has one CTA per work item, and a CTA that is done with an item cancels one
// that has not started yet and takes its place (cluster launch control), so that the hardware's own
// dispatch order stays the schedule. The TMA warp runs ahead: it takes over the next item as soon as
// the loads of this one are issued, its Q and first K / V tiles arrive while the softmax warps write
// this item's output, and the MMA warp issues its first scores. TMEM, barriers and descriptors are
// set up once. The producer hands an item over with what the others need of it (number of tiles, first segments), and
// issues a CTA's first loads while tensor memory is being allocated: 512 causal tokens, 8 heads 21.3 -> 14.8 us,
// 12 documents in 16k tokens 406 -> 365. One item per CTA -> this (B200, us): 64
// sequences of 512 keys, one query, 32 heads 184 -> 143; 12 documents in 16k tokens 599 -> 546; window
// 4096 in 16k tokens 1140 -> 1090; 4 x 2000 tokens 192 -> 182; causal 8k 609 -> 588, 16k 2010 -> 1978.
// Launches that stage peers' blocks run one item per CTA (p.persist = 0): their CTAs must be able to
// wait for each other's copies.
template <bool FEW>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ FwdParams p) {
  constexpr int STAGES = FwdSmem<FEW>::STAGES;
  extern __shared__ uint8_t smem_raw[];
  FwdSmem<FEW>& s = *reinterpret_cast<FwdSmem<FEW>*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int psh = p.pack_shift;

  if (p.stage.flags != nullptr) {
    grid_wait();
    // does this CTA read a staged block? then it first helps to empty the copy queue
    const FwdItem it = fwd_item<FEW>(p, blockIdx.x, blockIdx.y);
    trace_stamp(p.trace, it.linear, 0);
    bool waits = it.row.q_wait_flag != 0;
    for (int e = it.row.seg_begin; e < it.row.seg_end && !waits; ++e) waits = fwd_seg(p, e).wait_flag != 0;
    drain_stage_queue(p.stage, waits, it.linear, &s.stage_slot);
  }
  // FEW: warps without a valid row have nothing to do (their scores are never read back). The number is the same for
  // all items of a launch: with more than one row tile all four warps are at work, also in the last one, where those behind
  // its rows see no key.
  const int act_warps = FEW ? (min(ATTN_TILE, p.dense_row.q_len << psh) + 31) / 32 : 4;

  // The producer sets the barriers up, looks up its first item and goes on to load it; the others meet at
  // a named barrier once tensor memory is there as well.
  FwdItem item0;
  if (warp == FWD_TMA_WARP && lane == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.q_full[i], 1);
      mbar_init(&s.s_full[i], 1);
      mbar_init(&s.p_full[i], act_warps);   // one arrival per softmax warp
      mbar_init(&s.pv_done[i], 1);
      mbar_init(&s.item_full[i], 1);
      mbar_init(&s.item_empty[i], (FEW ? 1 : 2) + 2 * act_warps);   // MMA and softmax warps
    }
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&s.k_full[i], 1);
      mbar_init(&s.k_empty[i], 1);
      mbar_init(&s.v_full[i], 1);
      mbar_init(&s.v_empty[i], 1);
    }
    mbar_init(&s.q_empty, 1);
    mbar_init(&s.s_free, act_warps);
    mbar_init(&s.stat_full, act_warps);
    mbar_init(&s.merged, act_warps);
    mbar_init(&s.clc_full, 1);
    s.abort_flag = 0;
    fence_mbar_init();
    grid_wait();
    item0 = fwd_item<FEW>(p, blockIdx.x, blockIdx.y);
    fwd_publish(p, item0, s.item[0]);
  }
  if (warp == 1) {
    if (lane < (FEW ? 1 : ATTN_MAX_SRC))
      s.hot.out[lane] = FwdOut{p.o_ptr[lane], p.lse_ptr[lane], p.o_row_stride[lane], p.o_batch_stride[lane],
                               p.lse_head_stride[lane], p.lse_batch_stride[lane]};
    if (lane == 31) {
      s.hot.part_o = p.part_o;
      s.hot.part_lse = p.part_lse;
      s.hot.n_parts = p.n_parts;
      s.hot.n_heads = p.n_heads;
      s.hot.pack_shift = p.pack_shift;
    }
  }
  if (warp == FWD_QK_WARP) {
    tmem_alloc(&s.tmem_base, 512);
    tmem_relinquish();
  }
  uint32_t tmem_base = 0;
  grid_wait();
  if (p.stage.flags == nullptr) trace_stamp(p.trace, blockIdx.y * gridDim.x + blockIdx.x, 0);
  if (warp == FWD_TMA_WARP) {
    __syncwarp();
    named_barrier_arrive(1, FWD_THREADS);
  } else {
    tc_fence_before_sync();
    named_barrier_sync(1, FWD_THREADS);
    tc_fence_after_sync();
    tmem_base = s.tmem_base;
  }
  WaitCtx wc{&s.abort_flag, p.status, 4000000000ull};
  auto wait = [&](uint64_t* bar, uint32_t parity, int where) -> bool {
    if (mbar_wait_quiet(bar, parity, wc)) return true;
    report_error_call(wc.abort_flag, wc.status, UA_ERR_MBAR_TIMEOUT, where, static_cast<int>(parity));
    return false;
  };

  // Consumers: true once item n + 1 is in its slot (false: there is none, or a wait gave up). They hand
  // item n back by an arrival on item_empty when they have read what they need of it.
  auto next_item = [&](uint32_t n) -> bool {
    const uint32_t m = n + 1;
    return p.persist && wait(&s.item_full[m & 1], ((m >> 1) - ((m & 1) ^ 1)) & 1, 120) && s.item[m & 1].exists != 0;
  };
  auto take_total = [&](uint32_t n) -> int {         // (the MMA issuers need nothing else of an item)
    const int total = s.item[n & 1].total;
    if (p.persist) mbar_arrive(&s.item_empty[n & 1]);
    return total;
  };

  if (warp >= FWD_SOFTMAX_WARPS) {
    reg_dealloc<FWD_REGS_LOAD>();
    if (warp == FWD_TMA_WARP) {
      // =============================== TMA producer and scheduler ==============================
      if (lane == 0) {
        bool ok = true;
        FwdItem it = item0;
        uint32_t j = 0;          // K / V tiles loaded so far
        uint32_t live = 0;       // items with keys so far
        for (uint32_t n = 0; ok; ++n) {
          if (s.item[n & 1].total > 0) {
            const CUtensorMap* tq = &p.tmQ[it.row.q_src];
            tma_prefetch_desc(tq);
            if (!wait_staged(p.stage.flags, it.row.q_wait_flag, it.row.q_wait_count * p.stage.epoch, wc.budget_ns)) {
              report_error_call(wc.abort_flag, wc.status, UA_ERR_FLAG_TIMEOUT, 110, it.row.q_wait_flag);
              ok = false;
            }
            // the previous item's last scores have been computed
            if (ok && live > 0 && !wait(&s.q_empty, (live - 1) & 1, 102)) ok = false;
            for (int w = 0; w < (FEW ? 1 : 2) && ok; ++w) {
              mbar_arrive_expect_tx(&s.q_full[w], FWD_TILE_BYTES);
              const int qrow = it.row.q_start + it.tok0 + ((w * ATTN_TILE) >> psh);
              tma_load_4d(s.q[w], tq, &s.q_full[w], 0, it.q_head, qrow, it.batch);
              tma_load_4d(s.q[w] + 16384, tq, &s.q_full[w], 64, it.q_head, qrow, it.batch);
            }
            ++live;
#pragma unroll 1
            for (int e = it.row.seg_begin; e < it.row.seg_end && ok; ++e) {
              const AttnSeg sg = fwd_seg(p, e);
              const TileRange tr = fwd_tiles(p, it, sg);
              const CUtensorMap* tk = &p.tmK[sg.src];
              const CUtensorMap* tv = &p.tmV[sg.src];
              if (tr.first < tr.end &&
                  !wait_staged(p.stage.flags, sg.wait_flag, sg.wait_count * p.stage.epoch, wc.budget_ns)) {
                report_error_call(wc.abort_flag, wc.status, UA_ERR_FLAG_TIMEOUT, 111, sg.wait_flag);
                ok = false;
                break;
              }
#pragma unroll 1
              for (int t = tr.first; t < tr.end; ++t, ++j) {
                const int st = j % STAGES;
                const uint32_t ph = (j / STAGES) & 1;
                const int krow = sg.start + t * ATTN_TILE;
                if (!wait(&s.k_empty[st], ph ^ 1, 100)) { ok = false; break; }
                mbar_arrive_expect_tx(&s.k_full[st], FWD_TILE_BYTES);
                tma_load_4d(s.k[st], tk, &s.k_full[st], 0, it.kv_head, krow, it.batch);
                tma_load_4d(s.k[st] + 16384, tk, &s.k_full[st], 64, it.kv_head, krow, it.batch);
                if (!wait(&s.v_empty[st], ph ^ 1, 101)) { ok = false; break; }
                mbar_arrive_expect_tx(&s.v_full[st], FWD_TILE_BYTES);
                tma_load_4d(s.v[st], tv, &s.v_full[st], 0, it.kv_head, krow, it.batch);
                tma_load_4d(s.v[st] + 16384, tv, &s.v_full[st], 64, it.kv_head, krow, it.batch);
              }
            }
          }
          if (!ok || !p.persist) break;
          // everything of this item is on its way: take over the next one
          mbar_arrive_expect_tx(&s.clc_full, 16);
          clc_try_cancel(&s.clc, &s.clc_full);
          if (!wait(&s.clc_full, n & 1, 104)) break;
          int bx, by;
          const bool got = clc_read(&s.clc, bx, by);
          if (!got) grid_trigger();               // (not before: with the next kernel pending no CTA can be taken over)
          fence_proxy_async_smem();               // read before the next response may overwrite it
          if (got) it = fwd_item<FEW>(p, bx, by);
          // the slot's previous item (n - 1) is done with
          const uint32_t slot = (n + 1) & 1;
          if (n >= 1 && !wait(&s.item_empty[slot], ((n - 1) >> 1) & 1, 103)) break;
          if (got) fwd_publish(p, it, s.item[slot]);
          else s.item[slot].exists = 0;
          mbar_arrive(&s.item_full[slot]);
          if (!got) break;
        }
      }
    } else if (warp == FWD_QK_WARP || (!FEW && warp == FWD_PV_WARP)) {
      // =============================== MMA issuers ============================================
      if (elect_one()) {             // (not lane == 0: the assembler knows that one thread is left)
        const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);   // S = Q K^T, both K-major
        const uint32_t idesc_o = make_idesc_bf16(128, 128, 0, 1);   // O += P V, V is N-major
        // one base descriptor per operand; a tile and an instruction add their offset (in 16-byte units) to the
        // address field, which cannot carry out of it for addresses inside shared memory
        const uint32_t q_desc = desc_lo(smem_u32(s.q[0]), 16), k_desc = desc_lo(smem_u32(s.k[0]), 16);
        const uint32_t v_desc = desc_lo(smem_u32(s.v[0]), 16384);
        constexpr uint32_t HI = desc_hi_sw128(1024);
        constexpr uint32_t TILE16 = FWD_TILE_BYTES >> 4;
        auto issue_s = [&](int w, int st) {
          const uint32_t qa = q_desc + (FEW ? 0 : w) * TILE16, ka = k_desc + st * TILE16;
          const uint32_t tS = tmem_base + (FEW ? w * 128 : 0);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
            umma_ss_lo<HI, HI>(tS, qa + off, ka + off, idesc_s, kk > 0 ? 1u : 0u);
          }
        };
        auto issue_pv = [&](int w, int st, bool acc) {
          const uint32_t va = v_desc + st * TILE16;
          const uint32_t tP = tmem_base + (FEW ? w * 128 : 128 + w * 64), tO = tmem_base + 256 + w * 128;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            // A: 16 keys = 8 packed columns of P; B: 16 key rows = 2048 B, d-halves 16384 B apart
            umma_ts_lo<HI>(tO, tP + kk * 8, va + ((kk * 2048) >> 4), idesc_o, (acc || kk > 0) ? 1u : 0u);
        };
        bool ok = true;
        uint32_t kv = 0;                  // K / V tiles so far
        uint32_t live = 0;
        // (that O of the previous item has been read out is implied by P of an item's first tile: the same warps
        // write it after their epilogue)
        if constexpr (FEW) {
          uint32_t phase = 0;             // bit w: parity of sub-tile w's next P
          for (uint32_t n = 0; ok; ++n) {
            const int n_total = take_total(n);
            if (n_total > 0) {
              if (!wait(&s.q_full[0], live & 1, 200)) break;
              // key tile j belongs to sub-tile j & 1; its scores are issued two tiles ahead
              auto next_s = [&](int j) -> bool {
                const uint32_t g = kv + j;
                if (!wait(&s.k_full[g % STAGES], (g / STAGES) & 1, 201)) return false;
                tc_fence_after_sync();
                issue_s(j & 1, g % STAGES);
                tc_commit(&s.s_full[j & 1]);
                tc_commit(&s.k_empty[g % STAGES]);
                if (j + 1 == n_total) tc_commit(&s.q_empty);
                return true;
              };
              ok = next_s(0) && (n_total < 2 || next_s(1));
              for (int j = 0; j < n_total && ok; ++j) {
                const int w = j & 1, st = (kv + j) % STAGES;
                if (!wait(&s.v_full[st], ((kv + j) / STAGES) & 1, 203)) { ok = false; break; }
                if (!wait(&s.p_full[w], (phase >> w) & 1, 204)) { ok = false; break; }
                phase ^= 1u << w;
                tc_fence_after_sync();
                issue_pv(w, st, j >= 2);
                tc_commit(&s.pv_done[w]);
                tc_commit(&s.v_empty[st]);
                if (j + 2 < n_total) ok = next_s(j + 2);
              }
              if (!ok) break;
              kv += n_total;
              ++live;
            }
            if (!next_item(n)) break;
          }
        } else if (warp == FWD_QK_WARP) {
          uint32_t use = 0;               // score tiles so far (of both sub-tiles)
          auto scores = [&](int w, int st) -> bool {
            if (use > 0 && !wait(&s.s_free, (use - 1) & 1, 206)) return false;
            ++use;
            tc_fence_after_sync();
            issue_s(w, st);
            tc_commit(&s.s_full[w]);
            return true;
          };
          for (uint32_t n = 0; ok; ++n) {
            const int n_total = take_total(n);
            if (n_total > 0) {
              if (!wait(&s.q_full[0], live & 1, 200)) break;
              if (!wait(&s.q_full[1], live & 1, 202)) break;
              for (int j = 0; j < n_total && ok; ++j, ++kv) {
                const int st = kv % STAGES;
                FWD_PROF(kv == FWD_PROF_TILE, 0);
                FWD_PROF(kv == FWD_PROF_TILE + FWD_PROF_SPAN, 5);
                ok = wait(&s.k_full[st], (kv / STAGES) & 1, 201) && scores(0, st) && scores(1, st);
                if (ok) tc_commit(&s.k_empty[st]);
              }
              if (!ok) break;
              tc_commit(&s.q_empty);
              ++live;
            }
            if (!next_item(n)) break;
          }
        } else {
          auto product = [&](int w, int st, bool acc) -> bool {
            if (!wait(&s.p_full[w], kv & 1, 204 + w)) return false;
            tc_fence_after_sync();
            issue_pv(w, st, acc);
            tc_commit(&s.pv_done[w]);
            return true;
          };
          for (uint32_t n = 0; ok; ++n) {
            const int n_total = take_total(n);
            for (int j = 0; j < n_total && ok; ++j, ++kv) {
              const int st = kv % STAGES;
              ok = wait(&s.v_full[st], (kv / STAGES) & 1, 203) && product(0, st, j > 0) && product(1, st, j > 0);
              if (ok) tc_commit(&s.v_empty[st]);
            }
            if (!ok || !next_item(n)) break;
          }
        }
      }
    }
  } else {
    reg_alloc<FWD_REGS_SOFTMAX>();
    if ((warp & 3) < act_warps) {
      // =============================== softmax + epilogue =====================================
      const int w = warp >> 2;                 // sub-tile
      const int quad = warp & 3;               // TMEM lane quadrant of this warp
      const int r_tile = quad * 32 + lane;     // row inside the 128-row sub-tile
      const int r_cta = (FEW ? 0 : w * ATTN_TILE) + r_tile;   // row inside the CTA's tile
      const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
      const uint32_t tS = tmem_base + lane_base + (FEW ? w * 128 : 0);
      const uint32_t tP = FEW ? tS : tmem_base + lane_base + 128 + w * 64;
      const uint32_t tO = tmem_base + lane_base + 256 + w * 128;
      const float NEG_INF = -INFINITY;
      uint32_t cnt = 0;                        // score tiles of this sub-tile so far
      for (uint32_t n = 0;; ++n) {
        const FwdWork& it = s.item[n & 1];       // (stays in shared memory: the score loop needs the registers)
        auto seg_of = [&](int e) -> AttnSeg {
          const int k = e - it.row.seg_begin;
          return k < FWD_SEG_CACHE ? it.seg[k] : fwd_seg(p, e);
        };
        if (n > 0) trace_stamp(p.trace, it.linear, 0);
        trace_stamp(p.trace, it.linear, 1);
        trace_ident(p.trace, it.linear, it.row_idx);
        float m_use = NEG_INF;   // running reference max, log2 units (already scaled)
        float l = 0.f;           // row sum
        bool ok = true;
        uint32_t j = 0;
#pragma unroll 1
        for (int e = it.row.seg_begin; e < it.row.seg_end && ok; ++e) {
          // Every row of the warp sees all of the tiles [clear_first, clear_end), and no row anything outside
          // [some_first, some_end).
          int t, t_end, clear_first, clear_end, some_first, some_end;
          {
            const AttnSeg sg = seg_of(e);
            const TileRange tr = fwd_tiles(p, it, sg);
            t = tr.first;
            t_end = tr.end;
            const int r_first = (it.r0 + r_cta - lane) >> psh, r_last = (it.r0 + r_cta - lane + 31) >> psh;
            clear_end = seg_end_of(sg, r_first) >> 7;
            some_end = (seg_end_of(sg, r_last) + ATTN_TILE - 1) >> 7;
            some_first = seg_first_of(sg, r_first) >> 7;
            clear_first = (seg_first_of(sg, r_last) + ATTN_TILE - 1) >> 7;
            if (r_cta - lane >= it.rows_here) some_end = 0;              // (rows behind the last one)
          }
#pragma unroll 1
          for (; t < t_end; ++t, ++j) {
            if (FEW && (j & 1) != static_cast<uint32_t>(w)) continue;
            const bool prof = (n == 0) && (j == FWD_PROF_TILE || j == FWD_PROF_TILE + 1) && quad == 0 && lane == 0;
            const int pslot = 8 + w * 24 + (static_cast<int>(j) - FWD_PROF_TILE) * 8;
            (void)prof; (void)pslot;
            FWD_PROF(prof, pslot + 0);
            ok = mbar_wait_quiet(&s.s_full[w], cnt & 1, wc);             // (looked at below)
            FWD_PROF(prof, pslot + 1);
            ++cnt;
            tc_fence_after_sync();
            if (t < some_first || t >= some_end) {
              // Nothing to see here for these 32 rows (a tile that only the other sub-tile, or another warp, needs): P = 0,
              // and neither the maximum nor the sum changes.
              if (!FEW) mbar_arrive_warp(&s.s_free);
              if (j >= (FEW ? 2u : 1u)) ok = mbar_wait_quiet(&s.pv_done[w], cnt & 1, wc) && ok;
              ok = __all_sync(0xFFFFFFFFu, ok);
              if (!ok) break;
              tc_fence_after_sync();
              uint32_t zero[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) zero[i] = 0u;
              tmem_st_x32(tP, zero);
              tmem_st_x32(tP + 32, zero);
              tmem_wait_st();
              tc_fence_before_sync();
              mbar_arrive_warp(&s.p_full[w]);
              continue;
            }
            float sv[ATTN_TILE];
            {
              uint32_t(&raw)[ATTN_TILE] = reinterpret_cast<uint32_t(&)[ATTN_TILE]>(sv);
#pragma unroll
              for (int c = 0; c < 4; ++c)
                tmem_ld_x32(tS + c * 32, reinterpret_cast<uint32_t(&)[32]>(raw[c * 32]));
              tmem_wait_ld();
            }
            if (!FEW) {
              tc_fence_before_sync();
              mbar_arrive_warp(&s.s_free);
              PIN
            }
            FWD_PROF(prof, pslot + 2);
            if (t < clear_first || t >= clear_end) {
              // Columns outside [low, lim) become -inf, 32 at a time and only where some row needs it (two instructions a
              // column with a mask in bits; in a loop over tensor memory, before the scores are read, a masked
              // tile took 1000 clocks more: window of 1024 with sinks, 32k tokens, 350 -> 332 us).
              const AttnSeg sg = seg_of(e);
              const int r = (it.r0 + r_cta) >> psh, r_first = (it.r0 + r_cta - lane) >> psh, r_last = (it.r0 + r_cta - lane + 31) >> psh;
              const int c0 = t * ATTN_TILE;
              const int low = seg_first_of(sg, r) - c0, lim = seg_end_of(sg, r) - c0;
              const int clear_lo = seg_first_of(sg, r_last) - c0, clear_hi = seg_end_of(sg, r_first) - c0;
#pragma unroll
              for (int c = 0; c < ATTN_TILE; c += 32) {
                if (c >= clear_lo && c + 32 <= clear_hi) continue;
                // bit i: column c + i is seen
                const int a = min(max(low - c, 0), 32), b = min(max(lim - c, 0), 32);
                const uint32_t seen = (b > 0 ? 0xFFFFFFFFu >> (32 - b) : 0u) & (a < 32 ? 0xFFFFFFFFu << a : 0u);
#pragma unroll
                for (int i = 0; i < 32; ++i) sv[c + i] = (seen >> i) & 1u ? sv[c + i] : NEG_INF;
              }
            }
            // eight independent running maxima, two new values per instruction: one dependent chain of
            // compares would cost more than the exponentials
            float mx8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) mx8[i] = fmaxf(sv[i], sv[8 + i]);
#pragma unroll
            for (int i = 16; i < ATTN_TILE; i += 16)
#pragma unroll
              for (int k = 0; k < 8; ++k) mx8[k] = fmax3(mx8[k], sv[i + k], sv[i + 8 + k]);
            float mx = fmaxf(fmax3(mx8[0], mx8[1], mx8[2]), fmax3(mx8[3], mx8[4], mx8[5]));
            mx = fmax3(mx, mx8[6], mx8[7]);
            PIN
            mx *= p.scale_log2;
            const float m_new = fmaxf(m_use, mx);
            FWD_PROF(prof, pslot + 6);
            // P V of the tile before is complete: P may be overwritten, and O rescaled
            bool need = false;
            if (j < (FEW ? 2u : 1u)) {
              m_use = m_new;
            } else {
              ok = mbar_wait_quiet(&s.pv_done[w], cnt & 1, wc) && ok;
              tc_fence_after_sync();
              // lazy rescale: only when the running max grew by more than 2^8
              need = (m_new - m_use > 8.0f) || (m_use == NEG_INF && m_new > NEG_INF);
            }
            // (one vote for all that is rare; warp-uniform, because accesses to tensor memory are warp-collective)
            if (__any_sync(0xFFFFFFFFu, need || !ok)) {
              ok = __all_sync(0xFFFFFFFFu, ok);
              if (!ok) break;
              const float alpha = need ? fast_exp2(m_use - m_new) : 1.0f;
              if (need) m_use = m_new;
              l *= alpha;
#pragma unroll 1
              for (int c = 0; c < 8; ++c) {
                uint32_t ov[16];
                tmem_ld_x16(tO + c * 16, ov);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                tmem_st_x16(tO + c * 16, ov);
              }
            }
            FWD_PROF(prof, pslot + 3);
            const float m_eff = (m_use == NEG_INF) ? 0.f : m_use;
            // multiply-add and row sum on packed pairs; four independent partial sums
            const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2);
            const uint64_t nm2 = f2_pack(-m_eff, -m_eff);
            uint64_t ls2[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) ls2[k] = f2_pack(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t pk[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                float x0, x1;
                f2_unpack(f2_fma(f2_pack(sv[c * 32 + 2 * i], sv[c * 32 + 2 * i + 1]), sc2, nm2), x0, x1);
                const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
                ls2[i & 3] = f2_add(ls2[i & 3], f2_pack(p0, p1));
                pk[i] = pack_bf16x2(p0, p1);
              }
              tmem_st_x16(tP + c * 16, pk);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive_warp(&s.p_full[w]);
            PIN
            FWD_PROF(prof, pslot + 4);
            float ls4[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float a, b;
              f2_unpack(ls2[k], a, b);
              ls4[k] = a + b;
            }
            l += (ls4[0] + ls4[1]) + (ls4[2] + ls4[3]);
            FWD_PROF(prof, pslot + 5);
          }
        }
        // ---------------------------------- epilogue --------------------------------------------
        const bool any = j > (FEW ? static_cast<uint32_t>(w) : 0u);
        auto ready = [&]() {
          if (any && ok) ok = mbar_wait_quiet(&s.pv_done[w], (cnt & 1) ^ 1, wc);
          tc_fence_after_sync();
        };
        if constexpr (FEW) {
          ready();
          if (w == 1) {
            s.stat[r_tile] = make_float2(any ? m_use : NEG_INF, any ? l : 0.f);
            tc_fence_before_sync();
            mbar_arrive_warp(&s.stat_full);
            ok = mbar_wait_quiet(&s.merged, n & 1, wc) && ok;      // (O is free for this sub-tile's next item)
          } else {
            ok = mbar_wait_quiet(&s.stat_full, n & 1, wc) && ok;
            tc_fence_after_sync();
            few_epilogue(s, n & 1, tO, any ? l : 0.f, any ? m_use : NEG_INF);
            tc_fence_before_sync();
            mbar_arrive_warp(&s.merged);
          }
        } else {
          fwd_epilogue(s, n & 1, tO, l, m_use, any, ready);
        }
        if (!ok) report_error_call(wc.abort_flag, wc.status, UA_ERR_MBAR_TIMEOUT, 300 + w, static_cast<int>(j));
        trace_stamp(p.trace, it.linear, 2);
        __syncwarp();                            // every lane is done reading the item
        if (lane == 0 && p.persist) mbar_arrive(&s.item_empty[n & 1]);
        if (!__all_sync(0xFFFFFFFFu, ok && next_item(n))) break;
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == FWD_QK_WARP) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// Merge the parts of a split dense launch: O = sum_i w_i O_i with w_i = exp(lse_i - lse), fp32 throughout,
// one warp per (token, head) row, 4 head-dim elements per lane. Bound by reading the parts (they
// mostly sit in L2: 0.5 KB per row and part).
__global__ void __launch_bounds__(256)
combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse, int n_parts, int tokens, int heads,
               __nv_bfloat16* __restrict__ o, long o_row_stride, long o_batch_stride, float* __restrict__ lse,
               long lse_head_stride, long lse_batch_stride, long n_rows) {
  grid_wait();
  grid_trigger();
  const long r = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= n_rows) return;
  const long per_part = static_cast<long>(tokens) * heads;
  const long batch = r / per_part, in = r % per_part;           // in = token * heads + head
  const long first = batch * n_parts * per_part + in;
  float mx = -INFINITY;
  bool bad = false;                    // a NaN score: the row comes out as in a launch without parts, O = 0 and lse = -inf
  for (int i = lane; i < n_parts; i += 32) {
    const float x = part_lse[first + i * per_part];
    bad |= x != x;
    mx = fmaxf(mx, x);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
  if (__any_sync(0xFFFFFFFFu, bad)) mx = -INFINITY;
  float tot = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (mx > -INFINITY) {
#pragma unroll 4
    for (int i = 0; i < n_parts; ++i) {
      const float w = __expf(part_lse[first + i * per_part] - mx);
      const float4 v = *reinterpret_cast<const float4*>(part_o + (first + i * per_part) * ATTN_D + lane * 4);
      tot += w;                          // (w = 0 also times what is not finite, as P V does with P = 0)
      acc.x += w * v.x;
      acc.y += w * v.y;
      acc.z += w * v.z;
      acc.w += w * v.w;
    }
  }
  const float inv = tot > 0.f ? 1.f / tot : 0.f;
  const long tok = in / heads, head = in % heads;
  uint2 ov;
  ov.x = pack_bf16x2(acc.x * inv, acc.y * inv);
  ov.y = pack_bf16x2(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(o + batch * o_batch_stride + tok * o_row_stride + head * ATTN_D + lane * 4) = ov;
  if (lane == 0)
    lse[batch * lse_batch_stride + head * lse_head_stride + tok] = tot > 0.f ? mx + __logf(tot) : -INFINITY;
}

}  // namespace ua

using namespace ua;

// Register (or, with buf = NULL, remove) the per-CTA trace buffer of the current device:
// which = 0 forward, 1 backward; buf = 4 * cap 64-bit words of device memory (see KernelTrace).
extern "C" int ua_set_kernel_trace(int which, unsigned long long* buf, int cap) {
  int dev = 0;
  UA_CUDA(cudaGetDevice(&dev));
  if (which < 0 || which > 1 || dev >= 64) UA_FAIL("ua_set_kernel_trace: bad kernel or device index");
  trace_registry()[which * 64 + dev] = TraceSlot{buf, buf != nullptr ? cap : 0};
  return 0;
}

// Hits and misses of the host-side tensor-map cache since the library was loaded.
extern "C" int ua_tmap_cache_stats(unsigned long long* hits, unsigned long long* misses) {
  TmapCache& c = tmap_cache();
  while (c.busy.test_and_set(std::memory_order_acquire)) {}
  *hits = c.hits;
  *misses = c.misses;
  c.busy.clear(std::memory_order_release);
  return 0;
}

#ifdef UA_FWD_PROF
extern "C" int ua_fwd_prof_read(long long* host64) {
  UA_CUDA(cudaMemcpyFromSymbol(host64, g_fwd_prof, sizeof(long long) * 64));
  return 0;
}
#endif

// rows_head / rows_tok: heads and tokens per 128-row tile (1 x 128, or a packed group of heads)
static int encode_src(CUtensorMap* tm, const UaTensorSrc& t, uint32_t rows_head = 1) {
  uint64_t dims[4] = {ATTN_D, static_cast<uint64_t>(t.heads), static_cast<uint64_t>(t.tokens),
                      static_cast<uint64_t>(t.batch)};
  uint64_t str[3] = {static_cast<uint64_t>(t.head_stride) * 2,
                     static_cast<uint64_t>(t.token_stride) * 2,
                     static_cast<uint64_t>(t.batch_stride > 0 ? t.batch_stride : t.token_stride * t.tokens) * 2};
  uint32_t box[4] = {64, rows_head, ATTN_TILE / rows_head, 1};
  return make_tmap_2byte(tm, t.ptr, 4, dims, str, box);
}

template <bool FEW>
static int launch_fwd(const FwdParams& p, int heads, int batch, cudaStream_t stream) {
  static int smem_set[64] = {0};
  const int smem_bytes = sizeof(FwdSmem<FEW>) + 1024;
  int dev = 0;
  UA_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !smem_set[dev]) {
    UA_CUDA(cudaFuncSetAttribute(attn_fwd_kernel<FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    if (dev < 64) smem_set[dev] = 1;
  }
  dim3 grid(p.n_tiles * heads, batch, 1);
  UA_CUDA(launch_kernel(attn_fwd_kernel<FEW>, grid, FWD_THREADS, smem_bytes, stream, p.stage.flags == nullptr, p));
  return 0;
}

static int set_trace(FwdParams& p) {
  int dev = 0;
  UA_CUDA(cudaGetDevice(&dev));
  const TraceSlot ts = dev < 64 ? trace_registry()[0 * 64 + dev] : TraceSlot{nullptr, 0};
  p.trace.buf = ts.buf;
  p.trace.cap = ts.cap;
  return 0;
}

// rows / segs / tiles are device pointers (prepared once per plan); q/k/v/out tables are host
// arrays of n_q / n_kv / n_out entries.
extern "C" int ua_attn_fwd(const UaTensorSrc* q_src, int n_q, const UaTensorSrc* k_src,
                           const UaTensorSrc* v_src, int n_kv, const UaOutDst* outs, int n_out,
                           const void* rows_dev, const void* segs_dev, const void* tiles_dev,
                           int n_tiles, int n_heads, int n_kv_heads, int batch,
                           float softmax_scale, int* status, const void* copy_tasks_dev,
                           int n_copy_tasks, int n_copy_ctas, unsigned int* stage_flags,
                           int stage_epoch, unsigned int* stage_ticket, cudaStream_t stream) {
  if (n_q > ATTN_MAX_SRC || n_kv > ATTN_MAX_SRC || n_out > ATTN_MAX_SRC)
    UA_FAIL("ua_attn_fwd: too many sources (max %d)", ATTN_MAX_SRC);
  if (n_tiles <= 0) return 0;
  if (check_sources("ua_attn_fwd", batch, n_heads, n_kv_heads, q_src, n_q, k_src, v_src, n_kv)) return -1;
  FwdParams p;
  memset(&p, 0, sizeof(p));
  for (int i = 0; i < n_q; ++i)
    if (encode_src(&p.tmQ[i], q_src[i])) return -1;
  for (int i = 0; i < n_kv; ++i) {
    if (encode_src(&p.tmK[i], k_src[i])) return -1;
    if (encode_src(&p.tmV[i], v_src[i])) return -1;
  }
  for (int i = 0; i < n_out; ++i) {
    p.o_ptr[i] = static_cast<__nv_bfloat16*>(outs[i].o_ptr);
    p.lse_ptr[i] = outs[i].lse_ptr;
    p.o_row_stride[i] = outs[i].o_row_stride;
    p.o_batch_stride[i] = outs[i].o_batch_stride;
    p.lse_head_stride[i] = outs[i].lse_head_stride;
    p.lse_batch_stride[i] = outs[i].lse_batch_stride;
  }
  p.rows = static_cast<const FwdRow*>(rows_dev);
  p.segs = static_cast<const AttnSeg*>(segs_dev);
  p.tiles = static_cast<const int2*>(tiles_dev);
  p.n_tiles = n_tiles;
  p.n_heads = n_heads;
  p.kv_group = n_heads / n_kv_heads;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  p.stage.tasks = static_cast<const CopyTask*>(copy_tasks_dev);
  p.stage.n_tasks = n_copy_tasks;
  {
    const long grid_ctas = static_cast<long>(n_tiles) * n_heads * batch;
    p.stage.n_copy_ctas = static_cast<int>(n_copy_ctas < grid_ctas ? n_copy_ctas : grid_ctas);
  }
  p.stage.flags = stage_flags;
  p.stage.epoch = stage_epoch;
  p.stage.ticket = stage_ticket;
  if (set_trace(p)) return -1;
  if (n_copy_tasks > 0) {
    if (stage_ticket == nullptr) UA_FAIL("ua_attn_fwd: copy tasks need a ticket counter");
    UA_CUDA(cudaMemsetAsync(stage_ticket, 0, sizeof(unsigned int), stream));
  }
  p.n_split = 1;
  p.persist = stage_flags == nullptr;
  p.tail_heads = stage_flags == nullptr ? tail_heads(n_tiles, n_heads, sm_count()) : 1;
  return launch_fwd<false>(p, n_heads, batch, stream);
}

// ---- dense launches -------------------------------------------------------------------------------
namespace ua {

// Rates of the estimate below (us, bytes per us). They are fitted to which cut was the fastest, with a kernel whose tiles were
// slower, and are no times of the present one: a tile of a 256-row CTA takes 1.5 us now, one of a FEW CTA with 128 rows 1.0.
// The choices still hold. Of 1, 2, 3, 4, 5, 6, 8 and 12 parts the chosen number was the fastest, or within 5 % of it, for 12 of 13
// shapes between 1 query behind 8192 keys and 1000 causal tokens; 512 queries behind 2000 keys, 8 heads, take 19.4 us in the chosen 5
// parts and 17.4 in 8.
constexpr int FEW_MIN_KEY_TILES = 4;
constexpr int MAX_SPLIT = 64;
constexpr int MAX_GIVEN_SPLIT = 1 << 16;      // (a caller's n_split; the shares of fwd_tiles are 32-bit products)
constexpr double TILE_US = 1.9;               // one 128-key tile of a 256-row CTA
constexpr double CTA_US = 6.0;                // start, first loads, epilogue
constexpr double FEW_FULL_TILE_US = 1.3;      // one 128-key tile of a FEW CTA with 128 rows
constexpr double FEW_TILE_US = 0.75;          // one 128-key tile of a FEW CTA that has the memory to itself
constexpr double FEW_BYTES_PER_US = 6.5e6;
constexpr double COMBINE_US = 3.0;
constexpr double COMBINE_BYTES_PER_US = 3.0e6;

struct DensePlan {
  bool few;
  int pack_shift;
  int heads;       // head indices of the grid: query heads, or key/value heads when packed
  int q_tiles;
  int n_split;
  int n_parts;     // partial results per row (0: written directly)
};

// How a dense problem is cut into CTAs. Rows first (query heads of a group packed when their number
// is a power of two: at 1000 tokens, 32 / 8 heads, a tile then spans 64 tokens instead of 256 and wastes
// less under the diagonal); then, if those leave SMs idle or the last wave nearly empty, the keys.
// The estimate of one choice: CTAs of equal cost run in whole waves, unequal ones (causal, heaviest
// first) fill up to about half a CTA of tail, whichever is shorter; plus what the extra fp32 parts
// cost to write and merge.
// Packing (us, kernel of the time, before -> after): 16 sequences, 1 query behind 8123 keys, 32 / 8 heads, 528 -> 107; 8192
// causal tokens, 32 / 8 heads, 589 -> 517. Splitting (us, B200, cold L2, present kernel, one part -> as planned here): 1 query behind
// 8192 keys, 32 / 8 heads, 64.5 -> 17.5 (10 parts); 512 queries behind 32768 keys 408 -> 217 (2). On the other side of the line: 16
// sequences of 8123 keys, one query, take 82 us unsplit (the time of the bytes) and 86 in two parts, 1000 causal tokens, 32 / 8
// heads, 25.5 and 44.7.
static DensePlan plan_dense(int batch, int sq, int skv, int n_heads, int n_kv_heads, int causal, int n_split, int sms) {
  DensePlan d{};
  const int group = n_heads / n_kv_heads;
  int sh = 0;
  while ((1 << sh) < group) ++sh;
  if ((1 << sh) != group || group > ATTN_TILE) sh = 0;
  d.pack_shift = sh;
  d.heads = sh > 0 ? n_kv_heads : n_heads;
  const long rows = static_cast<long>(sq) << sh;
  const int key_tiles = (skv + ATTN_TILE - 1) / ATTN_TILE;
  d.few = rows <= ATTN_TILE && key_tiles >= FEW_MIN_KEY_TILES;
  const int cta_rows = d.few ? ATTN_TILE : 2 * ATTN_TILE;
  d.q_tiles = static_cast<int>((rows + cta_rows - 1) / cta_rows);
  // key tiles of the heaviest tile and of all tiles together
  double total = 0;
  const AttnSeg sg{0, 0, skv, causal ? SEG_UPPER : 0, skv - sq, 0, 0, 0};
  if (causal && d.q_tiles > 1) {
    for (int t = 0; t < d.q_tiles; ++t) {
      const long last = ((static_cast<long>(t) + 1) * cta_rows < rows ? (static_cast<long>(t) + 1) * cta_rows : rows) - 1;
      total += seg_tiles(sg, 0, static_cast<int>(last >> sh)).end;
    }
  } else {
    total = static_cast<double>(key_tiles) * d.q_tiles;
  }
  const double per_head = static_cast<double>(d.heads) * batch;
  total *= per_head;
  const double base = d.q_tiles * per_head;
  double best = 0;
  int best_z = 1;
  const int max_z = n_split > 0 ? 1 : (key_tiles < MAX_SPLIT ? key_tiles : MAX_SPLIT);
  for (int z = 1; z <= max_z; ++z) {
    const double ctas = base * z;
    const double active = ctas < sms ? ctas : sms;
    double tile_us = TILE_US;
    if (d.few) {
      const double mem_us = active * (2.0 * FWD_TILE_BYTES) / FEW_BYTES_PER_US;
      tile_us = mem_us > FEW_TILE_US ? mem_us : FEW_TILE_US;
    }
    const double heavy = CTA_US + (static_cast<double>(key_tiles) / z) * tile_us;
    const double waves = static_cast<double>(static_cast<long>((ctas + sms - 1) / sms)) * heavy;
    const double filled = (ctas * CTA_US + total * tile_us) / sms + 0.5 * heavy;
    double us = ctas <= sms ? heavy : (waves < filled ? waves : filled);
    const int parts = z > 1 ? z : 0;
    if (parts > 0)
      us += COMBINE_US + static_cast<double>(parts) * batch * sq * n_heads * (2.0 * ATTN_D * 4) / COMBINE_BYTES_PER_US;
    if (z == 1 || us < best) {
      best = us;
      best_z = z;
    }
  }
  const int most = key_tiles < MAX_GIVEN_SPLIT ? key_tiles : MAX_GIVEN_SPLIT;
  d.n_split = n_split > 0 ? (n_split < most ? n_split : most) : best_z;
  d.n_parts = d.n_split > 1 ? d.n_split : 0;
  // Few items leave SMs idle, and the launch lasts as long as its longest item, whose two sub-tiles go through all keys. With
  // items of 128 rows each sub-tile takes half of them: 1.0 us per key tile for 1.5 us (the issuing warp has one chain
  // less to overlap with, so a launch that fills the device is slower that way: 1000 causal tokens, 32 heads over 8, by 7 %,
  // and the rule asks for items that all run at once). It beats splitting too, unless the parts are many. Before -> now (B200,
  // us): causal 1000 tokens, 8 heads 19.1 -> 15.1; 512 13.4 -> 11.2; 2000 tokens, 8 over 2 28.7 -> 23.6; 1000 tokens,
  // 8 heads, not causal 18.7 -> 15.6. Left as it was: 512 of 2000 tokens, 8 heads (5 parts) 19.1, this 22.8; up to 3
  // tiles, equal. (FEW_FULL_TILE_US is compared with the estimate above, so it is as much above its 1.0 us as TILE_US above 1.5.)
  const int few_q_tiles = static_cast<int>((rows + ATTN_TILE - 1) / ATTN_TILE);
  if (!d.few && n_split == 0 && key_tiles >= FEW_MIN_KEY_TILES && few_q_tiles * per_head <= sms && CTA_US + key_tiles * FEW_FULL_TILE_US < best) {
    d.few = true;
    d.q_tiles = few_q_tiles;
    d.n_split = 1;
    d.n_parts = 0;
  }
  return d;
}

}  // namespace ua

// Partial results per (batch, token, head) that ua_attn_fwd_dense needs room for: the caller's
// workspace holds n * batch * sq * n_heads rows of 129 floats. n_split = 0 leaves the choice here.
extern "C" int ua_attn_fwd_dense_parts(int batch, int sq, int skv, int n_heads, int n_kv_heads, int causal, int n_split) {
  if (batch <= 0 || sq <= 0 || skv <= 0 || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return 0;
  return plan_dense(batch, sq, skv, n_heads, n_kv_heads, causal, n_split, sm_count()).n_parts;
}

// All queries of `q` against all keys: O and lse of softmax(scale Q K^T) V; causal: key c is visible
// to query r iff c <= r + skv - sq.
extern "C" int ua_attn_fwd_dense(const UaDenseFwd* t, int causal, float softmax_scale, int n_split, float* workspace,
                                 int* status, cudaStream_t stream) {
  const UaTensorSrc *q = &t->q, *k = &t->k, *v = &t->v;
  const UaOutDst* out = &t->out;
  const int batch = static_cast<int>(q->batch), sq = static_cast<int>(q->tokens), skv = static_cast<int>(k->tokens);
  const int n_heads = static_cast<int>(q->heads), n_kv_heads = static_cast<int>(k->heads);
  if (sq <= 0 || batch <= 0) return 0;
  if (check_sources("ua_attn_fwd_dense", batch, n_heads, n_kv_heads, q, 1, k, v, 1)) return -1;
  if (v->tokens < skv) UA_FAIL("ua_attn_fwd_dense: %ld values for %d keys", v->tokens, skv);
  const DensePlan d = plan_dense(batch, sq, skv, n_heads, n_kv_heads, causal, n_split, sm_count());
  if (d.n_parts > 0 && workspace == nullptr) UA_FAIL("ua_attn_fwd_dense: a split launch needs a workspace");
  FwdParams p;
  memset(&p, 0, sizeof(p));
  if (encode_src(&p.tmQ[0], *q, 1u << d.pack_shift)) return -1;
  if (encode_src(&p.tmK[0], *k) || encode_src(&p.tmV[0], *v)) return -1;
  p.o_ptr[0] = static_cast<__nv_bfloat16*>(out->o_ptr);
  p.lse_ptr[0] = out->lse_ptr;
  p.o_row_stride[0] = out->o_row_stride;
  p.o_batch_stride[0] = out->o_batch_stride;
  p.lse_head_stride[0] = out->lse_head_stride;
  p.lse_batch_stride[0] = out->lse_batch_stride;
  p.dense_row.q_len = sq;
  p.dense_row.seg_end = 1;
  p.dense_seg.len = skv;
  p.dense_seg.causal = causal ? SEG_UPPER : 0;
  p.dense_seg.diag = skv - sq;
  p.pack_shift = d.pack_shift;
  p.n_split = d.n_split;
  p.n_tiles = d.q_tiles * d.n_split;
  p.n_heads = n_heads;
  p.kv_group = n_heads / n_kv_heads;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  p.stage.epoch = 1;
  p.persist = 1;
  p.tail_heads = causal ? tail_heads(p.n_tiles, d.heads, sm_count()) : 1;
  const long n_rows = static_cast<long>(batch) * sq * n_heads;
  if (d.n_parts > 0) {
    p.n_parts = d.n_parts;
    p.part_o = workspace;
    p.part_lse = workspace + static_cast<long>(d.n_parts) * n_rows * ATTN_D;
  }
  if (set_trace(p)) return -1;
  if (d.few ? launch_fwd<true>(p, d.heads, batch, stream) : launch_fwd<false>(p, d.heads, batch, stream)) return -1;
  if (d.n_parts > 0) {
    UA_CUDA(launch_kernel(combine_kernel, static_cast<unsigned>((n_rows + 7) / 8), 256, 0, stream, true, p.part_o, p.part_lse, d.n_parts,
                          sq, n_heads, p.o_ptr[0], p.o_row_stride[0], p.o_batch_stride[0], p.lse_ptr[0], p.lse_head_stride[0],
                          p.lse_batch_stride[0], n_rows));
  }
  return 0;
}
