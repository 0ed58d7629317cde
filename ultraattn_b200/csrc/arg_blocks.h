// Argument blocks of the library's C entries that callers fill in: the launchers (*.cu), the native host part
// (host_ext.cpp) and, field by field, ops/attention.py (_src_fields, _DENSE_FWD, _LOCAL_BWD). All fields are 64 bits wide.
#pragma once

// One tensor source: [batch, tokens, heads, 128] bf16 with the given strides (elements).
struct UaTensorSrc {
  const void* ptr;
  long tokens;
  long heads;
  long batch;
  long token_stride;
  long head_stride;
  long batch_stride;
};

struct UaOutDst {
  void* o_ptr;
  float* lse_ptr;
  long o_row_stride;
  long o_batch_stride;
  long lse_head_stride;
  long lse_batch_stride;
};

// The tensors of a dense forward launch in one block, so that a caller marshals one argument.
struct UaDenseFwd {
  UaTensorSrc q, k, v;
  UaOutDst out;
};

// The same of a whole backward on one device.
struct UaLocalBwd {
  UaTensorSrc q, k, v, d_o;
  const void* o;
  long o_row_stride, o_batch_stride;
  const float* lse;              // [batch, heads, tokens], contiguous; dvec alike
  float* dvec;
  float* dq32;                   // [batch, tokens, heads, 128] workspace
  void* dq;                      // bf16, contiguous
  void* dk;                      // bf16
  void* dv;
  long dkv_row_stride, dkv_batch_stride;
  const void* cols;              // tables as in ua_attn_bwd, not read if dense
  const void* segs;
  const void* tiles;
  long n_tiles, dense, skewed;
};
static_assert(sizeof(UaDenseFwd) == 27 * 8 && sizeof(UaLocalBwd) == 45 * 8, "ops/attention.py packs 27 and 45 words");
