// Argument blocks of the product-chain kernel (chain_sm100.cu).
#pragma once
#include <stdint.h>

extern "C" {

#define DMUON_CHAIN_MAX_OPS 76
#define DMUON_CHAIN_MAX_GROUPS 16
#define DMUON_CHAIN_MAX_MAPS 128

// One batched product of a chain (device array; same meaning of the fields as in DmuonGemmArgs).
// What it reads and writes lies in the work memory that a launch names, so one list serves every
// stream: alpha_vec, C, D and partials are byte offsets into it, -1 where there is none.
struct DmuonChainOp {
  int map_a, map_b;            // indices into the chain's tensor maps; map_a < 0: sum of partial products
  int a_mn_major, b_mn_major, ab_fp16;
  int M, N, K;
  int kb_per_split;            // > 0: split over K, every split stores its own fp32 partial product
  int splits;                  // number of partial products (split product and its sum)
  int out_kind;
  int final_slot;              // >= 0: output, scale and pointer tables come from the launch (DmuonChainFinal)
  float alpha, beta, diag;
  int pad_;
  long long alpha_vec, C, D;
  long long partials;          // input of a sum
  long long ldc, ldd, strideC, strideD;
};

// What a launch supplies for the last product of a group.  Pointers (those in the tables
// too) are multiples of 16 bytes, pitches and strides of 8 elements.
struct DmuonChainFinal {
  const void* C;
  void* D;
  const void* const* C_tab;
  void* const* D_tab;
  void* const* D2_tab;
  const float* alpha_vec;
  long long ldc, ldd, ldd2, strideC, strideD;
  float alpha, beta;
  int out_kind;
  int pad_;
};

struct DmuonChainMap {
  const void* base;
  long long rows, cols, batch, ld, batch_stride;
  int fp16, box_cols, box_rows, pad_;
};

struct DmuonChainArgs {
  const void* ops;             // device: n_ops DmuonChainOp
  const void* maps;            // host: n_maps encoded tensor maps (128 bytes each), copied into the launch's parameters
  const int* tab;              // device: total entries of four ints, see chain_sm100.cu
  int* counters;               // device, zero between launches: ticket, exits, one per matrix
  void* work;                  // device: what the operations' offsets count from
  int* status;
  int n_ops, n_maps, total, n_counters, n_final;
  int bn;                      // 64 or 128: 128 x bn tiles; 256: CTA pairs on 256 x 256 tiles
  int wide;                    // CTA pairs: entries may be two tiles side by side
  struct DmuonChainFinal fin[DMUON_CHAIN_MAX_GROUPS];
};

int dmuon_chain_encode_maps(const struct DmuonChainMap* maps, int n, void* out_host);
int dmuon_chain_launch(const struct DmuonChainArgs* args, void* stream);
}
