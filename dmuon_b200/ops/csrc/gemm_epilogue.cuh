// Pieces shared by the tcgen05 GEMM kernels: tile constants, the per-product
// parameters and the epilogue that turns accumulator rows into stored rows.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace dmuon {

constexpr int BM = 128;
constexpr int BK = 64;       // 64 two-byte elements = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int kThreads = 192;
constexpr int kBlockBytes = 64 * 128;  // one 64 x 64 swizzled block (MN-major staging)

struct KParams {
  int M, N, K, batch;
  const int4* tile_tab;
  int tiles_per_batch;
  int a_mn_major, b_mn_major, ab_fp16;
  float alpha, beta, diag;
  const float* alpha_vec;
  const void* C;
  void* D;
  void* D2;
  const void* const* C_tab;
  void* const* D_tab;
  void* const* D2_tab;
  long long ldc, ldd, ldd2;
  long long strideC, strideD, strideD2;
  int out_kind;
  const int* b_ready;
  int b_ready_epoch;
  int* status;
  int d2_multimem;
};

// ---- epilogue helpers -------------------------------------------------------

template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <>
__device__ __forceinline__ float to_f32<float>(float x) { return x; }

template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ float from_f32<float>(float x) { return x; }

template <typename T>
__device__ __forceinline__ void load_row32(const T* src, float (&c)[32], int nvalid, bool vec) {
  if (vec && nvalid == 32) {
    constexpr int kPerVec = 16 / sizeof(T);
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int i = 0; i < 32 / kPerVec; ++i) {
      uint4 raw = s4[i];
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int j = 0; j < kPerVec; ++j) c[i * kPerVec + j] = to_f32<T>(e[j]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) c[j] = (j < nvalid) ? to_f32<T>(src[j]) : 0.f;
  }
}

template <typename T>
__device__ __forceinline__ void store_row32(T* dst, const float (&v)[32], int nvalid, bool vec) {
  if (vec && nvalid == 32) {
    constexpr int kPerVec = 16 / sizeof(T);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int i = 0; i < 32 / kPerVec; ++i) {
      uint4 raw;
      T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int j = 0; j < kPerVec; ++j) e[j] = from_f32<T>(v[i * kPerVec + j]);
      d4[i] = raw;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < nvalid) dst[j] = from_f32<T>(v[j]);
  }
}

// bf16 row chunk to a multicast address: every rank's copy of the buffer
// receives it (multimem.st through the switch).  The host only selects this
// path when every row start is 16-byte aligned and N is a multiple of 8.
__device__ __forceinline__ void store_row32_multicast(__nv_bfloat16* mc_dst, const float (&v)[32], int nvalid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i * 8 < nvalid) {
      uint4 raw;
      __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&raw);
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = __float2bfloat16_rn(v[i * 8 + j]);
      multimem_st_16B(mc_dst + i * 8, raw);
    }
  }
}

template <typename T>
__device__ __forceinline__ void store_col32(T* dst, long long ld, const float (&v)[32], int nvalid) {
  // dst points at element (col0, row) of the transposed tile; consecutive
  // lanes hold consecutive rows, so each store instruction is contiguous
  // across the warp.
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j < nvalid) dst[static_cast<long long>(j) * ld] = from_f32<T>(v[j]);
}

template <typename T>
__device__ __forceinline__ void epilogue_chunk(const KParams& p, const T* Cb, T* Db,
                                               __nv_bfloat16* D2b, float (&v)[32], int row, int col0,
                                               bool mirror) {
  const int nvalid = min(32, p.N - col0);
  const bool row_ok = row < p.M;
  if (p.beta != 0.f && row_ok) {
    float c[32];
    const T* src = Cb + static_cast<long long>(row) * p.ldc + col0;
    const bool vec = ((p.ldc * sizeof(T)) % 16 == 0) && ((reinterpret_cast<uintptr_t>(Cb) & 15) == 0);
    load_row32<T>(src, c, nvalid, vec);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = fmaf(p.beta, c[j], v[j]);
  }
  if (p.diag != 0.f) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (col0 + j == row) v[j] += p.diag;
  }
  if (!row_ok) return;
  {
    T* dst = Db + static_cast<long long>(row) * p.ldd + col0;
    const bool vec = ((p.ldd * sizeof(T)) % 16 == 0) && ((reinterpret_cast<uintptr_t>(Db) & 15) == 0);
    store_row32<T>(dst, v, nvalid, vec);
    if (mirror) store_col32<T>(Db + static_cast<long long>(col0) * p.ldd + row, p.ldd, v, nvalid);
  }
  if (D2b != nullptr && p.d2_multimem) {
    store_row32_multicast(D2b + static_cast<long long>(row) * p.ldd2 + col0, v, nvalid);
  } else if (D2b != nullptr) {
    __nv_bfloat16* dst = D2b + static_cast<long long>(row) * p.ldd2 + col0;
    const bool vec = ((p.ldd2 * 2) % 16 == 0) && ((reinterpret_cast<uintptr_t>(D2b) & 15) == 0);
    store_row32<__nv_bfloat16>(dst, v, nvalid, vec);
    if (mirror)
      store_col32<__nv_bfloat16>(D2b + static_cast<long long>(col0) * p.ldd2 + row, p.ldd2, v, nvalid);
  }
}

// Pointers and scale of one matrix of a batch.
struct EpiloguePtrs {
  const char* C;
  char* D;
  __nv_bfloat16* D2;
  float alpha;
};

__device__ __forceinline__ EpiloguePtrs epilogue_ptrs(const KParams& p, int b) {
  EpiloguePtrs e;
  e.C = reinterpret_cast<const char*>(p.C_tab ? p.C_tab[b] : p.C);
  e.D = reinterpret_cast<char*>(p.D_tab ? p.D_tab[b] : p.D);
  e.D2 = reinterpret_cast<__nv_bfloat16*>(p.D2_tab ? p.D2_tab[b] : p.D2);
  const int esz = (p.out_kind == 2) ? 4 : 2;
  if (!p.C_tab && e.C) e.C += static_cast<long long>(b) * p.strideC * esz;
  if (!p.D_tab) e.D += static_cast<long long>(b) * p.strideD * esz;
  if (!p.D2_tab && e.D2) e.D2 += static_cast<long long>(b) * p.strideD2;
  e.alpha = p.alpha_vec ? p.alpha * p.alpha_vec[b] : p.alpha;
  return e;
}

// Straight from the lanes.
__device__ __forceinline__ void epilogue_store32(const KParams& p, const EpiloguePtrs& e, float (&v)[32], int row,
                                                 int col0, bool mirror) {
  if (p.out_kind == 0) {
    epilogue_chunk<__nv_bfloat16>(p, reinterpret_cast<const __nv_bfloat16*>(e.C),
                                       reinterpret_cast<__nv_bfloat16*>(e.D), e.D2, v, row, col0, mirror);
  } else if (p.out_kind == 1) {
    epilogue_chunk<__half>(p, reinterpret_cast<const __half*>(e.C), reinterpret_cast<__half*>(e.D), e.D2, v, row,
                                col0, mirror);
  } else {
    epilogue_chunk<float>(p, reinterpret_cast<const float*>(e.C), reinterpret_cast<float*>(e.D), e.D2, v, row,
                               col0, mirror);
  }
}

// One warp's share (32 accumulator rows, `row` = this lane's) of an output tile of `cols` columns.
__device__ __forceinline__ void epilogue_rows32(const KParams& p, uint32_t tmem_addr, int row, int n0, int cols, int b,
                                                bool mirror) {
  const EpiloguePtrs e = epilogue_ptrs(p, b);
  for (int c = 0; c < cols; c += 32) {
    const int col0 = n0 + c;
    if (col0 >= p.N) break;  // uniform across the warp
    uint32_t r[32];
    tmem_ld_32x32(tmem_addr + static_cast<uint32_t>(c), r);
    tmem_ld_wait();
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = e.alpha * __uint_as_float(r[j]);
    epilogue_store32(p, e, v, row, col0, mirror);
  }
}

// ---- staged stores -------------------------------------------------------------
//
// After tcgen05.ld a lane holds 32 columns of ONE row.  Stored from there, every
// 16-byte store of a warp touches 32 lines, and the transposed copy of a symmetric
// tile needs 32 two-byte stores of 64 contiguous bytes each.  Measured on a B200 with
// those stores: 3.1 us from the accumulator to the last store of a mirrored 128 x 64
// tile, three times as long as without the mirror, and longer than the tile's product
// for K <= 1024.  Here each warp passes 32 x 32 two-byte (or 32 x 16 four-byte)
// elements through 2 KB of shared memory, so that four lanes share the 64 bytes of a
// row: a store instruction covers eight rows, the mirror is four stores instead of 32,
// and C is read the same way (fetched before the accumulator is ready).
// Takes outputs whose dimensions and pitches are multiples of 8 elements and whose
// pointers are multiples of 16 bytes, and no mirror of 32-bit outputs.
// Layout: 64 bytes per row, 16-byte piece c of row r at c ^ ((r >> 1) & 3), which makes
// both the row-wise and the piece-wise accesses free of bank conflicts.
constexpr int kStageWarpBytes = 2048;

__device__ __forceinline__ uint4* stage_at(uint8_t* st, int row, int piece) {
  return reinterpret_cast<uint4*>(st + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
}

// two 16-bit elements of a 32-bit word (no pointers into registers: those would put the
// arrays into local memory)
template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 x = __floats2bfloat162_rn(a, b);
  return static_cast<uint32_t>(__bfloat16_as_ushort(x.x)) | (static_cast<uint32_t>(__bfloat16_as_ushort(x.y)) << 16);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  const __half2 x = __floats2half2_rn(a, b);
  return static_cast<uint32_t>(__half_as_ushort(__low2half(x))) |
         (static_cast<uint32_t>(__half_as_ushort(__high2half(x))) << 16);
}
template <typename T>
__device__ __forceinline__ float unpack_lo(uint32_t w);
template <typename T>
__device__ __forceinline__ float unpack_hi(uint32_t w);
template <>
__device__ __forceinline__ float unpack_lo<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w << 16); }
template <>
__device__ __forceinline__ float unpack_hi<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
template <>
__device__ __forceinline__ float unpack_lo<__half>(uint32_t w) {
  return __half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu)));
}
template <>
__device__ __forceinline__ float unpack_hi<__half>(uint32_t w) {
  return __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16)));
}

// C of 32 columns of the warp's 32 rows as fetched: pieces 0..3 are all of them for
// two-byte elements, the first 16 columns for four-byte ones (4..7 the other 16).
struct RawC {
  uint4 r[8];
};

// How one warp's 32 rows of a tile leave the tensor memory.
struct TileEpilogue {
  // Values, not a reference: the parameters lie in shared memory, and a store to the staging
  // memory would make the compiler read them again.
  float alpha, beta, diag;
  int N, out_kind, ldc, ldd, ldd2;
  uint8_t* st;          // this warp's staging memory
  int row0, lane;
  int rows;             // rows of the matrix from this lane's first staged row (row0 + lane / 4) on
  const char* c_lane;   // C, D and D2 at this lane's first staged row and piece, column 0
  char *d_lane, *t_lane, *d2_lane;    // t_lane: the mirror, at column row0 + 8 * (lane % 4) of row lane / 4
  bool mirror, add_c, copy;

  __device__ __forceinline__ TileEpilogue(const KParams& p, int b, int row0_, bool mirror_, uint8_t* st_, int lane_)
      : beta(p.beta), diag(p.diag), N(p.N), out_kind(p.out_kind), ldc(static_cast<int>(p.ldc)),
        ldd(static_cast<int>(p.ldd)), ldd2(static_cast<int>(p.ldd2)), st(st_), row0(row0_), lane(lane_),
        mirror(mirror_), add_c(p.beta != 0.f) {
    const EpiloguePtrs e = epilogue_ptrs(p, b);
    const int esz = out_kind == 2 ? 4 : 2;
    const int r = row0 + (lane >> 2), piece = (lane & 3) * 16;
    alpha = e.alpha;
    rows = p.M - r;
    c_lane = e.C + static_cast<long long>(r) * ldc * esz + piece;
    d_lane = e.D + static_cast<long long>(r) * ldd * esz + piece;
    t_lane = e.D + (static_cast<long long>(lane >> 2) * ldd + row0) * 2 + piece;
    copy = e.D2 != nullptr;
    d2_lane = reinterpret_cast<char*>(e.D2) + static_cast<long long>(r) * ldd2 * 2 + (out_kind == 2 ? piece / 2 : piece);
  }

  // pieces first..first+3 of C, in the order in which the stores need them
  template <int first>
  __device__ __forceinline__ void fetch4(RawC& c, int col0, int esz) const {
    const bool in = col0 + (lane & 3) * (16 / esz) < N;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // past the L1 cache: C may have been stored by another SM earlier in the same launch
      if (in && 8 * i < rows)
        c.r[first + i] = __ldcg(reinterpret_cast<const uint4*>(c_lane + (static_cast<long long>(8 * i) * ldc + col0) * esz));
    }
  }

  // C of the 32 columns at col0
  __device__ __forceinline__ void fetch_c(RawC& c, int col0) const {
    if (!add_c) return;
    if (out_kind == 2) {
      fetch4<0>(c, col0, 4);
      fetch4<4>(c, col0 + 16, 4);
    } else {
      fetch4<0>(c, col0, 2);
    }
  }

  // rows held one per lane (32 two-byte elements as words) -> rows at `dst`
  __device__ __forceinline__ void put_rows(const uint32_t (&w)[16], char* dst, int ld, int col0) const {
#pragma unroll
    for (int k = 0; k < 4; ++k) *stage_at(st, lane, k) = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    __syncwarp();
    const bool in = col0 + 8 * (lane & 3) < N;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const uint4 x = *stage_at(st, it * 8 + (lane >> 2), lane & 3);
      if (in && 8 * it < rows)
        *reinterpret_cast<uint4*>(dst + (static_cast<long long>(8 * it) * ld + col0) * 2) = x;
    }
    __syncwarp();
  }

  template <typename T>
  __device__ __forceinline__ void store16(float (&v)[32], RawC& c, int col0, bool more) const {
    if (add_c) {
#pragma unroll
      for (int it = 0; it < 4; ++it) *stage_at(st, it * 8 + (lane >> 2), lane & 3) = c.r[it];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 x = *stage_at(st, lane, k);
        v[8 * k + 0] = fmaf(beta, unpack_lo<T>(x.x), v[8 * k + 0]);
        v[8 * k + 1] = fmaf(beta, unpack_hi<T>(x.x), v[8 * k + 1]);
        v[8 * k + 2] = fmaf(beta, unpack_lo<T>(x.y), v[8 * k + 2]);
        v[8 * k + 3] = fmaf(beta, unpack_hi<T>(x.y), v[8 * k + 3]);
        v[8 * k + 4] = fmaf(beta, unpack_lo<T>(x.z), v[8 * k + 4]);
        v[8 * k + 5] = fmaf(beta, unpack_hi<T>(x.z), v[8 * k + 5]);
        v[8 * k + 6] = fmaf(beta, unpack_lo<T>(x.w), v[8 * k + 6]);
        v[8 * k + 7] = fmaf(beta, unpack_hi<T>(x.w), v[8 * k + 7]);
      }
      __syncwarp();
      if (more) fetch4<0>(c, col0 + 32, 2);
    }
    if (diag != 0.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j == row0 + lane) v[j] += diag;
    }
    uint32_t w[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) w[k] = pack2<T>(v[2 * k], v[2 * k + 1]);
    put_rows(w, d_lane, ldd, col0);
    if (mirror) {
      unsigned short* tr = reinterpret_cast<unsigned short*>(st) + lane;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        tr[(2 * k) * 32] = static_cast<unsigned short>(w[k] & 0xffffu);
        tr[(2 * k + 1) * 32] = static_cast<unsigned short>(w[k] >> 16);
      }
      __syncwarp();
      // the matrix is square and its size a multiple of 8, so N bounds the columns of the mirror as well
      const bool in = row0 + 8 * (lane & 3) < N;
      const int cols = N - col0 - (lane >> 2);
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const uint4 x = reinterpret_cast<const uint4*>(st)[it * 32 + lane];
        if (in && 8 * it < cols)
          *reinterpret_cast<uint4*>(t_lane + static_cast<long long>(col0 + 8 * it) * ldd * 2) = x;
      }
      __syncwarp();
    }
    if (copy) {
#pragma unroll
      for (int k = 0; k < 16; ++k) w[k] = pack2<__nv_bfloat16>(v[2 * k], v[2 * k + 1]);
      put_rows(w, d2_lane, ldd2, col0);
    }
  }

  // 16 columns, the lane's values of them from v[first] on
  template <int first>
  __device__ __forceinline__ void store32(const float (&v)[32], RawC& c, int col0, bool more) const {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *stage_at(st, lane, k) = make_uint4(__float_as_uint(v[first + 4 * k]), __float_as_uint(v[first + 4 * k + 1]),
                                          __float_as_uint(v[first + 4 * k + 2]), __float_as_uint(v[first + 4 * k + 3]));
    __syncwarp();
    const int col = col0 + 4 * (lane & 3);
    const bool in = col < N;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const uint4 raw = *stage_at(st, it * 8 + (lane >> 2), lane & 3);
      float4 x = make_float4(__uint_as_float(raw.x), __uint_as_float(raw.y), __uint_as_float(raw.z), __uint_as_float(raw.w));
      if (in && 8 * it < rows) {
        if (add_c) {
          x.x = fmaf(beta, __uint_as_float(c.r[first / 4 + it].x), x.x);
          x.y = fmaf(beta, __uint_as_float(c.r[first / 4 + it].y), x.y);
          x.z = fmaf(beta, __uint_as_float(c.r[first / 4 + it].z), x.z);
          x.w = fmaf(beta, __uint_as_float(c.r[first / 4 + it].w), x.w);
        }
        if (diag != 0.f) {
          const int row = row0 + it * 8 + (lane >> 2);
          if (col == row) x.x += diag;
          if (col + 1 == row) x.y += diag;
          if (col + 2 == row) x.z += diag;
          if (col + 3 == row) x.w += diag;
        }
        *reinterpret_cast<float4*>(d_lane + (static_cast<long long>(8 * it) * ldd + col0) * 4) = x;
        if (copy)
          *reinterpret_cast<uint2*>(d2_lane + (static_cast<long long>(8 * it) * ldd2 + col0) * 2) =
              make_uint2(pack2<__nv_bfloat16>(x.x, x.y), pack2<__nv_bfloat16>(x.z, x.w));
      }
    }
    __syncwarp();
    if (more && add_c) fetch4<first / 4>(c, col0 + 32, 4);
  }

  // v: alpha-scaled values of the 32 columns at col0 of this lane's row; c: C as fetched for col0.
  // If more columns follow, c holds C of the next ones afterwards.
  template <int kind>
  __device__ __forceinline__ void store_kind(float (&v)[32], RawC& c, int col0, bool more) const {
    if constexpr (kind == 0) {
      store16<__nv_bfloat16>(v, c, col0, more);
    } else if constexpr (kind == 1) {
      store16<__half>(v, c, col0, more);
    } else {
      store32<0>(v, c, col0, more);
      store32<16>(v, c, col0 + 16, more);
    }
  }

  __device__ __forceinline__ void store(float (&v)[32], RawC& c, int col0) const {
    if (out_kind == 0) store_kind<0>(v, c, col0, false);
    else if (out_kind == 1) store_kind<1>(v, c, col0, false);
    else store_kind<2>(v, c, col0, false);
  }

  template <int kind>
  __device__ __forceinline__ void run_kind(uint32_t tmem_addr, int n0, int cols, RawC c) const {
#pragma unroll 1
    for (int k = 0; k < cols; k += 32) {
      const int col0 = n0 + k;
      if (col0 >= N) break;  // uniform across the warp
      uint32_t r[32];
      tmem_ld_32x32(tmem_addr + static_cast<uint32_t>(k), r);
      tmem_ld_wait();
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = alpha * __uint_as_float(r[j]);
      store_kind<kind>(v, c, col0, k + 32 < cols);
    }
  }

  // `cols` accumulator columns at tmem_addr -> columns n0.. of the output; c holds C as fetched for n0.
  // One loop per output type: the types differ in what has to stay in registers.
  __device__ __forceinline__ void run(uint32_t tmem_addr, int n0, int cols, const RawC& c) const {
    if (out_kind == 0) run_kind<0>(tmem_addr, n0, cols, c);
    else if (out_kind == 1) run_kind<1>(tmem_addr, n0, cols, c);
    else run_kind<2>(tmem_addr, n0, cols, c);
  }
};

}  // namespace dmuon
