// C-ABI entry points of the block-sparse matrix products: argument checks,
// metadata decoding and kernel family selection.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include "common.h"

namespace bsp {

template <typename T>
int sdd_mma_t(const void* a, const void* b, void* c, int block, int Z, int K,
              int64_t a_sz, int64_t a_sh, int64_t a_sm, int64_t a_sk,
              int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
              int64_t c_sz, const Meta& m, cudaStream_t st);
template <typename T>
int dsd_mma_t(const void* s, const void* b, void* c, int block, int Z, int N,
              int64_t s_sz, int trans_s,
              int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
              int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn,
              const Meta& m, cudaStream_t st);

int dsd_tc_tile_width(int N, int64_t row_tiles, int sms);
bool dsd_tc_eligible(const void* s, const void* b, const void* c, int dtype, int block, int Z, int H, int N, int64_t s_sz,
                     int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
                     int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn);
int dsd_tc(const void* s, const void* b, void* c, int dtype, int block, int Z, int N, int64_t s_sz, int trans_s,
           int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
           int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn, const Meta& m, cudaStream_t st);

bool sdd_tc_eligible(const void* a, const void* b, const void* c, int dtype, int block, int Z, int H,
                     int64_t a_sz, int64_t a_sh, int64_t a_sm, int64_t a_sk,
                     int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn, int64_t c_sz);
int sdd_tc(const void* a, const void* b, void* c, int dtype, int block, int Z, int K,
           int64_t a_sz, int64_t a_sh, int64_t a_sm, int64_t a_sk,
           int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn, int64_t c_sz, const Meta& m, cudaStream_t st);

namespace {

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int decode_meta(const int32_t* hdr, const int32_t* dev, Meta& m) {
  if (!hdr || !dev) return fail(BSP_ERR_INVALID, "metadata pointer is NULL");
  if (hdr[0] != BSP_META_MAGIC) return fail(BSP_ERR_INVALID, "metadata header is corrupt (bad magic)");
  if (hdr[1] <= 0 || hdr[2] <= 0 || hdr[3] <= 0 || hdr[4] < 0) return fail(BSP_ERR_INVALID, "metadata header is corrupt");
  m = meta_view(dev, hdr[1], hdr[2], hdr[3], hdr[4], hdr[5], hdr[6]);
  return BSP_OK;
}

int check_basic(const char* op, int dtype, int block, int Z, int H, const Meta& m) {
  if (!valid_dtype(dtype)) return fail(BSP_ERR_INVALID, "%s: unknown dtype %d", op, dtype);
  if (!valid_block(block)) return fail(BSP_ERR_INVALID, "%s: block must be 16, 32, 64 or 128 (got %d)", op, block);
  if (Z <= 0 || Z > 65535) return fail(BSP_ERR_INVALID, "%s: batch %d outside [1, 65535]", op, Z);
  if (H != m.H) return fail(BSP_ERR_INVALID, "%s: operand has %d heads, layout has %d", op, H, m.H);
  return BSP_OK;
}

// A dense operand must have one unit inner stride; everything else has to keep
// 16-byte alignment for the vector copies.
int check_dense(const char* op, const char* name, const void* p, int dtype, int64_t sz, int64_t sh,
                int64_t s0, int64_t s1) {
  const int vec = dtype == BSP_F32 ? 4 : 8;
  if (!p) return fail(BSP_ERR_INVALID, "%s: %s is NULL", op, name);
  if (!aligned16(p)) return fail(BSP_ERR_INVALID, "%s: %s must be 16-byte aligned", op, name);
  if (s0 != 1 && s1 != 1) return fail(BSP_ERR_INVALID, "%s: %s needs a unit stride on one of its two inner dimensions", op, name);
  const int64_t other = s0 == 1 ? s1 : s0;
  if (sz % vec || sh % vec || (other != 1 && other % vec))
    return fail(BSP_ERR_INVALID, "%s: strides of %s must be multiples of %d elements", op, name, vec);
  return BSP_OK;
}

int check_sparse(const char* op, const char* name, const void* p, int dtype, int64_t sz) {
  const int vec = dtype == BSP_F32 ? 4 : 8;
  if (!p) return fail(BSP_ERR_INVALID, "%s: %s is NULL", op, name);
  if (!aligned16(p)) return fail(BSP_ERR_INVALID, "%s: %s must be 16-byte aligned", op, name);
  if (sz % vec) return fail(BSP_ERR_INVALID, "%s: batch stride of %s must be a multiple of %d elements", op, name, vec);
  return BSP_OK;
}

// Which forms run on the tcgen05 kernels (0 none, 1 by size, 2 all that they cover); see bsp_matmul_use_tcgen05.
std::atomic<int> g_matmul_tc{1};

// Whether a product is left to the tcgen05 kernels, by its size.  Whole tiles of several batch entries
// and heads always are.  Where tiles are padded (a reduction of sdd that is no multiple of 64, a width of
// dsd / dds that is no multiple of 128) or few (one batch entry, one head) the mma.sync kernels can be
// faster: they walk the blocks that exist in steps that fit them, while a tcgen05 tile of 128 rows pays
// its set-up, the union of its block-rows' columns and the padding (FP16, us, tcgen05 / mma.sync: sdd
// block 32, 4 x 8 heads of 4096 x 32 x 4096, fixed layout 362 / 145; dsd block 32, 12 heads of 1024 x 1024,
// density 0.25, width 64: 15 / 8, width 320: 19 / 29).
// The device time of both is estimated from the layout's counts, with coefficients fitted to 10 284 forms
// (blocks 32 to 128, densities 0.1 to 0.5 and structured layouts, 128 to 4096 rows, free sizes 16 to 4096,
// 1 to 32 heads in all; mean error 6 to 18 %); the number of columns in a tile's union is taken as if the
// blocks lay at random, which overrates it for structured layouts.  mma.sync keeps what it would do
// nearly as fast.  Of the 9 671 padded or few forms 2 % then take over 5 % longer than on mma.sync (with
// all of them on tcgen05 48 % did, up to 4.4 times as long), and their mean is 1.7 % above the faster kernel's.
struct Cost { double tc, mma; };
double ceil_div(double a, double b) { return std::ceil(a / b); }

Cost sdd_cost(int block, int Z, int K, const Meta& m) {
  const double tc[2][4] = {{1.55, 0.173, 6.26, 0.291}, {1.67, 0.118, 6.01, 0.293}};
  const double mma[2][4] = {{2.83, 0.0106, 0.0170, 0.0123}, {2.99, 0.0077, 0.0217, 0.0056}};
  const double *t = tc[block == 64], *q = mma[block == 64];
  const int R = 128 / block;
  const double density = m.nnz / ((double)m.H * m.Mb * m.Nb), cols = m.Nb * (1 - std::pow(1 - density, R));
  const double tiles = (double)Z * m.H * ceil_div(m.Mb, R) * std::max(1.0, cols / (2 * R));   // groups of 2 R columns
  const double waves = std::max(1.0, tiles / 148), stages = ceil_div(K, 64), area = (double)Z * m.nnz * block * block;
  return {t[0] + t[1] * stages + t[2] * waves + t[3] * waves * stages, q[0] + q[1] * K + q[2] * area / 1e4 + q[3] * area * K / 1e6};
}
Cost dsd_cost(int block, int Z, int N, int trans_s, const Meta& m) {
  const double tc[3][4] = {{3.76, 0.960, 8.58, 0.049}, {2.14, 1.051, 9.40, 0.0}, {6.15, 0.609, 4.21, 0.041}};
  const double mma[3][4] = {{3.75, 0.313, 0.0090, 0.187}, {4.65, 0.413, 0.0065, 0.177}, {7.00, 0.526, 0.0054, 0.173}};
  const double *t = tc[block == 32 ? 0 : block == 64 ? 1 : 2], *q = mma[block == 32 ? 0 : block == 64 ? 1 : 2];
  const int R = 128 / block, out_b = trans_s ? m.Nb : m.Mb, red_b = trans_s ? m.Mb : m.Nb;
  const double density = m.nnz / ((double)m.H * m.Mb * m.Nb), cols = red_b * (1 - std::pow(1 - density, R));
  const double rows_t = (double)Z * m.H * ceil_div(out_b, R);
  const bool narrow = dsd_tc_tile_width(N, (int64_t)rows_t, 148) == 128;
  const double waves = std::max(1.0, rows_t * ceil_div(N, narrow ? 128 : 256) / (block == 128 ? 148 : 296)) * (narrow ? 0.6 : 1.0);
  const double stages = cols * (block == 32 ? 0.5 : block == 64 ? 1 : 2);
  const double width = N <= 64 ? 64 : 128 * ceil_div(N, 128);              // what the mma.sync kernel computes
  return {t[0] + t[1] * stages * waves + t[2] * waves + t[3] * stages,
          q[0] + q[1] * (m.nnz / ((double)m.H * out_b)) * block / 32 + q[2] * Z * (double)m.nnz * block * block * width / 1e6 +
              q[3] * Z * (double)m.H * out_b * block * N / 1e5};
}
bool sdd_prefers_tc(int block, int Z, int K, const Meta& m) {
  if (block == 128 || (K % 64 == 0 && Z > 1 && m.H > 1)) return true;      // (block 128: at most 1.1 x mma.sync's time, 0.64 in the mean)
  const Cost c = sdd_cost(block, Z, K, m);
  return 1.2 * c.tc < c.mma;
}
bool dsd_prefers_tc(int block, int Z, int N, int trans_s, const Meta& m) {
  if (N % 128 == 0 && Z > 1 && m.H > 1) return true;
  const Cost c = dsd_cost(block, Z, N, trans_s, m);
  return 1.1 * c.tc < c.mma;
}

int run_dsd(const void* s, const void* b, void* c, int dtype, int block, int Z, int N,
            int64_t s_sz, int trans_s,
            int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
            int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn,
            const Meta& m, cudaStream_t st) {
  // (a layout without any block has no sparse tensor to describe to the tensor-map encoder: the
  // mma.sync kernel writes the zeros)
  // (the tcgen05 kernel plans a tile with one bit per block of the reduction side, 1024 at most)
  const int tc = g_matmul_tc.load();
  if (tc && m.nnz > 0 && (trans_s ? m.Mb : m.Nb) <= 1024 &&
      dsd_tc_eligible(s, b, c, dtype, block, Z, m.H, N, s_sz, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn) &&
      (tc == 2 || dsd_prefers_tc(block, Z, N, trans_s, m)))
    return dsd_tc(s, b, c, dtype, block, Z, N, s_sz, trans_s, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn, m, st);
  if (dtype == BSP_F32)
    return dsd_mma_t<float>(s, b, c, block, Z, N, s_sz, trans_s, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn, m, st);
  if (dtype == BSP_F16)
    return dsd_mma_t<__half>(s, b, c, block, Z, N, s_sz, trans_s, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn, m, st);
  return dsd_mma_t<__nv_bfloat16>(s, b, c, block, Z, N, s_sz, trans_s, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn, m, st);
}

}  // namespace
}  // namespace bsp

using namespace bsp;

extern "C" int bsp_sdd(const void* a, const void* b, void* c, int dtype, int block,
                       int Z, int H, int K,
                       int64_t a_sz, int64_t a_sh, int64_t a_sm, int64_t a_sk,
                       int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
                       int64_t c_sz, const int32_t* meta_hdr, const int32_t* meta, void* stream) {
  Meta m;
  if (int rc = decode_meta(meta_hdr, meta, m)) return rc;
  if (int rc = check_basic("sdd", dtype, block, Z, H, m)) return rc;
  // (k-contiguous operands are read in pieces of 16; with both operands k-strided any K is fine)
  if (K <= 0 || (K % 16 && !(a_sk != 1 && b_sk != 1))) return fail(BSP_ERR_INVALID, "Reduction size for SDD must be a multiple of 16");
  if (int rc = check_dense("sdd", "a", a, dtype, a_sz, a_sh, a_sm, a_sk)) return rc;
  if (int rc = check_dense("sdd", "b", b, dtype, b_sz, b_sh, b_sk, b_sn)) return rc;
  if (int rc = check_sparse("sdd", "c", c, dtype, c_sz)) return rc;
  if (m.nnz == 0) return BSP_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // (the tcgen05 kernel's grid: groups of 128 rows per head in y, the batch in z)
  const int tc = g_matmul_tc.load();
  if (tc && Z <= 65535 && (int64_t)m.H * ((m.Mb * block + 127) / 128) <= 65535 &&
      sdd_tc_eligible(a, b, c, dtype, block, Z, m.H, a_sz, a_sh, a_sm, a_sk, b_sz, b_sh, b_sk, b_sn, c_sz) &&
      (tc == 2 || sdd_prefers_tc(block, Z, K, m)))
    return sdd_tc(a, b, c, dtype, block, Z, K, a_sz, a_sh, a_sm, a_sk, b_sz, b_sh, b_sk, b_sn, c_sz, m, st);
  if (dtype == BSP_F32)
    return sdd_mma_t<float>(a, b, c, block, Z, K, a_sz, a_sh, a_sm, a_sk, b_sz, b_sh, b_sk, b_sn, c_sz, m, st);
  if (dtype == BSP_F16)
    return sdd_mma_t<__half>(a, b, c, block, Z, K, a_sz, a_sh, a_sm, a_sk, b_sz, b_sh, b_sk, b_sn, c_sz, m, st);
  return sdd_mma_t<__nv_bfloat16>(a, b, c, block, Z, K, a_sz, a_sh, a_sm, a_sk, b_sz, b_sh, b_sk, b_sn, c_sz, m, st);
}

extern "C" int bsp_dsd(const void* s, const void* b, void* c, int dtype, int block,
                       int Z, int H, int N, int64_t s_sz, int trans_s,
                       int64_t b_sz, int64_t b_sh, int64_t b_sk, int64_t b_sn,
                       int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn,
                       const int32_t* meta_hdr, const int32_t* meta, void* stream) {
  Meta m;
  if (int rc = decode_meta(meta_hdr, meta, m)) return rc;
  if (int rc = check_basic("dsd", dtype, block, Z, H, m)) return rc;
  const int vec = dtype == BSP_F32 ? 4 : 8;
  if (N <= 0 || (N % vec && !(b_sk == 1 && b_sn != 1)))
    return fail(BSP_ERR_INVALID, "dsd: dense width %d must be positive, and a multiple of %d where b has unit stride along it", N, vec);
  if (m.nnz > 0)                 // (a layout without blocks has an empty sparse operand, never dereferenced)
    if (int rc = check_sparse("dsd", "a", s, dtype, s_sz)) return rc;
  if (int rc = check_dense("dsd", "b", b, dtype, b_sz, b_sh, b_sk, b_sn)) return rc;
  if (!c) return fail(BSP_ERR_INVALID, "dsd: c is NULL");
  return run_dsd(s, b, c, dtype, block, Z, N, s_sz, trans_s, b_sz, b_sh, b_sk, b_sn, c_sz, c_sh, c_sm, c_sn, m,
                 reinterpret_cast<cudaStream_t>(stream));
}

// C = A . op(S) is computed as C^T = op(S)^T . A^T: the sparse operand is used
// with the opposite transposition and the dense operand / result swap the
// roles of their two inner strides.
extern "C" int bsp_dds(const void* a, const void* s, void* c, int dtype, int block,
                       int Z, int H, int M,
                       int64_t a_sz, int64_t a_sh, int64_t a_sm, int64_t a_sk,
                       int64_t s_sz, int trans_s,
                       int64_t c_sz, int64_t c_sh, int64_t c_sm, int64_t c_sn,
                       const int32_t* meta_hdr, const int32_t* meta, void* stream) {
  Meta m;
  if (int rc = decode_meta(meta_hdr, meta, m)) return rc;
  if (int rc = check_basic("dds", dtype, block, Z, H, m)) return rc;
  const int vec = dtype == BSP_F32 ? 4 : 8;
  if (M <= 0 || (M % vec && !(a_sk == 1 && a_sm != 1)))
    return fail(BSP_ERR_INVALID, "dds: dense height %d must be positive, and a multiple of %d where a has unit stride along it", M, vec);
  if (int rc = check_dense("dds", "a", a, dtype, a_sz, a_sh, a_sm, a_sk)) return rc;
  if (m.nnz > 0)
    if (int rc = check_sparse("dds", "b", s, dtype, s_sz)) return rc;
  if (!c) return fail(BSP_ERR_INVALID, "dds: c is NULL");
  return run_dsd(s, a, c, dtype, block, Z, M, s_sz, !trans_s, a_sz, a_sh, a_sk, a_sm, c_sz, c_sh, c_sn, c_sm, m,
                 reinterpret_cast<cudaStream_t>(stream));
}

// Chooses the kernel family of MatMul for blocks 32, 64 and 128 with FP16 / BF16 operands.
extern "C" int bsp_matmul_use_tcgen05(int enable) {
  if (enable < 0 || enable > 2) return fail(BSP_ERR_INVALID, "bsp_matmul_use_tcgen05: 0, 1 or 2 (got %d)", enable);
  g_matmul_tc.store(enable);
  return BSP_OK;
}

extern "C" int bsp_matmul_prefers_tcgen05(int op, int block, int Z, int free_size, int trans_s, const int32_t* meta_hdr, int* prefers) {
  Meta m;
  if (op < 0 || op > 2 || !prefers) return fail(BSP_ERR_INVALID, "bsp_matmul_prefers_tcgen05: op must be 0 (sdd), 1 (dsd) or 2 (dds)");
  if (int rc = decode_meta(meta_hdr, meta_hdr, m)) return rc;              // (only the counts of the header are read)
  if (int rc = check_basic("matmul", BSP_F16, block, Z, m.H, m)) return rc;
  if (free_size <= 0) return fail(BSP_ERR_INVALID, "bsp_matmul_prefers_tcgen05: the free size must be positive");
  *prefers = block == 16 || m.nnz == 0 ? 0 : op == 0 ? sdd_prefers_tc(block, Z, free_size, m)
                                                     : dsd_prefers_tc(block, Z, free_size, op == 1 ? trans_s : !trans_s, m);
  return BSP_OK;
}
