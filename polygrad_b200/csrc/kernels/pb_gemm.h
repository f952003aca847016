/*
 * pb_gemm.h -- the planned contraction shared by the fp32 kernel (pb_gemm.cu)
 * and the tensor-core kernel (pb_gemm_tc.cu).
 */
#ifndef PB_GEMM_H
#define PB_GEMM_H

#include "../runtime/pb_runtime.h"
#include <cuda_bf16.h>
#include <vector>

enum { PB_F32 = 0, PB_BF16 = 1, PB_F16 = 2 };      /* storage type of a contraction's operands */
#define PB_PACK_MAX_AXES 12
#define PB_TC_UNSUPPORTED 77
#define PB_TC_NO_SCRATCH 78      /* float32 modes: the operands' parts did not fit the pool; nothing was computed */

/* A launch that may start while the work before it on the stream drains (programmatic dependence): its blocks set up
 * barriers and tensor memory and then wait in pb_grid_wait() for all of that work, results included, before they
 * touch global memory.  pb_grid_release() lets the next such launch do the same; called at the start, since a
 * kernel's blocks must all have started before the next one's do.  A kernel launched like this calls
 * pb_grid_wait() on every path.  197 x 2304 x 768 under the bfloat16 policy, a copy
 * and a contraction: 14.3 us one after the other, 11.2 like this.  (Not for kernels of which an SM holds several blocks, unless they are many:
 * blocks are dealt out as slots come free, unevenly.  8 x 12 x 1024 x 64 attention released early 89 -> 92 us, a small contraction 27 -> 50.) */
template <class F, class... Args>
static inline cudaError_t pb_launch_chained(F *kernel, dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, unsigned cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();        /* returned here: not the next launch's error as well */
  return e;
}
#ifdef __CUDACC__
__device__ __forceinline__ void pb_grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pb_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

/* dst[i] (dense, axis 0 fastest) = (dst type) src[sum_d x_d * sstride[d]] */
int pb_pack_launch(const void *src, void *dst, int naxes, const long long *ext, const long long *sstride,
                   int src_dtype, int dst_dtype, long long inner, long long dpitch, cudaStream_t stream);

/* One axis of the contraction: kind m/n/k/b, extent, and the stride it has in
 * the output C, in A, in B and in the addend X (0 where it does not appear). */
struct PbGemmAxis { char kind; long long ext, sc, sa, sb, sx; };

/* A copy of one operand for the tensor cores, kept while the source is unchanged.  form: what `data` holds, 16-bit
 * elements or the two tf32 parts of float32 ones (one program makes either, as the policy says at the call). */
enum { PB_TC_FORM_16 = 1, PB_TC_FORM_TF32 = 2 };
struct PbTcOperand {
  void *data = nullptr; size_t bytes = 0; int form = 0;
  const void *src = nullptr; uint64_t version = 0;
  int misses = 0;      /* conversions done; an operand that changes every call stops being cached */
};

struct PbGemmProgram : PbAotProgram {
  int p_c = -1, p_a = -1, p_b = -1, p_x = -1;
  int dtype = PB_F32;                 /* storage type of A and B */
  long long off_c = 0, off_a = 0, off_b = 0, off_x = 0;
  bool relu = false, has_x = false;
  float alpha = 1.0f;                 /* C = X + alpha * sum (relu); 1 except for fused optimizer updates */
  bool a_bf16 = false;                /* A's buffer holds bfloat16 (same element layout) although dtype is f32 */
  bool c_bf16 = false;                /* C is written as bfloat16 (round to nearest even) into the same element layout */
  bool gelu = false;                  /* tanh-GELU applied after the addend, before the bfloat16 store (needs c_bf16) */
  std::vector<PbGemmAxis> m_ax, n_ax, k_ax, b_ax;   /* m, n by output stride (largest first); k by A stride */
  long long M = 1, N = 1, K = 1, nbatch = 1;
  bool a_direct = false, b_direct = false;          /* strides nest: usable without packing */
  long long a_sm = 0, a_sk = 0, b_sk = 0, b_sn = 0, c_sm = 0, c_sn = 0, x_sm = 0, x_sn = 0;
  int launches = 1;
  PbTcOperand tc_a, tc_b;

  ~PbGemmProgram() override;
  int n_launches() const override { return launches; }
  int launch(void *const *bufs, cudaStream_t stream) override;
  bool stale(void *const *bufs) override;

  /* Dense [batch.., rows.., k..] copy (k fastest) of A or B in dst_dtype into dst. */
  int pack_into(void *dst, const void *src, long long off, bool is_a, int src_dtype, int dst_dtype,
                long long kpitch, cudaStream_t stream);
  void *pack_operand(const void *src, long long off, bool is_a, int src_dtype, int dst_dtype, cudaStream_t stream);
};

/* Builds the planned contraction from header lines whose keys start with `prefix`. */
PbGemmProgram *pb_parse_gemm(const PbHeader &h, const char *prefix, std::string &err);

/* Fused attention (pb_attention.cu). */
bool pb_attention_supported(long long T, long long hd);
/* A bfloat16 matrix of 64-element rows: element (batch.., row, d) at
 * ptr[sum_i batch_i * bstride[i] + row * row_stride + d]. */
struct PbAttnOperand { const void *ptr; long long row_stride; long long bstride[3]; };
int pb_attention_launch(const PbAttnOperand &q, const PbAttnOperand &k, const PbAttnOperand &v,
                        const float *mask, long long mask_sq, long long mask_sk,
                        float scale, void *out, bool out_bf16, int nb, const int *bext, const long long *o_sb, long long o_sm,
                        long long BH, long long T, cudaStream_t stream, float *tiles = nullptr, int tiles_mode = 0,
                        const float *norms_ready = nullptr);
/* tiles_mode 1: the mask classification (a record of eight floats per 128 x 128 tile of the mask) is computed into `tiles`,
 * 2: it is read from there; 0: the launch uses scratch of its own.  norms_ready: the row-norm bounds of q's blocks and
 * then of k's, where they have been computed already. */

/* Can the tensor-core kernel run this problem whatever the buffer addresses are
 * (16-byte aligned bases assumed), reading A in place when a_bf16 and writing
 * bfloat16 when c_bf16? */
bool pb_gemm_tc_static_ok(const PbGemmProgram &p);

/* Tensor-core path: returns 0 / -1, or PB_TC_UNSUPPORTED when the shape is not handled. */
/* fp32_mode 0: 16-bit operands.  1: float32 operands as three tf32 products, summed in tensor memory.
 * 2: the same with the partial sums moved to registers every two k-blocks (float32-accurate), 3: every block. */
int pb_gemm_tc_run(PbGemmProgram &p, void *const *bufs, cudaStream_t stream, int fp32_mode = 0);

/* The tensor-core kernel on ready-made bfloat16 K-major operands; touches no
 * memory beyond its arguments. */
int pb_gemm_tc_launch_raw(const void *a_bf16, long long a_pitch, const void *b_bf16, long long b_pitch,
                          float *C, long long c_sm, long long M, long long N, long long K,
                          const float *bias, int relu, cudaStream_t stream);

/* One-time set-up of everything pb_gemm_tc_launch_raw may need (shared-memory attribute of
 * each tile-width variant, the tensor-map encoder, the SM count).  0 / -1. */
int pb_gemm_tc_prepare_raw(void);

/* POLY_B200_GEMM=bf16: run fp32 contractions with operands rounded to bf16
 * (round-to-nearest-even), products and sums in fp32, on the tensor cores. */
bool pb_gemm_policy_bf16(void);

#endif
