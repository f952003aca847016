/*
 * pb_gather.cu -- embedding lookup and its gradient.
 *
 * polygrad expresses  out[t, d] = table[ids[t], d]  as a one-hot contraction
 *   out[t, d] = sum_v  (ids[t] == arange[v]) ? table[v, d] : 0
 * over the whole table (reference: src/modelzoo/models/gpt2.c:93-153), where ids
 * and arange are float32 buffers.  The kernels keep those semantics for any
 * buffer contents: a token's id selects every v with arange[v] equal to it (none
 * for NaN, out-of-range or fractional ids, which therefore give a row of +0), and
 * the matching rows are added in ascending v starting from +0, exactly like the
 * reference accumulation, so a -0.0f table entry comes out as +0.0f there and here.
 *
 * Where `arange` is strictly increasing (true for the 0..V-1 buffer the builders
 * make; false for anything with NaNs or duplicates) an id matches at most one v,
 * found by trying v = id and otherwise by bisection.  The first kernel takes that
 * for granted while it copies the rows, a warp per token, and its blocks check a
 * slice of `arange` each on the side; the second kernel returns at once if no
 * slice objected, and otherwise redoes every token by searching all of `arange`.
 * Either way the result is the reference's.  (Checking first and copying after
 * cost two dependent kernels with a single block in the first: 8192 tokens of a
 * 50257 x 768 table took 61 us, of which the copy, a block per token and an element
 * per thread, was 51; 14 us like this.)
 *
 * HBM traffic is the table rows read plus the output rows written.
 */
#include "../runtime/pb_runtime.h"
#include <cstdio>

struct GatherArgs {
  float *out; const float *ids; const float *arange; const float *table;
  long long vocab, table_vstride;
  long long out_off, ids_off, table_off;
  int ntok; long long tok_ext[4], tok_out[4], tok_ids[4];
  int nfeat; long long feat_ext[3], feat_out[3], feat_tab[3];
  long long n_tokens, n_feat;
};

#define GATHER_THREADS 256
#define GATHER_MAX_MATCH 8

/* [0] set when a slice of `arange` is not strictly increasing, [1] blocks of the second kernel that are
 * done with a call for which it was; both zero between calls (the library launches on one stream). */
static __device__ int pb200_gather_state[2];

/* FLAT: at most one token axis and one feature axis of unit strides (after merging): no index needs a division */
template <bool FLAT>
__device__ __forceinline__ void gather_token(const GatherArgs &a, long long tok, long long *o_out, long long *o_ids) {
  if (FLAT) { *o_out = a.out_off + tok * a.tok_out[0]; *o_ids = a.ids_off + tok * a.tok_ids[0]; return; }
  *o_out = a.out_off; *o_ids = a.ids_off;
  if (a.ntok == 1) { *o_out += tok * a.tok_out[0]; *o_ids += tok * a.tok_ids[0]; return; }
  for (int i = 0; i < a.ntok; i++) {
    const long long x = tok % a.tok_ext[i]; tok /= a.tok_ext[i];
    *o_out += x * a.tok_out[i]; *o_ids += x * a.tok_ids[i];
  }
}

/* A warp per token.  VEC: a row is one run of 16-byte aligned float4s in the table and in the result, six of
 * them per lane in flight (a 768-wide row at once); otherwise sixteen single elements of the row, or (not FLAT) one through the axes. */
template <bool VEC, bool FLAT>
__global__ void __launch_bounds__(GATHER_THREADS) pb200_gather_rows(const GatherArgs a) {
  const int lane = threadIdx.x & 31;
  const long long step = (long long)gridDim.x * (GATHER_THREADS / 32);
  for (long long tok = (long long)blockIdx.x * (GATHER_THREADS / 32) + (threadIdx.x >> 5); tok < a.n_tokens; tok += step) {
    long long o_out, o_ids;
    gather_token<FLAT>(a, tok, &o_out, &o_ids);
    const float id = a.ids[o_ids];
    long long v = -1;
    if (id == id) {
      const long long guess = (id >= 0.0f && id < (float)a.vocab) ? (long long)id : -1;
      if (guess >= 0 && guess < a.vocab && a.arange[guess] == id) v = guess;
      else {
        long long lo = 0, hi = a.vocab - 1;
        while (lo <= hi) {
          const long long mid = (lo + hi) >> 1;
          const float x = a.arange[mid];
          if (x == id) { v = mid; break; }
          if (x < id) lo = mid + 1; else hi = mid - 1;
        }
      }
    }
    if (VEC) {
      float4 *o = reinterpret_cast<float4 *>(a.out + o_out);
      const float4 *t = reinterpret_cast<const float4 *>(a.table + a.table_off + (v >= 0 ? v : 0) * a.table_vstride);
      const int nq = (int)(a.n_feat >> 2);
      for (int f0 = 0; f0 < nq; f0 += 192) {
        float4 x[6];
#pragma unroll
        for (int i = 0; i < 6; i++) {
          const int f = f0 + i * 32 + lane;
          x[i] = (v >= 0 && f < nq) ? __ldg(t + f) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 6; i++) {
          const int f = f0 + i * 32 + lane;
          if (f < nq) o[f] = make_float4(0.0f + x[i].x, 0.0f + x[i].y, 0.0f + x[i].z, 0.0f + x[i].w);
        }
      }
    } else if (FLAT) {
      const float *t = a.table + a.table_off + (v >= 0 ? v : 0) * a.table_vstride + lane;
      float *o = a.out + o_out + lane;
      const int nf = (int)a.n_feat - lane;
      for (int f0 = 0; f0 < nf; f0 += 512) {
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] = (v >= 0 && f0 + i * 32 < nf) ? __ldg(t + f0 + i * 32) : 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) if (f0 + i * 32 < nf) o[f0 + i * 32] = 0.0f + x[i];
      }
    } else {
      for (long long f = lane; f < a.n_feat; f += 32) {
        long long fr = f, o = o_out, t = a.table_off;
        for (int i = 0; i < a.nfeat; i++) {
          const long long x = fr % a.feat_ext[i]; fr /= a.feat_ext[i];
          o += x * a.feat_out[i]; t += x * a.feat_tab[i];
        }
        a.out[o] = v >= 0 ? 0.0f + a.table[t + v * a.table_vstride] : 0.0f;
      }
    }
  }
  /* this block's slice of the pairs (arange[i], arange[i + 1]) */
  const long long pairs = a.vocab - 1, slice = (pairs + gridDim.x - 1) / gridDim.x, p0 = blockIdx.x * slice;
  const long long p1 = p0 + slice < pairs ? p0 + slice : pairs;
  bool ok = true;
#pragma unroll 4
  for (long long p = p0 + threadIdx.x; p < p1; p += GATHER_THREADS) ok = ok & (a.arange[p] < a.arange[p + 1]);
  if (a.vocab == 1) ok = a.arange[0] == a.arange[0];
  if (!ok) pb200_gather_state[0] = 1;
}

/* Any `arange`: a block searches all of it for up to four tokens at a time, eight values per thread in flight and eight being
 * compared; its warps then share the rows.  Bound by the compares and L2 round trips.  8192 tokens of a 50257 x 768 table, numbering permuted, the
 * first kernel's 11 us included: 196 us with one token and value at a time, 86 like this (172 where a block per token
 * searched at once and no rows had been copied before); 16 tokens 24 and 18 (25). */
#define GATHER_SEARCH_TOKENS 4
#define GATHER_SEARCH_DEEP 8
template <bool FLAT>
__global__ void __launch_bounds__(GATHER_THREADS) pb200_gather_search(const GatherArgs a) {
  __shared__ int s_count[GATHER_SEARCH_TOKENS];
  __shared__ long long s_out[GATHER_SEARCH_TOKENS], s_match[GATHER_SEARCH_TOKENS][GATHER_MAX_MATCH];
  __shared__ float s_id[GATHER_SEARCH_TOKENS];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (*(volatile int *)pb200_gather_state == 0) return;
  const int per = (int)min((long long)GATHER_SEARCH_TOKENS, (a.n_tokens + gridDim.x - 1) / gridDim.x);
  for (long long tok0 = (long long)blockIdx.x * per; tok0 < a.n_tokens; tok0 += (long long)gridDim.x * per) {
    const int n = (int)min((long long)per, a.n_tokens - tok0);
    if (threadIdx.x < GATHER_SEARCH_TOKENS) {
      s_count[threadIdx.x] = 0;
      s_id[threadIdx.x] = __int_as_float(0x7fc00000);        /* matches nothing */
      if ((int)threadIdx.x < n) {
        long long o_ids;
        gather_token<false>(a, tok0 + threadIdx.x, &s_out[threadIdx.x], &o_ids);
        s_id[threadIdx.x] = a.ids[o_ids];
      }
    }
    __syncthreads();
    float id[GATHER_SEARCH_TOKENS];
#pragma unroll
    for (int i = 0; i < GATHER_SEARCH_TOKENS; i++) id[i] = s_id[i];
    float x[GATHER_SEARCH_DEEP], next[GATHER_SEARCH_DEEP];
    auto fetch = [&](long long v0) {                         /* values v0 + threadIdx.x + j * 256 */
      const float *p = a.arange + v0 + threadIdx.x;
      const int left = (int)min((long long)(GATHER_THREADS * GATHER_SEARCH_DEEP), a.vocab - v0) - (int)threadIdx.x;
#pragma unroll
      for (int j = 0; j < GATHER_SEARCH_DEEP; j++) next[j] = j * GATHER_THREADS < left ? __ldg(p + j * GATHER_THREADS) : __int_as_float(0x7fc00000);
    };
    fetch(0);
    for (long long v0 = 0; v0 < a.vocab; v0 += GATHER_THREADS * GATHER_SEARCH_DEEP) {
#pragma unroll
      for (int j = 0; j < GATHER_SEARCH_DEEP; j++) x[j] = next[j];
      if (v0 + GATHER_THREADS * GATHER_SEARCH_DEEP < a.vocab) fetch(v0 + GATHER_THREADS * GATHER_SEARCH_DEEP);
      bool any = false;
#pragma unroll
      for (int j = 0; j < GATHER_SEARCH_DEEP; j++) any |= x[j] == id[0] || x[j] == id[1] || x[j] == id[2] || x[j] == id[3];
      if (any) {
#pragma unroll
        for (int j = 0; j < GATHER_SEARCH_DEEP; j++)
#pragma unroll 1
          for (int i = 0; i < n; i++)
            if (x[j] == s_id[i]) {
              const int slot = atomicAdd(&s_count[i], 1);
              if (slot < GATHER_MAX_MATCH) s_match[i][slot] = v0 + threadIdx.x + j * GATHER_THREADS;
            }
      }
    }
    __syncthreads();
    if ((int)threadIdx.x < n && s_count[threadIdx.x] <= GATHER_MAX_MATCH) {
      /* ascending v: the order the reference adds in */
      long long *m = s_match[threadIdx.x];
      for (int i = 1; i < s_count[threadIdx.x]; i++) {
        long long x = m[i]; int j = i - 1;
        while (j >= 0 && m[j] > x) { m[j + 1] = m[j]; j--; }
        m[j + 1] = x;
      }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, parts = GATHER_THREADS / 32 / n, k = warp % n, part = warp / n;      /* warps share the rows */
    const int count = s_count[k];
    if (part < parts) {
      const long long step = parts * 32, f0 = part * 32 + (threadIdx.x & 31);
      if (FLAT && count <= 1) {
        const float *t = a.table + a.table_off + (count ? s_match[k][0] : 0) * a.table_vstride;
        float *o = a.out + s_out[k];
        for (long long f = f0; f < a.n_feat; f += step * 8) {
          float x[8];
#pragma unroll
          for (int i = 0; i < 8; i++) x[i] = count && f + i * step < a.n_feat ? __ldg(t + f + i * step) : 0.0f;
#pragma unroll
          for (int i = 0; i < 8; i++) if (f + i * step < a.n_feat) o[f + i * step] = 0.0f + x[i];
        }
      } else {
        for (long long f = f0; f < a.n_feat; f += step) {
          long long fr = f, o = s_out[k], t = a.table_off;
          if (FLAT) { o += f; t += f; }
          else for (int i = 0; i < a.nfeat; i++) {
            const long long x = fr % a.feat_ext[i]; fr /= a.feat_ext[i];
            o += x * a.feat_out[i]; t += x * a.feat_tab[i];
          }
          float acc = 0.0f;
          if (count <= GATHER_MAX_MATCH) {
            for (int i = 0; i < count; i++) acc = acc + a.table[t + s_match[k][i] * a.table_vstride];
          } else {
            /* pathological arange with many duplicates: plain ordered scan */
            for (long long v = 0; v < a.vocab; v++)
              if (a.arange[v] == s_id[k]) acc = acc + a.table[t + v * a.table_vstride];
          }
          a.out[o] = acc;
        }
      }
    }
    __syncthreads();
  }
  /* the last block to get here clears the state for the next call (every block has read it by then) */
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&pb200_gather_state[1], 1) == (int)gridDim.x - 1) { pb200_gather_state[0] = 0; pb200_gather_state[1] = 0; }
  }
}

/* Axis i + 1 continues axis i in both stride sets: one axis (batch and position of a dense token buffer). */
static void merge_axes(int &n, long long *ext, long long *s0, long long *s1) {
  int w = 0;
  for (int i = 0; i < n; i++) {
    if (ext[i] == 1) continue;
    if (w > 0 && s0[i] == s0[w - 1] * ext[w - 1] && s1[i] == s1[w - 1] * ext[w - 1]) { ext[w - 1] *= ext[i]; continue; }
    ext[w] = ext[i]; s0[w] = s0[i]; s1[w] = s1[i]; w++;
  }
  if (w == 0) s0[0] = s1[0] = 0;
  n = w;
}
static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct GatherProgram : PbAotProgram {
  GatherArgs a{};
  int n_launches() const override { return 2; }
  int p_out, p_ids, p_arange, p_table;
  int launch(void *const *bufs, cudaStream_t stream) override {
    GatherArgs g = a;
    g.out = (float *)bufs[p_out]; g.ids = (const float *)bufs[p_ids];
    g.arange = (const float *)bufs[p_arange]; g.table = (const float *)bufs[p_table];
    if (g.n_tokens <= 0 || g.n_feat <= 0) return 0;
    const bool flat = g.ntok <= 1 && g.nfeat == 1 && g.feat_out[0] == 1 && g.feat_tab[0] == 1 && g.n_feat < (1LL << 31);
    bool vec = flat && g.n_feat % 4 == 0 &&
               g.table_vstride % 4 == 0 && g.out_off % 4 == 0 && g.table_off % 4 == 0 && aligned16(g.out) && aligned16(g.table);
    for (int i = 0; i < g.ntok; i++) if (g.tok_out[i] % 4) vec = false;
    /* a warp per token; with few tokens, enough blocks that checking `arange` takes each a few loads per thread */
    long long grid = (g.n_tokens + GATHER_THREADS / 32 - 1) / (GATHER_THREADS / 32);
    const long long check = g.vocab / 1024 < 148 ? g.vocab / 1024 : 148;
    if (grid < check) grid = check;
    if (grid > (1LL << 20)) grid = 1LL << 20;
    if (vec) pb200_gather_rows<true, true><<<(unsigned)grid, GATHER_THREADS, 0, stream>>>(g);
    else if (flat) pb200_gather_rows<false, true><<<(unsigned)grid, GATHER_THREADS, 0, stream>>>(g);
    else pb200_gather_rows<false, false><<<(unsigned)grid, GATHER_THREADS, 0, stream>>>(g);
    /* launched while the first kernel drains (programmatic dependence: it waits for that kernel's results itself) */
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(g.n_tokens < 592 ? g.n_tokens : 592)); cfg.blockDim = dim3(GATHER_THREADS); cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, flat ? pb200_gather_search<true> : pb200_gather_search<false>, g);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { pb_set_error("gather launch: %s", cudaGetErrorString(e)); return -1; }
    return 0;
  }
};

PbAotProgram *pb_make_gather(const PbHeader &h, std::string &err) {
  auto params = h.getv("params"), vocab = h.getv("vocab"), off = h.getv("offsets");
  auto tok = h.getv("tok"), feat = h.getv("feat");
  if (params.size() != 4 || vocab.size() != 2 || off.size() != 3 || tok.size() % 3 || feat.size() % 3 ||
      tok.size() > 12 || feat.size() > 9) { err = "malformed gather header"; return nullptr; }
  GatherProgram *p = new GatherProgram();
  p->n_params = (int)h.geti("nparams");
  p->p_out = (int)params[0]; p->p_ids = (int)params[1]; p->p_arange = (int)params[2]; p->p_table = (int)params[3];
  p->rw.assign((size_t)p->n_params, '-');
  for (int i = 1; i < 4; i++) p->rw[(size_t)params[i]] = 'r';
  p->rw[(size_t)params[0]] = 'w';
  GatherArgs &a = p->a;
  a.vocab = vocab[0]; a.table_vstride = vocab[1];
  a.out_off = off[0]; a.ids_off = off[1]; a.table_off = off[2];
  a.ntok = (int)tok.size() / 3; a.nfeat = (int)feat.size() / 3;
  a.n_tokens = 1; a.n_feat = 1;
  for (int i = 0; i < a.ntok; i++) { a.tok_ext[i] = tok[3 * i]; a.tok_out[i] = tok[3 * i + 1]; a.tok_ids[i] = tok[3 * i + 2]; a.n_tokens *= a.tok_ext[i]; }
  if (a.n_tokens > 0) merge_axes(a.ntok, a.tok_ext, a.tok_out, a.tok_ids);
  for (int i = 0; i < a.nfeat; i++) { a.feat_ext[i] = feat[3 * i]; a.feat_out[i] = feat[3 * i + 1]; a.feat_tab[i] = feat[3 * i + 2]; a.n_feat *= a.feat_ext[i]; }
  /* feature axes: smallest output stride first so that consecutive threads write consecutive floats */
  for (int i = 1; i < a.nfeat; i++)
    for (int j = i; j > 0 && llabs(a.feat_out[j]) < llabs(a.feat_out[j - 1]); j--) {
      std::swap(a.feat_ext[j], a.feat_ext[j - 1]); std::swap(a.feat_out[j], a.feat_out[j - 1]); std::swap(a.feat_tab[j], a.feat_tab[j - 1]);
    }
  if (a.n_feat > 0) merge_axes(a.nfeat, a.feat_ext, a.feat_out, a.feat_tab);
  return p;
}

/* ── the lookup's gradient ───────────────────────────────────────────── */
/* out[v, d] = sum_t (ids[t] == arange[v]) ? src[t, d] : 0 for every table row v (reference: the backward
 * of the one-hot lookup, which polygrad runs as a contraction over all tokens for every row).  A block
 * owns up to SCATTER_ROWS consecutive rows (and, where the table has few, a part of the features).  It writes
 * zeros to all of them -- most rows have no token, and the writes drain while it looks -- and goes through the
 * tokens SCATTER_CHUNK at a time, each warp through consecutive ones, noting in token order which token
 * matches which of its rows; a stable counting sort brings the matches of a row together, still in token order;
 * then a warp per (row with matches, 128 features of it) adds the source rows one by one, starting from +0 (from
 * the result so far in later chunks) -- the order and the value of the reference's accumulation, in which the
 * non-matching tokens add +0 -- with SCATTER_DEEP rows' loads in flight.
 *
 * A token finds its row by subtraction where the block's part of `arange` is consecutive integers, otherwise by
 * comparing with every row (NaNs match nothing); where values repeat, the tokens go to the last row of their value, whose
 * sum the others copy.  A warp's list holds every token of its part
 * of a chunk, so it cannot overflow.
 *
 * HBM traffic: the output written once, the ids read once per block (from L2), the matching source rows.  8192
 * tokens (ids distributed as words in text) into a 50257 x 768 table: 1000 us with blocks of 16 rows that compared
 * one id at a time with all of them, sorted the matches by insertion on one thread and added one load at a time; 65 us like this, of which the zeros
 * are 33 (4.7 TB/s) and the longest chains (a word 272 times) most of the rest. */
struct ScatterArgs {
  float *out; const float *ids; const float *arange; const float *src;
  long long vocab, out_vstride;
  long long out_off, ids_off, src_off;
  int ntok; long long tok_ext[4], tok_ids[4], tok_src[4];
  int nfeat; long long feat_ext[3], feat_out[3], feat_src[3];
  long long n_tokens, n_feat;
  int rows_per_block;
  int ids_vec;                    /* ids are one run of 16-byte aligned floats */
  long long feat_per_block;       /* a multiple of 128 */
};

#define SCATTER_THREADS 256
#define SCATTER_WARPS 8
#define SCATTER_ROWS 128
#define SCATTER_CHUNK 4096
#define SCATTER_DEEP 6

/* MODE 1: one token axis and one feature axis of unit strides; 2: and 16-byte aligned rows; 0: any axes */
template <int MODE>
__global__ void __launch_bounds__(SCATTER_THREADS, 4) pb200_scatter_rows(const ScatterArgs a) {
  constexpr int PER_WARP = SCATTER_CHUNK / SCATTER_WARPS;
  __shared__ float s_ar[SCATTER_ROWS];
  __shared__ unsigned s_list[SCATTER_WARPS][PER_WARP];            /* row << 16 | token within the chunk */
  __shared__ unsigned short s_tok[SCATTER_CHUNK];                 /* tokens of the chunk by row, in token order */
  __shared__ __align__(16) int s_off[SCATTER_ROWS * SCATTER_WARPS];   /* matches of (row, warp): their number, then where they go in s_tok */
  __shared__ int s_begin[SCATTER_ROWS + 1];                       /* where those of the row begin */
  __shared__ unsigned char s_rows[SCATTER_ROWS];                  /* rows with matches */
  __shared__ int s_matched;
  __shared__ unsigned char s_some[SCATTER_ROWS];                  /* rows that had matches in any chunk */
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long v0 = (long long)blockIdx.x * a.rows_per_block;
  const int rows = (int)min((long long)a.rows_per_block, a.vocab - v0);
  const long long f_begin = (long long)blockIdx.y * a.feat_per_block;
  const int nf = (int)(min(f_begin + a.feat_per_block, a.n_feat) - f_begin), segs = (nf + 127) / 128;
  float *const out = a.out + a.out_off + v0 * a.out_vstride;
  const float *const src = a.src + a.src_off;

  /* feature f of this block: offset in a row of the result and of the source */
  auto feature = [&](int f, long long *oo, long long *so) {
    if (MODE) { *oo = *so = f_begin + f; return; }
    long long fr = f_begin + f;
    *oo = *so = 0;
    for (int d = 0; d < a.nfeat; d++) { const long long x = fr % a.feat_ext[d]; fr /= a.feat_ext[d]; *oo += x * a.feat_out[d]; *so += x * a.feat_src[d]; }
  };
  for (int r = warp; r < rows; r += SCATTER_WARPS) {
    float *orow = out + r * a.out_vstride;
    long long oo, so;
    if (MODE == 2) for (int f = lane * 4; f < nf; f += 128) *reinterpret_cast<float4 *>(orow + f_begin + f) = make_float4(0.f, 0.f, 0.f, 0.f);
    else for (int f = lane; f < nf; f += 32) { feature(f, &oo, &so); orow[oo] = 0.0f; }
  }
  if (threadIdx.x < SCATTER_ROWS) {
    s_ar[threadIdx.x] = (int)threadIdx.x < rows ? a.arange[v0 + threadIdx.x] : __int_as_float(0x7fc00000);
    s_some[threadIdx.x] = 0;
  }
  __syncthreads();
  const float ar0 = s_ar[0];
  bool consecutive = truncf(ar0) == ar0 && fabsf(ar0) < 8388608.0f;        /* differences of such values are exact */
  if ((int)threadIdx.x < rows) consecutive &= s_ar[threadIdx.x] == ar0 + (float)threadIdx.x;
  consecutive = __syncthreads_and(consecutive ? 1 : 0) != 0;
  /* the last row of the token's value */
  auto row_of = [&](float x) {
    if (consecutive) { const float dlt = x - ar0; return dlt >= 0.0f && dlt < (float)rows && ar0 + dlt == x && truncf(dlt) == dlt ? (int)dlt : -1; }
    int row = -1;
    for (int r = 0; r < rows; r++) if (x == s_ar[r]) row = r;
    return row;
  };
  for (long long c0 = 0; c0 < a.n_tokens; c0 += SCATTER_CHUNK) {
    /* matches of this warp's tokens: four consecutive tokens per lane and step, all steps' loads in flight */
    const long long w0 = c0 + warp * PER_WARP;
    const int nw = (int)max(0LL, min((long long)PER_WARP, a.n_tokens - w0));
    float id[PER_WARP / 128][4];
#pragma unroll
    for (int s = 0; s < PER_WARP / 128; s++) {
      const int t = s * 128 + lane * 4;
      if (a.ids_vec && t + 3 < nw) {
        const float4 x = __ldg(reinterpret_cast<const float4 *>(a.ids + a.ids_off + w0 + t));
        id[s][0] = x.x; id[s][1] = x.y; id[s][2] = x.z; id[s][3] = x.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          id[s][i] = __int_as_float(0x7fc00000);                         /* matches nothing */
          if (t + i < nw) {
            long long rem = w0 + t + i, o = a.ids_off;
            if (MODE) o += rem * a.tok_ids[0];
            else for (int d = 0; d < a.ntok; d++) { const long long x = rem % a.tok_ext[d]; rem /= a.tok_ext[d]; o += x * a.tok_ids[d]; }
            id[s][i] = a.ids[o];
          }
        }
      }
    }
    for (int i = threadIdx.x; i < SCATTER_ROWS * SCATTER_WARPS / 4; i += SCATTER_THREADS) reinterpret_cast<int4 *>(s_off)[i] = make_int4(0, 0, 0, 0);
    __syncthreads();
    int n = 0;                                                           /* entries of this warp's list */
#pragma unroll
    for (int s = 0; s < PER_WARP / 128; s++) {
      int row[4];
#pragma unroll
      for (int i = 0; i < 4; i++) row[i] = row_of(id[s][i]);
      const int mine = (row[0] >= 0) + (row[1] >= 0) + (row[2] >= 0) + (row[3] >= 0);
      if (__any_sync(0xffffffffu, mine)) {
        int at = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, at, o); if (lane >= o) at += y; }
        const int total = __shfl_sync(0xffffffffu, at, 31);
        at += n - mine;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (row[i] >= 0) {
            s_list[warp][at++] = ((unsigned)row[i] << 16) | (unsigned)(warp * PER_WARP + s * 128 + lane * 4 + i);
            atomicAdd(&s_off[row[i] * SCATTER_WARPS + warp], 1);
          }
        n += total;
      }
    }
    __syncthreads();
    /* counts -> positions, by row and, within a row, by warp (which is by token); a lane per row */
    if (warp == 0) {
      int base = 0, found = 0;
#pragma unroll 1
      for (int rb = 0; rb < SCATTER_ROWS && rb < rows; rb += 32) {
        int4 *cp = reinterpret_cast<int4 *>(s_off + (rb + lane) * SCATTER_WARPS);
        const int4 c = cp[0], d = cp[1];
        const int sum = c.x + c.y + c.z + c.w + d.x + d.y + d.z + d.w;
        int at = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, at, o); if (lane >= o) at += y; }
        const int total = __shfl_sync(0xffffffffu, at, 31);
        at += base - sum;
        s_begin[rb + lane] = at;
        const unsigned some = __ballot_sync(0xffffffffu, sum > 0);
        if (sum > 0) { s_rows[found + __popc(some & ((1u << lane) - 1u))] = (unsigned char)(rb + lane); s_some[rb + lane] = 1; }
        int4 p, q;
        p.x = at; p.y = p.x + c.x; p.z = p.y + c.y; p.w = p.z + c.z; q.x = p.w + c.w; q.y = q.x + d.x; q.z = q.y + d.y; q.w = q.z + d.z;
        cp[0] = p; cp[1] = q;
        base += total; found += __popc(some);
      }
      if (lane == 0) { s_begin[min(SCATTER_ROWS, (rows + 31) / 32 * 32)] = base; s_matched = found; }
    }
    __syncthreads();
    /* every warp places its list; s_off[row, warp] moves on with it */
    for (int i0 = 0; i0 < n; i0 += 32) {
      const bool have = i0 + lane < n;
      const unsigned e = have ? s_list[warp][i0 + lane] : 0xffffffffu;
      const unsigned peers = __match_any_sync(0xffffffffu, e >> 16);
      const int before = __popc(peers & ((1u << lane) - 1u));
      int *slot = &s_off[(e >> 16) * SCATTER_WARPS + warp];
      int at = 0;
      if (have) { at = *slot; s_tok[at + before] = (unsigned short)(e & 0xffffu); }
      __syncwarp();
      if (have && before == 0) *slot = at + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    auto token_row = [&](int m) {
      long long rem = c0 + s_tok[m];
      if (MODE) return src + rem * a.tok_src[0];
      const float *p = src;
      for (int d = 0; d < a.ntok; d++) { const long long x = rem % a.tok_ext[d]; rem /= a.tok_ext[d]; p += x * a.tok_src[d]; }
      return p;
    };
    const int matched = s_matched;
    /* the source rows of the commonest words are requested from memory beforehand: their sum is one serial chain */
    if (MODE) {
      const unsigned lines = ((unsigned)nf + 31) / 32;
      for (int k = 0; k < matched; k++) {
        const int m0 = s_begin[s_rows[k]], m1 = s_begin[s_rows[k] + 1];
        if (m1 - m0 <= SCATTER_DEEP) continue;
        for (unsigned i = threadIdx.x; i < (unsigned)(m1 - m0) * lines; i += SCATTER_THREADS) {
          const unsigned m = i / lines;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(token_row(m0 + (int)m) + f_begin + (i - m * lines) * 32));
        }
      }
    }
    for (unsigned item = warp; item < (unsigned)(matched * segs); item += SCATTER_WARPS) {
      const unsigned k = item / (unsigned)segs;
      const int r = s_rows[k], f = (int)(item - k * segs) * 128 + (MODE == 2 ? lane * 4 : lane);
      const int m0 = s_begin[r], m1 = s_begin[r + 1];
      float *orow = out + r * a.out_vstride;
      if (MODE == 2) {
        if (f >= nf) continue;
        float4 *op = reinterpret_cast<float4 *>(orow + f_begin + f);
        float4 acc = c0 == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *op;
        for (int m = m0; m < m1; m += SCATTER_DEEP) {
          float4 x[SCATTER_DEEP];
#pragma unroll
          for (int i = 0; i < SCATTER_DEEP; i++) if (m + i < m1) x[i] = __ldg(reinterpret_cast<const float4 *>(token_row(m + i) + f_begin + f));
#pragma unroll
          for (int i = 0; i < SCATTER_DEEP; i++) if (m + i < m1) { acc.x += x[i].x; acc.y += x[i].y; acc.z += x[i].z; acc.w += x[i].w; }
        }
        *op = acc;
      } else {
        /* four features 32 apart per lane */
        long long oo[4], so[4];
        float acc[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          feature(f + j * 32, &oo[j], &so[j]);
          acc[j] = (c0 == 0 || f + j * 32 >= nf) ? 0.0f : orow[oo[j]];
        }
        constexpr int DEEP = MODE ? 4 : 1;
        for (int m = m0; m < m1; m += DEEP) {
          float x[DEEP][4];
#pragma unroll
          for (int i = 0; i < DEEP; i++)
            if (m + i < m1) {
              const float *p = token_row(m + i);
#pragma unroll
              for (int j = 0; j < 4; j++) if (f + j * 32 < nf) x[i][j] = __ldg(p + so[j]);
            }
#pragma unroll
          for (int i = 0; i < DEEP; i++)
            if (m + i < m1) {
#pragma unroll
              for (int j = 0; j < 4; j++) if (f + j * 32 < nf) acc[j] += x[i][j];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) if (f + j * 32 < nf) orow[oo[j]] = acc[j];
      }
    }
    __syncthreads();
  }
  if (consecutive) return;
  bool repeats = false;
  if ((int)threadIdx.x < rows) for (int r = 0; r < (int)threadIdx.x; r++) repeats |= s_ar[r] == s_ar[threadIdx.x];
  if (!__syncthreads_or(repeats ? 1 : 0)) return;
  for (int r = warp; r < rows; r += SCATTER_WARPS) {
    int last = r;
    for (int r2 = r + 1; r2 < rows; r2++) if (s_ar[r2] == s_ar[r]) last = r2;
    if (last == r || !s_some[last]) continue;
    float *to = out + r * a.out_vstride;
    const float *from = out + last * a.out_vstride;
    if (MODE == 2) {
#pragma unroll 4
      for (int f = lane * 4; f < nf; f += 128) *reinterpret_cast<float4 *>(to + f_begin + f) = *reinterpret_cast<const float4 *>(from + f_begin + f);
    } else for (int f = lane; f < nf; f += 32) { long long oo, so; feature(f, &oo, &so); to[oo] = from[oo]; }
  }
}

struct ScatterProgram : PbAotProgram {
  ScatterArgs a{};
  int n_launches() const override { return 1; }
  int p_out, p_ids, p_arange, p_src;
  int launch(void *const *bufs, cudaStream_t stream) override {
    ScatterArgs g = a;
    g.out = (float *)bufs[p_out]; g.ids = (const float *)bufs[p_ids];
    g.arange = (const float *)bufs[p_arange]; g.src = (const float *)bufs[p_src];
    if (g.vocab <= 0 || g.n_feat <= 0) return 0;
    const bool flat = g.ntok <= 1 && g.nfeat == 1 && g.feat_out[0] == 1 && g.feat_src[0] == 1;
    bool vec = flat && g.n_feat % 4 == 0 && g.out_vstride % 4 == 0 &&
               g.out_off % 4 == 0 && g.src_off % 4 == 0 && aligned16(g.out) && aligned16(g.src);
    for (int i = 0; i < g.ntok; i++) if (g.tok_src[i] % 4) vec = false;
    g.ids_vec = g.ntok == 1 && g.tok_ids[0] == 1 && aligned16(g.ids + g.ids_off) ? 1 : 0;
    /* every block reads all ids and the blocks should run as one wave (four fit on an SM), so as many rows per block as
     * that takes; where the table has too few rows for that many blocks, parts of the features each */
    const long long want = 148 * 4;
    long long rows = (g.vocab + want - 1) / want;
    g.rows_per_block = (int)(rows < 4 ? 4 : rows > SCATTER_ROWS ? SCATTER_ROWS : rows);
    const long long grid = (g.vocab + g.rows_per_block - 1) / g.rows_per_block;
    if (grid > 2147483647LL) { pb_set_error("scatter: too many table rows"); return -1; }
    const long long segs = (g.n_feat + 127) / 128;
    long long parts = grid < want ? want / grid : 1;
    if (parts > segs) parts = segs;
    if (parts > 65535) parts = 65535;
    g.feat_per_block = (segs + parts - 1) / parts * 128;
    const dim3 blocks((unsigned)grid, (unsigned)((g.n_feat + g.feat_per_block - 1) / g.feat_per_block));
    if (vec) pb200_scatter_rows<2><<<blocks, SCATTER_THREADS, 0, stream>>>(g);
    else if (flat) pb200_scatter_rows<1><<<blocks, SCATTER_THREADS, 0, stream>>>(g);
    else pb200_scatter_rows<0><<<blocks, SCATTER_THREADS, 0, stream>>>(g);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { pb_set_error("scatter launch: %s", cudaGetErrorString(e)); return -1; }
    return 0;
  }
};

PbAotProgram *pb_make_scatter(const PbHeader &h, std::string &err) {
  auto params = h.getv("params"), vocab = h.getv("vocab"), off = h.getv("offsets");
  auto tok = h.getv("tok"), feat = h.getv("feat");
  if (params.size() != 4 || vocab.size() != 2 || off.size() != 3 || tok.size() % 3 || feat.size() % 3 ||
      tok.empty() || tok.size() > 12 || feat.size() > 9) { err = "malformed scatter header"; return nullptr; }
  ScatterProgram *p = new ScatterProgram();
  p->n_params = (int)h.geti("nparams");
  p->p_out = (int)params[0]; p->p_ids = (int)params[1]; p->p_arange = (int)params[2]; p->p_src = (int)params[3];
  p->rw.assign((size_t)p->n_params, '-');
  for (int i = 1; i < 4; i++) p->rw[(size_t)params[i]] = 'r';
  p->rw[(size_t)params[0]] = 'w';
  ScatterArgs &a = p->a;
  a.vocab = vocab[0]; a.out_vstride = vocab[1];
  a.out_off = off[0]; a.ids_off = off[1]; a.src_off = off[2];
  a.ntok = (int)tok.size() / 3; a.nfeat = (int)feat.size() / 3;
  a.n_tokens = 1; a.n_feat = 1;
  for (int i = 0; i < a.ntok; i++) { a.tok_ext[i] = tok[3 * i]; a.tok_ids[i] = tok[3 * i + 1]; a.tok_src[i] = tok[3 * i + 2]; a.n_tokens *= a.tok_ext[i]; }
  if (a.n_tokens > 0) merge_axes(a.ntok, a.tok_ext, a.tok_ids, a.tok_src);
  for (int i = 0; i < a.nfeat; i++) { a.feat_ext[i] = feat[3 * i]; a.feat_out[i] = feat[3 * i + 1]; a.feat_src[i] = feat[3 * i + 2]; a.n_feat *= a.feat_ext[i]; }
  if (a.n_tokens >= (1LL << 40)) { err = "scatter: too many tokens"; delete p; return nullptr; }
  /* feature axes: smallest output stride first so that consecutive threads write consecutive floats */
  for (int i = 1; i < a.nfeat; i++)
    for (int j = i; j > 0 && llabs(a.feat_out[j]) < llabs(a.feat_out[j - 1]); j--) {
      std::swap(a.feat_ext[j], a.feat_ext[j - 1]); std::swap(a.feat_out[j], a.feat_out[j - 1]); std::swap(a.feat_src[j], a.feat_src[j - 1]);
    }
  if (a.n_feat > 0) merge_axes(a.nfeat, a.feat_ext, a.feat_out, a.feat_src);
  return p;
}
