// The fused dequant-GEMM forward with the dequantised weights in TENSOR MEMORY (tcgen05.mma with its A operand
// in TMEM).  Included by q4_gemm.cu after q4_gemm2.cuh.
//
// The pair kernel of q4_gemm2.cuh keeps both operands in shared memory: a dequant task there is eight swizzled
// 16-byte stores behind scale and zero-term vectors of eight columns, a proxy fence and a barrier, and per 64
// contraction elements an SM takes 16 KiB of dequant stores on top of 16 KiB of TMA writes and 32 KiB of tensor-core
// reads.  Here the product is transposed,
// y^T = W^T x^T: the weights are the A operand (M side: 256 output columns per pair, 128 per CTA = one TMEM lane
// each), the activations the B operand (N side: a tile of up to 384 rows of x, half per CTA, K-major by TMA exactly as
// before).  A dequant thread owns one output column: the eight packed words of its column and a stage are eight
// coalesced 4-byte loads, one word is eight consecutive k of that column = four half2 in contraction order, and the
// stage's 64 halves leave as one `tcgen05.st` of 32 columns.  Nothing of W touches shared memory.
//   Sequential groups (by the caller's word): scale and zero term are scalars of the thread.
//   Act-order (ACT): every weight has the scale and zero term of its own row's group.  A table in shared memory holds the
//   two as one word per group and column of this CTA; the lanes' columns lie on different banks whatever the group, and
//   the 64 rows' offsets into it are the same for all lanes of a warp.  (The pair kernel looks whole vectors of eight
//   columns up row by row: 333 rows of 5120 x 5120 take 43 us there and 28 here, 77 rows 32 and 22.)
//
// Tiles follow the rows: as many as of 384 or 256 rows, whichever takes less time (gemm3_plan), all of one height, a
// multiple of 32.  77 rows are one tile of 96 and 333 one of 352 - two MMAs, of 192 and 160 rows, on the same dequantised
// operand (TALL), which used to be dequantised for two tiles of 256.  (Each a multiple of 32: an MMA with A in TMEM has N in
// steps of 32.  The activation stage then holds twice the larger part, and the copies of the smaller one bring rows that
// nothing reads.)
// TMEM (512 columns): accumulator [128 lanes = output columns][columns = rows of x] fp32, and four to eight operand
// stages of 32 columns (lane = output column, column c of a stage = contraction elements 2c, 2c+1 as a half2).
// Roles (640 threads per CTA): warp 0 TMA producer of this CTA's half of the activation rows; warp 1 owns TMEM, its elected
// lane in the even CTA issues the MMAs; warps 4-15 dequantise (warp & 3 = its TMEM lane quarter; three groups of
// four warps take every third stage use: a task is a chain of loads, arithmetic, the wait for the slot, the TMEM
// store and its completion, about 1500 cycles where the MMAs of 256 rows take 540, so three tasks have to be in
// flight); warps 16-19 epilogue.  Whole tiles per pair round after round, or (SPLIT) equal runs of tiles x stages.
// The accumulator's lanes are output columns, so a thread of the epilogue holds 32 rows of one column: a warp turns blocks
// of 32 rows x 32 columns over in shared memory as fp16 and stores rows of 64 bytes, four lanes each.  In the plain form
// (sequential, up to 256 rows) there is room for all blocks, and the accumulator is handed back before the stores.
// Every wait is bounded as in the pair kernel.
// Where the pairs that share a tile form a cluster (p.cluster_pairs, few tiles), each adds up a part of the tile's rows from
// the others' shared memory: through the workspace the exchange took 5-7 us (write, fence, count, wait, and the
// contributors' sums one after the other from L2), in the cluster 1-2.
// Launched with the programmatic-dependent-launch attribute: the set-up runs before the wait for the earlier kernel, and
// every warp waits before its first read or write of global memory.  That holds for the layer's own tensors too: the
// kernel just ahead may be the one that fills the zero-term table of a layer's first call, or casts its scales or bias.
// (An L2 prefetch delivers no value, so the first words may be asked for before the wait.)
#pragma once

namespace q4 {

constexpr int G3_MAX_STAGES = 8;              // operand stages in TMEM = activation stages in shared memory
constexpr int G3_MAX_ROWS = 384;              // of a tile: its accumulator and four operand stages are all of TMEM
constexpr int G3_BAR_BYTES = 512;
constexpr int G3_MAX_CLUSTER = 4;             // pairs: eight CTAs, the portable size
constexpr int G3_GROUPS = 3;                  // dequant groups of four warps
constexpr int G3_THREADS = 32 * (4 + 4 * G3_GROUPS + 4);
constexpr int G3_OFFS_BYTES = 4 * G3_GROUPS * 256;   // act-order: per dequant warp the table offsets of a stage's 64 rows
constexpr int G3_PLAIN_AREA = G3_MAX_STAGES * 128 * GM_TILE_C * 2;
constexpr int G3_TURN_BLOCK = 32 * 64;         // a warp's 32 columns of 32 rows, fp16

// A tile of more than 256 rows is two MMAs: the rows of the first, a multiple of 32 and no fewer than the second's.
__host__ __device__ constexpr int gemm3_first_rows(int tile_rows) { return (tile_rows / 2 + 31) / 32 * 32; }

__device__ __forceinline__ void umma_f16_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp writes lane (lane base + i).
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]),
        "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
        "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

// Loads that the compiler may neither move nor take for loads of memory that nobody writes while the kernel lives (an
// earlier kernel of the stream may still be writing it when this one is launched).
__device__ __forceinline__ uint32_t ld_pinned_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_pinned_u16(const void* p) {
  uint16_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}

// One packed word = eight consecutive contraction elements of one output column -> four half2 in order.
// Byte j of the word holds levels 2j (low nibble) and 2j+1 (high nibble): the byte is copied to bytes 0 and 2,
// the low nibble becomes the mantissa of 1024 + q, the high nibble stays in place as the mantissa of 64 + q
// (exponent 0x5400, ulp 1/16), and one fused multiply-add with (-1024 s, -64 s) leaves rn(s q) in both halves.
template <bool FOLD>
__device__ __forceinline__ void deq_word_k(uint32_t w, uint32_t s2, uint32_t c2, uint32_t z2, uint32_t* o) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t u = prmt(w, w, j | (j << 8));
    const uint32_t v = and_or(u, 0x00F0000Fu, 0x54006400u);
    if (FOLD) o[j] = as_u32(__hsub2_rn(__hfma2(as_h2(v), as_h2(s2), as_h2(c2)), as_h2(z2)));
    else o[j] = as_u32(__hsub2_rn(__hmul2_rn(as_h2(s2), __hsub2(as_h2(v), as_h2(0x54006400u))), as_h2(z2)));
  }
}

// SPLIT as in the pair kernel: whole tiles per pair, or equal runs of the sequence of all tiles x stages with the
// partial sums of a shared tile meeting in the workspace (added in pair order by the pair whose run starts the tile).
// The launch gives the cluster's size: one pair or, with p.cluster_pairs = n > 1 (SPLIT only), the n pairs that share a tile.
// ACT: act-order.  Every weight has the scale and zero term of its own row's group: a table in shared memory holds, per group
// and column of this CTA, the two as one word, a lane's loads of it lie on its own bank whatever the groups are, and the
// rows' table offsets of a stage are the same for all lanes.
template <bool SPLIT, bool ACT, bool TALL>
__global__ void __launch_bounds__(G3_THREADS, 1)
q4_gemm3_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap umap, const GemmParams p) {
  extern __shared__ unsigned char smem_raw[];
  pdl_launch_dependents();
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int S = ACT || TALL ? p.stages : G3_MAX_STAGES;
  const int TR = p.tile_rows;                          // rows of x per tile, a multiple of 32
  constexpr int nh = TALL ? 2 : 1;                     // MMAs per 16 contraction elements
  const int HR = TALL ? gemm3_first_rows(TR) : TR;     // rows of the first, which takes no fewer than the second
  constexpr bool PLAIN = !ACT && !TALL;                // one layout for all: stages of 128 rows, a place to turn every block over
  const int x_bytes = PLAIN ? 128 * GM_TILE_C * 2 : nh * HR * GM_TILE_C;        // this CTA's half of a tile's rows of a stage
  unsigned char* tab = smem + S * x_bytes;             // act-order: [G][128 columns] scale | zero term
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (PLAIN ? G3_PLAIN_AREA : p.area));                  // even CTA: activation bytes + 4 dequant warps, of both CTAs
  uint64_t* empty = full + 8;                                                   // both CTAs: stage read by the MMAs
  uint64_t* acc_full = empty + 8;                                               // both CTAs: accumulator complete
  uint64_t* acc_empty = acc_full + 1;                                           // even CTA: 4 epilogue warps x 2 CTAs
  uint64_t* last_full = acc_empty + 1;                                          // both CTAs: the pair's last accumulator complete (one use)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned char* offs_all = reinterpret_cast<unsigned char*>(full) + G3_BAR_BYTES;
  unsigned char* turn = offs_all + (ACT ? G3_OFFS_BYTES : 0);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cluster_rank = cluster_ctarank(), rank = cluster_rank & 1, even_cta = cluster_rank & ~1u;
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int T = p.n_contract_tiles;
  const int lora_ks = (p.lora_r + 15) >> 4;
  const int N = p.N;
  const int m_tiles = (p.M + TR - 1) / TR;
  const int n_tiles = m_tiles * (N / G2_TILE_N);
  const WorkRange wr = work_range<SPLIT>(pair, n_pairs, n_tiles, T);
  const int n_items = wr.n_items;

  // where a warp turns a block of 32 rows over: a place per block (the accumulator can be handed back before the stores) or,
  // where shared memory is short, one per warp
  auto turn_of = [&](int quarter, int cb) __attribute__((always_inline)) {
    return turn + (PLAIN ? quarter * 8 + cb : p.turn_blocks ? quarter * p.turn_blocks + cb : warp - 4) * G3_TURN_BLOCK;
  };
  struct TaskRegs { uint32_t w[8]; uint32_t s, z; };             // (act-order: s and z are the groups of rows lane and 32 + lane)
  const bool is_deq = warp >= 4 && warp < 4 + 4 * G3_GROUPS;
  auto column_of = [&](int tile) { return (tile / m_tiles) * G2_TILE_N + 128 * (int)rank + 32 * (warp & 3) + lane; };
  auto prefetch = [&](int n, int j, TaskRegs& R) __attribute__((always_inline)) {
    if (j >= T) return;
    const uint32_t* wcol = p.qw + n;
    const uint32_t* src = wcol + (size_t)(j * (GM_TILE_C >> 3)) * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) R.w[i] = ld_pinned_u32(src + (size_t)i * N);
    if (ACT) {
      R.s = ld_pinned_u32(p.g_idx + j * GM_TILE_C + lane);
      R.z = ld_pinned_u32(p.g_idx + j * GM_TILE_C + 32 + lane);
    } else {
      const size_t at = (size_t)((j * GM_TILE_C) >> p.seq_shift) * N + n;
      R.s = ld_pinned_u16(p.scales + at);
      R.z = ld_pinned_u16(p.zp_table + at);
    }
    // the words of the group's task after the next, asked into L2 (eight rows of 128 bytes per warp)
    if (j + 2 * G3_GROUPS < T && lane < 8) prefetch_l2(wcol - lane + (size_t)((j + 2 * G3_GROUPS) * (GM_TILE_C >> 3) + lane) * N);
  };
  // A dequant warp asks for its first two tasks before the set-up below (barriers, TMEM, the cluster's meeting: about a
  // microsecond) and before the wait for the earlier kernel: into L2, where they are read once both are over.
  if (is_deq && n_items > 0) {
    const WorkItem w0 = work_item<SPLIT>(p, wr, 0, n_pairs, T);
    const int n = column_of(w0.tile) - lane;                       // the warp's 32 columns: 128 bytes of words, 64 of scales
#pragma unroll
    for (int ahead = 0; ahead < 2; ++ahead) {
      const int j = w0.kb + ((warp - 4) >> 2) + ahead * G3_GROUPS;
      if (j >= w0.ke) break;
      const size_t at = (size_t)((j * GM_TILE_C) >> p.seq_shift) * N + n;
      if (lane < 8) prefetch_l2(p.qw + (size_t)(j * (GM_TILE_C >> 3) + lane) * N + n);
      else if (ACT && lane < 10) prefetch_l2(p.g_idx + j * GM_TILE_C + 32 * (lane - 8));
      else if (!ACT && lane == 8) prefetch_l2(p.scales + at);
      else if (!ACT && lane == 9) prefetch_l2(p.zp_table + at);
    }
    if (ACT)
      for (int i = threadIdx.x - 128; i < 3 * p.G; i += 128 * G3_GROUPS) {
        const int c0 = (w0.tile / m_tiles) * G2_TILE_N + 128 * (int)rank, g = i / 3;
        if (i % 3 < 2) prefetch_l2(p.scales + (size_t)g * N + c0 + 64 * (i % 3));
        else prefetch_l2(p.qzeros + (size_t)g * (N >> 3) + (c0 >> 3));
      }
  }

  if (threadIdx.x == 0) {
    gm_mark_ns(p.trace, 100);
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 1 + 8); mbar_init(&empty[i], 1); }
    mbar_init(acc_full, 1); mbar_init(acc_empty, 8); mbar_init(last_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&amap);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, G2_TMEM_COLS); tmem_relinquish_pair(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) gm_mark_ns(p.trace, 101);

  // One block of 32 rows of a warp's 32 output columns: (+bias) -> fp16 -> shared memory, one half per row and lane.
  auto block_to_smem = [&](unsigned char* buf, const uint32_t (&v)[32], float bv) __attribute__((always_inline)) {
#pragma unroll
    for (int t = 0; t < 32; ++t)
      *reinterpret_cast<__half*>(buf + t * 64 + lane * 2) = __float2half_rn(__uint_as_float(v[t]) + bv);
  };
  // ... and from there to global memory: rows of 64 bytes, four lanes each, with the skip-path add
  auto block_to_global = [&](const unsigned char* buf, int m0, int n0) __attribute__((always_inline)) {
    const int rr = lane >> 2, cc = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = rr + 8 * i, m = m0 + r;
      uint4 o = *reinterpret_cast<const uint4*>(buf + r * 64 + cc * 16);
      if (m < p.M) {
        const size_t at = (size_t)m * N + n0 + 8 * cc;
        if (p.residual) {                                          // rounded first, as the separate add of the decoder layer would see it
          const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + at);      // (an earlier kernel's output: no read-only load)
          uint32_t* ov = reinterpret_cast<uint32_t*>(&o);
          const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 a = __half22float2(as_h2(ov[e])), b = __half22float2(as_h2(rw[e]));
            ov[e] = as_u32(__floats2half2_rn(a.x + b.x, a.y + b.y));
          }
        }
        *reinterpret_cast<uint4*>(p.out + at) = o;
      }
    }
  };
  // The pair's last item: nothing follows it, so the dequant warps (three per TMEM lane quarter) share its epilogue
  // with the epilogue warp of their quarter, blocks of 32 rows dealt round robin - the output of a whole tile, and the
  // writing or the adding up of the partial sums of a shared one.  (On short prompts, where every item is a piece of a
  // tile, one warp per quarter did the exchange block by block, a trip to L2 each: 128 rows of 4096 x 4096 took 23.2 us
  // and 18.9 shared, of 11008 x 4096 32.5 and 28.2; since the launch is programmatic 16.9 and 25.6.)
  // Not the items before: the dequant warps run ahead into the next one's stages instead (tall tiles, whose blocks may have
  // to be stored one by one, took 5 to 20 % longer with every epilogue shared).

  // A shared tile of this run: who contributes, its arrival counter (per CTA of the pair and lane quarter) and the
  // place of a contributor's sums: a warp's 32 columns x the tile's rows as [block][j][lane][4 floats] (512 contiguous bytes
  // per 16-byte access of the warp), indexed [contributing pair][CTA of the pair][lane quarter].
  struct Shared { bool shared, reducer; int c_first, c_last; unsigned* cnt; };
  auto shared_of = [&](const WorkItem& wi, int quarter) {
    Shared s = {SPLIT && wi.split, false, 0, 0, nullptr};
    if (s.shared) {
      const long long total = (long long)n_tiles * T;
      s.reducer = wi.kb == 0;
      s.c_first = stage_owner((long long)wi.tile * T, n_pairs, total);
      s.c_last = stage_owner((long long)wi.tile * T + T - 1, n_pairs, total);
      s.cnt = p.ws_counters + ((size_t)s.c_first * 2 + rank) * 4 + quarter;
    }
    return s;
  };
  auto part_of = [&](int cpair, int quarter) -> float* { return p.ws_partials + (((size_t)cpair * 2 + rank) * 4 + quarter) * (size_t)(TR * 32); };
  auto await_partials = [&](const Shared& s) {
    if (lane == 0) {
      const unsigned want = (unsigned)(s.c_last - s.c_first);
      bool ok = false;
      const uint32_t lim = *abort_flag ? 4u : 500000u;                    // x 200 ns
      for (uint32_t i = 0; i < lim && !ok; ++i) {
        unsigned have;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(s.cnt) : "memory");
        ok = have >= want;
        if (!ok) __nanosleep(200);
      }
      if (!ok) { *abort_flag = 1; atomicExch(&g_gemm_status, Q4_STATUS_WAIT_EXPIRED); }
    }
    __syncwarp();
    __threadfence();
  };
  // One block of the accumulator: to the workspace, or - with the other contributors' sums added - to shared memory.
  auto take_block = [&](const Shared& s, int quarter, int cb, uint32_t tsrc, unsigned char* buf, float bv) __attribute__((always_inline)) {
    uint32_t v[32];
    tmem_ld32(tsrc + cb * 32, v);
    tmem_ld_wait();
    if (s.shared && !s.reducer) {
      float* part = part_of(pair, quarter);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<uint4*>(part + ((cb * 8 + q) * 32 + lane) * 4) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      return;
    }
    if (s.reducer) {
      for (int c2 = s.c_first + 1; c2 <= s.c_last; ++c2) {
        const float* src = part_of(c2, quarter);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 a = __ldcg(reinterpret_cast<const float4*>(src + ((cb * 8 + q) * 32 + lane) * 4));
          v[4 * q] = __float_as_uint(__uint_as_float(v[4 * q]) + a.x); v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + a.y);
          v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + a.z); v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + a.w);
        }
      }
    }
    block_to_smem(buf, v, bv);
  };

  // The exchange inside a cluster (every pair has one item, a piece of the cluster's tile): a pair adds up the blocks of
  // 32 rows b % n == its own number and leaves its sums of the others in its shared memory, in the place of the activation
  // stages, which the last MMAs have read.  `w4` is the warp's number among the four of its lane quarter.
  const int n_cl = SPLIT ? p.cluster_pairs : 1;
  auto exchange_in_cluster = [&](int quarter, int w4) __attribute__((always_inline)) {
    const int me = (int)(cluster_rank >> 1);
    const WorkItem w_last = work_item<SPLIT>(p, wr, 0, n_pairs, T);
    const int n0 = (w_last.tile / m_tiles) * G2_TILE_N + 128 * (int)rank + 32 * quarter, m_base = (w_last.tile % m_tiles) * TR;
    const int nb = (min(TR, p.M - m_base) + 31) >> 5;
    const float bv = p.bias ? __half2float(p.bias[n0 + lane]) : 0.f;
    // [lane quarter][block that is not the pair's own][q][lane][4 floats]
    const int slots = (TR >> 5) - (TR >> 5) / n_cl;
    unsigned char* sums = smem + (size_t)quarter * slots * 4096 + lane * 16;
    const uint32_t tsrc = tmem_base + ((uint32_t)(32 * quarter) << 16);
    if (lane == 0) wait_bar_idle(last_full, 0, abort_flag, 40);
    __syncwarp();
    tc_fence_after();
#pragma unroll 1
    for (int cb = w4; cb < nb; cb += 4) {
      const int whose = cb % n_cl, slot = cb / n_cl * (n_cl - 1) + whose - (whose > me);
      if (whose == me) continue;
      uint32_t v[32];
      tmem_ld32(tsrc + cb * 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<uint4*>(sums + slot * 4096 + q * 512) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
    cluster_sync_all();
#pragma unroll 1
    for (int cb = me + n_cl * w4; cb < nb; cb += 4 * n_cl) {
      uint32_t v[32];
      tmem_ld32(tsrc + cb * 32, v);
      tmem_ld_wait();
#pragma unroll 1
      for (int c = 1; c < n_cl; ++c) {
        const int from = me + c < n_cl ? me + c : me + c - n_cl;
        const uint32_t src = mapa_u32(smem_u32(sums + (cb / n_cl * (n_cl - 1) + me - (me > from)) * 4096), 2 * from + rank);
        float4 t[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) t[q] = ld_cluster_f4(src + q * 512);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          v[4 * q] = __float_as_uint(__uint_as_float(v[4 * q]) + t[q].x); v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + t[q].y);
          v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + t[q].z); v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + t[q].w);
        }
      }
      unsigned char* mine = turn_of(quarter, cb);
      block_to_smem(mine, v, bv);
      __syncwarp();
      block_to_global(mine, m_base + cb * 32, n0);
      __syncwarp();
    }
  };

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's 128 rows of x (or of lora_u) of every stage ----------------
    if (lane == 0) {
      int st = 0, use = 0;
      const uint32_t full0 = mapa_u32(smem_u32(full), even_cta);
      pdl_wait();
      for (int item = 0; item < n_items; ++item) {
        const WorkItem wi = work_item<SPLIT>(p, wr, item, n_pairs, T);
        const int m0 = (wi.tile % m_tiles) * TR;
        const int at[2] = {m0 + (HR >> 1) * (int)rank, m0 + HR + ((TR - HR) >> 1) * (int)rank};
        const int nst = wi.ke - wi.kb + (wi.lora ? 1 : 0);
        for (int j = 0; j < nst; ++j) {
          const int it = wi.kb + j;
          if (use > 0) wait_bar_idle(&empty[st], (use - 1) & 1, abort_flag, 40);
          if (rank == 0) mbar_arrive_expect_tx(&full[st], nh * HR * GM_TILE_C * 2);
#pragma unroll
          for (int h = 0; h < nh; ++h) {
            unsigned char* dst = smem + (size_t)st * x_bytes + h * HR * GM_TILE_C;
            if (it < wi.ke) tma_load_2d_pair(dst, &amap, it * GM_TILE_C, at[h], full0 + 8 * st);
            else tma_load_2d_pair(dst, &umap, 0, at[h], full0 + 8 * st);
          }
          if (++st == S) { st = 0; ++use; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA only) ----------------
    // The whole warp walks the loop, so that stage counters, descriptors and TMEM addresses are warp-uniform values
    // (uniform registers, which the tensor-core instructions take their operands from); one elected lane issues.
    if (rank == 0) {
      uint32_t leader;
      asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(leader));
      const uint32_t idesc[2] = {idesc_f16(256, HR, false), idesc_f16(256, TR - HR, false)};
      const uint16_t both = (uint16_t)(3u << even_cta);
      // B: this CTA's 128 rows of x, K-major, 128-byte rows, 8-row groups 1024 B apart, 16 contraction elements = 32 B
      const uint64_t bd0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
      constexpr uint64_t B_STEP = 32 >> 4;
      const uint64_t ST_STEP = (uint64_t)(x_bytes >> 4), H_STEP = (uint64_t)((HR * GM_TILE_C) >> 4);
      const uint32_t a0_tmem = tmem_base + G2_TMEM_COLS - 32 * S;
      int st = 0, use = 0;
      uint64_t bd = bd0;
      for (int item = 0; item < n_items; ++item) {
        const WorkItem wi = work_item<SPLIT>(p, wr, item, n_pairs, T);
        const int ncon = wi.ke - wi.kb, nst = ncon + (wi.lora ? 1 : 0);
        if (item > 0) wait_bar_cluster(acc_empty, (item - 1) & 1, abort_flag);
        tc_fence_after();
        for (int it = 0; it < nst; ++it) {
          wait_bar_cluster(&full[st], use & 1, abort_flag);
          if (p.trace && lane == 0 && item == 0 && (it & 7) == 0 && it < 64) gm_mark_ns(p.trace, 110 + (it >> 3));
          tc_fence_after();
          const uint32_t a_tmem = a0_tmem + 32 * st;
          const int nks = it < ncon ? 4 : lora_ks;
          if (leader) {
            for (int ks = 0; ks < nks; ++ks)
#pragma unroll
              for (int h = 0; h < nh; ++h)
                umma_f16_pair_ts(tmem_base + h * HR, a_tmem + 8 * ks, bd + ks * B_STEP + h * H_STEP, idesc[h], (it > 0 || ks > 0) ? 1u : 0u);
            umma_commit_pair(&empty[st], both);
          }
          __syncwarp();
          bd += ST_STEP;
          if (++st == S) { st = 0; ++use; bd = bd0; }
        }
        if (leader) { umma_commit_pair(acc_full, both); if (item == n_items - 1) umma_commit_pair(last_full, both); }
        __syncwarp();
        if (lane == 0 && item == 0) gm_mark_ns(p.trace, 102);
        if (lane == 0 && item == n_items - 1) gm_mark_ns(p.trace, 103);
      }
    }
  } else if (warp >= 4 && warp < 4 + 4 * G3_GROUPS) {
    // ---------------- dequantisers: one output column per thread, 64 contraction elements per task ----------------
    const int grp = (warp - 4) >> 2;                               // takes the stage uses u with u % G3_GROUPS == grp
    const int quarter = warp & 3;
    const uint32_t full0 = mapa_u32(smem_u32(full), even_cta);
    const uint32_t tdst0 = tmem_base + ((uint32_t)(32 * quarter) << 16) + G2_TMEM_COLS - 32 * S;
    int gbase = 0;                                                 // stage uses of all earlier tiles
    int next_st = grp, next_use = 0;                               // of this group's next stage use (PLAIN: u & 7, u >> 3)
    int tab_n0 = -1;
    uint32_t* offs = reinterpret_cast<uint32_t*>(offs_all) + 64 * (warp - 4);
    const unsigned char* tabl = tab + 4 * (32 * quarter + lane);
    TaskRegs R0, R1;
    pdl_wait();                                                    // scales, zero terms, adapters, bias, workspace
    for (int item = 0; item < n_items; ++item) {
      const WorkItem wi = work_item<SPLIT>(p, wr, item, n_pairs, T);
      const int n = column_of(wi.tile);
      const int ncon = wi.ke - wi.kb, nst = ncon + (wi.lora ? 1 : 0);       // stages of this item: j = 0 .. nst-1, contraction stage kb + j
      auto task = [&](int j, const TaskRegs& C) __attribute__((always_inline)) {
        const int st = PLAIN ? (gbase + j) & (G3_MAX_STAGES - 1) : next_st, use = PLAIN ? (gbase + j) / G3_MAX_STAGES : next_use;
        uint32_t o[32];
        if (j == ncon) {
          // low-rank stage: lane = column n holds lora_B[n][0..r), zero beyond
          const __half* src = p.lora_w + (size_t)n * p.lora_r;
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const __half lo = 2 * c < p.lora_r ? src[2 * c] : __float2half(0.f);
            const __half hi = 2 * c + 1 < p.lora_r ? src[2 * c + 1] : __float2half(0.f);
            o[c] = as_u32(__halves2half2(lo, hi));
          }
        } else if (ACT) {
          offs[lane] = min(C.s, (uint32_t)(p.G - 1)) * 512;
          offs[lane + 32] = min(C.z, (uint32_t)(p.G - 1)) * 512;
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 oa = *reinterpret_cast<const uint4*>(offs + 8 * i), ob = *reinterpret_cast<const uint4*>(offs + 8 * i + 4);
            const uint32_t at[8] = {oa.x, oa.y, oa.z, oa.w, ob.x, ob.y, ob.z, ob.w};
            uint32_t e[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) e[k] = *reinterpret_cast<const uint32_t*>(tabl + at[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t v = and_or(prmt(C.w[i], C.w[i], k | (k << 8)), 0x00F0000Fu, 0x54006400u);
              const uint32_t s2 = prmt(e[2 * k], e[2 * k + 1], 0x5410), z2 = prmt(e[2 * k], e[2 * k + 1], 0x7632);
              o[4 * i + k] = as_u32(__hsub2_rn(__hmul2_rn(as_h2(s2), __hsub2(as_h2(v), as_h2(0x54006400u))), as_h2(z2)));
            }
          }
        } else {
          const uint32_t s2 = prmt(C.s, C.s, 0x1010), z2 = prmt(C.z, C.z, 0x1010);
          if ((C.s & 0x4000u) == 0) {                    // |s| < 2: 1024 s is exact
            const uint32_t c2 = as_u32(__hmul2_rn(as_h2(s2), as_h2(0xD400E400u) /* (-1024, -64) */));
#pragma unroll
            for (int i = 0; i < 8; ++i) deq_word_k<true>(C.w[i], s2, c2, z2, o + 4 * i);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) deq_word_k<false>(C.w[i], s2, 0u, z2, o + 4 * i);
          }
        }
        if (use > 0 && lane == 0) wait_bar_idle(&empty[st], (use - 1) & 1, abort_flag, 40);
        __syncwarp();
        tc_fence_after();
        tmem_st32(tdst0 + 32 * st, o);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(full0 + 8 * st);
        if (!PLAIN) {
          next_st += G3_GROUPS;
          if (next_st >= S) { next_st -= S; ++next_use; }
        }
      };
      int j = (grp + G3_GROUPS - gbase % G3_GROUPS) % G3_GROUPS;   // this group's first stage of the tile
      auto ask = [&](int jj, TaskRegs& R) __attribute__((always_inline)) { if (jj < ncon) prefetch(n, wi.kb + jj, R); };
      ask(j, R0);
      const int c0 = (wi.tile / m_tiles) * G2_TILE_N + 128 * (int)rank;
      if (ACT && c0 != tab_n0) {
        if (tab_n0 >= 0) named_bar_sync_warps(5, 128 * G3_GROUPS);       // the readers of the table before are done
#pragma unroll 1
        for (int i0 = threadIdx.x - 128; i0 < p.G * 16; i0 += 4 * 128 * G3_GROUPS) {
          uint4 sv[4];
          uint32_t zw[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) {                            // (nothing else covers their trips to L2: all four at once)
            const int i = i0 + b * 128 * G3_GROUPS, g = i >> 4, c8 = i & 15;
            if (i >= p.G * 16) break;
            sv[b] = ld_pinned_u4(p.scales + (size_t)g * N + c0 + 8 * c8);
            zw[b] = ld_pinned_u32(p.qzeros + (size_t)g * (N >> 3) + (c0 >> 3) + c8);
          }
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int i = i0 + b * 128 * G3_GROUPS;
            if (i >= p.G * 16) break;
            const uint4 s8 = sv[b], z8 = zero_terms(s8, zw[b]);
            uint4* to = reinterpret_cast<uint4*>(tab + 32 * i);
            to[0] = make_uint4(prmt(s8.x, z8.x, 0x5410), prmt(s8.x, z8.x, 0x7632), prmt(s8.y, z8.y, 0x5410), prmt(s8.y, z8.y, 0x7632));
            to[1] = make_uint4(prmt(s8.z, z8.z, 0x5410), prmt(s8.z, z8.z, 0x7632), prmt(s8.w, z8.w, 0x5410), prmt(s8.w, z8.w, 0x7632));
          }
        }
        named_bar_sync_warps(5, 128 * G3_GROUPS);
        tab_n0 = c0;
      }
      while (j < nst) {
        ask(j + G3_GROUPS, R1);
        task(j, R0);
        j += G3_GROUPS;
        if (j >= nst) break;
        ask(j + G3_GROUPS, R0);
        task(j, R1);
        j += G3_GROUPS;
      }
      gbase += nst;
    }
    if (n_cl == 1 && n_items > 0) {                      // the last item's epilogue, with the epilogue warp of the quarter
      const WorkItem w_last = work_item<SPLIT>(p, wr, n_items - 1, n_pairs, T);
      const int n0 = (w_last.tile / m_tiles) * G2_TILE_N + 128 * (int)rank + 32 * quarter;
      const int m_base = (w_last.tile % m_tiles) * TR;
      const int nb = (min(TR, p.M - m_base) + 31) >> 5;
      const float bv = p.bias ? __half2float(p.bias[n0 + lane]) : 0.f;
      // the quarter's shared-memory rows are free once its epilogue warp has stored the item before (a meeting of
      // the quarter's four warps: named barrier 1 + quarter)
      named_bar_sync_warps(1 + quarter, 128);
      if (lane == 0) wait_bar_idle(last_full, 0, abort_flag, 100);
      __syncwarp();
      tc_fence_after();
      const Shared sh = shared_of(w_last, quarter);
      if (sh.reducer) {
        await_partials(sh);
        named_bar_sync_warps(1 + quarter, 128);                        // all four warps have seen the count: the epilogue warp may clear it
      }
#pragma unroll 1
      for (int cb = grp; cb < nb; cb += G3_GROUPS + 1) {
        unsigned char* mine = turn_of(quarter, cb);
        take_block(sh, quarter, cb, tmem_base + ((uint32_t)(32 * quarter) << 16), mine, bv);
        __syncwarp();
        if (!sh.shared || sh.reducer) block_to_global(mine, m_base + cb * 32, n0);
        __syncwarp();
      }
      if (sh.shared && !sh.reducer) {
        __threadfence();
        named_bar_sync_warps(1 + quarter, 128);                        // this warp's sums are out: the epilogue warp counts for all four
      }
    }
  } else if (warp >= 4 + 4 * G3_GROUPS) {
    // ---------------- epilogue: TMEM -> registers -> (+bias) -> fp16 -> turned over in shared memory -> (+residual) -> global ----------------
    const int quarter = warp & 3;
    const uint32_t acc_empty0 = mapa_u32(smem_u32(acc_empty), even_cta);
    pdl_wait();
    for (int item = 0; item < (n_cl > 1 ? 0 : n_items); ++item) {
      const WorkItem wi = work_item<SPLIT>(p, wr, item, n_pairs, T);
      const int n0 = (wi.tile / m_tiles) * G2_TILE_N + 128 * (int)rank + 32 * quarter;     // this warp's 32 output columns
      const int m_base = (wi.tile % m_tiles) * TR;
      const int rows = min(TR, p.M - m_base);                     // rows of x the tile really has
      const float bv = p.bias ? __half2float(p.bias[n0 + lane]) : 0.f;
      if (item == n_items - 1) named_bar_sync_warps(1 + quarter, 128);   // the helpers may use this quarter's rows from here
      if (lane == 0) wait_bar_idle(acc_full, item & 1, abort_flag, 100);
      __syncwarp();
      tc_fence_after();
      if (lane == 0 && item == n_items - 1) gm_mark_ns(p.trace, 105);
      const uint32_t tsrc = tmem_base + ((uint32_t)(32 * quarter) << 16);
      const int nb = (rows + 31) >> 5;                             // blocks of 32 rows that hold anything
      const bool shared_out = item == n_items - 1;                 // the dequant warps take the blocks cb % 4 = 0, 1, 2
      const int cb0 = shared_out ? G3_GROUPS : 0, cbs = shared_out ? G3_GROUPS + 1 : 1;
      const Shared sh = shared_of(wi, quarter);
      if (sh.reducer) {
        await_partials(sh);
        if (shared_out) named_bar_sync_warps(1 + quarter, 128);
      }
#pragma unroll 1
      for (int cb = cb0; cb < nb; cb += cbs) {
        unsigned char* mine = turn_of(quarter, cb);
        take_block(sh, quarter, cb, tsrc, mine, bv);
        if (PLAIN || p.turn_blocks || (sh.shared && !sh.reducer)) continue;
        __syncwarp();
        block_to_global(mine, m_base + cb * 32, n0);
        __syncwarp();
      }
      // this warp has read its part of the accumulator: the even CTA may start the next item
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty0);
      if (!sh.shared || sh.reducer) {
        if (PLAIN || p.turn_blocks)
#pragma unroll 1
          for (int cb = cb0; cb < nb; cb += cbs) block_to_global(turn_of(quarter, cb), m_base + cb * 32, n0);
        __syncwarp();                                      // the rows are read before the next item overwrites them
      } else {                                             // publish: sums, then the count
        __threadfence();
        __syncwarp();
        if (shared_out) named_bar_sync_warps(1 + quarter, 128);
        if (lane == 0) atomicAdd(sh.cnt, 1u);
      }
      if (sh.reducer && lane == 0) *sh.cnt = 0;            // every contributor has been counted: ready for the next launch
    }
  }
  if (n_cl > 1) {
    if (warp >= 4) exchange_in_cluster(warp & 3, (warp - 4) >> 2);
    else cluster_sync_all();                           // the meeting of the exchange
  }
  if (threadIdx.x == G3_THREADS - 128) gm_mark_ns(p.trace, 106);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (threadIdx.x == 0) gm_mark_ns(p.trace, 107);
  if (warp == 1) tmem_dealloc_pair(tmem_base, G2_TMEM_COLS);
}

// How a launch lays its shared memory out: the stages that TMEM leaves room for beside a tile's accumulator, fewer (no less
// than four) where the act-order table of G groups needs the room; a place to turn over for every block of a tile where
// that fits.  bytes = 0: no room.
struct Gemm3Layout { int stages, area, turn_blocks; size_t bytes; };
static Gemm3Layout gemm3_layout(int tile_rows, int G, bool act, int cluster) {
  Gemm3Layout l = {0, 0, 0, 0};
  if (!act && tile_rows <= 256) {
    l.stages = G3_MAX_STAGES; l.area = G3_PLAIN_AREA; l.turn_blocks = 8;
    l.bytes = 1024 + (size_t)G3_PLAIN_AREA + G3_BAR_BYTES + 4 * 8 * G3_TURN_BLOCK;
    return l;
  }
  const int nb = tile_rows / 32, x_bytes = (tile_rows > 256 ? 2 * gemm3_first_rows(tile_rows) : tile_rows) * GM_TILE_C, table = act ? G * 512 : 0, limit = 227 * 1024;
  const int sums = cluster > 1 ? 4 * (nb - nb / cluster) * 4096 : 0;
  for (int s = (G2_TMEM_COLS - tile_rows) / 32 < G3_MAX_STAGES ? (G2_TMEM_COLS - tile_rows) / 32 : G3_MAX_STAGES; s >= 4; --s) {
    const int used = s * x_bytes + table > sums ? s * x_bytes + table : sums;
    l.stages = s;
    l.area = (used + 1023) & ~1023;
    const int rest = 1024 + G3_BAR_BYTES + (act ? G3_OFFS_BYTES : 0);
    for (int full = 1; full >= 0; --full) {
      l.turn_blocks = full ? nb : 0;
      l.bytes = (size_t)rest + l.area + (size_t)(full ? 4 * nb : 4 * G3_GROUPS + 4) * G3_TURN_BLOCK;
      if (l.bytes <= (size_t)limit) return l;
    }
  }
  l.bytes = 0;
  return l;
}

// How many pairs the device's SMs make, and how many clusters of 1 .. G3_MAX_CLUSTER pairs of this kernel it holds at once.
struct GemmResident { int sm_pairs, clusters[G3_MAX_CLUSTER + 1]; };

// Asked once per device, for the most shared memory there is (which the kernel's forms are allowed here).
static int gemm3_resident(int dev, GemmResident* r) {
  static std::atomic<int> known[64][G3_MAX_CLUSTER + 1];           // the answer and one
  if (!known[dev][G3_MAX_CLUSTER].load(std::memory_order_acquire)) {
    for (const void* f3 : {(const void*)q4_gemm3_kernel<false, false, false>, (const void*)q4_gemm3_kernel<true, false, false>,
                           (const void*)q4_gemm3_kernel<false, true, false>, (const void*)q4_gemm3_kernel<true, true, false>,
                           (const void*)q4_gemm3_kernel<false, false, true>, (const void*)q4_gemm3_kernel<true, false, true>,
                           (const void*)q4_gemm3_kernel<false, true, true>, (const void*)q4_gemm3_kernel<true, true, true>})
      if (int e = check_cuda(cudaFuncSetAttribute(f3, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024), "gemm smem attribute")) return e;
    for (int n = 1; n <= G3_MAX_CLUSTER; ++n) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * n * 64); cfg.blockDim = dim3(G3_THREADS); cfg.dynamicSmemBytes = 227 * 1024;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2 * n; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
      cfg.attrs = at; cfg.numAttrs = 1;
      int nc = 0;
      if (cudaOccupancyMaxActiveClusters(&nc, (const void*)q4_gemm3_kernel<true, false, false>, &cfg) != cudaSuccess || nc < 0) { cudaGetLastError(); nc = 0; }
      known[dev][n].store(nc + 1, std::memory_order_release);
    }
  }
  for (int n = 1; n <= G3_MAX_CLUSTER; ++n) r->clusters[n] = known[dev][n].load(std::memory_order_acquire) - 1;
  return Q4_OK;
}

}  // namespace q4
