// Grouped GEMM with the weights on the accumulator's lanes: D[weight row, token] = W_e[N, K] . X_e[rows, K]^T, with FP8
// weights (W8A16) and with bf16 weights.  What follows is about the FP8 form; the bf16 form has no converters, takes both
// operands from shared memory and uses all 512 columns of tensor memory for accumulators.
//
// A cluster of two CTAs (one SM pair, tcgen05 cta_group::2, M = 256) computes 256 weight rows against up to
// 384 tokens of one expert.  Compared with tokens on the lanes (gemm.cu):
//   * the token side is the MMA's N, a multiple of 32 chosen per job, so an expert with few rows costs what it
//     has and an expert with 130 rows is one job, not two 128-row tiles;
//   * an FP8 weight is converted once per 384 tokens, by the SM whose lane holds it, and the bf16 operand goes
//     straight into tensor memory (tcgen05.st; the A operand of the MMA is read from there).  Shared memory
//     carries the FP8 bytes and the tokens only: per 64-element K step and SM 8 KiB + 8 KiB FP8 in and out and
//     N/2 * 128 B of tokens in and out, where a bf16 tile built in shared memory adds 16-32 KiB each way.
//
// What bounds it.  Decode: the weights' bytes and the conversion, which share the step.  DeepSeek-V3 shape, 64 tokens,
// gate/up + down products: 2.30 ms before and 1.80 ms with the changes below, 5.6 TB/s of the measured 6.5 (without
// the conversion 1.49 ms, the HBM rate).  From a few thousand tokens on: the 1000 W cap (SM clock 1.1-1.3 GHz), where
// every weight byte moved and converted once more costs time: 16384 tokens 11.4 and 10.5 ms (10.0 by the counter).  Jobs of at
// most 320, 256 and 192 tokens were 1, 9 and 14 % slower there; prefetching tokens or weights into L2 ahead of the rings 2 to
// 15 %.
//   * two products by one packed multiplication (convert16): the converters are bound by issue slots, 2.8 instructions
//     per element of which 2.5 are conversions and the product: 64 tokens 2.30 and 2.10 ms;
//   * 128 K elements per hand-over: half as many waits, votes and commits per element, on both sides;
//   * the list of jobs is made by one warp, ahead: a look-up by every role between two jobs stopped the pipeline for
//     two thousand cycles, 13 % of a job of the down product (these two: 2.10 and 1.80 ms);
//   * the epilogue reads the accumulator in the layout of 8x8 fragments, so that SwiGLU's two halves meet in one thread
//     and stmatrix transposes: half the instructions and no shuffles (16384 tokens, down product 4.05 and 3.85 ms);
//   * one copy per token stage, through a map that sees the rows as [K / 64][rows][64], instead of one per step and per 64
//     or 16 tokens (4096 skewed tokens 4.89 and 4.77 ms);
//   * jobs alternate between the two ends of the accumulator columns and the next one starts as soon as the columns that
//     both need have been read (3.85 and 3.80 ms; the clock falls as the tensor cores idle less).
//   * jobs are handed out by a counter (next_job, where the caller has memory for one), not in fixed turns: pairs that
//     start late or get long jobs take fewer, and the jobs under way stay neighbours in the list, whose weights and tokens
//     L2 then holds: V3 layer 16384 tokens 13.1 and 11.9 ms, 65536 tokens 51 and 44, 4096 skewed 4.94 and 4.79; both
//     products alone, V2-236B 11000 tokens 3.97 and 3.31.
// Direct stores of the output from registers were slower than pieces staged for TMA (down product, 16384 tokens 4.5
// against 4.0 ms).
//
// Roles per CTA: warp 0 = weight TMA, warp 1 = token TMA, warp 2 = MMA issuer (leader CTA), warp 3 = job list and
// TMEM owner, warps 4-11 = epilogue (two per lane quarter, alternate 32-token chunks), warps 12-27 = converters: a
// thread owns one lane = one weight row and 64 K elements of a stage; warps 12-19 take the even stages of 128 K elements,
// 20-27 the odd ones.  Eight warps with all 128 elements each had less to issue while one of two per scheduler waits: V3, us,
// 64 tokens 2116 and 2107, 1024 tokens 2873 and 2844, 333 skewed 1608 and 1595; level from 4096 tokens on.
//
// Barriers (per CTA unless said otherwise):
//   wfull/wempty   weight ring, stages of 128 rows x 128 K bytes, released by the eight converter warps that read it
//   tfull/tempty   token ring; leader's tfull counts both CTAs' bytes, tempty by commit to both
//   aready/afree   the two 64-column slots of converted weights in TMEM, one per converter group; aready on the leader
//                  counts the eight warps of both CTAs, afree by commit to both
//   dfull/dempty   accumulators of even and odd jobs, dempty once an epilogue has read all of one
//   dpart          an epilogue has read the columns that the next job's accumulator shares with its own
//   jfull/jempty   the next job, for the roles of a CTA; mfull: its number, from the leader's list to the other CTA's
// Every wait is bounded (mbar_wait); on expiry the roles leave their loops and the kernel ends.  The lanes of a
// warp-wide role leave by the vote on a wait only, all at once: a lane that read the abort flag on its own would wait
// at the closing barrier for lanes that wait for it in a warp-wide instruction, without a limit.  A role that gives
// up has waited for the limit while the others could run ahead by a ring's length at most, so the loads still in
// flight then were issued about as long ago and have landed.
#include "tc.cuh"

namespace mg {

namespace {

constexpr int WL_GROUP_T = 8;                  // token tiles per L2 reuse group (weight tiles vary slower inside)
constexpr int WL_K = 64;                       // K elements per MMA step (one 128-byte swizzle row of bf16)
constexpr int WL_W_STAGE = 128 * 128;          // 16 KiB: 128 rows of 64 bf16 or of 128 FP8
constexpr int WL_A_SLOTS = 2;                  // FP8: converted weights, one slot per converter group of eight warps
constexpr int WL_A_COLS = 64;                  // 128 bf16 per lane
constexpr int WL_EPI_WARPS = 8, WL_CONV_WARPS = 16;
constexpr int WL_PIECE = 1024;                 // epilogue staging: 32 tokens x 16 outputs or 16 tokens x 32 outputs
constexpr int WL_JOBS = 1;                     // announced ahead: few, so that the last jobs go to whoever is free
constexpr int WL_AHEAD = 8;                     // weight stages brought into L2 while the kernel before still runs
constexpr int WL_MAIL = 4;                     // job numbers on their way from the leader to the other CTA
template <bool FP8>
struct WlCfg {
  static constexpr int MAX_TOKENS = 384;                       // per job
  // Weight and token stages.  bf16, ms at 8 and 3, 6 and 4, 5 and 5 stages: V2-236B 512 tokens 1.265, 1.302, 1.31, 2048
  // tokens 1.55, 1.59, 1.63, 32768 tokens 11.3, -, 11.9; Mixtral 2048 tokens 1.54, 1.52, 1.53.  With jobs of at most 256
  // tokens (8 and 4) V2-236B 8192 tokens 4.2 against 3.3.
  static constexpr int SW = FP8 ? 6 : 8, ST = FP8 ? 4 : 3;
  static constexpr int T_STAGE = MAX_TOKENS / 2 * WL_K * 2;    // this CTA's half of the tokens
  static constexpr int THREADS = (4 + WL_EPI_WARPS + (FP8 ? WL_CONV_WARPS : 0)) * 32;
  static constexpr int ACC_COLS = FP8 ? MAX_TOKENS : 512;      // accumulator columns; FP8: converted weights above them
  static constexpr int RING_BYTES = SW * WL_W_STAGE + ST * T_STAGE;
  static constexpr int BARS = 5 + 2 * WL_JOBS + 2 * (SW + ST + WL_A_SLOTS) + WL_MAIL;
  static constexpr size_t SMEM = 1024 + RING_BYTES + WL_EPI_WARPS * 2 * WL_PIECE + 8 * BARS + 32 + 32 * WL_JOBS + 4 * WL_MAIL +
                                 4 * (3 * kMaxExperts + 3);
  static_assert(SMEM <= 232448, "shared memory exceeds the 227 KiB a CTA may have");
};
static_assert(WlCfg<true>::SW % 2 == 0, "the two converter groups take alternate stages of the weight ring");

struct WlArgs {
  const int32_t* pad_offsets;
  const int32_t* counts;
  int n_groups;
  int n_tiles;                  // 256-row weight tiles per group
  int n_per_group;
  int k_steps;                  // K / 64
  const float* scales;          // [rows / 128][K / 128]
  int scale_cols;
  int32_t* next_job;            // counts the jobs handed out beyond each pair's first; nullptr: every n_pairs-th job
  int32_t* status;
  int rows;                     // of the token matrix: the first row number behind it
  int chained;                  // launched while the kernel before may still run (launch_chained)
};

struct Ring {
  uint32_t i = 0, ph = 0;
  __device__ __forceinline__ void next(uint32_t n) {
    if (++i == n) { i = 0; ph ^= 1u; }
  }
};

struct alignas(16) Job {
  int row0;      // first token row
  int left;      // live tokens
  int n_tok;     // left rounded up to 32: the MMA's N; 0: no further job
  int b_row;     // first of the 256 weight rows
  int n_idx;
  int pad[3];
};

// K steps that share a token stage, for h tokens per CTA: a job of few tokens packs several, so that the ring holds as
// many bytes in flight as a job of many
template <bool FP8>
__host__ __device__ constexpr int steps_per_stage(int h) {
  const int fit = WlCfg<FP8>::T_STAGE / (h * WL_K * 2);
  return fit >= 8 ? 8 : fit >= 4 ? 4 : fit >= 2 ? 2 : 1;
}

// Tokens of a job's first MMA per K step; the second takes the rest.  256, but 160 where 32 or 64 would be left: an MMA of few
// tokens with A in shared memory is bound by reading A (M256 K16, cycles at N = 32, 64, 96, 128: 39, 43, 50, 64, where the
// flop rate is N / 2), so that 256 + 32 tokens took 167 cycles, where 160 + 128 take 144.  V2-236B (320 tokens per job), layer,
// ms, 256 + rest and this: 32768 tokens 11.51 and 11.36, 8192 tokens 3.35 and 3.31.
// FP8 weights come from tensor memory, where an MMA takes N / 2 at any width.
template <bool FP8>
__device__ __forceinline__ int first_part(int n_tok) { return n_tok <= 256 ? n_tok : FP8 || n_tok >= 352 ? 256 : 160; }

// s_jp[e] = token tiles of the experts before e
__device__ __forceinline__ Job locate_job(int job, const int* s_pad, const int* s_cnt, const int* s_jp, const WlArgs& g) {
  int lo = 0, hi = g.n_groups;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_jp[mid] * g.n_tiles <= job) lo = mid; else hi = mid;
  }
  const int e = lo;
  const int local = job - s_jp[e] * g.n_tiles;
  const int nt = s_jp[e + 1] - s_jp[e];
  const int per_group = WL_GROUP_T * g.n_tiles;
  const int grp = local / per_group;
  const int rem = local - grp * per_group;
  const int gt = min(WL_GROUP_T, nt - grp * WL_GROUP_T);
  const int n = rem / gt;
  const int m = grp * WL_GROUP_T + (rem - n * gt);
  const int units = (s_cnt[e] + 31) >> 5;                  // 32 tokens each, dealt out evenly over the expert's tiles
  const int base = units / nt, more = units - base * nt;
  const int first = (m * base + min(m, more)) * 32;
  Job j;
  j.row0 = s_pad[e] + first;
  j.n_tok = (base + (m < more ? 1 : 0)) * 32;
  j.left = min(j.n_tok, s_cnt[e] - first);
  j.b_row = e * g.n_per_group + n * 256;
  j.n_idx = n;
  return j;
}

// D += A(tensor memory) * B(shared memory) on the SM pair
__device__ __forceinline__ void tc_mma_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
      "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
      "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 FP8 values -> 16 words of bf16 pairs, kept where they stand: without the empty statement the compiler moves the
// conversion below the next wait
__device__ __forceinline__ void convert32(const uint4& q0, const uint4& q1, float s, uint32_t* o) {
  uint4 w[4];
  convert16(q0, s, w[0], w[1]);
  convert16(q1, s, w[2], w[3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    asm volatile("" : "+r"(w[i].x), "+r"(w[i].y), "+r"(w[i].z), "+r"(w[i].w));
    o[4 * i] = w[i].x; o[4 * i + 1] = w[i].y; o[4 * i + 2] = w[i].z; o[4 * i + 3] = w[i].w;
  }
}

// Arrival on the leader CTA's barrier with the default semantics (release at CTA scope).  What it announces is tensor
// memory, ordered by tcgen05 fences; at cluster scope the release would first wait until every global store of
// the warp has reached L2, microseconds per tile in the epilogue.
__device__ __forceinline__ void arrive_at_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(smem_u32(bar), 0)) : "memory");
}

// 16 lanes (weight rows) x 32 columns (tokens) of the accumulator in the layout of 8x8 fragments: registers 4x, 4x + 1
// hold row lane / 4, tokens 8x + 2 (lane mod 4) and the next; 4x + 2, 4x + 3 the same of row lane / 4 + 8.
__device__ __forceinline__ void tc_ld_16x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// four 8x8 fragments, transposed: fragment m's column i goes to the 16 bytes that lane 8m + i points at
__device__ __forceinline__ void store_fragments(uint32_t addr, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(m0), "r"(m1),
               "r"(m2), "r"(m3)
               : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// a value that another kernel may be writing: some value, for a guess only
__device__ __forceinline__ int peek(const int32_t* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <int EPI, bool FP8>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WlCfg<FP8>::THREADS, 1)
grouped_gemm_wl_kernel(const __grid_constant__ WlMaps maps, const WlArgs g) {
  using C = WlCfg<FP8>;
  constexpr bool SWIGLU = EPI == EPI_SWIGLU_BF16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* pieces = smem + C::RING_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(pieces + WL_EPI_WARPS * 2 * WL_PIECE);
  uint64_t* dfull = bars;
  uint64_t* dempty = dfull + 2;
  uint64_t* dpart = dempty + 2;
  uint64_t* jfull = dpart + 1;
  uint64_t* jempty = jfull + WL_JOBS;
  uint64_t* wfull = jempty + WL_JOBS;
  uint64_t* wempty = wfull + C::SW;
  uint64_t* tfull = wempty + C::SW;
  uint64_t* tempty = tfull + C::ST;
  uint64_t* aready = tempty + C::ST;                 // FP8
  uint64_t* afree = aready + WL_A_SLOTS;
  uint64_t* mfull = afree + WL_A_SLOTS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  Job* s_job = reinterpret_cast<Job*>((reinterpret_cast<uintptr_t>(tmem_slot + 2) + 15) & ~uintptr_t(15));
  int* s_mail = reinterpret_cast<int*>(s_job + WL_JOBS);
  int* s_pad = s_mail + WL_MAIL;
  int* s_cnt = s_pad + kMaxExperts + 1;
  int* s_jp = s_cnt + kMaxExperts + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();           // 0 = leader
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::SW; ++s) { mbar_init(smem_u32(&wfull[s]), 1); mbar_init(smem_u32(&wempty[s]), FP8 ? WL_CONV_WARPS / 2 : 1); }
    for (int s = 0; s < C::ST; ++s) { mbar_init(smem_u32(&tfull[s]), 1); mbar_init(smem_u32(&tempty[s]), 1); }
    if (FP8)
      for (int s = 0; s < WL_A_SLOTS; ++s) { mbar_init(smem_u32(&aready[s]), WL_CONV_WARPS); mbar_init(smem_u32(&afree[s]), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&dfull[s]), 1); mbar_init(smem_u32(&dempty[s]), 2 * WL_EPI_WARPS); }
    mbar_init(smem_u32(dpart), 2 * WL_EPI_WARPS);
    for (int s = 0; s < WL_JOBS; ++s) {
      mbar_init(smem_u32(&jfull[s]), 1);
      mbar_init(smem_u32(&jempty[s]), 2 + (rank == 0 ? 1 : 0) + WL_EPI_WARPS + (FP8 ? WL_CONV_WARPS : 0));
    }
    for (int s = 0; s < WL_MAIL; ++s) mbar_init(smem_u32(&mfull[s]), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // token tiles before each expert: lane sums of runs of 16 experts, warp scan, runs written out
  auto count_tiles = [&]() {
    constexpr int RUN = kMaxExperts / 32;
    int sum = 0;
    for (int i = 0; i < RUN; ++i) {
      const int e = lane * RUN + i;
      if (e < g.n_groups) sum += (s_cnt[e] + C::MAX_TOKENS - 1) / C::MAX_TOKENS;
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= o) inc += v;
    }
    int run = inc - sum;
    for (int i = 0; i < RUN; ++i) {
      const int e = lane * RUN + i;
      if (e < g.n_groups) {
        s_jp[e] = run;
        run += (s_cnt[e] + C::MAX_TOKENS - 1) / C::MAX_TOKENS;
        if (e == g.n_groups - 1) s_jp[g.n_groups] = run;
      }
    }
  };
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // barriers of both CTAs initialised, TMEM allocated on both SMs
  tc_fence_after();
  // Until the wait, nothing that an earlier kernel of the forward wrote is known to be visible.  The counts seen just before it
  // (last of all here: the plan may still be storing them when this kernel begins) say which weights this pair will most likely
  // read first, and these are brought into L2 meanwhile; whatever the counts hold, the job they give is one of the layer's.
  // Layer, us, routing changing from call to call, without this, with 4, 8 and 16 stages: V2-Lite 8 tokens 137.7, 136.5, 136.5
  // and 137.0, 512 tokens 257, 237, 237 and 239; Mixtral 61 tokens 469, 465, 465 and 465; V2-236B 512 tokens 1241, 1228, 1225
  // and 1228; V3, where converting bounds it, 8 tokens 591, 595, 595 and 596, 64 tokens 2124, 2143, 2149 and 2143.
  if (g.chained) {
    for (int i = threadIdx.x; i < g.n_groups; i += blockDim.x) s_cnt[i] = min(max(peek(g.counts + i), 0), 1 << 16);
    __syncthreads();
    if (warp == 3) count_tiles();
    __syncthreads();
  }
  if (g.chained && warp == 0 && pair < s_jp[g.n_groups] * g.n_tiles && elect_one()) {
    const int blk = locate_job(pair, s_cnt, s_cnt, s_jp, g).b_row >> 7, r0 = static_cast<int>(rank);
    const int steps = min(g.k_steps / (FP8 ? 2 : 1), WL_AHEAD);
    for (int kb = 0; kb < steps; ++kb) {
      if (FP8) tma_prefetch_3d(&maps.w, kb * 128, SWIGLU ? r0 * 64 : 0, SWIGLU ? blk : blk + r0);
      else tma_prefetch_4d(&maps.w, kb * WL_K, 0, SWIGLU ? blk : blk + r0, SWIGLU ? r0 * 4 : 0);
    }
  }
  chain_wait();
  chain_go();
  bool same = g.chained;
  for (int i = threadIdx.x; i < g.n_groups; i += blockDim.x) {
    s_pad[i] = g.pad_offsets[i];
    same = same && g.counts[i] == s_cnt[i];
  }
  if (!__syncthreads_and(same)) {
    for (int i = threadIdx.x; i < g.n_groups; i += blockDim.x) s_cnt[i] = g.counts[i];
    __syncthreads();
    if (warp == 3) count_tiles();
    __syncthreads();
  }
  const uint32_t tmem_base = *tmem_slot;
  const int total_jobs = s_jp[g.n_groups] * g.n_tiles;
  const uint32_t w_base = smem_u32(smem);
  const uint32_t t_base = w_base + C::SW * WL_W_STAGE;

  // the next job, for a role of one thread and for a role of a warp; false: none left, or the kernel is being left
  auto take_job = [&](Job& j, Ring& r) {
    if (*abort_flag || !mbar_wait(smem_u32(&jfull[r.i]), r.ph, abort_flag, g.status, 60)) return false;
    j = s_job[r.i];
    mbar_arrive(smem_u32(&jempty[r.i]));
    r.next(WL_JOBS);
    return j.n_tok != 0;
  };
  auto take_job_warp = [&](Job& j, Ring& r) {
    if (!wait_warp(smem_u32(&jfull[r.i]), r.ph, abort_flag, g.status, 61)) return false;
    j = s_job[r.i];
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&jempty[r.i]));
    r.next(WL_JOBS);
    return j.n_tok != 0;
  };

  if (warp == 0) {
    // ---------------- weight TMA (both CTAs, own 128 rows) ----------------
    if (elect_one()) {
      Ring r, rj;
      Job j;
      while (take_job(j, rj)) {
        const int blk = j.b_row >> 7, r0 = static_cast<int>(rank);
        if (FP8) {
          // SwiGLU rows come in blocks of 128 gate then 128 up; this CTA takes 64 of each
          for (int kb = 0; kb < g.k_steps / 2; ++kb, r.next(C::SW)) {
            if (!mbar_wait(smem_u32(&wempty[r.i]), r.ph ^ 1u, abort_flag, g.status, 51)) break;
            const uint32_t fb = smem_u32(&wfull[r.i]), dst = w_base + r.i * WL_W_STAGE;
            mbar_expect_tx(fb, WL_W_STAGE);
            if (SWIGLU) tma_load_3d(dst, &maps.w, kb * 128, r0 * 64, blk, fb);
            else tma_load_3d(dst, &maps.w, kb * 128, 0, blk + r0, fb);
          }
        } else {
          for (int kb = 0; kb < g.k_steps; ++kb, r.next(C::SW)) {
            if (!mbar_wait(smem_u32(&wempty[r.i]), r.ph ^ 1u, abort_flag, g.status, 51)) break;
            const uint32_t fb = smem_u32(&wfull[r.i]), dst = w_base + r.i * WL_W_STAGE;
            if (rank == 0) mbar_expect_tx(fb, 2 * WL_W_STAGE);           // of both CTAs
            // SwiGLU: 16 gate rows, the 16 up rows of the same outputs, the next 16 gate rows ...
            if (SWIGLU) tma_load_4d_pair(dst, &maps.w, kb * WL_K, 0, blk, r0 * 4, fb);
            else tma_load_4d_pair(dst, &maps.w, kb * WL_K, 0, blk + r0, 0, fb);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- token TMA (both CTAs, own half of each MMA's N) ----------------
    if (elect_one()) {
      Ring r, rj;
      Job j;
      while (take_job(j, rj)) {
        const int h1 = first_part<FP8>(j.n_tok) >> 1, h2 = (j.n_tok >> 1) - h1;
        const int row1 = j.row0 + static_cast<int>(rank) * h1, row2 = j.row0 + 2 * h1 + static_cast<int>(rank) * h2;
        const int kpt = steps_per_stage<FP8>(j.n_tok >> 1);
        if (j.n_tok == 32) {
          // Two groups of eight rows, each with all steps of the stage, or zeros for a group without a live one: a box
          // that begins behind the last row reads nothing.  Rows that nobody wrote cost their bytes and, at the power cap,
          // the multipliers' work on whatever they hold: layer, us, all 32 rows and this, workspace full of random values:
          // V3 16 tokens 1112 and 1064, 64 tokens 2244 and 2139, 256 tokens 2659 and 2555; zeros there already: 2152 and
          // 2146; Mixtral 61 tokens 476 and 472, V2-236B 512 tokens 1238 and 1229.
          const int live = j.left - 16 * static_cast<int>(rank);
          const int g0 = live > 0 ? row1 : g.rows, g1 = live > 8 ? row1 + 8 : g.rows;
          for (int kb = 0; kb < g.k_steps; kb += kpt, r.next(C::ST)) {
            if (!mbar_wait(smem_u32(&tempty[r.i]), r.ph ^ 1u, abort_flag, g.status, 52)) break;
            const uint32_t fb = smem_u32(&tfull[r.i]);
            const uint32_t dst = t_base + r.i * C::T_STAGE;
            if (rank == 0) mbar_expect_tx(fb, kpt * 32 * 128);
            tma_load_3d_pair(dst, &maps.t8, 0, g0, kb, fb);
            tma_load_3d_pair(dst + kpt * 1024, &maps.t8, 0, g1, kb, fb);
          }
          continue;
        }
        const CUtensorMap* m1 = h2 > 0 && h1 < 128 ? &maps.t2[(h1 >> 4) - 1] : &maps.t[(h1 >> 4) - 1];
        const CUtensorMap* m2 = &maps.t2[(max(h2, 16) >> 4) - 1];
        for (int kb = 0; kb < g.k_steps; kb += kpt, r.next(C::ST)) {
          if (!mbar_wait(smem_u32(&tempty[r.i]), r.ph ^ 1u, abort_flag, g.status, 52)) break;
          const uint32_t fb = smem_u32(&tfull[r.i]);
          const uint32_t dst = t_base + r.i * C::T_STAGE;
          if (rank == 0) mbar_expect_tx(fb, kpt * j.n_tok * 128);      // steps beyond K arrive as zeros
          tma_load_3d_pair(dst, m1, 0, row1, kb, fb);
          if (h2 > 0) tma_load_3d_pair(dst + h1 * 128, m2, 0, row2, kb, fb);
        }
      }
    }
  } else if (warp == 2) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (rank == 0 && elect_one()) {
      Ring rt, ra, rj;
      uint32_t seq = 0u, parts = 0u;       // jobs, and waits for a part of the accumulator
      int n_before = 0;
      // kind::f16: D fp32 (bit 4), A bf16 (bit 7), B bf16 (bit 10), both K-major, N>>3 at 17, M>>4 at 24
      const uint32_t id0 = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(256 >> 4) << 24);
      bool ok = true;
      Job j;
      while (take_job(j, rj)) {
        const uint32_t h = seq & 1u;
        ok = mbar_wait(smem_u32(&dempty[h]), ((seq >> 1) & 1u) ^ 1u, abort_flag, g.status, 53);
        if (ok && n_before + j.n_tok > C::ACC_COLS) ok = mbar_wait(smem_u32(dpart), parts++ & 1u, abort_flag, g.status, 62);
        if (!ok) break;
        ++seq;
        n_before = j.n_tok;
        tc_fence_after();
        const int n1 = first_part<FP8>(j.n_tok), n2 = j.n_tok - n1;
        const uint32_t id1 = id0 | (static_cast<uint32_t>(n1 >> 3) << 17), id2 = id0 | (static_cast<uint32_t>(n2 >> 3) << 17);
        const uint32_t d = tmem_base + (h ? C::ACC_COLS - j.n_tok : 0);
        const int kpt = steps_per_stage<FP8>(j.n_tok >> 1), step_bytes = j.n_tok == 32 ? 1024 : j.n_tok * 64;
        const uint32_t group_bytes = j.n_tok == 32 ? kpt * 1024 : 1024;      // see the token role
        int in_stage = 0;
        if (FP8) {
          for (int kb = 0; kb < g.k_steps; kb += 2) {
            ok = mbar_wait(smem_u32(&aready[ra.i]), ra.ph, abort_flag, g.status, 55);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              if (in_stage == 0) {
                ok = mbar_wait(smem_u32(&tfull[rt.i]), rt.ph, abort_flag, g.status, 54);
                if (!ok) break;
                tc_fence_after();
              }
              const uint32_t tb = t_base + rt.i * C::T_STAGE + in_stage * step_bytes;
              const uint64_t db = make_smem_desc(tb, group_bytes);
              const uint64_t db2 = make_smem_desc(tb + n1 * 64);
              const uint32_t a = tmem_base + C::ACC_COLS + ra.i * WL_A_COLS + half * (WL_A_COLS / 2);
#pragma unroll
              for (int k = 0; k < WL_K / 16; ++k) {
                // 16 bf16 = 32 bytes = 2 sixteen-byte units inside the swizzle row, or 8 columns of tensor memory
                const uint32_t accumulate = (kb | half | k) != 0 ? 1u : 0u;
                tc_mma_pair_ts(d, a + 8 * k, db + 2 * k, id1, accumulate);
                if (n2 > 0) tc_mma_pair_ts(d + n1, a + 8 * k, db2 + 2 * k, id2, accumulate);
              }
              if (++in_stage == kpt || kb + half + 1 == g.k_steps) {
                tc_commit_pair(smem_u32(&tempty[rt.i]));
                rt.next(C::ST);
                in_stage = 0;
              }
            }
            if (!ok) break;
            tc_commit_pair(smem_u32(&afree[ra.i]));
            ra.next(WL_A_SLOTS);
          }
        } else {
          for (int kb = 0; kb < g.k_steps; ++kb, ra.next(C::SW)) {
            ok = (in_stage != 0 || mbar_wait(smem_u32(&tfull[rt.i]), rt.ph, abort_flag, g.status, 54)) &&
                 mbar_wait(smem_u32(&wfull[ra.i]), ra.ph, abort_flag, g.status, 57);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tb = t_base + rt.i * C::T_STAGE + in_stage * step_bytes;
            const uint64_t da = make_smem_desc(w_base + ra.i * WL_W_STAGE);
            const uint64_t db = make_smem_desc(tb, group_bytes), db2 = make_smem_desc(tb + n1 * 64);
#pragma unroll
            for (int k = 0; k < WL_K / 16; ++k) {
              const uint32_t accumulate = (kb | k) != 0 ? 1u : 0u;
              tc_mma_bf16_pair(d, da + 2 * k, db + 2 * k, id1, accumulate);
              if (n2 > 0) tc_mma_bf16_pair(d + n1, da + 2 * k, db2 + 2 * k, id2, accumulate);
            }
            tc_commit_pair(smem_u32(&wempty[ra.i]));
            if (++in_stage == kpt || kb + 1 == g.k_steps) {
              tc_commit_pair(smem_u32(&tempty[rt.i]));
              rt.next(C::ST);
              in_stage = 0;
            }
          }
        }
        if (!ok) break;
        tc_commit_pair(smem_u32(&dfull[h]));
      }
    }
  } else if (warp == 3) {
    // ---------------- job list of this pair ----------------
    // A look-up costs a binary search over the experts and two divisions, a thousand cycles and more where the issue
    // slots are busy: done once here and ahead, not by every role between two jobs.  The leader draws the number once all
    // roles have begun the job before, and passes it to the other CTA; the latter cannot be WL_MAIL jobs behind, since
    // the leader's MMAs of a job need that CTA's weights and tokens.
    if (elect_one()) {
      Ring rj, rm;
      int job = pair;
      for (;; rj.next(WL_JOBS)) {
        if (!mbar_wait(smem_u32(&jempty[rj.i]), rj.ph ^ 1u, abort_flag, g.status, 59)) break;
        if (job < 0) {
          if (g.next_job == nullptr) {
            job = ~job + n_pairs;
          } else if (rank == 0) {
            job = n_pairs + atomicAdd(g.next_job, 1);
            st_cluster(map_to_cta(smem_u32(&s_mail[rm.i]), 1), job);
            mbar_arrive_cluster(map_to_cta(smem_u32(&mfull[rm.i]), 1));
          } else {
            if (!mbar_wait_cluster(smem_u32(&mfull[rm.i]), rm.ph, abort_flag, g.status, 63)) break;
            job = *reinterpret_cast<volatile int*>(&s_mail[rm.i]);
          }
          rm.next(WL_MAIL);
        }
        Job j;
        j.n_tok = 0;
        if (job < total_jobs) j = locate_job(job, s_pad, s_cnt, s_jp, g);
        s_job[rj.i] = j;
        mbar_arrive(smem_u32(&jfull[rj.i]));
        if (j.n_tok == 0) break;
        job = ~job;
      }
    }
  } else if (warp >= 4 && warp < 4 + WL_EPI_WARPS) {
    // ---------------- epilogue (both CTAs, own 128 lanes) ----------------
    const int quarter = warp & 3;
    // two pieces of output rows per warp: one is filled while the other leaves
    const uint32_t piece0 = smem_u32(pieces + (warp - 4) * 2 * WL_PIECE);
    uint32_t piece = 0u;
    auto next_piece = [&]() {
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      __syncwarp();
      return piece0 + piece * WL_PIECE;
    };
    auto send_piece = [&](int col, int row) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tma_store_2d(&maps.c, col, row, piece0 + piece * WL_PIECE);
      piece ^= 1u;
    };
    uint32_t seq = 0u;
    Ring rj;
    Job next;
    bool more = take_job_warp(next, rj);
    while (more) {
      const Job j = next;
      more = take_job_warp(next, rj);
      const uint32_t h = seq & 1u;
      if (!wait_warp(smem_u32(&dfull[h]), (seq >> 1) & 1u, abort_flag, g.status, 56)) break;
      ++seq;
      tc_fence_after();
      const int col0 = SWIGLU ? j.n_idx * 128 + static_cast<int>(rank) * 64 + quarter * 16
                              : j.n_idx * 256 + static_cast<int>(rank) * 128 + quarter * 32;
      const uint32_t taddr = tmem_base + (h ? C::ACC_COLS - j.n_tok : 0) + (static_cast<uint32_t>(quarter * 32) << 16);
      auto release = [&](uint64_t* bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_leader(bar);
      };
      // chunks of 32 tokens, those first that lie in the next job's columns: once all warps have read them, the next
      // job's MMAs may start
      const int chunks = j.n_tok >> 5, shared = more ? max(0, j.n_tok + next.n_tok - C::ACC_COLS) >> 5 : 0;
      const int i0 = (warp - 4) >> 2;
      if (shared > 0 && i0 >= shared) release(dpart);
      if (i0 >= chunks) release(&dempty[h]);
      for (int i = i0; i < chunks; i += 2) {
        const int c = 32 * (h ? i : chunks - 1 - i);
        uint32_t va[16], vb[16];                // lanes 0-15 and 16-31 of the quarter
        tc_ld_16x32(taddr + c, va);
        tc_ld_16x32(taddr + (16u << 16) + c, vb);
        tc_ld_wait();
        // this warp's share is in registers
        if (i < shared && i + 2 >= shared) release(dpart);
        if (i + 2 >= chunks) release(&dempty[h]);
        if (SWIGLU) {
          // va: gate rows, vb: the up rows of the same 16 outputs; a piece is 32 tokens x 16 outputs
          uint32_t p[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            p[i] = pack_bf16(silu_f(__uint_as_float(va[2 * i])) * __uint_as_float(vb[2 * i]),
                             silu_f(__uint_as_float(va[2 * i + 1])) * __uint_as_float(vb[2 * i + 1]));
          const uint32_t dst = next_piece() + (8 * (lane >> 4) + (lane & 7)) * 32 + ((lane >> 3) & 1) * 16;
          store_fragments(dst, p[0], p[1], p[2], p[3]);
          store_fragments(dst + 512, p[4], p[5], p[6], p[7]);
          send_piece(col0, j.row0 + c);
        } else {
          // two pieces of 16 tokens x 32 outputs, in the 64-byte swizzle of the store's tensor map
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (c + 16 * t >= j.left) break;
            const uint32_t tok = lane & 7, m = lane >> 3;
            const uint32_t dst = next_piece() + tok * 64 + ((m ^ ((tok >> 1) & 3)) << 4);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int i = 8 * t + 4 * x;
              store_fragments(dst + x * 512, pack_bf16(__uint_as_float(va[i]), __uint_as_float(va[i + 1])),
                              pack_bf16(__uint_as_float(va[i + 2]), __uint_as_float(va[i + 3])),
                              pack_bf16(__uint_as_float(vb[i]), __uint_as_float(vb[i + 1])),
                              pack_bf16(__uint_as_float(vb[i + 2]), __uint_as_float(vb[i + 3])));
            }
            send_piece(col0, j.row0 + c + 16 * t);
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  } else if (FP8 && warp >= 4 + WL_EPI_WARPS) {
    // ---------------- FP8 -> bf16 converters: shared -> registers -> tensor memory ----------------
    const int quarter = warp & 3;
    const uint32_t grp = (warp - 4 - WL_EPI_WARPS) >> 3;   // even / odd stages, counted over all jobs
    const uint32_t half = (warp - 4 - WL_EPI_WARPS) >> 2 & 1u;          // 64 K elements of a stage
    const int row = !SWIGLU ? quarter * 32 + lane : quarter * 16 + (lane & 15) + (lane & 16) * 4;
    const int block = SWIGLU ? lane >> 4 : static_cast<int>(rank);      // scale block row of this lane's weights
    const uint32_t a_slot = tmem_base + C::ACC_COLS + grp * WL_A_COLS + half * (WL_A_COLS / 2) +
                            (static_cast<uint32_t>(quarter * 32) << 16);
    const int stages = g.k_steps / 2;
    Ring rw, rj;
    rw.i = grp;
    uint32_t ph = 0u;
    int first = static_cast<int>(grp);
    Job j;
    bool ok = true;
    while (ok && take_job_warp(j, rj)) {
      const float* srow = g.scales + static_cast<long long>((j.b_row >> 7) + block) * g.scale_cols;
      float s16 = 0.f;
      for (int kb = first; kb < stages; kb += 2) {
        // the scales of this group's next 16 stages, spread over a lane's half of the warp and handed out by shuffle
        const int in16 = ((kb - first) >> 1) & 15;
        if (in16 == 0) s16 = kb + 2 * (lane & 15) < stages ? __ldg(srow + kb + 2 * (lane & 15)) : 0.f;
        const float s = __shfl_sync(0xFFFFFFFFu, s16, (lane & 16) | in16);
        ok = wait_warp(smem_u32(&wfull[rw.i]), rw.ph, abort_flag, g.status, 57);
        if (!ok) break;
        const uint8_t* src = smem + rw.i * WL_W_STAGE + row * 128;
        uint4 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const uint4*>(src + (((half * 4 + i) ^ (row & 7)) << 4));
        uint32_t o[32];
        convert32(q[0], q[1], s, o);
        convert32(q[2], q[3], s, o + 16);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&wempty[rw.i]));
        ok = wait_warp(smem_u32(&afree[grp]), ph ^ 1u, abort_flag, g.status, 58);
        if (!ok) break;
        ph ^= 1u;
        tc_fence_after();
        tc_st32(a_slot, o);
        rw.i += 2;
        if (rw.i >= C::SW) { rw.i -= C::SW; rw.ph ^= 1u; }
        tc_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_leader(&aready[grp]);
      }
      first = (first + stages) & 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // neither CTA leaves while the other may still signal it or use its TMEM
  if (warp == 3) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

template <int EPI, bool FP8>
int launch_kernel(const Handle* h, const WlMaps& maps, const WlArgs& a, int grid, cudaStream_t st) {
  using C = WlCfg<FP8>;
  static bool done[64];
  if (!(h->device >= 0 && h->device < 64 && done[h->device])) {
    MG_CUDA(cudaFuncSetAttribute(grouped_gemm_wl_kernel<EPI, FP8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(C::SMEM)));
    if (h->device >= 0 && h->device < 64) done[h->device] = true;
  }
  MG_CUDA(launch_chained(h, grouped_gemm_wl_kernel<EPI, FP8>, grid, C::THREADS, C::SMEM, st, maps, a));
  return MG_OK;
}

// From the handle's cache, by what the maps are made of: a forward's launches are few and the same ones again.  Encoding the
// maps anew, as for a batch size not seen lately, takes a forward 3 us more on the host (V2-Lite 36 and 39 us).
template <bool FP8>
int wl_maps(const Handle* h, const GemmProblem& p, bool swiglu, const WlMaps** out) {
  WlMapCache& cache = h->wl_maps;
  const WlMapCache::Key key{p.a, p.b, p.out, p.a_rows, static_cast<int64_t>(p.n_groups) * p.n_per_group, p.ldo, p.K, FP8, swiglu};
  for (int i = 0; i < cache.used; ++i)
    if (cache.e[i].key == key) { *out = &cache.e[i].maps; return MG_OK; }
  WlMaps m;
  const uint64_t K = static_cast<uint64_t>(p.K), blocks = static_cast<uint64_t>(key.w_rows) / 128;
  const uint32_t both = swiglu ? 2 : 1;
  int rc = FP8 ? encode_map(&m.w, p.b, true, 3, {K, 128, blocks}, {K, 128 * K}, {128, 128 / both, both})
               : encode_map(&m.w, p.b, false, 4, {K, 16, blocks, 8}, {2 * K, 256 * K, 32 * K}, {WL_K, 16, both, 8 / both});
  const uint64_t rows = static_cast<uint64_t>(p.a_rows), steps = K / WL_K;
  for (int i = 0; i < 13 && rc == MG_OK; ++i) {
    const uint32_t n = 16 * (i < 8 ? i + 1 : i - 7);
    rc = encode_map(i < 8 ? &m.t[i] : &m.t2[i - 8], p.a, false, 3, {WL_K, rows, steps}, {2 * K, 2 * WL_K},
                    {WL_K, n, i < 8 ? static_cast<uint32_t>(steps_per_stage<FP8>(n)) : 1u});
  }
  if (rc == MG_OK)
    rc = encode_map(&m.t8, p.a, false, 3, {WL_K, rows, steps}, {2 * K, 2 * WL_K}, {WL_K, 8, steps_per_stage<FP8>(16)});
  if (rc == MG_OK)
    rc = encode_2d(h, &m.c, p.out, rows, static_cast<uint64_t>(p.ldo), swiglu ? 32 : 16, swiglu ? TM_OUT_16 : TM_OUT_PIECE);
  if (rc != MG_OK) return rc;
  WlMapCache::Entry& e = cache.e[cache.next];
  e.key = key;
  e.maps = m;
  cache.next = (cache.next + 1) % WlMapCache::kEntries;
  if (cache.used < WlMapCache::kEntries) ++cache.used;
  *out = &e.maps;
  return MG_OK;
}

}  // namespace

int launch_gemm_wl(const Handle* h, const GemmProblem& p, cudaStream_t st) {
  const bool swiglu = p.epilogue == EPI_SWIGLU_BF16;
  MG_REQUIRE(p.pad_offsets != nullptr && (!p.b_fp8 || p.scales != nullptr) && (swiglu || p.epilogue == EPI_PLAIN_BF16),
             MG_ERR_CONFIG, "weight-lane GEMM: grouped weights, FP8 with scales, and bf16 outputs only");
  MG_REQUIRE(p.K % (p.b_fp8 ? 128 : WL_K) == 0 && p.n_per_group % 256 == 0 && p.ldo % 16 == 0, MG_ERR_SHAPE,
             "weight-lane GEMM: K=%d, N per expert=%d", p.K, p.n_per_group);
  const WlMaps* maps = nullptr;
  const int rc = p.b_fp8 ? wl_maps<true>(h, p, swiglu, &maps) : wl_maps<false>(h, p, swiglu, &maps);
  if (rc != MG_OK) return rc;
  WlArgs a;
  a.pad_offsets = p.pad_offsets;
  a.counts = p.counts;
  a.n_groups = p.n_groups;
  a.n_tiles = p.n_per_group / 256;
  a.n_per_group = p.n_per_group;
  a.k_steps = p.K / WL_K;
  a.scales = p.scales;
  a.scale_cols = p.K / 128;
  a.next_job = p.next_job;
  a.status = h->d_status;
  a.rows = static_cast<int>(p.a_rows);
  a.chained = h->chain ? 1 : 0;
  const int max_tokens = p.b_fp8 ? WlCfg<true>::MAX_TOKENS : WlCfg<false>::MAX_TOKENS;
  const int64_t tiles = (p.a_rows + max_tokens - 1) / max_tokens + p.n_groups;
  int64_t pairs = h->sm_count / 2;
  if (tiles * a.n_tiles < pairs) pairs = tiles * a.n_tiles;
  const int grid = static_cast<int>(2 * pairs);
  if (p.b_fp8)
    return swiglu ? launch_kernel<EPI_SWIGLU_BF16, true>(h, *maps, a, grid, st)
                  : launch_kernel<EPI_PLAIN_BF16, true>(h, *maps, a, grid, st);
  return swiglu ? launch_kernel<EPI_SWIGLU_BF16, false>(h, *maps, a, grid, st)
                : launch_kernel<EPI_PLAIN_BF16, false>(h, *maps, a, grid, st);
}

}  // namespace mg
