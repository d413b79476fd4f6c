// Grouped BF16 products on the 5th-generation tensor cores (tcgen05 + TMEM),
// operands staged by TMA, for the prefill expert and shared-expert products.
//
// Replaces the two fused_moe_kernel launches of the reference prefill path
// (native/aot/gfx1151/q8192-output2/manifest.json:1398-1415, 4672-4689; launched
// at native/src/native_moe_prefill.hip.cpp:862-876), expert_silu_multiply_kernel
// (:384-402), and the five hipBLASLt plans of the shared expert with their
// pointwise kernels (:790-826) -- the epilogues are fused.
//
// Two kernels.  The two-SM one (grouped_gemm_pair_kernel, below) runs the expert, shared-expert, dense and router-logits
// products of one GPU.  The one-SM one, described here, serves expert parallelism (its epilogue stores to peers, and its
// launches can be split into parts).
//
// Work unit = one 128-row tile of one expert x one 256-wide slice of the output
// columns.  D[128, 256] (FP32) lives in tensor memory, two buffers of 256
// columns, so the epilogue of a unit overlaps the main loop of the next.
//   warp 0   TMA producer: per 64-wide K block one 128x64 tile of A and two
//            128x64 tiles of B into a 4-stage shared-memory ring (128-byte swizzle)
//   warp 1   issues tcgen05.mma (M128 N256 K16, 4 per K block) and
//            commits to the ring's "empty" barriers / the accumulator's "full" barrier
//   warp 2   allocates and frees the 512 tensor-memory columns
//   warps 2-3 with fused dispatch (gate_up only): gather the tile's 128 activation rows BY TOKEN
//            INDEX with 16-byte cp.async copies that arrive on the stage's barrier when complete
//   warps 4-11 epilogue (two per quarter of the TMEM lanes, half of the columns each): tcgen05.ld 32 rows x 32 columns per warp, SwiGLU or
//            scaling; the BF16 results of 64 output columns are turned in shared memory so that
//            every store instruction writes whole 128-byte pieces of four rows (a thread storing
//            its own row would touch 32 different lines per instruction)
// Every mbarrier wait is bounded; on expiry the block sets the status word,
// stops issuing, waits for its copies in flight, frees tensor memory and returns.
#include "grouped_gemm.cuh"

#include <cuda.h>
#include <mutex>
#include <unordered_map>
#include <cudaTypedefs.h>

namespace aima {
namespace {

constexpr int kBM = 128;           // rows per tile (= kTileRows of the plan)
constexpr int kBN = 256;           // accumulator columns per unit
constexpr int kBK = 64;            // K elements per stage: 128 bytes = one swizzle row
constexpr int kStages = 4;
constexpr int kUmmaK = 16;
constexpr int kStageABytes = kBM * kBK * 2;        // 16 KB
constexpr int kStageBBytes = kBN * kBK * 2;        // 32 KB
constexpr int kStageBytes = kStageABytes + kStageBBytes;
constexpr int kEpilogueWarps = 8;   // two per quarter of the 128 TMEM lanes, each taking half of the columns
constexpr int kTcThreads = (4 + kEpilogueWarps) * 32;
constexpr int kTmemColumns = 512;
constexpr int kStoreStageBytes = 32 * 128;          // per epilogue warp: 32 rows x 64 BF16 outputs
constexpr int kTcSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/ +
                             kEpilogueWarps * kStoreStageBytes;

struct TcMaps {
  CUtensorMap a;    // [rows, k]      box 64 x 128
  CUtensorMap b0;   // gate half / only weight matrix, [n_rows, k]
  CUtensorMap b1;   // up half (may equal b0)
};

struct TcProblem {
  GroupedGemm g;
  int n_chunks;           // output column slices of kBN accumulator columns
  int b_rows_per_expert;  // rows between experts in b0 / b1
  int up_row_offset;      // row offset of the "up" half inside an expert (gate_up modes)
  int n_valid;            // valid output columns (plain mode masks beyond)
  int* status;            // device status word
  unsigned long long wait_limit_ns;
  // two-SM form
  int dense_tile;         // dense modes: rows per tile
  int k_splits;           // kGemmPlainF32: runs of K, each a unit of its own
  SharedProblem shared;   // expert modes: the shared expert's rows, in the same launch
  int shared_tiles;
};

// ---- PTX wrappers ---------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];"
      :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// The producer and MMA loops below are run by their WHOLE warp and only the issuing instructions are guarded by
// elect_one().  With a branch on lane == 0 around the loops a stage cost its TMA thread 680 cycles (two loads) and its MMA
// thread 320 (four MMAs) of issue time -- more than the 512 cycles the tensor cores need for it.
constexpr int kGatherThreads = 64;     // warps 2 and 3
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}
// the barrier receives one arrival (already part of its expected count) once all cp.async copies this
// thread has issued so far are complete
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
               :: "r"(smem_dst), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major tile whose rows are 128 bytes
// (64 BF16) with the 128-byte swizzle TMA applies: 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k_major_sw128(uint32_t smem_addr) {
  uint64_t desc = 0;
  desc |= static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4);          // start address
  desc |= static_cast<uint64_t>(1) << 16;                               // leading byte offset (unused)
  desc |= static_cast<uint64_t>(1024 >> 4) << 32;                       // stride byte offset
  desc |= static_cast<uint64_t>(1) << 46;                               // descriptor version (sm_100)
  desc |= static_cast<uint64_t>(2) << 61;                               // SWIZZLE_128B
  return desc;
}

// Instruction descriptor: D = F32, A = B = BF16, both K-major, M = 128, N = 256.
constexpr uint32_t kInstrDesc =
    (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kBN >> 3) << 17) |
    (static_cast<uint32_t>(kBM >> 4) << 24);

// 32 results of this thread's row into half `half` (0/1) of the warp's 32 x 128-byte staging
// tile; 16-byte pieces are XOR-swizzled by the row so that neither side has bank conflicts.
__device__ __forceinline__ void stage_32(uint8_t* stage, int lane, int half, const float* v) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 w;
    w.x = static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 0])) | (static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 1])) << 16);
    w.y = static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 2])) | (static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 3])) << 16);
    w.z = static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 4])) | (static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 5])) << 16);
    w.w = static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 6])) | (static_cast<uint32_t>(float_to_bf16_bits(v[8 * i + 7])) << 16);
    const int piece = (4 * half + i) ^ (lane & 7);
    *reinterpret_cast<uint4*>(stage + lane * 128 + piece * 16) = w;
  }
}

// The staged 32 x 64 tile to global memory: instruction i writes rows 4i .. 4i+3, eight lanes per
// row.  dst = first row of the warp's 32, first of the 64 columns; rows_ok = valid rows of the 32;
// cols_ok = valid columns of the 64 (a multiple of 8).
__device__ __forceinline__ void store_staged(const uint8_t* stage, int lane, __nv_bfloat16* dst, size_t ldc,
                                             int rows_ok, int cols_ok) {
  __syncwarp();
  const int piece = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = 4 * i + (lane >> 3);
    const uint4 w = *reinterpret_cast<const uint4*>(stage + row * 128 + ((piece ^ (row & 7)) * 16));
    if (row < rows_ok && piece * 8 < cols_ok)
      *reinterpret_cast<uint4*>(dst + static_cast<size_t>(row) * ldc + piece * 8) = w;
  }
  __syncwarp();
}


// The same with one destination per row: rows[i] is the address of the first of the 64 columns in the row
// instruction i writes for this lane (row 4 i + lane / 8 of the warp's 32), nullptr for a row past the tile's end.
__device__ __forceinline__ void store_staged_rows(const uint8_t* stage, int lane, __nv_bfloat16* const* rows, int cols_ok) {
  __syncwarp();
  const int piece = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = 4 * i + (lane >> 3);
    const uint4 w = *reinterpret_cast<const uint4*>(stage + row * 128 + ((piece ^ (row & 7)) * 16));
    if (rows[i] != nullptr && piece * 8 < cols_ok) *reinterpret_cast<uint4*>(rows[i] + piece * 8) = w;
  }
  __syncwarp();
}

// One epilogue warp drains its part of a 128-row x 256-column FP32 accumulator: TMEM lanes
// 32 ew .. 32 ew + 31 (rows row0 + 32 ew ... of the output), half `eh` of the unit's columns.
template <int MODE>
__device__ __forceinline__ void drain_accumulator(const GroupedGemm& g, const TcProblem& pb, uint32_t tmem_base,
                                                  int buf, int ew, int eh, int lane, uint8_t* stage, int chunk,
                                                  int row0, int rows) {
  constexpr bool kDual = (MODE == kGemmExpertGateUp || MODE == kGemmSharedGateUp);
  const int r = ew * 32 + lane;                // row inside the tile
  const bool row_ok = r < rows;
  const int row = row0 + r;
  const uint32_t taddr = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + static_cast<uint32_t>(buf * kBN);
  const int rows_ok = min(32, rows - ew * 32);           // valid rows among this warp's 32 (may be <= 0)
  if (kDual) {
    // columns [0,128) gate, [128,256) up  ->  128 activations per row, stored 64 at a time
    __nv_bfloat16* dst = g.c + static_cast<size_t>(row0 + ew * 32) * g.ldc + chunk * (kBN / 2);
#pragma unroll 1
    for (int c0 = eh * (kBN / 4); c0 < (eh + 1) * (kBN / 4); c0 += 64) {
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t gr[32], ur[32];
        tmem_ld32(taddr + c0 + 32 * half, gr);
        tmem_ld32(taddr + kBN / 2 + c0 + 32 * half, ur);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float gate = round_bf16(__uint_as_float(gr[j]));
          const float up = round_bf16(__uint_as_float(ur[j]));
          const float s = det_silu(gate);
          v[j] = (MODE == kGemmExpertGateUp) ? __fmul_rn(round_bf16(s), up) : __fmul_rn(s, up);
        }
        stage_32(stage, lane, half, v);
      }
      store_staged(stage, lane, dst + c0, static_cast<size_t>(g.ldc), rows_ok, 64);
    }
  } else if (MODE != kGemmPlainF32) {
    float scale = 1.0f;
    if (row_ok) {
      scale = g.row_scale[MODE == kGemmExpertDown ? g.sorted_rows[row] : row];
    }
    const int col_base = chunk * kBN;
    __nv_bfloat16* dst = g.c + static_cast<size_t>(row0 + ew * 32) * g.ldc + col_base;
    const bool scatter = MODE == kGemmExpertDown && g.scatter_tokens_per_rank > 0;
    __nv_bfloat16* scatter_rows[8];
    if (scatter) {
      // where the eight rows this lane stores live: on the GPU that owns the row's token
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3);
        scatter_rows[i] = nullptr;
        if (rr < rows_ok) {
          const int flat = g.sorted_rows[row0 + ew * 32 + rr];
          const int owner = (flat >> 3) / g.scatter_tokens_per_rank;
          const int local_flat = flat - owner * g.scatter_tokens_per_rank * 8;
          scatter_rows[i] = reinterpret_cast<__nv_bfloat16*>(g.scatter_region[owner] + g.scatter_offset) +
                            static_cast<size_t>(local_flat) * g.ldc + col_base;
        }
      }
    }
#pragma unroll 1
    for (int c0 = eh * (kBN / 2); c0 < (eh + 1) * (kBN / 2); c0 += 64) {
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t ar[32];
        tmem_ld32(taddr + c0 + 32 * half, ar);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float acc = __uint_as_float(ar[j]);
          v[j] = (MODE == kGemmExpertDown) ? __fmul_rn(acc, scale) : __fmul_rn(scale, round_bf16(acc));
        }
        stage_32(stage, lane, half, v);
      }
      const int cols_ok = max(0, min(64, pb.n_valid - col_base - c0));
      if (scatter) {
        __nv_bfloat16* at[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) at[i] = scatter_rows[i] != nullptr ? scatter_rows[i] + c0 : nullptr;
        store_staged_rows(stage, lane, at, cols_ok);
      } else {
        store_staged(stage, lane, dst + c0, static_cast<size_t>(g.ldc), rows_ok, cols_ok);
      }
    }
  } else {
    // FP32 output (approximate router logits): every thread stores its own row
    const int col_base = chunk * kBN;
#pragma unroll 1
    for (int c0 = eh * (kBN / 2); c0 < (eh + 1) * (kBN / 2); c0 += 32) {
      uint32_t ar[32];
      tmem_ld32(taddr + c0, ar);
      tmem_ld_wait();
      if (row_ok) {
        float4* out = reinterpret_cast<float4*>(g.c_f32 + static_cast<size_t>(row) * g.ldc + col_base + c0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (col_base + c0 + 4 * j + 4 <= pb.n_valid)
            out[j] = make_float4(__uint_as_float(ar[4 * j]), __uint_as_float(ar[4 * j + 1]),
                                 __uint_as_float(ar[4 * j + 2]), __uint_as_float(ar[4 * j + 3]));
        }
      }
    }
  }
}

template <int MODE, bool kGather = false>
__global__ void __launch_bounds__(kTcThreads, 1)
grouped_gemm_tc_kernel(const __grid_constant__ TcMaps maps, const TcProblem pb) {
  constexpr bool kDual = (MODE == kGemmExpertGateUp || MODE == kGemmSharedGateUp);
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: the swizzled descriptors assume base offset 0
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kStages * kStageBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kStages + 2 + b); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + kStages * kStageBytes + 8 * (2 * kStages + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + kStages * kStageBytes + 8 * (2 * kStages + 4) + 8);
  const uint32_t drain_bar = bar_base + 8u * (2 * kStages + 6);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // known to be the same in all lanes
  const int lane = threadIdx.x & 31;
  const GroupedGemm& g = pb.g;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar(s), kGather ? 1 + kGatherThreads : 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), kEpilogueWarps);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemColumns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Programmatic dependent launch: the kernel is launched with stream serialisation relaxed, so its
  // blocks may become resident -- and run the set-up above (barriers, TMEM) -- while the kernel
  // before it in the stream is still draining.  Nothing above reads or writes global memory;
  // everything below does, so this is where the kernel waits for its predecessor to complete and
  // for that kernel's writes to be visible.  The kernel after this one may be scheduled likewise.
  pdl_enter();

  const int n_tiles_all = g.tile_count != nullptr ? *g.tile_count : g.max_tiles;
  const int parts = g.parts > 1 ? g.parts : 1;
  const int tile_lo = static_cast<int>(static_cast<long long>(n_tiles_all) * g.part / parts);
  const int tile_hi = static_cast<int>(static_cast<long long>(n_tiles_all) * (g.part + 1) / parts);
  // a bounded wait that ran out earlier in this call (a peer that never answered, a barrier of a kernel before
  // this one) leaves a status: nothing that follows can be right, so the products are skipped rather than run on
  // incomplete data until the host reads the status
  // (one thread samples it for the block, so that all warp roles see the same verdict)
  volatile int* poison_slot = abort_flag + 1;
  if (threadIdx.x == 0) *poison_slot = *reinterpret_cast<volatile const int*>(pb.status);
  __syncthreads();
  const bool poisoned = *poison_slot != 0;
  const int total_units = poisoned ? 0 : (tile_hi - tile_lo) * pb.n_chunks;
  const int k_blocks = g.k / kBK;

  auto unit_tile = [&](int unit, int& tile, int& chunk, int& expert, int& row0, int& rows) {
    tile = unit / pb.n_chunks;
    chunk = unit - tile * pb.n_chunks;
    tile += tile_lo;
    if (g.tile_expert != nullptr) {
      expert = g.tile_expert[tile] - g.expert_base;
      row0 = g.tile_row0[tile];
      rows = g.tile_rows[tile];
    } else {
      expert = 0;
      row0 = tile * kBM;
      rows = min(kBM, g.dense_rows - row0);
    }
  };
  auto timeout = [&]() {
    atomicCAS(pb.status, 0, kStatusTimeoutMbarrier);
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool alive = true;
    for (int unit = blockIdx.x; unit < total_units && alive; unit += gridDim.x) {
      int tile, chunk, expert, row0, rows;
      unit_tile(unit, tile, chunk, expert, row0, rows);
      int b0_row, b1_row;
      if (kDual) {
        b0_row = expert * pb.b_rows_per_expert + chunk * (kBN / 2);
        b1_row = expert * pb.b_rows_per_expert + pb.up_row_offset + chunk * (kBN / 2);
      } else {
        b0_row = expert * pb.b_rows_per_expert + chunk * kBN;
        b1_row = b0_row + kBN / 2;
      }
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(empty_bar(stage), phase ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        if (elect_one()) {
          const uint32_t a_dst = smem_base + stage * kStageBytes;
          const uint32_t b_dst = a_dst + kStageABytes;
          mbar_arrive_expect_tx(full_bar(stage), kGather ? kStageBBytes : kStageBytes);
          if (!kGather) tma_load_2d(a_dst, &maps.a, kb * kBK, row0, full_bar(stage));
          tma_load_2d(b_dst, &maps.b0, kb * kBK, b0_row, full_bar(stage));
          tma_load_2d(b_dst + kStageBBytes / 2, kDual ? &maps.b1 : &maps.b0, kb * kBK, b1_row, full_bar(stage));
        }
        __syncwarp();
        ++issued;
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    // drain on abort: wait (bounded) for the stages whose copies are still in flight
    if (lane == 0 && *abort_flag != 0) {
      volatile int ignore = 0;
      int s = stage;
      uint32_t ph = phase;
      for (int i = 0; i < min(issued, kStages); ++i) {
        if (--s < 0) { s = kStages - 1; ph ^= 1u; }
        mbar_wait_bounded(full_bar(s), ph, &ignore);
      }
    }
  } else if (kGather && (warp == 2 || warp == 3)) {
    // ------------------------------ A-row gather -------------------------------
    // Eight neighbouring threads copy the eight 16-byte pieces of one row per K block (a warp
    // instruction then touches four 128-byte lines, not 32): thread t owns piece t % 8 of rows
    // t / 8 + 8 j, j = 0 .. 15, fetched by token index; piece c of row r goes to piece position
    // c ^ (r & 7) (the 128-byte swizzle).  The copies are asynchronous and the thread never waits for
    // them: an arrive-on-completion on the stage's "full" barrier (already counted in the barrier's
    // arrival count) follows each batch, so the only wait is for a free stage and up to kStages
    // batches per thread stay in flight.
    const int lt = (warp - 2) * 32 + lane;
    const int piece = lt & 7;
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    for (int unit = blockIdx.x; unit < total_units && alive; unit += gridDim.x) {
      int tile, chunk, expert, row0, rows;
      unit_tile(unit, tile, chunk, expert, row0, rows);
      int source[16];            // element offset of this thread's piece in each of its 16 rows
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int r = (lt >> 3) + 8 * j;
        source[j] = r < rows ? (g.sorted_rows[row0 + r] >> 3) * g.lda + piece * 8 : -1;   // nothing past the tile's end
      }
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1u, abort_flag)) { alive = false; timeout(); break; }
        const uint32_t base = smem_base + stage * kStageBytes;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int r = (lt >> 3) + 8 * j;
          if (source[j] >= 0) cp_async_16(base + r * 128 + ((piece ^ (r & 7)) << 4), g.gather_src + source[j] + kb * kBK);
        }
        cp_async_arrive_noinc(full_bar(stage));
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    cp_async_wait_all();     // nothing of this thread's may be in flight when the block exits
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    int stage = 0;
    uint32_t phase = 0;
    int local = 0;
    bool alive = true;
    for (int unit = blockIdx.x; unit < total_units && alive; unit += gridDim.x, ++local) {
      const int buf = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      // the epilogue must have drained this accumulator buffer (first use: free)
      if (!mbar_wait_bounded_warp(tempty_bar(buf), (use & 1u) ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
      tc_fence_after();
      const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buf * kBN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(full_bar(stage), phase, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        if (kGather) fence_async_proxy();     // rows written by cp.async are read through the async proxy
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = smem_base + stage * kStageBytes;
          const uint64_t adesc = smem_desc_k_major_sw128(a_addr);
          const uint64_t bdesc = smem_desc_k_major_sw128(a_addr + kStageABytes);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            // advancing 16 elements (32 bytes) along K inside the swizzled row
            umma_bf16(tmem_d, adesc + static_cast<uint64_t>(k * 2), bdesc + static_cast<uint64_t>(k * 2),
                      kInstrDesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(empty_bar(stage));      // frees the stage when the MMAs above retire
          if (kb + 1 == k_blocks) umma_commit(tfull_bar(buf));
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------ epilogue ----------------------------------
    const int ew = (warp - 4) & 3;                 // TMEM lanes 32 ew .. 32 ew + 31 (a warp reaches the quarter warp % 4)
    const int eh = (warp - 4) >> 2;                // which half of the unit's columns this warp drains
    int local = 0;
    bool alive = true;
    for (int unit = blockIdx.x; unit < total_units && alive; unit += gridDim.x, ++local) {
      int tile, chunk, expert, row0, rows;
      unit_tile(unit, tile, chunk, expert, row0, rows);
      const int buf = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      if (!mbar_wait_bounded_warp(tfull_bar(buf), use & 1u, abort_flag, pb.wait_limit_ns)) { alive = false; if (lane == 0) timeout(); break; }
      tc_fence_after();
      drain_accumulator<MODE>(g, pb, tmem_base, buf, ew, eh, lane,
                              smem_gen + kStages * kStageBytes + 256 + (warp - 4) * kStoreStageBytes, chunk, row0, rows);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(buf));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    // a wait ran out: the copies have been waited for above, and so are the MMAs under way, by a last commit
    volatile int ignore = 0;
    if (warp == 1 && elect_one()) umma_commit(drain_bar);
    if (threadIdx.x == 0) mbar_wait_bounded(drain_bar, 0, &ignore);
    __syncthreads();
  }
  if (warp == 2) tmem_dealloc(tmem_base, kTmemColumns);
}

// ---------------------------------------------------------------------------
// Two-SM form with the WEIGHTS on the M side.  A pair of blocks (a cluster of two) computes 256 weight rows x one
// tile of N <= 256 rows of A, transposed: D^T[256, N] = W[256, K] . A[N, K]^T with tcgen05.mma.cta_group::2.  Block r
// of the pair stages 128 weight rows and N / 2 rows of A per K block; the leader (block 0) issues the MMAs for both;
// each block drains the 128 weight rows (= output columns) in its own tensor memory.
//
// Why this way round: the tile height of the instruction is fixed at 256 (or 128 in one block), its width N goes in
// steps of 32.  With the rows of an expert on the M side every expert pads its last tile to 128 or 256 rows -- at
// T = 8192 and balanced routing 1.25 x (128-row tiles) or 1.5 x (256) of the useful products, and with few rows per
// expert nearly all of them -- while the weights, always whole multiples of 256 rows, pad nothing.  Here a tile costs
// what its rows cost, rounded up to 32, and each weight byte enters shared memory once per up to 256 rows.
//
//   full[s]    leader only.  Completed by the TMA loads of BOTH blocks (cta_group::2 loads signal the
//              leader's barrier), and with fetched rows by an arrival for the second block's rows[s].
//   rows[s]    fetched rows: this block's rows of stage s have landed (cp.async arrives by itself).
//   empty[s]   both blocks: the MMAs reading stage s have retired (tcgen05.commit, multicast to the pair).
//   tfull[b]   both blocks: accumulator b is complete (commit, multicast).
//   tempty[b]  leader only: the eight epilogue warps of each block have drained accumulator b.
// No load uses cluster multicast: each block fetches its own operands.
// ---------------------------------------------------------------------------
constexpr int kStages2 = 6;
constexpr int kPairRows = 256;                            // rows of A per tile at most = accumulator columns of a buffer
constexpr int kPlainBand = 8;                             // row tiles the units of a dense product walk together
constexpr int kPairN = 256;                               // weight rows per unit (128 per block)
constexpr int kStage2ABytes = 128 * kBK * 2;              // 16 KB: this block's 128 weight rows
constexpr int kStage2BBytes = (kPairRows / 2) * kBK * 2;  // up to 16 KB: this block's half of the tile's rows
constexpr int kStage2Bytes = kStage2ABytes + kStage2BBytes;
constexpr int kGatherTableBytes = 32 * 16;                // per gather warp: token indices of 128 rows, in fours
constexpr int kTc2BarrierBytes = 512;
constexpr int kPairEpilogueWarps = 16;                    // four per quarter of the 128 TMEM lanes
constexpr int kPairThreads = (4 + kPairEpilogueWarps) * 32;
constexpr int kStoreStage2Bytes = 32 * 64;                // per epilogue warp: 32 rows x 32 BF16 outputs
constexpr int kTc2SmemBytes = kStages2 * kStage2Bytes + 1024 /*alignment slack*/ + kTc2BarrierBytes +
                              kPairEpilogueWarps * kStoreStage2Bytes + 2 * kGatherTableBytes;
static_assert(kTc2SmemBytes <= 227 * 1024, "two-SM product kernel exceeds 227 KB of shared memory");

struct TcPairMaps {
  CUtensorMap w;        // weights: [rows, k] box 64 x 128, or the 5-D view of a gate_up tensor (make_gate_up_map)
  CUtensorMap shared_w[2];     // the shared expert's gate and up matrices (box 64 x 16), or its down matrix (box 64 x 128)
  CUtensorMap shared_rows[4];  // its rows, like `rows`
  CUtensorMap rows[4];  // A: boxes of 64 x 16, 32, 64 and 128 rows (any multiple of 16 rows is at most four loads)
  CUtensorMap one_row;  // gather: the box of one row of the rows by token
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory location in block `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of either block that publishes what this thread has done or waited for -- shared-memory writes of a
// block's own threads, tensor-memory reads -- to the other block, which takes it over with mbar_wait_bounded_warp<true>.  Both
// fences are restricted to shared memory: a release of everything first waits for the thread's global stores (3000 cycles per
// unit in the epilogue).  us per layer for the row relay with them / with arrive.release.cluster and try_wait.acquire.cluster:
// 286 / 588 at 333 tokens, 364 / 690 at 2047 with the norms, 714 / 1198 at 8192; without any order at cluster scope 286, 364 and
// 716.  For the drained accumulators, with / without: 310 / 310 at 1024 tokens, 367 / 367 at 2047, 1802 / 1800 for four layers of
// 4096, 322 / 323 for the dense product of 8192 x 12352 x 2048.
__device__ __forceinline__ void mbar_publish_cluster(uint32_t cluster_addr) {
  asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" :: "r"(cluster_addr) : "memory");
}
// TMA tile loads of one block of the pair; the bytes are accounted on the LEADER's barrier
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];"
      :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar) : "memory");
}
// The same for weights that are read once, or by neighbouring units at the same time: marked to leave L2 first, so that the
// stream of weights does not push out the rows, the activations and the outputs that are read again.  us per layer with the
// mark / with the normal priority, timed in turn, balanced routing, weights of three layers in rotation: 118 / 124 at 16
// tokens, 270 / 282 at 333, 300 / 307 at 1024, 332 / 341 at 2047, 414 / 428 at 4096.  No difference beyond the spread of 5 %
// and more at 8192 tokens (728 / 729) and with eight hot experts, whose weights many tiles share (182 / 189 at 2047, 514 / 511
// at 8192).
__device__ __forceinline__ uint64_t policy_stream() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ void tma_load_2d_pair_stream(uint32_t dst, const CUtensorMap* map, int x, int y,
                                                        uint32_t leader_bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;"
      :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(uint32_t dst, const CUtensorMap* map, int x, int group, int expert,
                                                 uint32_t leader_bar, uint64_t policy) {
  const int zero = 0;
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %3, %4, %5}], [%6], %7;"
      :: "r"(dst), "l"(map), "r"(x), "r"(zero), "r"(group), "r"(expert), "r"(leader_bar), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_gather4_pair(uint32_t dst, const CUtensorMap* map, int x, int r0, int r1, int r2,
                                                 int r3, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      :: "r"(dst), "l"(map), "r"(x), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
               :: "r"(smem_dst), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(columns) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at the same shared-memory offset in both blocks of the pair once the MMAs issued so far retire
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  const uint16_t both = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               :: "r"(bar), "h"(both) : "memory");
}

// D = F32, A = B = BF16, both K-major, M = 256 (128 weight rows per block), N = the tile's rows rounded up to 32
__device__ __forceinline__ uint32_t pair_instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | ((256u >> 4) << 24);
}
__host__ __device__ inline int pair_width(int rows) { return (rows + 31) & ~31; }
// groups of four rows a block gathers for `rows` rows of its own (<= 0: none): one for each gather warp at least
__device__ __forceinline__ int gather_fours(int rows) { return max(2, (rows + 3) / 4); }

// 16 lanes x 32 columns of the accumulator in the fragment layout: v[4 i + 2 p + c] of thread t is lane t / 4 + 8 p,
// column 8 i + 2 (t % 4) + c
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// four 8 x 8 blocks of BF16 fragments, transposed: lane 8 m + j gives the address of row j of block m
__device__ __forceinline__ void stmatrix_trans4(uint32_t smem_row, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
               :: "r"(smem_row), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  return static_cast<uint32_t>(float_to_bf16_bits(lo)) | (static_cast<uint32_t>(float_to_bf16_bits(hi)) << 16);
}

// One epilogue warp drains its share of D^T[128, rows]: TMEM lanes 32 q .. 32 q + 31 (output columns), every
// `groups`-th 32-row batch of the tile.  Fragments of eight columns x eight rows are turned by stmatrix.trans into the
// warp's own shared memory (16-byte pieces XOR-swizzled by the row: no bank conflicts on either side), from where a row
// is written in whole 32- or 64-byte pieces.
// `drained` is the leader's barrier for the accumulator: the warp arrives on it as soon as its last values are in
// registers.
template <int MODE>
__device__ __forceinline__ void drain_transposed(const GroupedGemm& g, const TcProblem& pb, uint32_t taddr, int rank,
                                                 int q, int h, int lane, uint8_t* stage, int chunk, int split, bool shared, int row0,
                                                 int rows, const float* scale, uint32_t drained) {
  constexpr int kStep = 32 * (kPairEpilogueWarps / 4);
  const uint32_t stage_s = smem_u32(stage);
  auto release = [&]() {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_publish_cluster(drained);
  };
  if (32 * h >= rows) {
    release();
    return;
  }
  if (MODE == kGemmExpertGateUp) {
    // lanes 0-15 of the quarter are gate columns, lanes 16-31 the up columns of the same sixteen outputs
    __nv_bfloat16* dst = (shared ? pb.shared.c : g.c) + static_cast<size_t>(row0) * g.ldc + chunk * (kPairN / 2) + rank * 64 + 16 * q;
#pragma unroll 1
    for (int c0 = 32 * h; c0 < rows; c0 += kStep) {
      uint32_t gr[16], ur[16];
      tmem_ld_16x32(taddr + c0, gr);
      tmem_ld_16x32(taddr + (16u << 16) + c0, ur);
      tmem_ld_wait();
      if (c0 + kStep >= rows) release();
      uint32_t packed[8];         // [2 i + p]: rows 8 i .. 8 i + 7 of the batch, columns 8 p .. 8 p + 7
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float gate = round_bf16(__uint_as_float(gr[2 * i + c]));
          const float up = round_bf16(__uint_as_float(ur[2 * i + c]));
          const float s = det_silu(gate);
          v[c] = __fmul_rn(shared ? s : round_bf16(s), up);
        }
        packed[i] = pack_bf16(v[0], v[1]);
      }
      // 32 bytes per row: block m = 2 i' + p of a call holds rows 8 (2 call + i') .., piece p
#pragma unroll
      for (int call = 0; call < 2; ++call) {
        const int row = 8 * (2 * call + (lane >> 4)) + (lane & 7);
        const int piece = ((lane >> 3) & 1) ^ ((row >> 2) & 1);
        stmatrix_trans4(stage_s + row * 32 + piece * 16, packed[4 * call], packed[4 * call + 1], packed[4 * call + 2],
                        packed[4 * call + 3]);
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = 16 * i + (lane >> 1);
        const uint4 w = *reinterpret_cast<const uint4*>(stage + row * 32 + (((lane & 1) ^ ((row >> 2) & 1)) * 16));
        if (c0 + row < rows)
          *reinterpret_cast<uint4*>(dst + static_cast<size_t>(c0 + row) * g.ldc + (lane & 1) * 8) = w;
      }
      __syncwarp();
    }
  } else if (MODE == kGemmPlainF32) {
    // FP32 as it is: a row's 32 columns are one 128-byte store
    const int col0 = chunk * kPairN + rank * 128 + 32 * q;
    float* dst = g.c_f32 + (static_cast<size_t>(split) * g.dense_rows + row0) * g.ldc + col0 + lane;
#pragma unroll 1
    for (int c0 = 32 * h; c0 < rows; c0 += kStep) {
      uint32_t r[32];
      tmem_ld32(taddr + c0, r);
      tmem_ld_wait();
      if (c0 + kStep >= rows) release();
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (c0 + j < rows && col0 + lane < pb.n_valid) dst[static_cast<size_t>(c0 + j) * g.ldc] = __uint_as_float(r[j]);
      }
    }
  } else {
    const int col0 = chunk * kPairN + rank * 128 + 32 * q;
    __nv_bfloat16* dst = (MODE == kGemmExpertDown && shared ? pb.shared.c : g.c) + static_cast<size_t>(row0) * g.ldc + col0;
    const bool piece_ok = col0 + 8 * (lane & 3) < pb.n_valid;
#pragma unroll
    for (int b = 0; b < kPairRows / kStep; ++b) {
      const int c0 = 32 * h + kStep * b;
      if (c0 < rows) {
        uint32_t r[32];           // [16 half + 4 i + 2 p + c]: column 16 half + 8 p + lane / 4, row 8 i + 2 (lane % 4) + c
        tmem_ld_16x32(taddr + c0, r);
        tmem_ld_16x32(taddr + (16u << 16) + c0, r + 16);
        tmem_ld_wait();
        if (c0 + kStep >= rows) release();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float s0 = 1.0f, s1 = 1.0f;
          if (MODE == kGemmExpertDown) {
            s0 = __shfl_sync(0xffffffffu, scale[b], 8 * i + 2 * (lane & 3));
            s1 = __shfl_sync(0xffffffffu, scale[b], 8 * i + 2 * (lane & 3) + 1);
          }
          uint32_t packed[4];     // columns 8 m .. 8 m + 7 of rows 8 i .. 8 i + 7
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            float lo = __uint_as_float(r[16 * (m >> 1) + 4 * i + 2 * (m & 1)]);
            float hi = __uint_as_float(r[16 * (m >> 1) + 4 * i + 2 * (m & 1) + 1]);
            if (MODE == kGemmExpertDown) {
              lo = __fmul_rn(shared ? round_bf16(lo) : lo, s0);
              hi = __fmul_rn(shared ? round_bf16(hi) : hi, s1);
            }
            packed[m] = pack_bf16(lo, hi);
          }
          const int row = 8 * i + (lane & 7);
          stmatrix_trans4(stage_s + row * 64 + (((lane >> 3) ^ ((row >> 1) & 3)) * 16), packed[0], packed[1], packed[2], packed[3]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = 8 * i + (lane >> 2);
          const uint4 w = *reinterpret_cast<const uint4*>(stage + row * 64 + (((lane & 3) ^ ((row >> 1) & 3)) * 16));
          if (c0 + row < rows && piece_ok)
            *reinterpret_cast<uint4*>(dst + static_cast<size_t>(c0 + row) * g.ldc + (lane & 3) * 8) = w;
        }
        __syncwarp();
      }
    }
  }
}

// Where the rows of A come from: they lie in the order of the plan already; by token index through TMA gathers; or by token
// index through cp.async.
enum RowFeed { kRowsInOrder = 0, kRowsGathered = 1, kRowsFetched = 2 };

template <int MODE, int kFeed>
__global__ void __launch_bounds__(kPairThreads, 1)
grouped_gemm_pair_kernel(const __grid_constant__ TcPairMaps maps, const TcProblem pb) {
  static_assert(MODE != kGemmSharedGateUp && MODE != kGemmSharedDown, "the shared expert runs inside the expert modes");
  constexpr bool kGather = kFeed == kRowsGathered;
  constexpr bool kFetch = kFeed == kRowsFetched;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kStages2 * kStage2Bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages2 + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kStages2 + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kStages2 + 2 + b); };
  uint8_t* tail = smem_gen + kStages2 * kStage2Bytes + 8 * (2 * kStages2 + 4);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);
  volatile int* issued_stages = reinterpret_cast<volatile int*>(tail + 16);      // by the producer and the two gather warps
  const uint32_t drain_bar = smem_u32(tail + 32);
  const uint32_t rows_bar0 = smem_u32(tail + 40);
  auto rows_bar = [&](int s) { return rows_bar0 + 8u * s; };
  uint8_t* store_stage = smem_gen + kStages2 * kStage2Bytes + kTc2BarrierBytes;
  uint8_t* gather_tables = store_stage + kPairEpilogueWarps * kStoreStage2Bytes;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // known to be the same in all lanes
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0: leader of the pair
  const bool leader = rank == 0;
  const GroupedGemm& g = pb.g;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages2; ++s) {
      mbar_init(full_bar(s), kFetch ? 2 : 1);
      mbar_init(empty_bar(s), 1);
      if (kFetch) mbar_init(rows_bar(s), kGatherThreads);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), 2 * kPairEpilogueWarps);
    }
    mbar_init(drain_bar, 1);
    for (int i = 0; i < 3; ++i) issued_stages[i] = 0;
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  if (warp == 2) tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemColumns);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // both blocks' barriers exist before either signals the other's
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  pdl_enter();

  constexpr bool kDense = MODE == kGemmPlain || MODE == kGemmPlainF32;
  const int n_tiles = kDense ? (g.dense_rows + pb.dense_tile - 1) / pb.dense_tile : pb.shared_tiles + *g.tile_count;
  // as in the one-SM kernel; the leader samples the status for the pair
  volatile int* poison_slot = abort_flag + 1;
  if (threadIdx.x == 0 && leader) {
    const int seen = *reinterpret_cast<volatile const int*>(pb.status);
    *poison_slot = seen;
    asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(map_to_rank(smem_u32(const_cast<int*>(poison_slot)), 1)), "r"(seen) : "memory");
  }
  __syncthreads();
  cluster_sync_all();
  const bool poisoned = *poison_slot != 0;
  constexpr bool kSplit = MODE == kGemmPlainF32;
  const int unit_chunks = kSplit ? pb.n_chunks * pb.k_splits : pb.n_chunks;
  const int total_units = poisoned ? 0 : n_tiles * unit_chunks;
  const int n_pairs = gridDim.x >> 1;
  const int pair = blockIdx.x >> 1;
  const int k_blocks = g.k / kBK / (kSplit ? pb.k_splits : 1);

  // unit -> chunk of 256 weight rows, expert (-1: the shared expert, whose tiles come first), first row and number of
  // rows (1 .. 256) of the tile.  Every role asks for
  // the unit after the one it works on (or later), so that these loads, and in the epilogue the two that follow from
  // them, are never waited for between two units: in the down product, whose units are eight stages long, they cost
  // half of a unit's time.
  struct Unit {
    int chunk, expert, row0, rows, split;
  };
  auto describe = [&](int unit) {
    Unit u{0, 0, 0, 0, 0};
    if (unit >= total_units) return u;
    if (kDense) {
      // eight row tiles x all chunks at a time: the pairs that run together then share both operands in L2
      const int band = unit / (kPlainBand * unit_chunks);
      const int height = min(kPlainBand, n_tiles - band * kPlainBand);
      const int within = unit - band * kPlainBand * unit_chunks;
      u.chunk = within / height;
      u.row0 = (band * kPlainBand + within - u.chunk * height) * pb.dense_tile;
      u.rows = min(pb.dense_tile, g.dense_rows - u.row0);
      if (kSplit) {
        u.split = u.chunk / pb.n_chunks;
        u.chunk -= u.split * pb.n_chunks;
      }
    } else {
      int tile = unit / pb.n_chunks;
      u.chunk = unit - tile * pb.n_chunks;
      if (tile < pb.shared_tiles) {
        u.expert = -1;
        u.row0 = tile * pb.dense_tile;
        u.rows = min(pb.dense_tile, pb.shared.rows - u.row0);
      } else {
        tile -= pb.shared_tiles;
        u.expert = g.tile_expert[tile] - g.expert_base;
        u.row0 = g.tile_row0[tile];
        u.rows = g.tile_rows[tile];
      }
    }
    return u;
  };
  // Rows that lie one after the other all the same -- the shared expert's, in the input -- come by tile loads: from the
  // gather warps (which then have a box of 16 rows each at least), or from the warp that loads the weights.
  auto tiled = [&](const Unit& u) { return u.rows > 32 && u.expert < 0; };
  auto fetched = [&](const Unit& u) { return kFetch && u.expert >= 0; };
  // a wait ran out in this warp (or it saw the flag of one that did): both blocks of the pair stop
  auto timeout = [&]() {
    if (lane == 0) {
      atomicCAS(pb.status, 0, kStatusTimeoutMbarrier);
      asm volatile("st.shared::cluster.u32 [%0], %1;"
                   :: "r"(map_to_rank(smem_u32(const_cast<int*>(abort_flag)), rank ^ 1u)), "r"(kStatusTimeoutMbarrier) : "memory");
    }
  };

  if (warp == 0) {
    // ------------------------------ TMA producer (both blocks) -----------------
    const uint32_t leader_full0 = map_to_rank(full_bar(0), 0);
    const uint64_t stream_policy = policy_stream();
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool alive = true;
    Unit next = describe(pair);
    for (int unit = pair; unit < total_units && alive; unit += n_pairs) {
      const Unit u = next;
      next = describe(unit + n_pairs);
      const bool shared = !kDense && u.expert < 0;
      const int half = pair_width(u.rows) / 2;      // a multiple of 16
      const int my_row0 = u.row0 + static_cast<int>(rank) * half;
      const int w_row = u.expert * pb.b_rows_per_expert + u.chunk * kPairN + static_cast<int>(rank) * 128;
      // what both blocks fetch for a stage: weights, and the tile's rows (gathered: in fours per block)
      uint32_t stage_bytes = 2 * (kStage2ABytes + half * kBK * 2);
      if (kGather && !tiled(u)) stage_bytes = 2 * kStage2ABytes + (gather_fours(min(half, u.rows)) + gather_fours(u.rows - half)) * (4 * kBK * 2);
      if (fetched(u)) stage_bytes = 2 * kStage2ABytes;
      const int k_first = kSplit ? u.split * k_blocks * kBK : 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(empty_bar(stage), phase ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        if (elect_one()) {
          const uint32_t w_dst = smem_base + stage * kStage2Bytes;
          const uint32_t leader_full = leader_full0 + 8u * stage;
          if (leader) mbar_arrive_expect_tx(full_bar(stage), stage_bytes);
          if (MODE == kGemmExpertGateUp && shared) {
            // two tensors: the interleaving of the 5-D view, sixteen rows at a time
#pragma unroll
            for (int i = 0; i < 8; ++i)
              tma_load_2d_pair(w_dst + i * (16 * kBK * 2), &maps.shared_w[i & 1], kb * kBK,
                               u.chunk * (kPairN / 2) + static_cast<int>(rank) * 64 + 16 * (i >> 1), leader_full);
          } else if (MODE == kGemmExpertGateUp)
            tma_load_5d_pair(w_dst, &maps.w, kb * kBK, u.chunk * 8 + static_cast<int>(rank) * 4, u.expert, leader_full, stream_policy);
          else if (MODE == kGemmExpertDown && shared)
            tma_load_2d_pair(w_dst, &maps.shared_w[0], kb * kBK, u.chunk * kPairN + static_cast<int>(rank) * 128, leader_full);
          else if (MODE == kGemmExpertDown)
            tma_load_2d_pair_stream(w_dst, &maps.w, kb * kBK, w_row, leader_full, stream_policy);
          else
            tma_load_2d_pair(w_dst, &maps.w, k_first + kb * kBK, w_row, leader_full);
          if (!kGather && !fetched(u)) {
            int done = 0;
#pragma unroll
            for (int b = 3; b >= 0; --b) {
              const int size = 16 << b;
              if (half & size) {
                tma_load_2d_pair(w_dst + kStage2ABytes + done * (kBK * 2), shared ? &maps.shared_rows[b] : &maps.rows[b],
                                 k_first + kb * kBK, my_row0 + done, leader_full);
                done += size;
              }
            }
          }
        }
        __syncwarp();
        ++issued;
        if (++stage == kStages2) { stage = 0; phase ^= 1u; }
      }
    }
    if (lane == 0) issued_stages[0] = issued;
  } else if (kGather && (warp == 2 || warp == 3)) {
    // ------------------------------ row gather (both blocks) -------------------
    // Rows by token index, four per TMA instruction (tile::gather4, a box of one row), the two warps in turn; those of a
    // tile whose rows lie in order (tiled) by tile loads, one part of the block's half per warp.  Only rows that exist are
    // gathered, the last group filled up with repeats; what a stage holds beyond them ends in accumulator columns that
    // nobody reads.  Each warp fetches at least one group per stage, an unneeded one if the tile has no row for it: a stage
    // then always waits for both, so that neither can fall behind the ring or run ahead of it by a whole round, which a
    // barrier's parity would not tell.  (One warp for all groups, or the warp that loads the weights, is slower: 456 against
    // 380 us per layer at 2048 tokens.)  Why tall tiles are not gathered: 256 rows are 1440 cycles of gather4 a stage against
    // 512 of tensor time.
    // The tile's token indices wait in shared memory, one private copy per warp.
    int4* table = reinterpret_cast<int4*>(gather_tables + (warp - 2) * kGatherTableBytes);
    const uint32_t leader_full0 = map_to_rank(full_bar(0), 0);
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool alive = true;
    // two units ahead: description; one unit ahead: token indices
    auto tokens = [&](const Unit& u) {
      const int half = pair_width(u.rows) / 2;
      const int mine = max(0, min(half, u.rows - static_cast<int>(rank) * half));
      int4 t = make_int4(0, 0, 0, 0);
      if (mine > 0 && lane < gather_fours(mine)) {
        const int first = u.row0 + static_cast<int>(rank) * half;
        auto flat = [&](int r) { return u.expert < 0 ? (first + r) << 3 : g.sorted_rows[first + r]; };
        t.x = flat(min(4 * lane, mine - 1));
        t.y = flat(min(4 * lane + 1, mine - 1));
        t.z = flat(min(4 * lane + 2, mine - 1));
        t.w = flat(min(4 * lane + 3, mine - 1));
      }
      return t;
    };
    Unit next = describe(pair), later = describe(pair + n_pairs);
    int4 next_tokens = tokens(next);
    for (int unit = pair; unit < total_units && alive; unit += n_pairs) {
      const Unit u = next;
      const int4 t4 = next_tokens;
      next = later;
      next_tokens = tokens(next);
      later = describe(unit + 2 * n_pairs);
      const int half = pair_width(u.rows) / 2;
      const bool by_tile = tiled(u);
      // boxes of 16 rows of this block's half: the first warp takes the larger part
      const int my_boxes = (half / 16 + 3 - warp) / 2;
      const int my_first = warp == 2 ? 0 : half - 16 * my_boxes;
      const int fours = gather_fours(min(half, u.rows - static_cast<int>(rank) * half));
      __syncwarp();
      table[lane] = make_int4(t4.x >> 3, t4.y >> 3, t4.z >> 3, t4.w >> 3);
      __syncwarp();
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(empty_bar(stage), phase ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        const uint32_t dst = smem_base + stage * kStage2Bytes + kStage2ABytes;
        const uint32_t leader_full = leader_full0 + 8u * stage;
        if (elect_one()) {
          if (by_tile) {
            int done = my_first;
#pragma unroll
            for (int b = 2; b >= 0; --b) {
              if (my_boxes & (1 << b)) {
                tma_load_2d_pair(dst + done * (kBK * 2), &maps.shared_rows[b], kb * kBK,
                                 u.row0 + static_cast<int>(rank) * half + done, leader_full);
                done += 16 << b;
              }
            }
          } else {
#pragma unroll 4
            for (int i = warp - 2; i < fours; i += 2) {
              const int4 t = table[i];
              tma_gather4_pair(dst + i * (4 * kBK * 2), &maps.one_row, kb * kBK, t.x, t.y, t.z, t.w, leader_full);
            }
          }
        }
        __syncwarp();
        ++issued;
        if (++stage == kStages2) { stage = 0; phase ^= 1u; }
      }
    }
    if (lane == 0) issued_stages[warp - 1] = issued;
  } else if (kFetch && (warp == 2 || warp == 3)) {
    // ------------------------------ row fetch (both blocks) --------------------
    // Rows by token index with cp.async, 16 bytes per thread: eight threads take the 64 columns of a row, the two warps groups
    // of four rows in turn.  The copies arrive on the block's own barrier by themselves; nobody waits for them here.  Moving
    // a stage's 128 rows takes the two warps no longer than the tensor cores need for them (512 cycles; 1440 by TMA gathers).
    // Only rows that exist are fetched; what a stage holds beyond them ends in accumulator columns that nobody reads.  Every
    // thread arrives once per stage, whatever it has fetched: a warp left out of a stage could fall behind by a whole round
    // of the ring, which a barrier's parity would not tell.
    const int sub = lane >> 3, piece = lane & 7;
    const int in_eight = 4 * (warp - 2) + sub;                   // row within every eight of this block's half
    const uint32_t dst0 = smem_base + kStage2ABytes + in_eight * 128 + ((piece ^ in_eight) << 4);
    const uint8_t* src0 = reinterpret_cast<const uint8_t*>(g.gather_src) + piece * 16;
    const uint32_t row_bytes = static_cast<uint32_t>(g.lda) * 2;
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    auto mine_of = [&](const Unit& u) { return max(0, min(pair_width(u.rows) / 2, u.rows - static_cast<int>(rank) * (pair_width(u.rows) / 2))); };
    // one unit ahead: token indices (-1: not a row of this tile)
    auto tokens = [&](const Unit& u, int* t) {
      const int mine = fetched(u) ? mine_of(u) : 0;
      const int first = u.row0 + static_cast<int>(rank) * (pair_width(u.rows) / 2);
#pragma unroll
      for (int j = 0; j < 16; ++j) t[j] = 8 * j + in_eight < mine ? g.sorted_rows[first + 8 * j + in_eight] >> 3 : -1;
    };
    Unit next = describe(pair), later = describe(pair + n_pairs);
    int token[16];
    tokens(next, token);
    for (int unit = pair; unit < total_units && alive; unit += n_pairs) {
      const Unit u = next;
      const uint8_t* src[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) src[j] = token[j] >= 0 ? src0 + static_cast<size_t>(token[j]) * row_bytes : nullptr;
      next = later;
      tokens(next, token);
      later = describe(unit + 2 * n_pairs);
      const int eights = fetched(u) ? (mine_of(u) + 7) / 8 : 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(empty_bar(stage), phase ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        const uint32_t dst = dst0 + stage * kStage2Bytes;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j < eights && src[j] != nullptr) cp_async_16(dst + j * 1024, src[j] + kb * (kBK * 2));
        }
        cp_async_arrive_noinc(rows_bar(stage));
        if (++stage == kStages2) { stage = 0; phase ^= 1u; }
      }
    }
    cp_async_wait_all();
  } else if (kFetch && warp == 1 && !leader) {
    // ------------------------------ relay (second block) -----------------------
    // Tells the leader, whose MMAs read this block's rows too, that a stage's rows have landed: acquired from this block's
    // threads by the wait, handed to the async proxy by the fence, and published to the leader by the arrival.
    const uint32_t leader_full0 = map_to_rank(full_bar(0), 0);
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    for (int unit = pair; unit < total_units && alive; unit += n_pairs) {
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_warp(rows_bar(stage), phase, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) mbar_publish_cluster(leader_full0 + 8u * stage);
        if (++stage == kStages2) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (leader) {
      // ------------------------------ MMA issuer (leader) ------------------------
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      bool alive = true;
      Unit next = describe(pair);
      for (int unit = pair; unit < total_units && alive; unit += n_pairs, ++local) {
        const uint32_t idesc = pair_instr_desc(pair_width(next.rows));
        next = describe(unit + n_pairs);
        const int buf = local & 1;
        const uint32_t use = static_cast<uint32_t>(local >> 1);
        if (!mbar_wait_bounded_warp<true>(tempty_bar(buf), (use & 1u) ^ 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buf * kPairRows);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait_bounded_warp<kFetch>(full_bar(stage), phase, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
          if (kFetch) {
            if (!mbar_wait_bounded_warp(rows_bar(stage), phase, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
            fence_async_proxy();                // rows of both blocks: written by cp.async, read by the tensor cores
          }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t w_addr = smem_base + stage * kStage2Bytes;
            const uint64_t wdesc = smem_desc_k_major_sw128(w_addr);
            const uint64_t rdesc = smem_desc_k_major_sw128(w_addr + kStage2ABytes);
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k) {
              umma_bf16_pair(tmem_d, wdesc + static_cast<uint64_t>(k * 2), rdesc + static_cast<uint64_t>(k * 2),
                             idesc, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit_pair(empty_bar(stage));
            if (kb + 1 == k_blocks) umma_commit_pair(tfull_bar(buf));
          }
          __syncwarp();
          if (++stage == kStages2) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------ epilogue (both blocks) ---------------------
    const int q = (warp - 4) & 3;                  // TMEM lanes 32 q .. 32 q + 31
    const int h = (warp - 4) >> 2;                 // which of the tile's 32-row batches
    uint8_t* my_stage = store_stage + (warp - 4) * kStoreStage2Bytes;
    int local = 0;
    bool alive = true;
    constexpr int kSharedRow = 1 << 30;            // flat index of row 0 of the shared expert
    // three units ahead: description; two: the rows' flat indices; one: their scales
    auto flats = [&](const Unit& u, int* flat) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int r = 32 * h + 128 * b + lane;
        flat[b] = -1;
        if (MODE == kGemmExpertDown && r < u.rows) flat[b] = u.expert < 0 ? kSharedRow + u.row0 + r : g.sorted_rows[u.row0 + r];
      }
    };
    auto scales = [&](const int* flat, float* scale) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        scale[b] = 0.0f;
        if (MODE == kGemmExpertDown && flat[b] >= 0)
          scale[b] = flat[b] >= kSharedRow ? pb.shared.row_scale[flat[b] - kSharedRow] : g.row_scale[flat[b]];
      }
    };
    Unit u1 = describe(pair), u2 = describe(pair + n_pairs), u3 = describe(pair + 2 * n_pairs);
    int flat[2];
    float scale[2];
    flats(u1, flat);
    scales(flat, scale);
    flats(u2, flat);
    for (int unit = pair; unit < total_units && alive; unit += n_pairs, ++local) {
      const Unit u = u1;
      const float scale_now[2] = {scale[0], scale[1]};
      scales(flat, scale);
      flats(u3, flat);
      u1 = u2;
      u2 = u3;
      u3 = describe(unit + 3 * n_pairs);
      const int buf = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      if (!mbar_wait_bounded_warp(tfull_bar(buf), use & 1u, abort_flag, pb.wait_limit_ns)) { alive = false; timeout(); break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * kPairRows);
      drain_transposed<MODE>(g, pb, taddr, static_cast<int>(rank), q, h, lane, my_stage, u.chunk, u.split, u.expert < 0, u.row0,
                             u.rows, scale_now, map_to_rank(tempty_bar(buf), 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // neither block leaves while the other may still signal it or read its memory
  if (*abort_flag != 0) {
    // Raised in both blocks, before the barrier above.  Nothing is issued any more; what is under way has to land before
    // shared memory and tensor memory are given up: the MMAs (a last commit, to both blocks) and the loads of the last
    // round of the ring (the leader's full barriers).  A stage that not every loader got to (or, with fetched rows, the
    // relay) never completes; its wait gives the copies that were issued the whole budget.  Fetched rows have been waited
    // for by the warps that fetch.
    volatile int ignore = 0;
    if (warp == 1 && leader && elect_one()) umma_commit_pair(drain_bar);
    if (threadIdx.x == 0) {
      mbar_wait_bounded(drain_bar, 0, &ignore);
      if (leader) {
        int last = 0;
        for (int i = 0; i < 3; ++i) {
          int theirs;
          asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(theirs) : "r"(map_to_rank(smem_u32(const_cast<int*>(issued_stages + i)), 1)) : "memory");
          last = max(last, max(theirs, static_cast<int>(issued_stages[i])));
        }
        for (int j = max(0, last - kStages2); j < last; ++j) {
          if (!mbar_wait_bounded(full_bar(j % kStages2), (j / kStages2) & 1, &ignore)) break;
        }
      }
    }
    __syncthreads();
    cluster_sync_all();
  }
  if (warp == 2) tmem_dealloc_pair(tmem_base, kTmemColumns);
}

// ---- host side --------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (fn == nullptr) {
    void* pointer = nullptr;
    cudaDriverEntryPointQueryResult query;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &pointer, cudaEnableDefault, &query) == cudaSuccess &&
        query == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(pointer);
    }
  }
  return fn;
}

// Descriptors of BF16 tensors, 128-byte swizzle.  A descriptor depends only on the base address and these numbers,
// and a layer's weights and the workspace keep their addresses from bind to release, so the encoded descriptors are
// kept: a prefill layer asks for about twenty of them per call, always the same ones.
struct MapKey {
  const void* base;
  uint64_t rows, cols, pitch;
  uint32_t box_rows;        // rows of the tile; 0: the 5-D view of make_gate_up_map
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && cols == o.cols && pitch == o.pitch && box_rows == o.box_rows;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    uint64_t h = reinterpret_cast<uint64_t>(k.base) * 0x9e3779b97f4a7c15ull;
    h ^= (k.rows + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2));
    h ^= (k.cols * 31 + k.pitch * 131 + k.box_rows + (h << 6) + (h >> 2));
    return static_cast<size_t>(h);
  }
};

bool cached_map(CUtensorMap* map, const MapKey& key, cuuint32_t rank, const cuuint64_t* dims, const cuuint64_t* strides,
                const cuuint32_t* box) {
  static std::mutex mutex;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  {
    std::lock_guard<std::mutex> lock(mutex);
    const auto hit = cache.find(key);
    if (hit != cache.end()) { *map = hit->second; return true; }
  }
  PFN_cuTensorMapEncodeTiled_v12000 encode = encode_fn();
  if (encode == nullptr) return false;
  const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(key.base), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  std::lock_guard<std::mutex> lock(mutex);
  if (cache.size() >= 8192) cache.clear();      // a host that keeps binding new tensors: start over rather than grow
  cache.emplace(key, *map);
  return true;
}

// [rows, cols] row-major, box of 64 columns x box_rows rows
bool make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_elems,
              uint32_t box_rows = kBM) {
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {pitch_elems * 2};
  const cuuint32_t box[2] = {kBK, box_rows};
  return cached_map(map, MapKey{base, rows, cols, pitch_elems, box_rows}, 2, dims, strides, box);
}

// [experts, 2 (gate, up), n, k] seen as (k, 16 rows, gate / up, groups of 16 rows, expert); the box takes 64 columns of
// four groups, gate and up: 128 rows that arrive as 16 gate rows, the 16 up rows that belong to them, 16 gate rows, ...,
// so that one warp of the transposed epilogue holds both halves of its sixteen outputs.
bool make_gate_up_map(CUtensorMap* map, const void* base, uint64_t experts, uint64_t n, uint64_t k) {
  const cuuint64_t dims[5] = {k, 16, 2, n / 16, experts};
  const cuuint64_t strides[4] = {k * 2, n * k * 2, 16 * k * 2, 2 * n * k * 2};
  const cuuint32_t box[5] = {kBK, 16, 2, 4, 1};
  return cached_map(map, MapKey{base, experts * 2 * n, k, k, 0}, 5, dims, strides, box);
}

template <int MODE, bool kGather = false>
cudaError_t launch_mode(const TcMaps& maps, const TcProblem& pb, int grid, cudaStream_t stream) {
  const cudaError_t e = opt_in_dynamic_smem<grouped_gemm_tc_kernel<MODE, kGather>>(kTcSmemBytes);
  if (e != cudaSuccess) return e;
  return launch_pdl(grouped_gemm_tc_kernel<MODE, kGather>, dim3(grid), dim3(kTcThreads), kTcSmemBytes, stream, maps, pb);
}

// two-SM form: clusters of two blocks, launched like launch_pdl
template <int MODE, int kFeed>
cudaError_t launch_pair_mode(const TcPairMaps& maps, const TcProblem& pb, int grid, cudaStream_t stream) {
  const cudaError_t e = opt_in_dynamic_smem<grouped_gemm_pair_kernel<MODE, kFeed>>(kTc2SmemBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(grid & ~1);
  config.blockDim = dim3(kPairThreads);
  config.dynamicSmemBytes = kTc2SmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = t_pdl_relaxed ? 1 : 0;
  config.attrs = attributes;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, grouped_gemm_pair_kernel<MODE, kFeed>, maps, pb);
}

// Rows per tile of a dense product over `chunks` chunks of 256 columns: the height whose last wave of units wastes
// least.  A unit's time goes with its rows, in steps of 32, but not below what issuing a stage costs (about 128 rows);
// smaller tiles then only help to spread a product over the chip.  Router logits (a run of K is a chunk here: four and two)
// at 1024 / 8192 rows: 64- / 224-row tiles.
int dense_tile_rows(int rows, int chunks, int pairs) {
  int best = kPairRows;
  long long best_cost = -1;
  for (int height = kPairRows; height >= 32; height -= 32) {
    const long long units = static_cast<long long>((rows + height - 1) / height) * chunks;
    const long long cost = (units + pairs - 1) / pairs * ((height > 128 ? height : 128) + 16);
    if (best_cost < 0 || cost < best_cost || (cost == best_cost && units <= pairs)) {
      best = height;
      best_cost = cost;
    }
  }
  return best;
}

cudaError_t launch_pair(GemmMode mode, const GroupedGemm& g, const TcExtra& extra, TcProblem pb, cudaStream_t stream) {
  TcPairMaps maps;
  const uint64_t experts = static_cast<uint64_t>(extra.experts_in_b);
  const bool fetch = mode == kGemmExpertGateUp && g.gather_src != nullptr && extra.fetch;
  const bool gather = mode == kGemmExpertGateUp && g.gather_src != nullptr && !fetch;
  bool ok = true;
  if (mode == kGemmExpertGateUp) {
    pb.n_chunks = g.n / (kPairN / 2);
    ok = make_gate_up_map(&maps.w, g.b0, experts, g.n, g.k);
  } else {
    pb.n_chunks = (g.n + kPairN - 1) / kPairN;
    pb.b_rows_per_expert = g.n;
    ok = make_map(&maps.w, g.b0, (mode == kGemmExpertDown ? experts : 1) * static_cast<uint64_t>(g.n), g.k, g.k);
  }
  if (ok && gather) ok = make_map(&maps.one_row, g.gather_src, extra.a_rows, g.k, g.lda, 1u);
  for (int b = 0; ok && !gather && !fetch && b < 4; ++b) ok = make_map(&maps.rows[b], g.a, extra.a_rows, g.k, g.lda, 16u << b);
  const SharedProblem& shared = extra.shared;
  if (mode == kGemmPlain || mode == kGemmPlainF32) {
    pb.k_splits = mode == kGemmPlainF32 ? extra.k_splits : 1;
    if (pb.k_splits < 1 || g.k / kBK % pb.k_splits != 0) return cudaErrorInvalidValue;
    pb.dense_tile = dense_tile_rows(g.dense_rows, pb.n_chunks * pb.k_splits, extra.sm_count / 2);
  } else if (shared.rows > 0) {
    // the shared expert's rows in equal tiles
    const int tiles = (shared.rows + kPairRows - 1) / kPairRows;
    pb.dense_tile = pair_width((shared.rows + tiles - 1) / tiles);
    pb.shared_tiles = tiles;
    pb.shared = shared;
    if (mode == kGemmExpertGateUp) {
      ok = ok && make_map(&maps.shared_w[0], shared.b0, g.n, g.k, g.k, 16) && make_map(&maps.shared_w[1], shared.b1, g.n, g.k, g.k, 16);
    } else {
      ok = ok && make_map(&maps.shared_w[0], shared.b0, g.n, g.k, g.k);
    }
    for (int b = 0; ok && b < (gather ? 3 : 4); ++b)
      ok = make_map(&maps.shared_rows[b], shared.a, shared.rows, g.k, g.k, 16u << b);
  }
  if (!ok) return cudaErrorNotSupported;
  if (mode == kGemmExpertGateUp)
    return fetch    ? launch_pair_mode<kGemmExpertGateUp, kRowsFetched>(maps, pb, extra.sm_count, stream)
           : gather ? launch_pair_mode<kGemmExpertGateUp, kRowsGathered>(maps, pb, extra.sm_count, stream)
                    : launch_pair_mode<kGemmExpertGateUp, kRowsInOrder>(maps, pb, extra.sm_count, stream);
  if (mode == kGemmExpertDown) return launch_pair_mode<kGemmExpertDown, kRowsInOrder>(maps, pb, extra.sm_count, stream);
  if (mode == kGemmPlain) return launch_pair_mode<kGemmPlain, kRowsInOrder>(maps, pb, extra.sm_count, stream);
  if (mode == kGemmPlainF32) return launch_pair_mode<kGemmPlainF32, kRowsInOrder>(maps, pb, extra.sm_count, stream);
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_grouped_gemm_tc(GemmMode mode, const GroupedGemm& g, const TcExtra& extra,
                                   cudaStream_t stream) {
  if (g.max_tiles <= 0) return cudaSuccess;
  if (g.k % kBK != 0 || extra.status == nullptr) return cudaErrorInvalidValue;
  const bool gather = (mode == kGemmExpertGateUp && g.gather_src != nullptr);
  if (gather && g.sorted_rows == nullptr) return cudaErrorInvalidValue;
  TcMaps maps{};
  TcProblem pb{};
  pb.g = g;
  pb.status = extra.status;
  pb.wait_limit_ns = extra.wait_limit_ns;
  pb.n_valid = g.n;
  if (extra.pair) return launch_pair(mode, g, extra, pb, stream);
  const uint64_t experts = static_cast<uint64_t>(extra.experts_in_b);
  // (gathered rows are copied one by one, without a descriptor)
  bool ok = gather || make_map(&maps.a, g.a, extra.a_rows, static_cast<uint64_t>(g.k), static_cast<uint64_t>(g.lda));
  if (mode == kGemmExpertGateUp) {
    pb.n_chunks = g.n / (kBN / 2);
    pb.b_rows_per_expert = 2 * g.n;
    pb.up_row_offset = g.n;
    ok = ok && make_map(&maps.b0, g.b0, experts * 2 * g.n, g.k, g.k);
    maps.b1 = maps.b0;
  } else if (mode == kGemmSharedGateUp) {
    pb.n_chunks = g.n / (kBN / 2);
    pb.b_rows_per_expert = 0;
    pb.up_row_offset = 0;
    ok = ok && make_map(&maps.b0, g.b0, g.n, g.k, g.k) && make_map(&maps.b1, g.b1, g.n, g.k, g.k);
  } else {
    pb.n_chunks = (g.n + kBN - 1) / kBN;
    pb.b_rows_per_expert = (mode == kGemmExpertDown) ? g.n : 0;
    pb.up_row_offset = 0;
    ok = ok && make_map(&maps.b0, g.b0, (mode == kGemmExpertDown ? experts : 1) * static_cast<uint64_t>(g.n), g.k, g.k);
    maps.b1 = maps.b0;
  }
  if (!ok) return cudaErrorNotSupported;
  const int grid = extra.sm_count;
  switch (mode) {
    case kGemmExpertGateUp:
      return gather ? launch_mode<kGemmExpertGateUp, true>(maps, pb, grid, stream)
                    : launch_mode<kGemmExpertGateUp>(maps, pb, grid, stream);
    case kGemmSharedGateUp: return launch_mode<kGemmSharedGateUp>(maps, pb, grid, stream);
    case kGemmExpertDown: return launch_mode<kGemmExpertDown>(maps, pb, grid, stream);
    case kGemmSharedDown: return launch_mode<kGemmSharedDown>(maps, pb, grid, stream);
    case kGemmPlain: break;              // two-SM form only
    case kGemmPlainF32: return launch_mode<kGemmPlainF32>(maps, pb, grid, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace aima
