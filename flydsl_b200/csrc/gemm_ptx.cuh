// PTX wrappers, tile constants and the tile walk shared by the tcgen05 grouped-GEMM kernels.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_args.cuh"

namespace flymoe {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 128;

constexpr int kScaleBlock128 = 0;
constexpr int kScalePerToken = 1;

constexpr int kATileBytes = BM * BK;            // 16 KB
constexpr int kBTileBytes = BN * BK;            // 32 KB
constexpr int kAccStages = 2;
constexpr int kTmemCols = 512;
constexpr int kNumThreads = 384;
constexpr int kEpilogueWarps = 8;
constexpr unsigned long long kWaitLimitNs = 4000000000ull;   // 4 s

// ------------------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrive without release ordering: for hand-offs that publish no memory (a TMEM stage whose
// loads have already completed), so the arrive need not wait for this thread's loads in flight.
__device__ __forceinline__ void mbar_arrive_relaxed(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait.  Returns false when the CTA is aborting or the time limit ran out.
// `backoff_ns` > 0 makes a role that has slack sleep between polls instead of competing for
// issue slots with the epilogue warps of its scheduler partition.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int code, unsigned backoff_ns = 0,
                                          unsigned long long limit_ns = kWaitLimitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_timer_ns();
#pragma unroll 1
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (backoff_ns) __nanosleep(backoff_ns);
    if ((it & 0xFF) == 0) {
      if (*abort_flag) return false;
      if (global_timer_ns() - t0 > limit_ns) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}
// One lane of a converged warp.  Code under this predicate is known to run in a single thread, so the descriptors
// and addresses of TMA and tcgen05 instructions stay in uniform registers; under `lane == 0` every one of them is
// moved there first.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// All lanes of a warp wait together.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code,
                                          unsigned backoff_ns = 0) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code, backoff_ns));
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// Routing of the cluster kernel.  Null sorted_ids: identity routing of the dense GEMM -- sorted row r is row r, every
// row block belongs to expert 0, and all row blocks are in use -- no tables to write first.
__device__ __forceinline__ int routed_rows(const GemmArgs& a) {
  const int cap = a.size_expert_ids * a.tile_m;
  return a.sorted_ids != nullptr ? min(__ldg(a.num_valid_ids), cap) : cap;
}
__device__ __forceinline__ int block_expert(const GemmArgs& a, int b) {
  return a.sorted_ids != nullptr ? __ldg(a.sorted_expert_ids + b) : 0;
}
__device__ __forceinline__ int sorted_id(const GemmArgs& a, int r) {
  return a.sorted_ids != nullptr ? __ldg(a.sorted_ids + r) : min(r, a.num_tokens);   // num_tokens: a pad row
}
// Four rows by index (a box of one row, 128 bytes of K each) to four consecutive 128-byte rows of the tile; the
// 128-byte swizzle goes by the shared-memory address, so dst only has to be a multiple of 512 bytes.
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, const int* r) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// Row of the activations that sorted row `first + i` stands for, i = 0..3 (row 0 for pad rows and rows beyond
// `end`: their results are never used).
__device__ __forceinline__ void gather_rows4(const GemmArgs& a, int first, int end, int* rows) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int id = first + i < end ? sorted_id(a, first + i) : a.num_tokens;
    const int tok = id_token(id), slot = id_slot(id);
    const bool valid = tok < a.num_tokens && slot < a.topk;
    rows[i] = !valid ? 0
            : a.a_layout == FLYMOE_ROWS_BY_TOKEN ? tok
            : a.a_layout == FLYMOE_ROWS_BY_SLOT ? slot * a.num_tokens + tok : tok * a.topk + slot;
  }
}
// Per-token scaling, one rule for every kernel: a null table (16-bit operands; each of the two may be null by itself)
// stands for ones.
__device__ __forceinline__ float row_scale(const float* table, long long row) { return table ? __ldg(table + row) : 1.f; }
__device__ __forceinline__ float4 col_scales4(const float* table, const float* at) {
  return table ? __ldg(reinterpret_cast<const float4*>(at)) : make_float4(1.f, 1.f, 1.f, 1.f);
}
__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// KIND: 0 = f8f6f4, 1 = i8, 2 = f16
template <int KIND>
__device__ __forceinline__ void umma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
  if (KIND == 0) umma_f8(d, ad, bd, idesc, accumulate);
  else if (KIND == 1) umma_i8(d, ad, bd, idesc, accumulate);
  else umma_f16(d, ad, bd, idesc, accumulate);
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ unsigned long long pack_f32x2(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
// acc.lo += v0 * c.lo ; acc.hi += v1 * c.hi  (one instruction on sm_100)
__device__ __forceinline__ void ffma2(unsigned long long& acc, uint32_t v0, uint32_t v1, unsigned long long c) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(v0), "r"(v1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(v), "l"(c));
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major, 128-byte-swizzled operand tile: 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= uint64_t((smem_addr >> 4) & 0x3FFF);          // start address
  d |= uint64_t(1) << 16;                            // leading byte offset (unused with swizzle)
  d |= uint64_t((1024 >> 4) & 0x3FFF) << 32;         // stride byte offset
  d |= uint64_t(1) << 46;                            // descriptor version (sm_100)
  d |= uint64_t(2) << 61;                            // SWIZZLE_128B
  return d;
}
// Instruction descriptors, both operands K-major, M=128, N=256:
// kind::f8f6f4 with A=B=e4m3 (format 0) and D=f32 (format 1); kind::i8 with A=B=s8 (format 1) and D=s32 (format 2);
// kind::f16 with A=B=f16 (format 0) or bf16 (format 1) and D=f32.  One instruction covers 32 bytes of K in
// every kind (32 one-byte or 16 two-byte elements), so a 128-byte K block is four instructions in all of them.
constexpr uint32_t kInstrDescShape = (uint32_t(BN >> 3) << 17) | (uint32_t(BM >> 4) << 24);
constexpr uint32_t kInstrDescF8 = (1u << 4) | (0u << 7) | (0u << 10) | kInstrDescShape;
constexpr uint32_t kInstrDescI8 = (2u << 4) | (1u << 7) | (1u << 10) | kInstrDescShape;
constexpr uint32_t kInstrDescF16 = (1u << 4) | (0u << 7) | (0u << 10) | kInstrDescShape;
constexpr uint32_t kInstrDescBF16 = (1u << 4) | (1u << 7) | (1u << 10) | kInstrDescShape;

// Bulk operations from a staging slot to a contiguous global row segment (16-byte aligned, size % 16 == 0).
__device__ __forceinline__ void bulk_reduce_add_bf16(void* g, uint32_t s, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.noftz.bf16 [%0], [%1], %2;"
               ::"l"(g), "r"(s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_reduce_add_f16(void* g, uint32_t s, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.noftz.f16 [%0], [%1], %2;"
               ::"l"(g), "r"(s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_store(void* g, uint32_t s, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(g), "r"(s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void red_add_v4_f32(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// ------------------------------------------------------------------------------ clusters
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_rank(uint32_t bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// Wait whose success also orders the other ranks' shared-memory writes (acquire at cluster scope).
__device__ __forceinline__ uint32_t mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                  int code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const unsigned long long t0 = global_timer_ns();
#pragma unroll 1
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if ((it & 0xFF) == 0) {
      if (*abort_flag) return false;
      if (global_timer_ns() - t0 > kWaitLimitNs) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}
// ------------------------------------------------------------------------------ tiles
struct TileSched {
  int num_mblocks, num_ntiles, total, group_m;
  __device__ __forceinline__ void decode(int t, int& mb, int& n) const {
    const int per_group = group_m * num_ntiles;
    const int bg = t / per_group;
    const int rem = t - bg * per_group;
    const int gs = min(group_m, num_mblocks - bg * group_m);
    n = rem / gs;
    mb = bg * group_m + (rem - n * gs);
  }
};

// Block-wide exclusive scan over THREADS threads: running maximum (from -1) or running sum.
template <bool MAX, int THREADS>
__device__ __forceinline__ int block_scan_excl(int v, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc = MAX ? max(inc, o) : inc + o;
  }
  if (lane == 31) scratch[warp] = inc;
  __syncthreads();
  int before = MAX ? -1 : 0, all = before;
  for (int w = 0; w < THREADS / 32; ++w) {
    if (w == warp) before = all;
    all = MAX ? max(all, scratch[w]) : all + scratch[w];
  }
  const int prev = __shfl_up_sync(0xffffffffu, inc, 1);
  *total = all;
  if (lane == 0) return before;
  return MAX ? max(before, prev) : before + prev;
}
// Row tiles of a launch: an expert's row blocks are contiguous in sorted order, and every `bpt`-th of them starts a
// tile of up to bpt blocks.  table[tile] = first row block | (row blocks - 1) << 12.  Returns the number of tiles; the
// caller synchronises the block before it reads the table.  scratch: two rows of 32 ints.
constexpr int kTileTable = 4096;                 // row blocks the table covers
template <int THREADS>
__device__ __forceinline__ int build_tile_table(const GemmArgs& a, int valid_rows, int bpt, uint16_t* table,
                                                int (*scratch)[32]) {
  const int* ex = a.sorted_expert_ids;
  const int nblk = min((valid_rows + a.tile_m - 1) / a.tile_m, kTileTable);
  const int per = (nblk + THREADS - 1) / THREADS;
  const int b0 = min(int(threadIdx.x) * per, nblk), b1 = min(b0 + per, nblk);
  int run = -1;                                  // last start of an expert's run inside this thread's blocks
  for (int b = b0; b < b1; ++b)
    if (b == 0 || __ldg(ex + b) != __ldg(ex + b - 1)) run = b;
  int unused, total;
  const int run_before = block_scan_excl<true, THREADS>(run, scratch[0], &unused);
  int starts = 0;
  run = run_before;
  for (int b = b0; b < b1; ++b) {
    const int e = __ldg(ex + b);
    if (b == 0 || e != __ldg(ex + b - 1)) run = b;
    if (((b - run) & (bpt - 1)) == 0 && e >= 0 && e < a.experts) ++starts;
  }
  int at = block_scan_excl<false, THREADS>(starts, scratch[1], &total);
  run = run_before;
  for (int b = b0; b < b1; ++b) {
    const int e = __ldg(ex + b);
    if (b == 0 || e != __ldg(ex + b - 1)) run = b;
    if (((b - run) & (bpt - 1)) == 0 && e >= 0 && e < a.experts) {
      int nb = 1;
      while (nb < bpt && b + nb < nblk && __ldg(ex + b + nb) == e) ++nb;
      table[at++] = uint16_t(b | ((nb - 1) << 12));
    }
  }
  return total;
}

// ------------------------------------------------------------------------------ host
// Tensor maps of both operands: boxes of `a_box_rows` rows of A and of `b_box_rows` weight rows, 128 bytes of K wide.
int make_gemm_maps(int stage, const GemmArgs& a, int a_box_rows, int b_box_rows, CUtensorMap* map_a, CUtensorMap* map_b);
// Cluster sizes 1, 2, 4, 8: how many CTAs share a tile's K range, given how many clusters of each size run at once
// (0 = that size cannot run); 1 = the one-CTA-per-tile kernel.
constexpr int kClusterSizes = 4;
int plan_ksplit(int stage, const GemmArgs& a, const int* clusters);
// Fills clusters[1..3] for the current device.
void split_residency(int stage, int scaling, int* clusters);
int launch_gemm_split(int stage, const GemmArgs& a, const CUtensorMap& map_a, const CUtensorMap& map_b, int group_m,
                      int split, cudaStream_t stream);
bool use_pair_kernel(const GemmArgs& a);
int launch_gemm_pair(int stage, const GemmArgs& a, int ctas, cudaStream_t stream);

}  // namespace flymoe
