// q4f16 matmul on the 5th-generation tensor cores (the dispatcher gives it 9 rows and more, and fewer with a long or a
// ragged K): y[M,N] = x[M,K] . decode(Wq,S)^T.
//
// Decode at batches up to 128 is still bound by streaming the weights once, so the roles of a plain GEMM are swapped:
// the MMA's M dimension is 128 WEIGHT rows (A operand), its N dimension are tokens (B operand = x, 16..192 columns).
//
// The A operand lives in TENSOR MEMORY: a dequantiser thread turns the packed words of one row into registers and
// stores them with tcgen05.st; the MMA reads them from there.  Shared memory then carries the packed words and x only
// (no 16 KB of stores and 16 KB of operand reads per 64 k), no proxy fence stands between conversion and MMA, and
// the room goes to the rings.
//
// Work: a tile is 128 weight rows by up to 192 tokens over the whole K (above 128 rows x is cut into equal token
// tiles).  The CTAs of a cluster share tiles: CTA r takes the r-th slice of K of every tile of the cluster's list (tile =
// cluster, cluster + clusters, ...), so the kernel starts once however many tiles there are (a second wave of CTAs
// cost 7 us), and x of a slice stays in shared memory for all tiles where it fits.  The accumulator is double-buffered: the next tile's MMAs run while the epilogue drains this one's.  The
// partial tiles are exchanged by 16-byte stores into the owners' shared memory (owner o of a tile: batch columns
// [o * cw, (o + 1) * cw)) and added up there in rank order: deterministic, no atomics, no scratch in global memory.
//
//   warps 0,2,3 TMA producers: x (two K blocks of {64 k, NB batch rows} per load, 128-byte swizzle), packed weights
//               (256 k per load: whole 128-byte lines of 128 rows, 128-byte swizzle), scales {8 groups = 256 k,
//               128 rows}; the first ring-full of weights is requested during set-up
//   warps 8-23  dequantisers, four groups of 4 warps; a group takes one half (two K blocks) of every second 256-k
//               span and owns one slot of the A ring (its wait -> load -> convert -> store -> arrive chain is
//               latency bound, so it moves 128 k per trip); thread = weight row (= TMEM lane): 8 packed words -> 64 fp16
//               (exact q-7, one HMUL2 by the scale: the reference's rounding) -> 32 columns, twice
//   warp 1      issues tcgen05.mma kind::f16 (M=128, N=NB, K=16), eight per pair of K blocks
//   warps 4-7, 24-27  epilogue: tcgen05.ld -> owners' inboxes -> sum over the K slices -> fp16 stores (or, with one
//               slice, straight to y); two warps per TMEM quadrant share the columns
//
// What bounds it (measured at a batch of 64): 0.56 us per 256-k span and CTA, of which 0.37-0.39 us is the delivery of
// the span's 18 KB (a copy of the kernel without the conversion) and the rest the conversion; the MMAs (45 clocks
// each or less) are hidden.  Before, with A in shared memory, the MMAs issued under a branch on one lane and a grid of
// one tile per CTA, us in a chain over more weights than the L2 holds: M = 64, N = 22016, K = 4096 46.1 -> 20.0; N = 12288
// 23.3 -> 13.0; N = K = 4096 11.0 -> 9.2; N = 4096, K = 11008 18.9 -> 13.8; M = 128, N = 22016 49.5 -> 24.8; M = 16, N = K = 4096
// 9.7 -> 6.9.  With many tokens the SMs' fetches of x from L2 (a tile's x serves 128 weight rows) are the limit, about
// 14 TB/s over all SMs, and at the largest sizes the power cap.  Against the prefill kernel, whose 256-token tiles leave
// SMs idle up to about 1000 tokens: K = 4096, N = 4096 at 129 tokens 44 -> 11.8 us, at 512 45 -> 15.8; N = 3584, K = 8192 at
// 777 84 -> 37; N = 11008 at 2048 164 -> 134-140 (1320-1380 TFLOP/s; 1249-1265 over 0.2 s).
//
// Launched with programmatic dependent launch: set-up and the weight loads run ahead of the previous
// kernel's end; the loads of x and the stores of y wait for it.
//
// Every mbarrier wait is bounded; a wait that runs out raises a block-wide abort flag and a device
// error word, all loops then run through without waiting (the cluster barriers are still reached by
// every thread), TMEM is freed and the kernel ends.
#include <atomic>
#include <cooperative_groups.h>

#include "internal.h"
#include "q4_common.cuh"
#include "sm100_ptx.cuh"
#include "tmap.h"
#include "ws_plan.h"

namespace b200 {

__device__ int g_gemm_ws_error = 0;

namespace {

namespace cg = cooperative_groups;
using namespace ptx;

constexpr int BR = 128;            // weight rows per tile (UMMA M)
constexpr int BK = 64;             // k per K block (one 128-byte swizzled row of fp16)
constexpr int kMaxXStages = 32;    // x stages (SKB K blocks each)
constexpr int kMaxRawStages = 8;
constexpr int kASlots = 4;         // A ring: slots of SKB K blocks (32 TMEM columns each), one per dequantiser group
constexpr int kRawBytes = BR * 128;           // 16384: 128 rows x 32 words = 256 k, one 128-byte line per row
constexpr int kScBytes = BR * 16;             // 2048:  128 rows x 8 scales  = 256 k
constexpr int kDequantWarps = 16;
static_assert(kRawBytes + kScBytes == kWsSpanBytes, "the plan counts these bytes");
constexpr int kNumThreads = 256 + kDequantWarps * 32 + 128;   // 896: warps 24-27 are a second set of epilogue warps
constexpr uint32_t kTmemCols = 512;           // two accumulators of 128 (SKB = 2) or 192 columns, then the A ring
constexpr uint64_t kWaitNs = 4000000000ull;   // 4 s

struct WsParams {
  CUtensorMap tm_x;    // fp16   {64, M, K/64},    box {64, NB, SKB},  SWIZZLE_128B: [K block][batch row][128 B]
  CUtensorMap tm_w;    // uint32 {K/8, N},         box {32, 128},      SWIZZLE_128B: [row][128 B] (whole lines: 64-byte pieces
                       //                                                    halve the rate the weights arrive at)
  CUtensorMap tm_s;    // fp16   {K/32, N},        box {8, 128}        (GU: rows as {N/2, 2}, boxes of 64 gate rows and their 64 up rows)
  const __half* scales;
  __half* y;
  int M, N, K;
  int NB;              // batch columns of the MMA: M rounded up to 16 (32 with 8 slices)
  int SX, SR;          // ring depths: x stages, packed 256-k spans (weights + scales; even)
  int x_resident;      // the x ring holds a whole slice: loaded once, kept for every tile
  int ksplit;          // CTAs per cluster = K slices
  int mt;              // token tiles of NB rows of x: tile t is row tile t / mt, token tile t % mt
  int tiles;           // ceil(N / 128) * mt   (GU: ceil(N / 2 / 64) * mt)
  int cw;              // batch columns per owner: NB / ksplit, a multiple of 4
};

struct Bars {
  uint64_t x_full[kMaxXStages], x_empty[kMaxXStages];
  uint64_t r_full[kMaxRawStages], r_empty[kMaxRawStages];
  uint64_t a_full[kASlots], a_empty[kASlots];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t inbox_full, inbox_free;
  uint32_t tmem_base;
  int abort_flag;
};

// The conversion, the MMAs and the refills of the rings wait for x, so for the kernels in front of this one, which may
// legitimately run for longer than the limit (a sum over ranks waits up to gemv.peer_wait_ms for a late one).  A
// limit that runs out is therefore started once more behind griddepcontrol.wait.
__device__ __forceinline__ void wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (mbar_try_wait(bar, parity)) return;   // completed barrier: no read of the flag on the fast path
  if (*abort_flag) return;
  if (mbar_wait_ns(bar, parity, kWaitNs)) return;
  pdl_wait();
  if (!mbar_wait_ns(bar, parity, kWaitNs)) {
    *abort_flag = 1;
    atomicExch(&g_gemm_ws_error, code);
  }
}
__device__ __forceinline__ void wait_or_abort_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (mbar_try_wait_cluster(bar, parity)) return;
  if (*abort_flag) return;
  if (!mbar_wait_cluster_ns(bar, parity, kWaitNs)) {
    *abort_flag = 1;
    atomicExch(&g_gemm_ws_error, code);
  }
}

// Position in a ring of `n` stages without divisions: stage index + wrap parity.
struct Ring {
  int s = 0;
  uint32_t phase = 0;      // number of completed wraps, mod 2
  bool wrapped = false;    // at least one wrap so far
  __device__ __forceinline__ void next(int n) {
    if (++s == n) { s = 0; phase ^= 1; wrapped = true; }
  }
};

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, int32_t c0, int32_t c1, int32_t c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// Shared memory (1024-aligned base): x ring [SX][SKB][NB][128 B] | raw ring [SR][16 KB] | scale ring [SR][2 KB] |
// inbox [ksplit source ranks][cw / 4][128 rows][4 columns] fp32 (ksplit > 1; a warp's 16-byte stores are then 512
// contiguous bytes: with rows 80 bytes apart, so 16-byte pieces on the SM-to-SM network, the exchange of a tile of 64
// columns took 3900 clocks instead of 1400) | barriers.
// PAIRED: nibble order of the packed words (q4_common.cuh).  RAGGED: K is not a multiple of 256, or the scales are not
// 16-byte aligned, so that the scales' rows cannot be a tensor map's: the dequantisers then read their scales from global
// memory one trip ahead, and x comes one K block per load through a map that ends at K.  What lies past K is zero
// on both sides (packed words, scales and x).  SKB: K blocks per x stage and A slot: 2 up to 128 batch
// columns (fewer waits and arrivals), 1 above (tensor memory holds two accumulators of 192 columns and four slots of 32).
// GU: W's rows are [gate: N / 2 | up: N / 2]; a tile takes 64 of each and silu(gate) * up is stored, [M, N / 2], formed as the
// separate kernel does from the fp16-rounded sums.  The two rows of a product are 64 apart in tensor memory, out of each other's warp's
// reach, so the sums travel through the inbox with one slice too.  A layer's step without the launch for SwiGLU and without the trip
// of gate | up to memory: 64 rows of hidden 1024 33.2 -> 32.6 us, 24 of 4096 at 401 89.8 -> 85.8, 16
// of 4096 at 2012 133.0 -> 130.3, 16 of 2560 the same.
template <bool PAIRED, int SKB, bool RAGGED, bool GU>
__global__ void __launch_bounds__(kNumThreads, 1)
q4f16_gemm_ws_tcgen05_kernel(const __grid_constant__ WsParams p) {
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* base = smem_unaligned + ((1024u - (smem_u32(smem_unaligned) & 1023u)) & 1023u);
  const int xstage = SKB * p.NB * 128;
  constexpr uint32_t kAccPitch = SKB == 2 ? 128 : 192, kTmemA = 2 * kAccPitch;
  unsigned char* x_ring = base;
  unsigned char* raw_ring = x_ring + (size_t)p.SX * xstage;
  unsigned char* sc_ring = raw_ring + (size_t)p.SR * kRawBytes;
  float* inbox = reinterpret_cast<float*>(sc_ring + (size_t)p.SR * kScBytes);
  const bool exchange = GU || p.ksplit > 1;
  Bars& bar = *reinterpret_cast<Bars*>(inbox + (exchange ? (size_t)BR * p.NB : 0));
  volatile int* abort_flag = &bar.abort_flag;
  cg::cluster_group cluster = cg::this_cluster();

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform, and known to be
  const int lane = tid & 31;
  const int krank = (int)cluster.block_rank();          // K slice of this CTA (gridDim.x == ksplit)
  const int tile0 = blockIdx.y, tstep = gridDim.y;
  // 256-k spans, the first slices one span longer (every slice has at least one)
  const int units = (p.K + 255) >> 8;
  const int ubase = units / p.ksplit, uextra = units % p.ksplit;
  const int span0 = krank * ubase + min(krank, uextra);
  const int nspans = ubase + (krank < uextra ? 1 : 0);
  const int nunits = 4 / SKB * nspans;                  // x stages = A slots of a tile

  auto load_rows = [](void* dst, const void* map, int col, int row_tile, uint64_t* full) {
    if (GU) tma_load_3d(dst, map, col, row_tile * (BR / 2), 0, full);
    else tma_load_2d(dst, map, col, row_tile * BR, full);
  };
  if (tid == 0) {
    bar.abort_flag = 0;
    for (int i = 0; i < p.SX; ++i) { mbar_init(&bar.x_full[i], 1); mbar_init(&bar.x_empty[i], 1); }
    for (int i = 0; i < kASlots; ++i) { mbar_init(&bar.a_full[i], 4); mbar_init(&bar.a_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.acc_full[i], 1); mbar_init(&bar.acc_empty[i], 8); }
    mbar_init(&bar.inbox_full, 1);
    mbar_init(&bar.inbox_free, 8 * p.ksplit);         // the epilogue warps of every CTA of the cluster, this one's too
    mbar_fence_init();
  }
  if (tid == 64) {
    // The weights depend on nothing: the thread that will stream them sets up the packed ring's barriers itself
    // and fills the ring at once, ahead of the rest of the set-up (barriers, TMEM allocation, the cluster-wide sync).
    for (int i = 0; i < p.SR; ++i) { mbar_init(&bar.r_full[i], RAGGED ? 1 : 2); mbar_init(&bar.r_empty[i], kDequantWarps / SKB); }
    mbar_fence_init();
    for (int i = 0; i < p.SR && i < nspans; ++i) {
      mbar_arrive_expect_tx(&bar.r_full[i], kRawBytes);
      load_rows(raw_ring + (size_t)i * kRawBytes, &p.tm_w, (span0 + i) * 32, tile0 / p.mt, &bar.r_full[i]);
      if (!RAGGED) {
        mbar_arrive_expect_tx(&bar.r_full[i], kScBytes);
        load_rows(sc_ring + (size_t)i * kScBytes, &p.tm_s, (span0 + i) * 8, tile0 / p.mt, &bar.r_full[i]);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(&bar.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before_sync();
  // The peers' barriers are initialised before anything arrives on them: the fence above orders the initialisation, so the
  // arrival need not (a releasing one, with the weight loads just requested, took 1.8 us).  One branch around both halves: with the
  // block's barrier between them a run of single CTAs was 1.5-2.8 % slower (us, this / that: 512 x 12288 x 11008 117.0 / 119.6,
  // 1024 x 16384 x 8192 242.5 / 248.5, 2048 x 11008 x 4096 156.7 / 158.8), and clusters no faster.
  if (p.ksplit > 1) {
    cluster_arrive_relaxed();
    cluster_wait();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, bar.tmem_base, 0);
  pdl_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: x (SKB K blocks per load)
    if (lane == 0) {
      prefetch_tmap(&p.tm_x);
      pdl_wait();                                     // x may be the previous kernel's output
      Ring rx;
      for (int tile = tile0; tile < p.tiles; tile += tstep) {
        const int tok0 = tile % p.mt * p.NB;
        for (int u = 0; u < nunits; ++u, rx.next(p.SX)) {
          // (not a sleeping wait: a nanosleep lasts far longer than the time a stage takes)
          if (rx.wrapped) wait_or_abort(&bar.x_empty[rx.s], rx.phase ^ 1, abort_flag, 1);
          mbar_arrive_expect_tx(&bar.x_full[rx.s], xstage);
          if (RAGGED) {
#pragma unroll
            for (int j = 0; j < SKB; ++j)
              tma_load_2d(x_ring + (size_t)rx.s * xstage + j * p.NB * 128, &p.tm_x, (span0 * 4 + SKB * u + j) * BK, tok0, &bar.x_full[rx.s]);
          } else {
            tma_load_3d(x_ring + (size_t)rx.s * xstage, &p.tm_x, 0, tok0, span0 * 4 + SKB * u, &bar.x_full[rx.s]);
          }
        }
        if (p.x_resident) break;                      // one trip: the stages stay
      }
    }
  } else if (warp == 2 || warp == 3) {
    // ------------------------------------------------------------------ TMA producers: packed weights (warp 2), scales (warp 3), 256 k per load
    if (lane == 0 && !(RAGGED && warp == 3)) {
      const int first = min(p.SR, nspans);            // requested during set-up
      Ring rr;
      for (int tile = tile0; tile < p.tiles; tile += tstep) {
        const int row_tile = tile / p.mt;
        for (int sp = 0; sp < nspans; ++sp, rr.next(p.SR)) {
          if (tile == tile0 && sp < first) continue;
          const int s = rr.s;
          if (rr.wrapped) wait_or_abort(&bar.r_empty[s], rr.phase ^ 1, abort_flag, 3);
          if (warp == 2) {
            mbar_arrive_expect_tx(&bar.r_full[s], kRawBytes);
            load_rows(raw_ring + (size_t)s * kRawBytes, &p.tm_w, (span0 + sp) * 32, row_tile, &bar.r_full[s]);
          } else {
            mbar_arrive_expect_tx(&bar.r_full[s], kScBytes);
            load_rows(sc_ring + (size_t)s * kScBytes, &p.tm_s, (span0 + sp) * 8, row_tile, &bar.r_full[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop, converged: its values are warp-uniform and the tcgen05 wrappers elect the lane
    // that issues (see there).  Straight-line code per stage, one branch for both waits, cursors advanced
    // by selects, descriptors by 32-bit adds (every shared-memory address is below 256 KB, so nothing carries out of
    // the address field).
    const uint32_t idesc = umma_idesc_f16_f32(BR, p.NB);
    const uint64_t dconst = umma_desc_k128(0);
    const uint32_t b0 = (smem_u32(x_ring) & 0x3FFFFu) >> 4;
    const uint32_t b_step = (uint32_t)xstage >> 4, b_kb = (uint32_t)(p.NB * 128) >> 4;
    const uint32_t SX = (uint32_t)p.SX;
    const bool resident = p.x_resident != 0;
    uint32_t as = 0, aphase = 0, xs = 0, xphase = 0, it = 0;
    for (int tile = tile0; tile < p.tiles; tile += tstep, ++it) {
      const uint32_t buf = it & 1;
      if (it >= 2) wait_or_abort(&bar.acc_empty[buf], ((it >> 1) - 1) & 1, abort_flag, 4);
      const uint32_t td = tmem_base + buf * kAccPitch;
      if (resident) xs = xphase = 0;
      for (int u = 0; u < nunits; ++u) {
        uint64_t* af = &bar.a_full[as];
        uint64_t* xf = &bar.x_full[xs];
        const bool ready = mbar_try_wait(af, aphase) & mbar_try_wait(xf, xphase);
        if (!ready) {
          wait_or_abort(af, aphase, abort_flag, 6);
          wait_or_abort(xf, xphase, abort_flag, 5);
        }
        tc_fence_after_sync();
        const uint32_t ta = tmem_base + kTmemA + as * (32 * SKB);
        const uint64_t db = dconst | (uint64_t)(b0 + xs * b_step);
#pragma unroll
        for (int j = 0; j < SKB; ++j) {
#pragma unroll
          for (int k16 = 0; k16 < 4; ++k16) {
            // +16 k = +8 columns of A, +32 bytes inside the swizzled 128-byte row of x (+2 in 16-byte units)
            umma_f16_ts(td, ta + j * 32 + k16 * 8, db + (uint64_t)(j * b_kb + 2 * k16), idesc,
                        (j | k16) == 0 ? (uint32_t)(u != 0) : 1u);
          }
        }
        if (!resident) umma_commit(&bar.x_empty[xs]);
        umma_commit(&bar.a_empty[as]);
        as = as + 1 == kASlots ? 0 : as + 1;
        aphase ^= (uint32_t)(as == 0);
        xs = xs + 1 == SX ? 0 : xs + 1;
        xphase ^= (uint32_t)(xs == 0);
      }
      umma_commit(&bar.acc_full[buf]);
    }
  } else if (warp >= 8 && warp < 24) {
    // ------------------------------------------------------------------ dequantisers
    // Unit n (SKB K blocks) of the CTA's whole run goes to slot n % 4, which group n % 4 fills.  SKB = 2: group `grp`
    // takes the half grp % 2 of the spans whose running index has the parity grp / 2; SKB = 1: K block grp of every span.
    const int grp = (warp - 8) >> 2;
    const int part = SKB == 2 ? grp & 1 : grp;
    const int r = (warp & 3) * 32 + lane;           // weight row inside the tile = TMEM lane (a warp reaches quadrant warp % 4)
    const int r8 = r & 7;
    const uint32_t tslot = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kTmemA + (uint32_t)grp * (32 * SKB);
    uint32_t off[2 * SKB];                          // this part's 16-byte chunks; 128-byte swizzle: chunk ^ (row % 8)
#pragma unroll
    for (int j = 0; j < 2 * SKB; ++j) off[j] = (uint32_t)(r * 128 + (((2 * SKB * part + j) ^ r8) << 4));
    const Q4Consts qc = q4_consts();
    const uint32_t total = (uint32_t)nspans * (uint32_t)((p.tiles - tile0 + tstep - 1) / tstep);
    const uint32_t first = SKB == 2 ? (uint32_t)(grp >> 1) : 0;
    int s = (int)first;                        // ring slot (the ring's depth is even: with SKB = 2 a group stays on slots of its parity)
    uint32_t phase = 0, use = 0;
    const int groups = p.K >> 5;
    auto global_scales = [&](uint32_t i, uint32_t (&out)[SKB]) {       // of the span with running index i
      const int row_tile = (tile0 + (int)(i / (uint32_t)nspans) * tstep) / p.mt;
      int row = row_tile * BR + r;
      if (GU) {
        row = row_tile * (BR / 2) + (r & 63);
        row = row < p.N / 2 ? row + (r >> 6) * (p.N / 2) : p.N;
      }
      const int g0 = (span0 + (int)(i % (uint32_t)nspans)) * 8 + 2 * SKB * part;
      const __half* src = p.scales + (int64_t)row * groups + g0;
#pragma unroll
      for (int j = 0; j < SKB; ++j) {
        uint32_t lo = 0, hi = 0;
        if (i < total && row < p.N && g0 + 2 * j < groups) lo = __half_as_ushort(__ldg(src + 2 * j));
        if (i < total && row < p.N && g0 + 2 * j + 1 < groups) hi = __half_as_ushort(__ldg(src + 2 * j + 1));
        out[j] = lo | (hi << 16);
      }
    };
    uint32_t next_sc[SKB];
    if (RAGGED) global_scales(first, next_sc);
    for (uint32_t sidx = first; sidx < total; sidx += SKB, ++use) {
      wait_or_abort(&bar.r_full[s], phase, abort_flag, 8);
      const unsigned char* rbase = raw_ring + (size_t)s * kRawBytes;
      uint4 pk[2 * SKB];
      uint32_t scw[SKB];
#pragma unroll
      for (int j = 0; j < 2 * SKB; ++j) pk[j] = *reinterpret_cast<const uint4*>(rbase + off[j]);
#pragma unroll
      for (int j = 0; j < SKB; ++j)
        scw[j] = RAGGED ? next_sc[j] : *reinterpret_cast<const uint32_t*>(sc_ring + (size_t)s * kScBytes + r * 16 + (SKB * part + j) * 4);
      if (RAGGED) global_scales(sidx + SKB, next_sc);
#pragma unroll
      for (int j = 0; j < 2 * SKB; ++j) pin_loaded(pk[j]);
#pragma unroll
      for (int j = 0; j < SKB; ++j) pin_loaded(scw[j]);
      fence_proxy_async_smem();                // generic reads ordered before the TMA refill (async proxy)
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.r_empty[s]);
#pragma unroll
      for (int j = 0; j < SKB; ++j) {          // K block of the unit
        const __half2 scp = u32_as_h2(scw[j]);
        const __half2 s_lo = __low2half2(scp), s_hi = __high2half2(scp);
        const uint32_t words[8] = {pk[2 * j].x, pk[2 * j].y, pk[2 * j].z, pk[2 * j].w,
                                   pk[2 * j + 1].x, pk[2 * j + 1].y, pk[2 * j + 1].z, pk[2 * j + 1].w};
        uint32_t o[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 q = q4_dequant_ordered<PAIRED>(words[c], c < 4 ? s_lo : s_hi, qc);
          o[4 * c] = q.x; o[4 * c + 1] = q.y; o[4 * c + 2] = q.z; o[4 * c + 3] = q.w;
        }
        if (j == 0) {                          // the MMAs of this slot's previous unit have read it
          if (use > 0) wait_or_abort(&bar.a_empty[grp], (use - 1) & 1, abort_flag, 10);
          tc_fence_after_sync();
        }
        tmem_st_32x32b_x32(tslot + j * 32, o);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.a_full[grp]);
      s += SKB;
      if (s >= p.SR) { s -= p.SR; phase ^= 1; }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    pdl_wait();                                      // y may still be read by the previous kernel
    const int ew = warp & 3;                         // TMEM lane quadrant this warp may read
    const int set = warp >= 24 ? 1 : 0;              // two warps per quadrant share the columns
    const int r = ew * 32 + lane;                    // weight row inside the tile
    const uint32_t inbox_mine = smem_u32(inbox) + (uint32_t)(krank * p.cw * BR + r * 4) * 4;   // row r of the block that this CTA fills, in every inbox
    const uint32_t full_addr = smem_u32(&bar.inbox_full), free_addr = smem_u32(&bar.inbox_free);
    const uint32_t cw_inv = (65536u + (uint32_t)p.cw - 1) / (uint32_t)p.cw;      // column / cw for columns below 256
    uint32_t it = 0, inbox_phase = 0;
    for (int tile = tile0; tile < p.tiles; tile += tstep, ++it) {
      const uint32_t buf = it & 1;
      const int row = GU ? tile / p.mt * (BR / 2) + (r & 63) : tile / p.mt * BR + r;
      const int out_rows = GU ? p.N / 2 : p.N;           // pitch of y
      const int tok0 = tile % p.mt * p.NB;
      const int ntok = min(p.NB, p.M - tok0);          // tokens of this tile
      const int ntok4 = (ntok + 3) & ~3;               // columns that are exchanged
      const int own = max(0, min(p.cw, ntok4 - krank * p.cw));     // columns that this CTA adds up and stores
      __half* yt = p.y + (int64_t)tok0 * out_rows + row;
      // The owners have read what this CTA sent for the tile before.  This CTA is an owner itself: the two warps of a
      // quadrant send and sum different columns of the same rows, so without its own eight warps among the arrivals
      // the faster of the two could overwrite what the slower one has yet to add up.
      if (p.ksplit > 1 && it > 0) wait_or_abort_cluster(&bar.inbox_free, (it - 1) & 1, abort_flag, 12);
      // (a phase of inbox_full ends with the bytes of all ranks; the next one cannot end before every warp here
      // has told all ranks that it is done with this one)
      if (p.ksplit > 1 && own > 0 && warp == 4 && lane == 0) mbar_arrive_expect_tx(&bar.inbox_full, (uint32_t)(p.ksplit * BR * own * 4));
      wait_or_abort(&bar.acc_full[buf], (it >> 1) & 1, abort_flag, 7);
      tc_fence_after_sync();
      if (GU && p.ksplit == 1 && it > 0) bar_sync(2, 256);     // (the tile before has been read)
      const uint32_t taddr = tmem_base + ((uint32_t)(ew * 32) << 16) + buf * kAccPitch;
      for (int c0 = 16 * set; c0 < ntok; c0 += 32) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(taddr + c0, v);
        tmem_ld_wait();
        if (!exchange) {
          if (row < p.N) {
            __half* dst_y = yt + (int64_t)c0 * p.N;
            if (c0 + 16 <= ntok) {
#pragma unroll
              for (int q = 0; q < 16; ++q, dst_y += p.N) *dst_y = __float2half_rn(__uint_as_float(v[q]));
            } else {
#pragma unroll
              for (int q = 0; q < 16; ++q, dst_y += p.N)
                if (c0 + q < ntok) *dst_y = __float2half_rn(__uint_as_float(v[q]));
            }
          }
        } else if (GU && p.ksplit == 1) {
#pragma unroll
          for (int q = 0; q < 16; q += 4)                      // (columns past the tokens too: there is room for NB)
            *reinterpret_cast<uint4*>(inbox + (c0 + q) * BR + r * 4) = make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < 16; q += 4) {
            if (c0 + q < ntok4) {
              const uint32_t owner = ((uint32_t)(c0 + q) * cw_inv) >> 16;
              const uint32_t lc = (uint32_t)(c0 + q) - owner * (uint32_t)p.cw;
              st_async_v4(map_to_rank(inbox_mine + lc * (BR * 4), owner), map_to_rank(full_addr, owner), v[q], v[q + 1], v[q + 2], v[q + 3]);
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.acc_empty[buf]);
      if (!exchange) continue;
      // ---- this CTA's columns: sum over the K slices in rank order
      if (GU && p.ksplit == 1) bar_sync(2, 256);
      else if (own > 0) wait_or_abort_cluster(&bar.inbox_full, inbox_phase, abort_flag, 11);
      inbox_phase ^= (uint32_t)(own > 0);            // (a CTA without columns in a tile's last tokens sits that phase out)
      auto total = [&](int l, int rr) {                // of columns l .. l + 3, row rr of the tile
        const float* src = inbox + l * BR + rr * 4;
        if (GU) {                                     // (one sum after the other: registers)
          float4 sum = *reinterpret_cast<const float4*>(src);
#pragma unroll 1
          for (int q = 1; q < p.ksplit; ++q) {
            const float4 v = *reinterpret_cast<const float4*>(src + (size_t)q * p.cw * BR);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
          return sum;
        }
        float4 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < p.ksplit) v[q] = *reinterpret_cast<const float4*>(src + (size_t)q * p.cw * BR);
        float4 sum = v[0];
#pragma unroll
        for (int q = 1; q < 8; ++q)
          if (q < p.ksplit) { sum.x += v[q].x; sum.y += v[q].y; sum.z += v[q].z; sum.w += v[q].w; }
        return sum;
      };
      // GU: the four warps that hold rows of one half of the tile share the columns of both halves
      const int first = GU ? 4 * (2 * set + (ew >> 1)) : 4 * set;
      for (int l = first; l < own; l += GU ? 16 : 8) {
        const int col = krank * p.cw + l;
        float4 sum = total(l, GU ? r & 63 : r);
        if (GU) {
          const float4 up = total(l, (r & 63) + 64);
          auto act = [](float g, float u) {
            g = __half2float(__float2half_rn(g));
            u = __half2float(__float2half_rn(u));
            return g / (1.f + __expf(-g)) * u;
          };
          sum = make_float4(act(sum.x, up.x), act(sum.y, up.y), act(sum.z, up.z), act(sum.w, up.w));
        }
        if (row < out_rows) {
          __half* dst_y = yt + (int64_t)col * out_rows;
          dst_y[0] = __float2half_rn(sum.x);
          if (col + 1 < ntok) dst_y[out_rows] = __float2half_rn(sum.y);
          if (col + 2 < ntok) dst_y[2 * (int64_t)out_rows] = __float2half_rn(sum.z);
          if (col + 3 < ntok) dst_y[3 * (int64_t)out_rows] = __float2half_rn(sum.w);
        }
      }
      // Not after the last tile: the arrival's release would wait for the stores to y.
      __syncwarp();
      if (p.ksplit > 1 && tile + tstep < p.tiles && lane < p.ksplit) mbar_arrive_cluster(map_to_rank(free_addr, lane));
    }
  }

  // ---------------------------------------------------------------------- teardown
  if (p.ksplit > 1) {
    // Nobody leaves while a peer still writes or arrives here.  What peers send this CTA has landed by now (its last tile's sums
    // waited for every byte, and that tile's exchange for every arrival on inbox_free), unless a wait was given up: the arrival
    // orders nothing, in particular not the stores to y, which a releasing one would wait for.
    __syncwarp();
    cluster_arrive_relaxed();
    cluster_wait();
  }
  if (*abort_flag) {
    // loads may still be in flight into this CTA's shared memory: let them land before it is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

using WsKernel = void (*)(const WsParams);
template <bool RAGGED>
WsKernel kernel_of(int nb, bool paired, bool gu) {
  if (gu) return paired ? q4f16_gemm_ws_tcgen05_kernel<true, 2, RAGGED, true> : q4f16_gemm_ws_tcgen05_kernel<false, 2, RAGGED, true>;
  return nb <= 128 ? (paired ? q4f16_gemm_ws_tcgen05_kernel<true, 2, RAGGED, false> : q4f16_gemm_ws_tcgen05_kernel<false, 2, RAGGED, false>)
                   : (paired ? q4f16_gemm_ws_tcgen05_kernel<true, 1, RAGGED, false> : q4f16_gemm_ws_tcgen05_kernel<false, 1, RAGGED, false>);
}
WsKernel kernel_for(int nb, bool paired, bool ragged, bool gu) { return ragged ? kernel_of<true>(nb, paired, gu) : kernel_of<false>(nb, paired, gu); }

constexpr size_t kSmemCap = 227 * 1024;
// More than half of an SM: one such CTA per SM, whatever its rings would need.  (It takes all of tensor memory; two
// of them on one SM, from clusters of two streams, could wait for each other's.)
constexpr size_t kSmemFloor = 116 * 1024;

// How many clusters of `ksplit` CTAs run at once (one CTA per SM; a cluster stays inside a GPC, so fewer than
// SMs / ksplit for the larger sizes).  Asked once per device and size.
int max_clusters(int ksplit, const void* kern) {
  static std::atomic<int> cache[64][4];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() / ksplit;
  const int slot = ksplit == 1 ? 0 : ksplit == 2 ? 1 : ksplit == 4 ? 2 : 3;
  int v = cache[dev][slot].load(std::memory_order_relaxed);
  if (v > 0) return v;
  v = sm_count() / ksplit;
  if (ksplit > 1 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ksplit, (unsigned)v);
    cfg.blockDim = dim3(kNumThreads);
    cfg.dynamicSmemBytes = kSmemCap;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ksplit;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) v = n < v ? n : v;
    else cudaGetLastError();
  }
  cache[dev][slot].store(v, std::memory_order_relaxed);
  return v;
}

}  // namespace

// Whether SwiGLU in the epilogue is faster than a launch of its own behind the matmul.  Up to 96 rows it is.  Above, the inbox
// takes so much of a CTA's shared memory that a long run of one slice is slower, unless it is one that fills the SMs: separate / in the
// epilogue in us, M x I x K 64 x 5632 x 4096 14.7 / 14.0, 96 x 11008 x 4096 27.7 / 26.4, 112 x 4096 x 5120 17.7 / 14.5 and 128 x 1024 x 4096
// 11.6 / 9.9 (four slices), 128 x 8192 x 3072 16.7 / 16.2, but 128 x 1024 x 2048 10.1 / 11.2, 128 x 5632 x 5120 19.5 / 21.4,
// 128 x 11008 x 1024 12.4 / 13.2, 112 x 8192 x 8192 31.1 / 34.4.
bool gemm_ws_gate_up_is_ahead(int64_t M, int64_t I, int64_t K, bool ragged) {
  if (M <= 96) return true;
  const int64_t tiles = (I + BR / 2 - 1) / (BR / 2);
  int clusters_of[4];
  for (int i = 0; i < 4; ++i) clusters_of[i] = max_clusters(1 << i, reinterpret_cast<const void*>(kernel_for(16, false, ragged, false)));
  if (tiles > 64) return 3 * tiles > 2 * clusters_of[0] && tiles <= clusters_of[0] && K <= 4096;
  return choose_ws_split(M, tiles, (int)((K + 255) / 256), (int)options().gemm_ws_ksplit, clusters_of).ksplit > 1;
}

// Returns B200_ENOTREADY when the shape is outside what this kernel takes, or one for the prefill kernel.  gate_up: SwiGLU in the
// epilogue (up to 128 rows, N even).
int launch_gemm_ws(const __half* x, const uint32_t* wq, const __half* scales, __half* y, int64_t M, int64_t N,
                   int64_t K, cudaStream_t stream, bool gate_up) {
  if (gate_up && (M > 128 || N % 2 != 0)) return B200_ENOTREADY;
  if (M < 1 || K < 32 || K % 32 != 0) return B200_ENOTREADY;
  const bool ragged = K % 256 != 0 || (reinterpret_cast<uintptr_t>(scales) & 15u) != 0;
  WsParams p;
  int rc;
  const bool paired = current_layout() == kLayoutPaired;
  p.scales = scales;
  p.y = y;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  const int units = (int)((K + 255) / 256);
  const int64_t row_tiles = gate_up ? (N / 2 + BR / 2 - 1) / (BR / 2) : (N + BR - 1) / BR;
  if (row_tiles * ((M + 15) / 16) > 0x3fffffff) return B200_ENOTREADY;      // (tile numbers are 32-bit)
  int clusters_of[4];
  for (int i = 0; i < 4; ++i) clusters_of[i] = max_clusters(1 << i, reinterpret_cast<const void*>(kernel_for(16, paired, ragged, false)));
  const WsSplit split = choose_ws_split(M, row_tiles, units, (int)options().gemm_ws_ksplit, clusters_of);
  if (options().gemm_ws_ksplit == 0 && prefill_kernel_is_ahead(M, N, K, split, row_tiles, clusters_of[0])) return B200_ENOTREADY;
  const int ksplit = split.ksplit, nb16 = split.nb;
  const int skb = nb16 <= 128 ? 2 : 1;
  auto kern = kernel_for(nb16, paired, ragged, gate_up);
  static SmemLimit limits[12];                           // (one per kernel variant)
  if ((rc = raise_smem_limit(limits[(gate_up ? 2 : nb16 <= 128) * 4 + ragged * 2 + paired], reinterpret_cast<const void*>(kern), kSmemCap, "gemm_ws")))
    return rc;
  // an owner's columns are exchanged four at a time
  if (ksplit == 8 || (ksplit > 1 && (nb16 / ksplit) % 4 != 0)) p.NB = (nb16 + 4 * ksplit - 1) / (4 * ksplit) * (4 * ksplit);
  else p.NB = nb16;
  p.ksplit = ksplit;
  p.cw = p.NB / ksplit;
  p.mt = (int)((M + p.NB - 1) / p.NB);
  p.tiles = (int)row_tiles * p.mt;
  int clusters = clusters_of[ksplit == 1 ? 0 : ksplit == 2 ? 1 : ksplit == 4 ? 2 : 3];
  if (clusters > p.tiles) clusters = p.tiles;

  // Shared memory: the inbox, four packed spans (72 KB in flight cover HBM's latency at one SM's share of its
  // rate), then x: the whole slice if it fits (it is then loaded once for all tiles), else up to six stages; what
  // is left goes to the packed ring.
  const size_t inbox = ksplit > 1 || gate_up ? (size_t)BR * p.NB * sizeof(float) : 0;
  const size_t xstage = (size_t)skb * p.NB * 128;
  const size_t span = kRawBytes + kScBytes;
  const size_t fixed = 1024 + inbox + sizeof(Bars) + 256;
  const int slice_stages = 4 / skb * ((units + ksplit - 1) / ksplit);
  int sr = 4;
  int fit = (int)((kSmemCap - fixed - sr * span) / xstage);
  if (fit < 3) { sr = 2; fit = (int)((kSmemCap - fixed - sr * span) / xstage); }
  if (fit < 2) return B200_ENOTREADY;     // (never: 192 columns in several slices leave three stages)
  p.x_resident = p.mt == 1 && slice_stages <= fit && slice_stages <= kMaxXStages && options().gemm_ws_x_stages == 0;
  p.SX = p.x_resident ? slice_stages : fit < 6 ? fit : 6;
  if (options().gemm_ws_x_stages > 1 && options().gemm_ws_x_stages < p.SX) p.SX = (int)options().gemm_ws_x_stages;
  sr = (int)((kSmemCap - fixed - p.SX * xstage) / span);
  if (sr > kMaxRawStages) sr = kMaxRawStages;
  if (options().gemm_ws_r_stages >= 2 && options().gemm_ws_r_stages < sr) sr = (int)options().gemm_ws_r_stages;
  // An even depth: the groups of one span parity take every second span, so every slot of the ring then belongs to the
  // same groups, which wait for its next load only after they have consumed the one before themselves (with an
  // odd depth two parities would share a slot, each would meet it with the same phase parity every time, and its
  // wait could pass on the load before last).
  sr &= ~1;
  if (sr < 2) return B200_ENOTREADY;
  p.SR = sr;
  size_t smem = fixed + p.SX * xstage + p.SR * span;
  if (smem < kSmemFloor) smem = kSmemFloor;

  if (ragged) {
    const uint64_t d[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t s[1] = {(uint64_t)K * 2};
    const uint32_t b[2] = {BK, (uint32_t)p.NB};
    if ((rc = make_tmap(&p.tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  } else {
    const uint64_t d[3] = {BK, (uint64_t)M, (uint64_t)(K / BK)};
    const uint64_t s[2] = {(uint64_t)K * 2, BK * 2};
    const uint32_t b[3] = {BK, (uint32_t)p.NB, (uint32_t)skb};
    if ((rc = make_tmap(&p.tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, x, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  }
  // rows of W and of the scales: {N}, or gate and up rows {N / 2, 2} with boxes of 64 of each
  const int rank = gate_up ? 3 : 2;
  const uint64_t rows = (uint64_t)(gate_up ? N / 2 : N);
  const uint32_t box_rows = gate_up ? BR / 2 : BR;
  {
    const uint64_t d[3] = {(uint64_t)(K / 8), rows, 2};
    const uint64_t s[2] = {(uint64_t)(K / 2), (uint64_t)(K / 2) * rows};
    const uint32_t b[3] = {32, box_rows, 2};
    if ((rc = make_tmap(&p.tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT32, rank, wq, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  }
  if (!ragged) {
    const uint64_t d[3] = {(uint64_t)(K / 32), rows, 2};
    const uint64_t s[2] = {(uint64_t)(K / 32) * 2, (uint64_t)(K / 32) * 2 * rows};
    const uint32_t b[3] = {8, box_rows, 2};
    if ((rc = make_tmap(&p.tm_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, scales, d, s, b, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ksplit, (unsigned)clusters);
  cfg.blockDim = dim3(kNumThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ksplit;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = options().gemv_pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "gemm_ws launch: %s", cudaGetErrorString(e));
  count_launch();
  return B200_OK;
}

int gemm_ws_error_read_and_clear() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemm_ws_error, sizeof(int)) != cudaSuccess) return 0xff;
  if (v) cudaMemcpyToSymbol(g_gemm_ws_error, &zero, sizeof(int));
  return v & 0xff;
}

}  // namespace b200
