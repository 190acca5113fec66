// rhs_tc.cuh -- fused DG Maxwell right-hand side with the element contractions
// on the tcgen05 tensor cores (3xTF32: hi*hi + hi*lo + lo*hi, FP32 accumulate
// in TMEM).  Orders 1..5.
//
// One persistent CTA per SM walks tiles of E elements.  The MMA M dimension is
// the rows (element, component), split into four lane quarters of QR = M/4
// rows; quarter q holds elements EQ q .. EQ q + EQ - 1, component by component
// (tc_row_in_quarter), so the six components of an element sit in one warp's TMEM
// lanes and the curl can be combined with warp shuffles, and neighbouring
// elements' rows of one component differ mod 8 (16-byte stores of the LIFT
// operand without replays).
//   orders 1-4: M = 128, EQ = 5 (E = 20; rows 30, 31 of a quarter are padding),
//               two TMEM accumulator sets side by side in the columns;
//   order 5:    M = 64, EQ = 2 (E = 8; rows 12..15 of a quarter are padding).
//               A 64-row MMA keeps row 16 q + r of its accumulator (and of a
//               TMEM A operand, which must sit at the accumulator's lane offset)
//               in lane 32 q + o + r, o = 0 or 16, so a quarter's rows stay in
//               its own TMEM sub-partition and the two accumulator sets (each
//               with its own volume A operand) take the two lane halves of the
//               same columns; TMEM is read and written with the 16-lane shapes,
//               a warp's two thread halves on two column ranges.  Order 5 at 128
//               rows would need 608 TMEM columns for two accumulator sets and
//               about 370 KB of shared memory for its operands and state slots.
//
//   volume:  C_v[(e,c)][(k,i)] = sum_j F[(e,c)][j] * D_k[i][j]        (rhs.rs:39-85)
//   LIFT:    C_l[(e,c)][i]     = sum_s Flux[(e,c)][s] * LIFT[i][s]    (rhs.rs:1433-1439)
//
// The CTA is warp-specialised so that two tiles are in flight:
//   volume warps    build tile t's volume operand (tf32 hi/lo of the state,
//                   written to TMEM by tcgen05.st);
//   flux warps      form its numerical fluxes (rhs.rs:1370-1441) into the LIFT
//                   operand in shared memory;
//   epilogue warps  finish tile t-1 from its TMEM accumulators: reference
//                   derivatives -> curl by shuffles, LIFT sum, material scaling
//                   (rhs.rs:1443-1454) and the mode's update in place (dy, or the
//                   LSERK4 stage of explicit.rs:122-133 on y and p);
//   control lane    issues the MMAs of both contractions into one of two TMEM
//                   accumulator sets;
//   copy lane       issues the bulk async loads (state + element records three
//                   tiles deep, residual register two deep) and stores.
// The LIFT operand is formed and multiplied in two halves (faces 0-1, 2-3) by
// separate warps, each half released by its own MMA completion.
//
// What bounds it: at order 4 the flux warps' chain of one tile (trace loads,
// fluxes, operand stores), nearly as long as the tile period, with the
// load/store pipe 76 % busy; at order 3 that pipe, 84 % busy, half of the
// shared-memory wavefronts replays (three quarters of them of loads).  HBM and
// the tensor pipe (31 % busy at order 4, 19 % at order 3) are not.  One thread per (element, face, node group) with
// vector operand stores, the loads of a face in neighbouring lanes, packed f32x2
// arithmetic, a copy lane that refills a slot as soon as it is read and volume
// warps of their own took five order-4 steps of the 48^3 box from 21.7 to 18.1
// ms, twenty order-3 steps of the graded 24^3 box from 10.6 to 8.1 ms, ten
// order-5 steps of 14,586 elements from 2.86 to 2.15 ms (one node per thread,
// 4-byte stores, the flux warps also writing the volume operand, copies issued
// between the MMAs).  Loading a tile's out-of-tile traces while the previous
// tile's fluxes are formed measured slower (8, 6 and 4 % more).
// All hand-offs are mbarriers; every wait is bounded and an expired wait stops
// the CTA cleanly with an error flag.  The element count is padded on the
// device to a multiple of E with inert records (PEC faces, zero metric), so
// every tile is full.
#pragma once
#include <cstdint>

#include "dgtd_common.cuh"
#include "tc_util.cuh"

// Phase timers: compiled in only with -DDGTD_TC_PHASE_TIMERS (an instrumented
// build); otherwise the marks are empty.  One thread per role records the cycles
// up to each of its marks: volume warps 0 waits, 1 work; flux warps 8 tile wait,
// 9 trace loads, 2 operand wait, 3 flux; epilogue 10 MMA wait, 4 slot waits,
// 5 work; control lane 6; copy lane 11 results wait, 7 store read.
#ifdef DGTD_TC_PHASE_TIMERS
#define DGTD_TC_MARK(i)                                     \
  do {                                                      \
    if (timer_thread) {                                     \
      const long long now__ = clock64();                    \
      clk_acc[i] += (unsigned long long)(now__ - clk_last); \
      clk_last = now__;                                     \
    }                                                       \
  } while (0)
#else
#define DGTD_TC_MARK(i) \
  do {                  \
  } while (0)
#endif

namespace dgtd {

constexpr int kTcMarks = 12;                 // phase timers (DGTD_TC_PHASE_COUNTERS)
constexpr uint32_t kTcWaitLimit = 1u << 19;  // polls per bounded wait (about 2 s)

__host__ __device__ constexpr int tc_r8(int x) { return (x + 7) & ~7; }
__host__ __device__ constexpr int tc_r16(int x) { return (x + 15) & ~15; }
__host__ __device__ constexpr int tc_r128(int x) { return (x + 127) & ~127; }

// Tile shape of an order: MMA rows and elements per lane quarter (the file
// header says why order 5 differs).
__host__ __device__ constexpr int tc_m(int n) { return n == 5 ? 64 : 128; }
__host__ __device__ constexpr int tc_eq(int n) { return n == 5 ? 2 : 5; }
__host__ __device__ constexpr int tc_tile_e(int n) { return 4 * tc_eq(n); }
// MMA N of the volume and LIFT B operands (a 128-row MMA takes N in steps of 16,
// a 64-row one in steps of 8); the host lays out the constant operands with these.
__host__ __device__ constexpr int tc_nv(int n) { return tc_m(n) == 64 ? tc_r8(3 * np_of(n)) : tc_r16(3 * np_of(n)); }
__host__ __device__ constexpr int tc_nl(int n) { return tc_m(n) == 64 ? tc_r8(np_of(n)) : tc_r16(np_of(n)); }

// Face nodes of a flux unit: two where the units then still fit one per thread
// beside the other roles (the chain of loads, flux and stores per thread is half
// as long: 82,944 order-3 elements 76.6 -> 70.8 us per stage, 279,936 order-2
// elements 167 -> 146 us, 14,586 order-5 elements 38.5 -> 37.7 us), four at
// order 4, where two would take 20 warps.
__host__ __device__ constexpr int tc_fn(int n) { return n == 4 ? 4 : 2; }
// Face node of LIFT column s of a face (>= Nfp: a padding column).  FN = 2 or 4
// consecutive columns are one flux unit, the nodes mg, mg + FG, .. of the face:
// the FG units of a face are neighbouring lanes, so each of their FN loads
// reads neighbouring nodes, which share 32-byte sectors (four consecutive nodes
// to a unit: 2.3 times the L1 sector accesses).
__host__ __device__ constexpr int tc_face_node(int n, int s) {
  const int fn = tc_fn(n), fg = (nfp_of(n) + fn - 1) / fn;
  return s >= fn * fg ? nfp_of(n) : fg * (s % fn) + s / fn;
}

template <int N>
struct TcCfg {
  static constexpr int NP = np_of(N), NFP = nfp_of(N), NF = 4 * NFP;
  static constexpr int M = tc_m(N);
  static constexpr int EQ = tc_eq(N);         // elements per lane quarter
  static constexpr int E = 4 * EQ;            // elements per tile
  static constexpr int QR = M / 4;            // MMA rows per lane quarter
  static constexpr int RL = 6 * EQ;           // real rows (lanes) per quarter
  // the two accumulator sets: side by side in the columns (M = 128), or in the
  // lane halves of the same columns (M = 64), each with its own A operand
  static constexpr bool LANE_SETS = M == 64;
  static constexpr int KV = tc_r8(NP);        // volume K (nodes)
  static constexpr int NV = tc_nv(N);         // volume N ((k,i) pairs)
  static constexpr int KLF = tc_r8(NFP);      // LIFT K per face
  static constexpr int KL = 4 * KLF;          // LIFT K (face nodes, per-face padded)
  static constexpr int NL = tc_nl(N);         // LIFT N (nodes)
  // The LIFT B operand stacks LIFT hi (rows 0..NL-1) over LIFT lo (rows NL..2NL-1),
  // so one MMA forms both products of an A half: N = 2 NL.
  static constexpr int NL2 = 2 * NL;
  // TMEM columns: the accumulator sets [vol | lift hi | lift lo], then the
  // volume A operand (hi, lo)
  static constexpr int ACC = NV + NL2;
  static constexpr int T_AHI = LANE_SETS ? ACC : 2 * ACC;
  static constexpr int T_ALO = T_AHI + KV;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TILE_F = E * 6 * NP;   // floats of state per tile
  static constexpr int TILE_B = TILE_F * 4;
  static constexpr int META_B = E * kMetaWords * 4;
  // per-thread work
  // flux units: (element, face, group of FN face nodes); faces 0-1 are one half
  // of the LIFT operand, faces 2-3 the other, each formed by its own warps
  static constexpr int FN = tc_fn(N);
  static constexpr int FG = (NFP + FN - 1) / FN;                                     // node groups per face
  static constexpr int UNITS_H = E * 2 * FG;                                   // units of a half
  static constexpr int WARPS_H = (UNITS_H + 31) / 32;                          // flux warps of a half
  // Warps by role: epilogue, 4 volume operand (both cover whole TMEM lane
  // quarters, quarter = warp % 4), then the order's flux warps, the control and
  // the copy warp.
  static constexpr int EPI_WARPS = 12;
  static constexpr int VOL_WARP = EPI_WARPS, VOL_WARPS = 4, EPI_GROUPS = EPI_WARPS / 4;
  static constexpr int FLUX_WARP = VOL_WARP + VOL_WARPS;
  static constexpr int CTL_WARP = FLUX_WARP + 2 * WARPS_H, COPY_WARP = CTL_WARP + 1;
  static constexpr int THREADS = (COPY_WARP + 1) * 32;
  static constexpr bool SLOT4 = N == 3;                                        // see tc_row_in_quarter
  static constexpr bool VEC = NP % 4 == 0;                                     // state rows are whole 16-byte vectors
  static constexpr int KS_H = KL / 16;                                         // LIFT k-steps per half
  static constexpr int VCH = KV / 8;                                           // volume-operand column chunks
  static constexpr int ECH = (NP + 3) / 4;                                     // epilogue node chunks of 4
  static constexpr int ECH_PER = (ECH + EPI_GROUPS - 1) / EPI_GROUPS;
  // M = 64: a 16-lane TMEM access serves two chunks of 4 columns (one per
  // thread half): the volume operand's K in VCH units of 8, the accumulator's
  // nodes in EPAIRS units of 8
  static constexpr int EPAIRS = (ECH + 1) / 2, EPAIR_PER = (EPAIRS + EPI_GROUPS - 1) / EPI_GROUPS;
  // byte sizes of the shared-memory operands (hi or lo)
  static constexpr int BV_B = NV * KV * 4;
  static constexpr int BL_B = NL2 * KL * 4;   // stacked hi/lo
  // bytes between the 4-column chunks of the LIFT A operand: a warp's flux
  // stores cover FG chunks of neighbouring elements' rows, and these 16-byte
  // units of padding spread them over the bank groups
  static constexpr int AL_CH = M * 16 + 16 * (N == 4 ? 2 : N == 2 ? 4 : N == 1 ? 0 : 3);
  static constexpr int AL_B = AL_CH * (KL / 4);
  static constexpr int YS_B = tc_r128(TILE_B);
  static constexpr int MS_B = tc_r128(META_B);
  // shared-memory map (bytes)
  static constexpr int O_BVH = 0;
  static constexpr int O_BVL = O_BVH + tc_r128(BV_B);
  static constexpr int O_BL = O_BVL + tc_r128(BV_B);
  static constexpr int O_ALH = O_BL + tc_r128(BL_B);
  static constexpr int O_ALL = O_ALH + tc_r128(AL_B);
  static constexpr int O_Y = O_ALL + tc_r128(AL_B);  // 3 state slots
  static constexpr int O_M = O_Y + 3 * YS_B;           // 3 element-record slots
  static constexpr int O_P = O_M + 3 * MS_B;           // 2 residual / output slots
  static constexpr int O_TAB = O_P + 2 * YS_B;
  // gather tables, each face's list padded to whole units
  static constexpr int TAB_B = kMaxGather * FN * FG;
  static constexpr int SMEM = O_TAB + tc_r128(TAB_B);
  static_assert(SMEM <= 232448 - 1024, "shared memory per CTA (dynamic + static)");
  static_assert(T_ALO + KV <= TMEM_COLS, "TMEM columns");
  static_assert((TILE_B % 16) == 0 && (META_B % 16) == 0, "bulk copies need 16-byte sizes");
  static_assert(NV <= 256 && NL2 <= 256 && (NV % (M == 128 ? 16 : 8)) == 0 && (NL2 % (M == 128 ? 16 : 8)) == 0,
                "MMA N limits");
  static_assert((M == 128 || M == 64) && RL <= QR && (!LANE_SETS || (VEC && ECH % 2 == 0)), "tile shape");
  static_assert(NP <= NL && 3 * NP <= NV, "accumulator columns");
  static_assert((KL % 16) == 0, "LIFT halves are whole k-steps");
};

// Constant operands prepared by the host: tf32 hi/lo of D (volume B) and LIFT,
// already in the chunk-major K-major byte layout (tc_util.cuh).
struct TcTables {
  const float* b_vol;    // [hi | lo], each NV*KV
  const float* b_lift;   // stacked [hi ; lo] rows, 2NL x KL (per-face padded K)
  const uint8_t* fnodes;
  const uint8_t* gtab;
  int n_gather;
};

// TMEM address offset of accumulator set s (and, at M = 64, of its A operand).
template <class C>
__device__ __forceinline__ uint32_t tc_set_off(int s) {
  return C::LANE_SETS ? ((uint32_t)(16 * s) << 16) : (uint32_t)(s * C::ACC);
}

// MMA row of (element le, component c) of a tile: slot EQ c + el of the element's
// lane quarter, rotated by EQ times the quarter.  At order 3 the slots are 4 c + el
// of the quarter's first four elements, then 24 + c of its fifth, rotated by 4 in
// the odd quarters: the state rows (5 c + 30 el 16-byte units) of eight neighbouring
// lanes then fall into eight bank groups, which the 16-byte accesses of the
// epilogue and the volume warps need, and the operand stores lose nothing (82,944
// elements: 70.7 -> 68.4 us per stage).  Padding the elements apart in shared
// memory instead, at the price of one bulk copy per element, measured 99 us.
template <class C>
__device__ __forceinline__ int tc_rot(int q) {
  return C::SLOT4 ? 4 * (q & 1) : C::EQ * q;
}
template <class C>
__device__ __forceinline__ int tc_row_in_quarter(int le, int c) {
  const int q = le / C::EQ, el = le - q * C::EQ;
  const int slot = !C::SLOT4 ? C::EQ * c + el : el < 4 ? 4 * c + el : 24 + c;
  return (slot + tc_rot<C>(q)) & (C::QR - 1);
}

// The slot of row r of quarter q (>= RL: a padding row), and what it holds.
template <class C>
__device__ __forceinline__ int tc_row_slot(int q, int r) {
  return (r - tc_rot<C>(q)) & (C::QR - 1);
}
template <class C>
__device__ __forceinline__ int tc_slot_el(int s) {
  return !C::SLOT4 ? s % C::EQ : s < 24 ? s & 3 : 4;
}
template <class C>
__device__ __forceinline__ int tc_slot_comp(int s) {
  return !C::SLOT4 ? s / C::EQ : s < 24 ? s >> 2 : s - 24;
}

// Nodes i0 .. i0 + 3 of a state row in shared or global memory (one 16-byte access where
// rows are whole vectors; Np = 10 and 35 go node by node).
template <class C>
__device__ __forceinline__ void tc_row_ld(const float* row, int i0, bool on, float (&v)[4]) {
  if constexpr (C::VEC) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) t = *reinterpret_cast<const float4*>(row + i0);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (on && i0 + u < C::NP) ? row[i0 + u] : 0.f;
  }
}
template <class C>
__device__ __forceinline__ void tc_row_st(float* row, int i0, bool on, const float (&v)[4]) {
  if (!on) return;
  if constexpr (C::VEC) {
    *reinterpret_cast<float4*>(row + i0) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u < C::NP) row[i0 + u] = v[u];
  }
}

// Bounded waits.  A wait gives up after `limit` polls or once another role has
// raised the abort flag; the warp form is warp-uniform.  A poll that finds the
// phase incomplete suspends the thread until the phase completes or a hardware
// time limit passes, measured at 3.98 us on B200, so kTcWaitLimit = 2^19 polls
// bounds a wait at about 2.1 s of wall time.  (A wall-clock check inside the
// loop was tried: any extra state in these inlined loops slows the stage
// kernel by 7 %.)
__device__ __forceinline__ bool tc_wait1(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                         uint32_t limit = kTcWaitLimit) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (tc::mbar_try_wait(bar, parity)) {
      return true;
    }
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ bool tc_waitw(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const bool ok = tc_wait1(bar, parity, abort_flag);
  return __all_sync(0xffffffffu, ok);
}

// Test hook for the bounded wait: one thread waits, with the kernels' own
// helper, on an mbarrier that expects one arrival that never comes.  It gives
// up after `limit` polls, records the time it waited (global timer) and raises
// `err` as a stage kernel does; nothing faults and the context stays usable.
__global__ void k_tc_wait_probe(uint32_t limit, int* err, unsigned long long* waited_ns) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_abort;
  if (threadIdx.x != 0) return;
  tc::mbar_init(&bar, 1);
  tc::mbar_fence_init();
  s_abort = 0;
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  const bool ok = tc_wait1(&bar, 0u, &s_abort, limit);
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  *waited_ns = t1 - t0;
  if (!ok) atomicExch(err, 1);
}

template <int N, int MODE>
__global__ void __launch_bounds__(TcCfg<N>::THREADS, 1)
rhs_tc_kernel(RhsParams P, TcTables T, int64_t n_tiles, int* err) {
  using C = TcCfg<N>;
  constexpr int NP = C::NP, NFP = C::NFP, E = C::E, M = C::M;
  constexpr int KV = C::KV, NV = C::NV, KLF = C::KLF, NL = C::NL, FG = C::FG, FN = C::FN;
  extern __shared__ __align__(1024) unsigned char tsm[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t bar_ld[3];   // state + records of a slot landed
  __shared__ __align__(8) uint64_t bar_p[2];    // residual / output slot ready (residual register landed)
  __shared__ __align__(8) uint64_t bar_avol;    // volume warps: volume operand in TMEM
  __shared__ __align__(8) uint64_t bar_alift[2];  // flux warps: LIFT operand half (faces 0-1 | 2-3) written
  __shared__ __align__(8) uint64_t bar_l0done;    // the MMAs of LIFT half 0 done (half 0 free)
  __shared__ __align__(8) uint64_t bar_vdone;   // volume MMAs done (TMEM operand free)
  __shared__ __align__(8) uint64_t bar_mma[2];  // all MMAs of an accumulator set done
  __shared__ __align__(8) uint64_t bar_epi[2];  // epilogue of a tile done (results staged)
  __shared__ int s_abort;
  volatile int* const abort_flag = &s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool is_epi = warp < C::EPI_WARPS;
  const bool is_vol = !is_epi && warp < C::FLUX_WARP;
  const bool is_flux = !is_epi && !is_vol && warp < C::CTL_WARP;
  const bool ctl0 = warp == C::CTL_WARP && lane == 0;
  const bool copy0 = warp == C::COPY_WARP && lane == 0;
  unsigned char* const alh = tsm + C::O_ALH;
  unsigned char* const all = tsm + C::O_ALL;
  float* const sY0 = reinterpret_cast<float*>(tsm + C::O_Y);
  float* const sM0 = reinterpret_cast<float*>(tsm + C::O_M);
  float* const sP0 = reinterpret_cast<float*>(tsm + C::O_P);
  constexpr int kYStride = C::YS_B / 4, kMStride = C::MS_B / 4;
  uint8_t* const sG = tsm + C::O_TAB;
  const bool use_p = MODE == kModeLserk && P.read_p;
  const int64_t tile0 = P.e_begin / E;  // the launch covers tiles [tile0, tile0 + n_tiles)

  // ---- set-up: TMEM, barriers, constant operands, tables (while the previous
  // launch still runs, on SMs that it leaves)
  if (warp == 0) tc::tmem_alloc(&s_tmem, C::TMEM_COLS);
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) tc::mbar_init(&bar_ld[i], 1);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bar_p[i], 1);
      tc::mbar_init(&bar_mma[i], 1);
      tc::mbar_init(&bar_epi[i], C::EPI_WARPS);
    }
    tc::mbar_init(&bar_avol, C::VOL_WARPS);
    tc::mbar_init(&bar_alift[0], C::WARPS_H);
    tc::mbar_init(&bar_alift[1], C::WARPS_H);
    tc::mbar_init(&bar_l0done, 1);
    tc::mbar_init(&bar_vdone, 1);
    tc::mbar_fence_init();
    s_abort = 0;
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(T.b_vol);
    for (int i = tid; i < C::BV_B / 16; i += C::THREADS) {
      reinterpret_cast<uint4*>(tsm + C::O_BVH)[i] = src[i];
      reinterpret_cast<uint4*>(tsm + C::O_BVL)[i] = src[C::BV_B / 16 + i];
    }
    src = reinterpret_cast<const uint4*>(T.b_lift);
    for (int i = tid; i < C::BL_B / 16; i += C::THREADS) reinterpret_cast<uint4*>(tsm + C::O_BL)[i] = src[i];
    // LIFT operand padding (the spare rows of each quarter, face-padding columns)
    // must hold finite values and is never written again: start from zero.
    for (int i = tid; i < C::AL_B / 16; i += C::THREADS) {
      reinterpret_cast<uint4*>(alh)[i] = make_uint4(0, 0, 0, 0);
      reinterpret_cast<uint4*>(all)[i] = make_uint4(0, 0, 0, 0);
    }
    for (int i = tid; i < T.n_gather * FN * FG; i += C::THREADS) {
      const int m = tc_face_node(N, i % (FN * FG));
      sG[i] = m < NFP ? T.gtab[(i / (FN * FG)) * NFP + m] : (uint8_t)0;
    }
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = s_tmem;
  // Only now, with this CTA's TMEM in hand: a CTA of the next launch that shared
  // its SM could otherwise take the columns first and wait for this grid, which
  // would wait for the columns, without a limit.  So a launch that waits for
  // columns lets no other in, and one that lets others in has all its columns,
  // whatever number of CTAs the compiler's register count lets an SM hold.
  pdl_launch();
  pdl_wait();
  // A launch flagged off (adaptive stepping past its last attempt, an Arnoldi step
  // past convergence) has no tiles.  It has set itself up all the same: the flag
  // belongs to an earlier kernel and is known only here.  In a queue of such
  // launches the set-ups overlap: an exponential step of 3,072 order-3 elements
  // with 9 of its 12 Arnoldi steps off takes 214 us, and took 340 us when each
  // launch began after its predecessor's end and an off stage returned at once.
  const bool off = P.skip != nullptr && *P.skip;
  const int64_t n_my = !off && n_tiles > (int64_t)blockIdx.x
                           ? (n_tiles - (int64_t)blockIdx.x + gridDim.x - 1) / gridDim.x
                           : 0;

#ifdef DGTD_TC_PHASE_TIMERS
  const bool timer_thread = lane == 0 && (warp == 0 || warp == C::VOL_WARP || warp == C::FLUX_WARP || warp >= C::CTL_WARP);
  unsigned long long clk_acc[kTcMarks] = {0};
  long long clk_last = clock64();
#endif

  if (is_vol) {
    // ================= volume warps: tf32 hi/lo of the state -> TMEM
    const int q4 = warp & 3;
    // the TMEM row this lane writes: its own lane, or (16-lane stores at M = 64)
    // lane & 15 of the set's lane half, the thread half choosing the columns
    const int v_slot = tc_row_slot<C>(q4, lane & (C::QR - 1));
    const bool lane_real = v_slot < C::RL;
    const int v_src = lane_real ? ((q4 * C::EQ + tc_slot_el<C>(v_slot)) * 6 + tc_slot_comp<C>(v_slot)) * NP : 0;
    const uint32_t v_taddr = tmem + ((uint32_t)(q4 * 32) << 16);
    int ys = 0;
    uint32_t ld_par = 0u;  // bit s: parity of the next wait on bar_ld[s]
    for (int64_t it = 0; it < n_my; ++it) {
      const float* const sY = sY0 + ys * kYStride;
      bool ok = tc_waitw(&bar_ld[ys], (ld_par >> ys) & 1u, abort_flag);
      ld_par ^= 1u << ys;
      if (ok && it > 0) ok = tc_waitw(&bar_vdone, (uint32_t)((it - 1) & 1), abort_flag);
      if (!ok) {
        *abort_flag = 1;
        break;
      }
      tc::tc_fence_after();
      DGTD_TC_MARK(0);
      // ---- volume operand: row (e,c) of this lane, K = nodes, tf32 hi/lo -> TMEM
      if constexpr (C::LANE_SETS) {
        // 8-column unit w: this thread half's 4 columns 8 w + 4 (lane >> 4) ..,
        // in the lane half of the tile's accumulator set
        const uint32_t a_taddr = v_taddr + tc_set_off<C>((int)(it & 1));
#pragma unroll
        for (int w = 0; w < C::VCH; ++w) {
          {
            const float4 v4 = *reinterpret_cast<const float4*>(sY + v_src + 8 * w + 4 * (lane >> 4));
            const float v[4] = {v4.x, v4.y, v4.z, v4.w};
            float h[4], l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float x = lane_real ? v[q] : 0.f;
              h[q] = tc::tf32_round(x);
              l[q] = x - h[q];
            }
            tc::tmem_st16x2_4(a_taddr + (uint32_t)(C::T_AHI + w * 8), h);
            tc::tmem_st16x2_4(a_taddr + (uint32_t)(C::T_ALO + w * 8), l);
          }
        }
      } else {
#pragma unroll
        for (int ch = 0; ch < C::VCH; ++ch) {
          {
            float x[8], h[8], l[8];
            if constexpr (C::VEC) {
#pragma unroll
              for (int w = 0; w < 2; ++w) {
                float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane_real && ch * 8 + 4 * w < NP) v4 = *reinterpret_cast<const float4*>(sY + v_src + ch * 8 + 4 * w);
                x[4 * w] = v4.x;
                x[4 * w + 1] = v4.y;
                x[4 * w + 2] = v4.z;
                x[4 * w + 3] = v4.w;
              }
            } else {
#pragma unroll
              for (int q = 0; q < 8; ++q) x[q] = (lane_real && ch * 8 + q < NP) ? sY[v_src + ch * 8 + q] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              // hi/lo split as for the LIFT operand (flux section below)
              h[q] = tc::tf32_round(x[q]);
              l[q] = x[q] - h[q];
            }
            tc::tmem_st8(v_taddr + (uint32_t)(C::T_AHI + ch * 8), h);
            tc::tmem_st8(v_taddr + (uint32_t)(C::T_ALO + ch * 8), l);
          }
        }
      }
      tc::tmem_st_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bar_avol);
      DGTD_TC_MARK(1);
      ys = ys == 2 ? 0 : ys + 1;
    }
  } else if (is_flux) {
    // ================= flux warps: numerical fluxes -> LIFT operand
    // This thread's flux unit: node group mg (tc_face_node) of face f of element
    // le.  One unit per thread and tile: what belongs to the face (normal,
    // scale, neighbour, face code) is read once for FN nodes, and the nodes of a
    // row are one vector of the LIFT operand.  The lanes of a face are
    // neighbours, so a load of an out-of-tile trace touches few cache lines
    // (neighbouring elements in neighbouring lanes: 28.1 against 21.3 ms for
    // five 48^3 order-4 steps).
    const int hh = (warp - C::FLUX_WARP) / C::WARPS_H;  // half of the LIFT operand
    const int uh = tid - (C::FLUX_WARP + hh * C::WARPS_H) * 32;
    const bool has_unit = uh < C::UNITS_H;
    const int mg = uh % FG, le = (uh / FG) % E, f = (2 * hh + uh / (FG * E)) & 3;
    int own[FN];  // offsets of the nodes' states in the tile (component 0)
#pragma unroll
    for (int i = 0; i < FN; ++i) {
      const int m = tc_face_node(N, FN * mg + i);
      own[i] = le * 6 * NP + (has_unit && m < NFP ? (int)T.fnodes[f * NFP + m] : 0);
    }
    const uint32_t a_off = (uint32_t)((f * (KLF / 4) + FN * mg / 4) * C::AL_CH + (FN * mg % 4) * 4 +
                                      (le / C::EQ) * C::QR * 16);
    int ys = 0;
    uint32_t ld_par = 0u;  // bit s: parity of the next wait on bar_ld[s]
    for (int64_t it = 0; it < n_my; ++it) {
      const int64_t e0 = (tile0 + blockIdx.x + it * gridDim.x) * E;
      const float* const sY = sY0 + ys * kYStride;
      const float* const sM = sM0 + ys * kMStride;
      bool ok = tc_waitw(&bar_ld[ys], (ld_par >> ys) & 1u, abort_flag);
      ld_par ^= 1u << ys;
      DGTD_TC_MARK(8);
      // The neighbour's traces at the unit's nodes, as pairs of nodes: from the
      // tile in shared memory when the neighbour is in it, else from L2.
      float tr[FN][6];
#pragma unroll
      for (int i = 0; i < FN; ++i)
#pragma unroll
        for (int c = 0; c < 6; ++c) tr[i][c] = 0.f;
      bool port = false, pec = false;
      if (ok && has_unit) {
        const float* Me = sM + le * kMetaWords;
        const uint32_t code = reinterpret_cast<const uint16_t*>(Me + 41)[f];
        const int kind = (int)(code >> 8) & 3;
        if (kind == kInterior) {
          int gn[FN];  // the neighbour's nodes
          if constexpr (FN == 4) {
            const uint32_t g = reinterpret_cast<const uint32_t*>(sG)[(code & 0xff) * FG + mg];
#pragma unroll
            for (int i = 0; i < FN; ++i) gn[i] = (g >> (8 * i)) & 0xff;
          } else {
            const uint32_t g = reinterpret_cast<const uint16_t*>(sG)[(code & 0xff) * FG + mg];
            gn[0] = g & 0xff;
            gn[1] = g >> 8;
          }
          const int nbr = __float_as_int(Me[37 + f]);
          const int lo = nbr - (int)e0;  // element ids fit in int
          if ((uint32_t)lo < (uint32_t)E) {
            const float* Z = sY + lo * 6 * NP;
#pragma unroll
            for (int c = 0; c < 6; ++c)
#pragma unroll
              for (int i = 0; i < FN; ++i) tr[i][c] = Z[gn[i] + c * NP];
          } else {
            const float* Z = P.y_in + (int64_t)nbr * (6 * NP);
#pragma unroll
            for (int c = 0; c < 6; ++c)
#pragma unroll
              for (int i = 0; i < FN; ++i) tr[i][c] = Z[gn[i] + c * NP];
          }
        } else if (kind == kPec) {
          // PEC ghost: [E] = 2 E_tan, [H] = 2 H_n (rhs.rs:1387-1402); both
          // products of the flux drop the normal [H].  The negated jump itself,
          // not the ghost: E is all but normal to a wall, and the rounding of a
          // difference with the ghost, or of a projection after it, is one of E
          // (relative error of an oblique wall's flux with 1 % of E tangential
          // 3e-6, against 6e-8 so).
          pec = true;
          const float nx = Me[9 + 3 * f], ny = Me[10 + 3 * f], nz = Me[11 + 3 * f];
#pragma unroll
          for (int i = 0; i < FN; ++i) {
            const float* Y = sY + own[i];
            const float ex = Y[0 * NP], ey = Y[1 * NP], ez = Y[2 * NP];
            const float edn = fmaf(nz, ez, fmaf(ny, ey, nx * ex));
            tr[i][0] = -2.f * fmaf(-edn, nx, ex);
            tr[i][1] = -2.f * fmaf(-edn, ny, ey);
            tr[i][2] = -2.f * fmaf(-edn, nz, ez);
          }
        } else {
          port = true;  // characteristic boundary against a zero incident field (rhs.rs:1380-1386)
        }
      }
      DGTD_TC_MARK(9);
      // ---- numerical flux (rhs.rs:1370-1441) into the unit's half of the LIFT
      // operand, which is free once the previous tile's MMAs of that half are
      // done; its own MMAs then run while the other half is formed.
      if (ok && it > 0)
        ok = hh == 0 ? tc_waitw(&bar_l0done, (uint32_t)((it - 1) & 1), abort_flag)
                     : tc_waitw(&bar_mma[(it - 1) & 1], (uint32_t)(((it - 1) >> 1) & 1), abort_flag);
      if (!ok) {
        *abort_flag = 1;
        break;
      }
      DGTD_TC_MARK(2);
      if (has_unit) {
        const float* Me = sM + le * kMetaWords;
        const float nx = Me[9 + 3 * f], ny = Me[10 + 3 * f], nz = Me[11 + 3 * f];
        const float coef = -0.5f * Me[21 + f], a = port ? 1.f : P.alpha;
        // fe = coef (-n x [H] + a n x (n x [E])), fh = coef (n x [E] + a n x (n x [H]))
        // (rhs.rs:1420-1432), with n x (n x v) = n (n.v) - v for the unit normal,
        // on the negated jumps j = trace - own and with k = -coef n:
        // a coef (n (n.[v]) - [v]) = (k.j) (a n) + a coef j.
        const uint64_t kx = tc::dup2(coef * nx), ky = tc::dup2(coef * ny), kz = tc::dup2(coef * nz);
        const uint64_t mx = tc::dup2(-coef * nx), my = tc::dup2(-coef * ny), mz = tc::dup2(-coef * nz);
        const uint64_t ax = tc::dup2(a * nx), ay = tc::dup2(a * ny), az = tc::dup2(a * nz);
        const uint64_t ca = tc::dup2(-coef * a);
        const uint64_t ow = tc::dup2(pec ? 0.f : -1.f);  // a PEC face's jump is formed above
#pragma unroll
        for (int i = 0; i < FN / 2; ++i) {
          const float* Y0 = sY + own[2 * i];
          const float* Y1 = sY + own[2 * i + 1];
          const uint64_t ex = tc::fma2(ow, tc::pack2(Y0[0 * NP], Y1[0 * NP]), tc::pack2(tr[2 * i][0], tr[2 * i + 1][0]));
          const uint64_t ey = tc::fma2(ow, tc::pack2(Y0[1 * NP], Y1[1 * NP]), tc::pack2(tr[2 * i][1], tr[2 * i + 1][1]));
          const uint64_t ez = tc::fma2(ow, tc::pack2(Y0[2 * NP], Y1[2 * NP]), tc::pack2(tr[2 * i][2], tr[2 * i + 1][2]));
          const uint64_t hx = tc::fma2(ow, tc::pack2(Y0[3 * NP], Y1[3 * NP]), tc::pack2(tr[2 * i][3], tr[2 * i + 1][3]));
          const uint64_t hy = tc::fma2(ow, tc::pack2(Y0[4 * NP], Y1[4 * NP]), tc::pack2(tr[2 * i][4], tr[2 * i + 1][4]));
          const uint64_t hz = tc::fma2(ow, tc::pack2(Y0[5 * NP], Y1[5 * NP]), tc::pack2(tr[2 * i][5], tr[2 * i + 1][5]));
          const uint64_t de = tc::fma2(kz, ez, tc::fma2(ky, ey, tc::mul2(kx, ex)));
          const uint64_t dh = tc::fma2(kz, hz, tc::fma2(ky, hy, tc::mul2(kx, hx)));
          tc::unpack2(tc::fma2(de, ax, tc::fma2(ca, ex, tc::fma2(kz, hy, tc::mul2(my, hz)))), tr[2 * i][0], tr[2 * i + 1][0]);
          tc::unpack2(tc::fma2(de, ay, tc::fma2(ca, ey, tc::fma2(kx, hz, tc::mul2(mz, hx)))), tr[2 * i][1], tr[2 * i + 1][1]);
          tc::unpack2(tc::fma2(de, az, tc::fma2(ca, ez, tc::fma2(ky, hx, tc::mul2(mx, hy)))), tr[2 * i][2], tr[2 * i + 1][2]);
          tc::unpack2(tc::fma2(dh, ax, tc::fma2(ca, hx, tc::fma2(ky, ez, tc::mul2(mz, ey)))), tr[2 * i][3], tr[2 * i + 1][3]);
          tc::unpack2(tc::fma2(dh, ay, tc::fma2(ca, hy, tc::fma2(kz, ex, tc::mul2(mx, ez)))), tr[2 * i][4], tr[2 * i + 1][4]);
          tc::unpack2(tc::fma2(dh, az, tc::fma2(ca, hz, tc::fma2(kx, ey, tc::mul2(my, ex)))), tr[2 * i][5], tr[2 * i + 1][5]);
        }
        // hi = tf32(flux), lo = flux - hi (exact, |lo| <= 2^-11 |flux|).  lo is
        // stored unrounded: the tf32 MMA reads only its top 19 bits, an error
        // below 2^-10 |lo| <= 2^-21 |flux|, under the 3xTF32 products' own
        // 2^-22-class terms in the sum of many products.
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const uint32_t off = a_off + (uint32_t)(tc_row_in_quarter<C>(le, c) * 16);
          float h[FN], l[FN];
#pragma unroll
          for (int i = 0; i < FN; ++i) {
            // the operand's padding columns stay zero whatever the fields hold
            if (tc_face_node(N, FN * (FG - 1) + i) >= NFP && tc_face_node(N, FN * mg + i) >= NFP) tr[i][c] = 0.f;
            h[i] = tc::tf32_round(tr[i][c]);
            l[i] = tr[i][c] - h[i];
          }
          if constexpr (FN == 4) {
            *reinterpret_cast<float4*>(alh + off) = make_float4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<float4*>(all + off) = make_float4(l[0], l[1], l[2], l[3]);
          } else {
            *reinterpret_cast<float2*>(alh + off) = make_float2(h[0], h[1]);
            *reinterpret_cast<float2*>(all + off) = make_float2(l[0], l[1]);
          }
        }
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bar_alift[hh]);
      DGTD_TC_MARK(3);
      ys = ys == 2 ? 0 : ys + 1;
    }
  } else if (is_epi) {
    // ================= epilogue warps: TMEM -> dy -> mode update, in place
    const int q4 = warp & 3, eg = warp >> 2;
    // the TMEM row of this lane: its own lane, or (16-lane loads at M = 64)
    // lane & 15, the thread half (hb = 0 | 16) reading the second chunk of a pair
    const int hb = C::LANE_SETS ? (lane & 16) : 0;
    const int e_slot = tc_row_slot<C>(q4, lane & (C::QR - 1));
    const bool lane_real = e_slot < C::RL;
    const int e_el = lane_real ? tc_slot_el<C>(e_slot) : C::EQ - 1, e_c = lane_real ? tc_slot_comp<C>(e_slot) : 5;
    const int e_le = q4 * C::EQ + e_el;
    const int e_fld = e_c / 3, e_t = e_c % 3;
    const int e_srcA = hb + tc_row_in_quarter<C>(e_le, 3 * (1 - e_fld) + (e_t + 2) % 3);
    const int e_srcB = hb + tc_row_in_quarter<C>(e_le, 3 * (1 - e_fld) + (e_t + 1) % 3);
    const float e_sign = e_fld == 0 ? 1.f : -1.f;
    const int e_cA = (e_t + 2) % 3, e_cB = (e_t + 1) % 3;
    const int e_row_off = (e_le * 6 + e_c) * NP;
    float kry_sig = 1.f, kry_g = 0.f;
    if (MODE == kModeKrylov) {
      kry_sig = (float)P.kry[0];
      kry_g = (float)P.kry[1];
    }
    float kcl_h = 0.f, kcl_gs = 0.f;
    if (MODE == kModeKcl) {
      kcl_h = *P.kcl_h;
      kcl_gs = P.kcl_g != nullptr ? P.kcl_g[*P.kcl_frame] : 0.f;
    }
    int ys = 0;
    uint32_t ld_par = 0u;
    for (int64_t it = 0; it < n_my; ++it) {
      const int64_t tile = tile0 + blockIdx.x + it * gridDim.x;
      const int ps = (int)(it & 1);
      const uint32_t ppar = (uint32_t)((it >> 1) & 1);
      bool ok = tc_waitw(&bar_mma[ps], ppar, abort_flag);
      DGTD_TC_MARK(10);
      if (ok) ok = tc_waitw(&bar_ld[ys], (ld_par >> ys) & 1u, abort_flag);
      ld_par ^= 1u << ys;
      if (ok) ok = tc_waitw(&bar_p[ps], ppar, abort_flag);
      if (!ok) {
        *abort_flag = 1;
        break;
      }
      tc::tc_fence_after();
      DGTD_TC_MARK(4);
      const float* Me = sM0 + ys * kMStride + e_le * kMetaWords;
      // curl partials (the B one negated) and material scaling with the curl sign folded in
      const uint64_t gA0 = tc::dup2(Me[0 * 3 + e_cA]), gA1 = tc::dup2(Me[1 * 3 + e_cA]), gA2 = tc::dup2(Me[2 * 3 + e_cA]);
      const uint64_t gB0 = tc::dup2(-Me[0 * 3 + e_cB]), gB1 = tc::dup2(-Me[1 * 3 + e_cB]), gB2 = tc::dup2(-Me[2 * 3 + e_cB]);
      const float inv_wf = Me[25 + 3 * e_fld + e_t];
      const uint64_t inv_w = tc::dup2(inv_wf), w_curl = tc::dup2(e_sign * inv_wf), sig_w = tc::dup2(-Me[31 + 3 * e_fld + e_t]);
      const float dt_e = P.dt * Me[43];  // the element's own step (batched instances)
      float* const yrow = sY0 + ys * kYStride + e_row_off;
      float* const prow = sP0 + ps * kYStride + e_row_off;  // p in, p out (LSERK) / dy out (Apply)
      const int64_t t0 = tile * C::TILE_F;
      // do the step's sources reach this tile? (uniform per tile)
      const bool src_here = (MODE == kModeLserk || MODE == kModeKrylov || MODE == kModeKcl) &&
                            (P.src_vec != nullptr || (P.src_idx >= t0 && P.src_idx < t0 + C::TILE_F));
      const int64_t g_row = t0 + e_row_off;  // SoA index of node 0 of this row
      const uint32_t acc = tmem + tc_set_off<C>(ps) + ((uint32_t)(q4 * 32) << 16);
      // node chunks of 4 (M = 128), or pairs of them, one per thread half (M = 64)
      constexpr int kIters = C::LANE_SETS ? C::EPAIR_PER : C::ECH_PER;
      constexpr int kUnits = C::LANE_SETS ? C::EPAIRS : C::ECH;
#pragma unroll
      for (int cc = 0; cc < kIters; ++cc) {
        const int ch = eg + C::EPI_GROUPS * cc;
        if (ch < kUnits) {
          const int c0 = C::LANE_SETS ? ch * 8 : ch * 4;  // first column of the access
          const int i0 = c0 + (hb >> 2);                  // this thread's first node
          float r0[4], r1[4], r2[4], lf[4], lg[4];
          if constexpr (C::LANE_SETS) {
            tc::tmem_ld16x2_4(acc + (uint32_t)c0, r0);
            tc::tmem_ld16x2_4(acc + (uint32_t)(NP + c0), r1);
            tc::tmem_ld16x2_4(acc + (uint32_t)(2 * NP + c0), r2);
            tc::tmem_ld16x2_4(acc + (uint32_t)(NV + c0), lf);
            tc::tmem_ld16x2_4(acc + (uint32_t)(NV + NL + c0), lg);
          } else {
            tc::tmem_ldw<4>(acc + (uint32_t)i0, r0);
            tc::tmem_ldw<4>(acc + (uint32_t)(NP + i0), r1);
            tc::tmem_ldw<4>(acc + (uint32_t)(2 * NP + i0), r2);
            tc::tmem_ldw<4>(acc + (uint32_t)(NV + i0), lf);
            tc::tmem_ldw<4>(acc + (uint32_t)(NV + NL + i0), lg);
          }
          tc::tmem_ld_wait();
          // dy at the four nodes: curl (the shuffles pair this row's partials
          // with the two other components'), LIFT, materials
          float dy[4], yv[4];
          tc_row_ld<C>(yrow, i0, lane_real, yv);
#pragma unroll
          for (int u = 0; u < 4; u += 2) {
            // my contributions: A to curl component (t+1)%3, B to (t+2)%3
            const uint64_t q0 = tc::pack2(r0[u], r0[u + 1]), q1 = tc::pack2(r1[u], r1[u + 1]), q2 = tc::pack2(r2[u], r2[u + 1]);
            float A0, A1, B0, B1;
            tc::unpack2(tc::fma2(gA2, q2, tc::fma2(gA1, q1, tc::mul2(gA0, q0))), A0, A1);
            tc::unpack2(tc::fma2(gB2, q2, tc::fma2(gB1, q1, tc::mul2(gB0, q0))), B0, B1);
            const uint64_t sa = tc::pack2(__shfl_sync(0xffffffffu, A0, e_srcA), __shfl_sync(0xffffffffu, A1, e_srcA));
            const uint64_t sb = tc::pack2(__shfl_sync(0xffffffffu, B0, e_srcB), __shfl_sync(0xffffffffu, B1, e_srcB));
            const uint64_t li = tc::add2(tc::pack2(lf[u], lf[u + 1]), tc::pack2(lg[u], lg[u + 1]));
            const uint64_t d = tc::fma2(w_curl, tc::add2(sa, sb),
                                        tc::fma2(inv_w, li, tc::mul2(sig_w, tc::pack2(yv[u], yv[u + 1]))));
            tc::unpack2(d, dy[u], dy[u + 1]);
          }
          if (MODE == kModeLserk) {
            // LSERK4 stage (explicit.rs:122-133): p = a p + dt (dy + src); y += b p
            if (src_here) {
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int i = i0 + u;
                if (lane_real && i < NP) {
                  if (P.src_vec != nullptr) dy[u] = fmaf(P.src_g, P.src_vec[g_row + i], dy[u]);
                  if (P.src_idx == g_row + i) dy[u] += P.src_g;
                }
              }
            }
            float pv[4];
            const uint64_t dt2 = tc::dup2(dt_e);
            uint64_t p01 = tc::mul2(dt2, tc::pack2(dy[0], dy[1])), p23 = tc::mul2(dt2, tc::pack2(dy[2], dy[3]));
            if (P.read_p) {
              tc_row_ld<C>(prow, i0, lane_real, pv);
              const uint64_t a2 = tc::dup2(P.a);
              p01 = tc::fma2(a2, tc::pack2(pv[0], pv[1]), p01);
              p23 = tc::fma2(a2, tc::pack2(pv[2], pv[3]), p23);
            }
            const uint64_t b2 = tc::dup2(P.b);
            tc::unpack2(p01, pv[0], pv[1]);
            tc::unpack2(p23, pv[2], pv[3]);
            tc::unpack2(tc::fma2(b2, p01, tc::pack2(yv[0], yv[1])), yv[0], yv[1]);
            tc::unpack2(tc::fma2(b2, p23, tc::pack2(yv[2], yv[3])), yv[2], yv[3]);
            tc_row_st<C>(prow, i0, lane_real, pv);
            tc_row_st<C>(yrow, i0, lane_real, yv);
          } else if (MODE == kModeKcl) {
            // KCL stage (explicit_adaptive.rs:84-152) straight to global
            // memory, in the operation order of the separate stage kernel
            // (kcl.cuh k_kcl_stage); nothing is staged for the bulk store
            const int64_t g = g_row + i0;
            float ky[4], ke[4], kn[4];
            tc_row_ld<C>(P.kcl_y + g_row, i0, lane_real, ky);
            if (P.kcl_stage != 0) tc_row_ld<C>(P.kcl_e + g_row, i0, lane_real, ke);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float kk = dy[u];
              if (src_here && lane_real && i0 + u < NP) {
                if (P.src_vec != nullptr) kk += P.src_vec[g + u] * kcl_gs;
                if (P.src_idx == g + u) kk += kcl_gs;
              }
              const float fk = kcl_h * kk;
              ky[u] = ky[u] + P.kcl_b * fk;
              ke[u] = P.kcl_stage == 0 ? P.kcl_ew * fk : ke[u] + P.kcl_ew * fk;
              kn[u] = ky[u] + P.kcl_amb * fk;
            }
            tc_row_st<C>(P.kcl_y + g_row, i0, lane_real, ky);
            tc_row_st<C>(P.kcl_e + g_row, i0, lane_real, ke);
            if (P.kcl_next != nullptr) tc_row_st<C>(P.kcl_next + g_row, i0, lane_real, kn);
          } else {
            if (MODE == kModeKrylov) {
              // Krylov matvec of a stored basis vector: its scale and the
              // augmented source coefficient from device memory
#pragma unroll
              for (int u = 0; u < 4; ++u) dy[u] *= kry_sig;
              if (src_here) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const int i = i0 + u;
                  if (lane_real && i < NP) {
                    if (P.src_vec != nullptr) dy[u] = fmaf(kry_g, P.src_vec[g_row + i], dy[u]);
                    if (P.src_idx == g_row + i) dy[u] += kry_g;
                  }
                }
              }
            }
            tc_row_st<C>(prow, i0, lane_real, dy);
          }
        }
      }
      tc::tc_fence_before();
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bar_epi[ps]);
      DGTD_TC_MARK(5);
      ys = ys == 2 ? 0 : ys + 1;
    }
  } else if (ctl0) {
    // ================= control lane: MMAs
    uint32_t n_mma[2] = {0u, 0u}, n_vd = 0u, n_l0 = 0u;
    const uint32_t idv = tc::idesc_tf32(M, NV), idl = tc::idesc_tf32(M, C::NL2);
    // Shared-memory descriptors of k-step 0, built once: a k-step adds two chunks
    // (in 16-byte units) to the start-address field, which cannot carry (shared
    // addresses are below 2^18).  With the k-steps fully unrolled the issue of an
    // MMA is an add and the instruction itself, so one thread keeps the tensor
    // pipe fed.
    const uint64_t dvh = tc::tf32_step_desc(tc::smem_u32(tsm + C::O_BVH), NV, 0);
    const uint64_t dvl = tc::tf32_step_desc(tc::smem_u32(tsm + C::O_BVL), NV, 0);
    const uint64_t dbl = tc::tf32_step_desc(tc::smem_u32(tsm + C::O_BL), C::NL2, 0);
    const uint64_t dah = tc::smem_desc(tc::smem_u32(alh), C::AL_CH, 128u);
    const uint64_t dal = tc::smem_desc(tc::smem_u32(all), C::AL_CH, 128u);
    bool ok = true;
    for (int64_t it = 0; it < n_my && ok; ++it) {
      const int as = (int)(it & 1);
      const uint32_t acc = tmem + tc_set_off<C>(as);
      // the volume A operand: one for both sets (M = 128) or the set's own (M = 64)
      const uint32_t a_base = tmem + (C::LANE_SETS ? tc_set_off<C>(as) : 0u);
      // volume MMAs: A = state hi/lo (TMEM), B = D hi/lo (shared); the accumulator
      // set is free once tile it-2's epilogue is done
      ok = tc_wait1(&bar_avol, (uint32_t)(it & 1), abort_flag);
      if (ok && it > 1) ok = tc_wait1(&bar_epi[as], (uint32_t)(((it - 2) >> 1) & 1), abort_flag);
      if (!ok) break;
      tc::tc_fence_after();
      DGTD_TC_MARK(6);
#pragma unroll
      for (int ks = 0; ks < KV / 8; ++ks) {
        const uint32_t a_h = a_base + (uint32_t)(C::T_AHI + 8 * ks), a_l = a_base + (uint32_t)(C::T_ALO + 8 * ks);
        const uint64_t bh = dvh + (uint64_t)(2 * NV * ks), bo = dvl + (uint64_t)(2 * NV * ks);
        tc::mma_tf32_ta(acc, a_h, bh, idv, ks > 0 ? 1u : 0u);
        tc::mma_tf32_ta(acc, a_h, bo, idv, 1u);
        tc::mma_tf32_ta(acc, a_l, bh, idv, 1u);
      }
      tc::mma_commit(&bar_vdone);
      ++n_vd;
      // LIFT MMAs by halves: A = flux hi/lo (shared), B = stacked LIFT hi/lo
      // (shared): columns [NV, NV+NL) collect hi*hi + lo*hi, [NV+NL, NV+2NL)
      // hi*lo + lo*lo.  Half 0's commit frees it for the next tile's flux.
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        ok = tc_wait1(&bar_alift[hh], (uint32_t)(it & 1), abort_flag);
        if (!ok) break;
        tc::tc_fence_after();
        DGTD_TC_MARK(6);
#pragma unroll
        for (int j = 0; j < C::KS_H; ++j) {
          const int ks = hh * C::KS_H + j;
          const uint64_t bd = dbl + (uint64_t)(2 * C::NL2 * ks);
          tc::mma_tf32(acc + (uint32_t)NV, dah + (uint64_t)(C::AL_CH / 8 * ks), bd, idl, ks > 0 ? 1u : 0u);
          tc::mma_tf32(acc + (uint32_t)NV, dal + (uint64_t)(C::AL_CH / 8 * ks), bd, idl, 1u);
        }
        if (hh == 0) {
          tc::mma_commit(&bar_l0done);
          ++n_l0;
        } else {
          tc::mma_commit(&bar_mma[as]);
          ++n_mma[as];
        }
      }
    }
    if (!ok) {
      *abort_flag = 1;
      // let the MMAs still in flight finish before the CTA exits
      for (int s = 0; s < 2; ++s)
        if (n_mma[s]) (void)tc::mbar_wait(&bar_mma[s], (n_mma[s] - 1) & 1u, kTcWaitLimit);
      if (n_vd) (void)tc::mbar_wait(&bar_vdone, (n_vd - 1) & 1u, kTcWaitLimit);
      if (n_l0) (void)tc::mbar_wait(&bar_l0done, (n_l0 - 1) & 1u, kTcWaitLimit);
    }
  } else if (copy0) {
    // ================= copy lane: bulk loads and stores.  A tile's slots are
    // refilled as soon as its results have been read out of them: the state
    // three tiles on, the residual two.
    uint32_t n_ld[3] = {0u, 0u, 0u}, n_p[2] = {0u, 0u};
    auto load_y = [&](int64_t j) {  // tile j of this CTA -> slot j % 3
      const int s = (int)(j % 3);
      const int64_t tile = tile0 + blockIdx.x + j * gridDim.x;
      tc::mbar_expect_tx(&bar_ld[s], C::TILE_B + C::META_B);
      tc::bulk_g2s(sM0 + s * kMStride, P.meta + tile * E * kMetaWords, C::META_B, &bar_ld[s]);
      tc::bulk_g2s(sY0 + s * kYStride, P.y_in + tile * C::TILE_F, C::TILE_B, &bar_ld[s]);
      ++n_ld[s];
    };
    auto load_p = [&](int64_t j) {  // slot j & 1: free for tile j's results, with its residual register
      const int s = (int)(j & 1);
      if (use_p) {
        const int64_t tile = tile0 + blockIdx.x + j * gridDim.x;
        tc::mbar_expect_tx(&bar_p[s], C::TILE_B);
        tc::bulk_g2s(sP0 + s * kYStride, P.p + tile * C::TILE_F, C::TILE_B, &bar_p[s]);
      } else {
        tc::mbar_arrive(&bar_p[s]);
      }
      ++n_p[s];
    };
    for (int64_t j = 0; j < 3 && j < n_my; ++j) load_y(j);
    for (int64_t j = 0; j < 2 && j < n_my; ++j) load_p(j);
    bool ok = true;
    for (int64_t j = 0; j < n_my; ++j) {
      ok = tc_wait1(&bar_epi[j & 1], (uint32_t)((j >> 1) & 1), abort_flag);
      if (!ok) break;
      DGTD_TC_MARK(11);
      const int64_t gb = (tile0 + (int64_t)blockIdx.x + j * gridDim.x) * C::TILE_F;
      const float* sy = sY0 + (int)(j % 3) * kYStride;
      const float* sp = sP0 + (int)(j & 1) * kYStride;
      if (MODE == kModeApply || MODE == kModeKrylov) {
        tc::bulk_s2g(P.out + gb, sp, C::TILE_B);
      } else if (MODE == kModeLserk) {
        tc::bulk_s2g(P.out + gb, sy, C::TILE_B);
        if (P.write_p) tc::bulk_s2g(P.p + gb, sp, C::TILE_B);
      }  // kModeKcl: the epilogue wrote global memory itself
      tc::bulk_commit();
      tc::bulk_wait_read0();
      DGTD_TC_MARK(7);
      if (j + 3 < n_my) load_y(j + 3);
      if (j + 2 < n_my) load_p(j + 2);
    }
    tc::bulk_wait0();
    if (!ok) {
      *abort_flag = 1;
      // let the copies still in flight finish before the CTA exits
      for (int s = 0; s < 3; ++s)
        if (n_ld[s]) (void)tc::mbar_wait(&bar_ld[s], (n_ld[s] - 1) & 1u, kTcWaitLimit);
      for (int s = 0; s < 2; ++s)
        if (n_p[s]) (void)tc::mbar_wait(&bar_p[s], (n_p[s] - 1) & 1u, kTcWaitLimit);
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(err, 1);
#ifdef DGTD_TC_PHASE_TIMERS
  if (timer_thread && P.phase_clk != nullptr)
    for (int i = 0; i < kTcMarks; ++i) atomicAdd(P.phase_clk + i, clk_acc[i]);
#endif
  if (warp == 0) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace dgtd
