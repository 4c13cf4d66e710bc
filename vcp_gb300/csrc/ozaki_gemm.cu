// ozaki_gemm.cu -- the slice GEMM of the Ozaki form on tcgen05 tensor cores.
//
// A work item is one output tile (128 x 256) and one group of digit / residue
// plane pairs (A_p, B_q).  Each pair is a bf16 GEMM over the whole (padded)
// inner dimension, split into chunks of 1024: every chunk accumulates in fp32
// in tensor memory, where it is an exact integer (|digit products| <= 2^14,
// 1024 of them <= 2^24).  Epilogue warps drain each finished chunk
// (double-buffered TMEM accumulators, so draining overlaps the next chunk's
// MMAs) and, per mode:
//   OZ_CRT       group g = modulus m_g: the residue of the integer product
//                mod m_g, one byte per entry in res[g][col][row] (reduced on
//                the FP32 pipe straight from TMEM; several chunks: the sum of
//                their reductions, reduced again);
//   OZ_RAD_SET / OZ_RAD_ADD  all digit pairs of one radius product form one
//                group: every chunk is weighted by its pair's 2^(8 (t_ref - t))
//                and summed upward in fp32, one fold per (product, tile) into
//                P (radius factors were rounded up, so the sum bounds them);
//   OZ_MID       (slice form) folds into an int64 fixed-point value
//                W = sum_t C_t 2^(8 (t_ref - t)) in global memory; the last
//                fold is merged into the final epilogue
//                [lo, up] = [RD(W unit) - e, RU((W + R) unit) + e].
//
// Grouped products (a batch bucket) load B in 64-row boxes and multiply only
// the 64-column blocks of a tile that hold columns of its problem (MMA N =
// 64 .. 256): a narrow problem moves and multiplies a quarter to three
// quarters of a full tile; the epilogue skips the blocks that were not
// multiplied (their columns are past N and never stored for reassembly).
//
// Warp roles (320 threads, one CTA per SM, persistent over tiles):
//   warp 0      TMA producer (4-stage ring of 48 KB A+B k-blocks; pairs: 6 of 32)
//   warp 1      TMEM owner + MMA issuer (one thread)
//   warps 2..9  epilogue: warp w reads TMEM lanes 32*(w%4).. and columns
//               128*((w-2)/4).. of each accumulator.
// Every mbarrier wait is bounded; a timeout sets flag[1] and the CTA winds
// down (waits for its copies and MMAs, frees TMEM, returns).
//
// CTA pairs (PAIR; use_pairs below says where): two CTAs work on a 256 x 256
// tile with cta_group::2 MMAs.  Each still owns 128 rows of the result and its
// epilogue, but loads only half of the B tile: 32 KB a k-block instead of 48,
// so that the ring holds six stages in place of four, shared memory is read
// less per MMA, and a third of the traffic from L2 goes away.  The issuer's
// cycles per 1024-deep chunk (8192 at the tensor peak), single CTAs -> pairs:
// 1225x1225x12544 11050 -> 9820, 4096^3 11430 -> 10830.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "swfp.cuh"
#include "tc_ptx.cuh"

#include <mutex>

namespace vcpcu {

namespace {

constexpr int NTHREADS = 320;
constexpr int A_STAGE = OZ_BM * OZ_BK * 2;  // 16 KB
constexpr int B_STAGE = OZ_BN * OZ_BK * 2;  // 32 KB
constexpr int B_SUB = 64 * OZ_BK * 2;       // 8 KB: one 64-column block of B
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
// A CTA of a pair: 128 rows of A, 128 of the tile's 256 columns of B
constexpr int PAIR_STAGE_BYTES = A_STAGE + B_STAGE / 2;
constexpr int PAIR_STAGES = 6;
static_assert(PAIR_STAGES * PAIR_STAGE_BYTES == OZ_STAGES * STAGE_BYTES, "one ring size");
constexpr int TMEM_COLS = 512;  // two 128 x 256 fp32 accumulators

template <int STAGES>
struct Smem {
  uint64_t full[STAGES], empty[STAGES];
  uint64_t tfull[2], tempty[2];
  uint64_t mma_done;
  uint32_t tmem_base;
  int abort;
};

template <class S>
__device__ __forceinline__ void raise_timeout(S* sm, int* flag, int where) {
  atomicOr(&flag[1], 1 << where);
  *(volatile int*)&sm->abort = 1;
}

// An epilogue warp hands an accumulator back to the issuer (the pair's leader);
// the issuer's wait for it.
template <bool PAIR>
__device__ __forceinline__ void release_acc(uint64_t* tempty) {
  if constexpr (PAIR)
    ptx::mbar_arrive_cluster(ptx::leader_addr(tempty));
  else
    ptx::mbar_arrive(tempty);
}
template <bool PAIR>
__device__ __forceinline__ bool wait_acc(uint64_t* tempty, uint32_t par, long long lim) {
  if constexpr (PAIR)
    return ptx::mbar_wait_cluster(tempty, par, lim);
  else
    return ptx::mbar_wait(tempty, par, lim);
}

__device__ __forceinline__ double scale_dir(double x, int e, bool up) {
  while (e > 1023) {
    x = up ? __dmul_ru(x, 0x1p1023) : __dmul_rd(x, 0x1p1023);
    e -= 1023;
  }
  while (e < -1022) {
    x = up ? __dmul_ru(x, 0x1p-1022) : __dmul_rd(x, 0x1p-1022);
    e += 1022;
  }
  const double p = __longlong_as_double((long long)(e + 1023) << 52);
  return up ? __dmul_ru(x, p) : __dmul_rd(x, p);
}

// Smallest double >= 2^e (e may be below the subnormal range).
__device__ __forceinline__ double pow2_ru(int e) {
  if (e >= -1022) return scale_dir(1.0, e, true);
  if (e >= -1074) return __longlong_as_double(1LL << (e + 1074));
  return __longlong_as_double(1LL);
}

// Tile order: groups of OZ_RASTER row blocks, column blocks outer inside a
// group, so the CTAs resident at one time share a few A row panels and
// B column panels (both stay in L2 across the CTAs of one group).
constexpr int OZ_RASTER = 16;
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int& tm, int& tn,
                                            int raster = OZ_RASTER) {
  const int per_group = raster * tiles_n;
  const int g = tile / per_group;
  const int rows = min(raster, tiles_m - g * raster);
  const int idx = tile - g * per_group;
  tn = idx / rows;
  tm = g * raster + idx % rows;
}

// Work items.  MID (slice form): one item per tile, all groups (the groups
// accumulate into one W).  CRT and radius modes: one item per (group, tile),
// group-major -- every group writes its own residue plane or fold slots, so
// items are independent, and the CTAs in flight share one group's planes
// (compact L2 working set; the tail is one group of one tile).  Grouped
// products: the items of problem p follow one another, group-major within p.
struct ItemInfo {
  int arow, bcol;   // TMA row of the A tile / of the B tile in the planes
  int tm, tn, g0, g1;
  int nb;           // 64-column blocks of B the tile multiplies (1..4)
  int kblocks;      // k-blocks of its problem
  int Mp, Np;       // output layout of this item's problem
  int M, N;         // its valid rows / columns
  uint8_t* res;
  int32_t* P;
};

// PAIR: ntiles and the tile index count pairs of row blocks; `rank` is this
// CTA's block of the pair.
template <bool PAIR, bool GROUP>
__device__ __forceinline__ ItemInfo item_info(const OzGemmArgs& a, int item, int ntiles,
                                              int rank) {
  ItemInfo f;
  f.kblocks = a.Kp / OZ_BK;
  if constexpr (GROUP) {
    const int p = a.gprob[item];
    const OzGProb& q = a.gp[p];
    f.kblocks = q.Kp / OZ_BK;
    const int nt = q.tiles_m * q.tiles_n;
    const int local = item - a.gitem[p];
    f.g0 = local / nt;
    f.g1 = f.g0 + 1;
    tile_coords(local - f.g0 * nt, q.tiles_m, q.tiles_n, f.tm, f.tn);
    f.arow = q.arow + f.tm * OZ_BM * f.kblocks;
    f.bcol = q.brow + f.tn * OZ_BN * f.kblocks;
    f.Mp = q.Mp;
    f.Np = q.Np;
    f.M = q.m;
    f.N = q.n;
    // only the 64-column blocks that hold columns of the problem are loaded and
    // multiplied (tmB has 64-row boxes; MMA N = 64 .. 256)
    f.nb = min(4, (f.N - f.tn * OZ_BN + 63) >> 6);
    f.res = a.res ? a.res + q.res_off : nullptr;
    f.P = a.P ? a.P + q.P_off : nullptr;
    return f;
  }
  int tile = item;
  if (!PAIR && !GROUP && a.mode == OZ_MID) {
    f.g0 = 0;
    f.g1 = a.pl.ngroups;
  } else {
    f.g0 = item / ntiles;
    f.g1 = f.g0 + 1;
    tile = item - f.g0 * ntiles;
  }
  if (PAIR) {
    tile_coords(tile, (a.tiles_m + 1) >> 1, a.tiles_n, f.tm, f.tn, OZ_RASTER / 2);
    f.tm = 2 * f.tm + rank;  // (past the last row block: loads give zeros, all rows are padding)
  } else {
    tile_coords(tile, a.tiles_m, a.tiles_n, f.tm, f.tn);
  }
  const int unit = a.tiled ? f.kblocks : 1;  // rows of the tensor map per line
  f.arow = f.tm * OZ_BM * unit;
  f.bcol = f.tn * OZ_BN * unit;
  f.Mp = a.Mp;
  f.Np = a.Np;
  f.M = a.M;
  f.N = a.N;
  f.nb = 4;
  f.res = a.res;
  f.P = a.P;
  return f;
}

__device__ __forceinline__ int chunks_of(int kblocks) {
  return (kblocks + OZ_CHUNK / OZ_BK - 1) / (OZ_CHUNK / OZ_BK);
}

// The CTA's (or pair's) place among those of the grid; read where it is used,
// so that the epilogue's registers stay free of it.
template <bool PAIR>
__device__ __forceinline__ int worker() {
  return PAIR ? blockIdx.x >> 1 : blockIdx.x;
}
template <bool PAIR>
__device__ __forceinline__ int nworkers() {
  return PAIR ? gridDim.x >> 1 : gridDim.x;
}

// Residue of a one-chunk CRT group on the FP32 pipe (no float-to-int
// conversion, which GB300 issues on its narrow XU pipe, and no integer
// reduction).  The chunk value x is an exact integer with |x| <= 2^24, so
// |RN(x RN(1/m)) - x/m| <= (2^24/m) 2^-23 (1 + 2^-25) and q = rint of it
// (the add and subtract of 1.5 2^23) is within 1/2 + 2.0000002/m of x/m:
// r = RN(q (-m) + x) (one FMA, exact) is an integer with |r| <= m/2 + 2,
// and adding m to a negative r gives [0, m) (m >= 107).  The epilogue
// evaluates it for two columns per paired FP32 instruction.

__device__ __forceinline__ long long shift_t(int c, int sh) {
  const long long v = (long long)c;
  return sh >= 0 ? (v << sh) : (v >> (-sh));
}

// GROUP: the products of a batch bucket (never pairs).
template <bool PAIR, bool GROUP>
__global__ void __launch_bounds__(NTHREADS, 1)
oz_slice_gemm_kernel(const __grid_constant__ OzGemmArgs args) {
  constexpr int STAGES = PAIR ? PAIR_STAGES : OZ_STAGES;
  constexpr int STAGE = PAIR ? PAIR_STAGE_BYTES : STAGE_BYTES;
  extern __shared__ uint8_t dsmem_raw[];
  __shared__ Smem<STAGES> sm;
  uint8_t* dsmem = (uint8_t*)(((uintptr_t)dsmem_raw + 1023) & ~(uintptr_t)1023);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = PAIR ? (int)ptx::cluster_rank() : 0;
  const int ntiles = (PAIR ? (args.tiles_m + 1) >> 1 : args.tiles_m) * args.tiles_n;
  const bool mid = !PAIR && !GROUP && args.mode == OZ_MID;
  const int nitems = GROUP ? args.gnitems : (mid ? ntiles : ntiles * args.pl.ngroups);
  const long long lim = args.timeout_cycles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      ptx::mbar_init(&sm.full[i], 1);
      ptx::mbar_init(&sm.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&sm.tfull[i], 1);
      ptx::mbar_init(&sm.tempty[i], PAIR ? 16 : 8);  // the epilogue warps of both CTAs
    }
    ptx::mbar_init(&sm.mma_done, 1);
    sm.abort = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      ptx::tmem_alloc_pair(&sm.tmem_base, TMEM_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(&sm.tmem_base, TMEM_COLS);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) ptx::cluster_sync();  // the peer's barriers are initialised
  ptx::tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  if constexpr (!GROUP) {
    dep_wait();  // the planes are there
    dep_ready();
  }
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      ptx::prefetch_tmap(&args.tmA);
      ptx::prefetch_tmap(&args.tmB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t used = 0, lastpar = 0;  // per-stage bit masks
      // a k-block further: the next tile of the line block (tiled planes), or
      // 64 entries along the lines
      const int kx = args.tiled ? 0 : OZ_BK;
      const int ka = args.tiled ? OZ_BM : 0, kbb = args.tiled ? OZ_BN : 0;
      for (int item = worker<PAIR>(); item < nitems && ok; item += nworkers<PAIR>()) {
        const ItemInfo f = item_info<PAIR, GROUP>(args, item, ntiles, rank);
        for (int pi = args.pl.gstart[f.g0]; pi < args.pl.gstart[f.g1] && ok; ++pi) {
          const int pa = args.pl.pa[pi], pb = args.pl.pb[pi];
          for (int kb = 0; kb < f.kblocks; ++kb) {
            if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.empty[stage], phase ^ 1, lim)) {
              if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 0);
              ok = false;
              break;
            }
            uint8_t* sA = dsmem + stage * STAGE;
            uint8_t* sB = sA + A_STAGE;
            if constexpr (PAIR) {
              // both CTAs' bytes count on the leader's barrier, which the
              // issuer waits for
              const uint32_t bar = ptx::leader_addr(&sm.full[stage]);
              if (rank == 0) ptx::mbar_expect_tx(&sm.full[stage], 2 * PAIR_STAGE_BYTES);
              ptx::tma_load_3d_pair(sA, &args.tmA, bar, kb * kx, f.arow + kb * ka, pa);
              ptx::tma_load_3d_pair(sB, &args.tmB, bar, kb * kx, f.bcol + kb * kbb + 128 * rank, pb);
            } else {
              ptx::mbar_expect_tx(&sm.full[stage], A_STAGE + f.nb * B_SUB);
              ptx::tma_load_3d(sA, &args.tmA, &sm.full[stage], kb * kx, f.arow + kb * ka, pa);
              if constexpr (GROUP) {
                // 64-row boxes land back to back: the same SW128 K-major
                // layout as one box of 64 nb rows
                for (int i = 0; i < f.nb; ++i)
                  ptx::tma_load_3d(sB + i * B_SUB, &args.tmB, &sm.full[stage], kb * kx,
                                   f.bcol + kb * kbb + 64 * i, pb);
              } else {
                ptx::tma_load_3d(sB, &args.tmB, &sm.full[stage], kb * kx, f.bcol + kb * kbb, pb);
              }
            }
            used |= 1u << stage;
            lastpar = (lastpar & ~(1u << stage)) | (phase << stage);
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
      // every issued copy has landed before the CTA may exit (immediate in
      // the normal case: the MMA thread consumed them all); of a pair, the
      // issuer's arrivals on this CTA's empty barriers too
      for (int i = 0; i < STAGES; ++i)
        if (used & (1u << i)) {
          if (rank == 0) ptx::mbar_wait(&sm.full[i], (lastpar >> i) & 1u, lim);
          if (PAIR) ptx::mbar_wait(&sm.empty[i], (lastpar >> i) & 1u, lim);
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0 && rank == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc = 0;  // global chunk counter
      bool ok = true;
      for (int item = worker<PAIR>(); item < nitems && ok; item += nworkers<PAIR>()) {
        const ItemInfo f = item_info<PAIR, GROUP>(args, item, ntiles, rank);
        const int nchunks = chunks_of(f.kblocks);
        const uint32_t idesc =
            PAIR ? ptx::idesc_bf16_f32(2 * OZ_BM, OZ_BN) : ptx::idesc_bf16_f32(OZ_BM, 64 * f.nb);
        for (int pi = args.pl.gstart[f.g0]; pi < args.pl.gstart[f.g1] && ok; ++pi) {
          for (int ch = 0; ch < nchunks && ok; ++ch, ++acc) {
            const int buf = acc & 1;
            const uint32_t par = (acc >> 1) & 1;
            if (*(volatile int*)&sm.abort || !wait_acc<PAIR>(&sm.tempty[buf], par ^ 1, lim)) {
              if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 1);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t dt = tmem + buf * OZ_BN;
            const int kb0 = ch * (OZ_CHUNK / OZ_BK);
            const int kb1 = min(f.kblocks, kb0 + OZ_CHUNK / OZ_BK);
            for (int kb = kb0; kb < kb1; ++kb) {
              if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.full[stage], phase, lim)) {
                if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 2);
                ok = false;
                break;
              }
              ptx::tc_fence_after();
              const uint32_t sA = ptx::smem_u32(dsmem + stage * STAGE);
              const uint32_t sB = sA + A_STAGE;
#pragma unroll
              for (int kk = 0; kk < OZ_BK / 16; ++kk) {
                const uint64_t ad = ptx::sw128_kmajor_desc(sA + kk * 32);
                const uint64_t bd = ptx::sw128_kmajor_desc(sB + kk * 32);
                if constexpr (PAIR)
                  ptx::mma_bf16_pair(dt, ad, bd, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
                else
                  ptx::mma_bf16(dt, ad, bd, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
              }
              if constexpr (PAIR)
                ptx::mma_commit_pair(&sm.empty[stage]);
              else
                ptx::mma_commit(&sm.empty[stage]);
              if (++stage == STAGES) {
                stage = 0;
                phase ^= 1;
              }
            }
            if (!ok) break;
            if constexpr (PAIR)
              ptx::mma_commit_pair(&sm.tfull[buf]);
            else
              ptx::mma_commit(&sm.tfull[buf]);
          }
        }
      }
      // all MMAs of this thread done before TMEM is released; of a pair, the
      // peer's last arrivals on this CTA's barriers too
      if constexpr (PAIR)
        ptx::mma_commit_pair(&sm.mma_done);
      else
        ptx::mma_commit(&sm.mma_done);
      ptx::mbar_wait(&sm.mma_done, 0, lim);
      if (PAIR && ok)
        for (uint32_t a = acc > 2 ? acc - 2 : 0; a < acc; ++a)
          wait_acc<PAIR>(&sm.tempty[a & 1], (a >> 1) & 1, lim);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int ew = warp - 2;
    const int quarter = warp & 3;
    const int half = ew >> 2;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    uint32_t acc = 0;
    bool ok = true;
    bool nonfinite = args.flag[0] != 0;
    for (int item = worker<PAIR>(); item < nitems && ok; item += nworkers<PAIR>()) {
      const ItemInfo f = item_info<PAIR, GROUP>(args, item, ntiles, rank);
      const int g0 = f.g0, g1 = f.g1;
      const int nchunks = chunks_of(f.kblocks);
      const int gi = f.tm * OZ_BM + row_in_tile;
      const int gj0 = f.tn * OZ_BN + half * 128;
      if (!mid && f.tm * OZ_BM + quarter * 32 >= f.M) {
        // this warp's 32 rows are all past M (padding of the tile): release
        // each accumulator of the item unread -- the reassembly reads no
        // padding row (midpoint folds keep every row)
        for (int g = g0; g < g1 && ok; ++g) {
          const int total = (args.gkind[g] == OZ_CRT && nchunks == 1)
                                ? 1
                                : (args.pl.gstart[g + 1] - args.pl.gstart[g]) * nchunks;
          for (int idx = 0; idx < total; ++idx, ++acc) {
            const int buf = acc & 1;
            const uint32_t par = (acc >> 1) & 1;
            if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.tfull[buf], par, lim)) {
              if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 3);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) release_acc<PAIR>(&sm.tempty[buf]);
          }
        }
        continue;
      }
      bool have_w = false;
      for (int g = g0; g < g1 && ok; ++g) {
        const int kind = args.gkind[g];
        if (kind == OZ_RAD_SET || kind == OZ_RAD_ADD) {
          // radius product (its digit pairs form one group): every chunk, an
          // exact integer in fp32, is weighted by its pair's 2^(8 (t_ref - t))
          // and summed upward -- S = RU(chunk 2^sh + S), an upper bound of
          // the exact weighted integer sum -- and one fold per (product, tile)
          // goes out, never read back here
          const int ncb = (f.nb * 64 - half * 128) >> 5;  // column blocks multiplied
          float S[128];
#pragma unroll
          for (int e = 0; e < 128; ++e) S[e] = 0.0f;
          int pi = args.pl.gstart[g], pc = 0;
          const int total = (args.pl.gstart[g + 1] - pi) * nchunks;
          for (int idx = 0; idx < total; ++idx, ++acc) {
            const int buf = acc & 1;
            const uint32_t par = (acc >> 1) & 1;
            if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.tfull[buf], par, lim)) {
              if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 3);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const float sc = __int_as_float((127 + 8 * (args.t_ref - args.pl.pt[pi])) << 23);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              if (c4 < ncb) {
                uint32_t r[32];
                ptx::tmem_ld_32x32(tmem + lane_addr + buf * OZ_BN + half * 128 + c4 * 32, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e)
                  S[c4 * 32 + e] = __fmaf_ru(__uint_as_float(r[e]), sc, S[c4 * 32 + e]);
              }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) release_acc<PAIR>(&sm.tempty[buf]);
            if (++pc == nchunks) {
              pc = 0;
              ++pi;
            }
          }
          if (!ok) break;
          int32_t* pp = f.P + ((size_t)(kind == OZ_RAD_ADD ? args.slot_add : 0) * f.Np + gj0) *
                                  f.Mp + gi;
#pragma unroll
          for (int e = 0; e < 128; ++e) pp[(size_t)e * f.Mp] = __float_as_int(S[e]);
          continue;
        }
        if (kind == OZ_CRT && nchunks == 1) {
          // residue group (one modulus) of one chunk: the residue goes
          // straight from TMEM to res on the FP32 pipe, for the valid rows
          // and columns only (the reassembly reads no other)
          const int buf = acc & 1;
          const uint32_t par = (acc >> 1) & 1;
          ++acc;
          if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.tfull[buf], par, lim)) {
            if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 3);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const float mf = (float)args.moduli[g];
          const float invf = __frcp_rn(mf);
          uint8_t* rp = f.res + (size_t)args.gres[g] * f.Np * f.Mp + (size_t)gj0 * f.Mp + gi;
          const size_t ld = (size_t)f.Mp;
          const int ncol = gi < f.M ? f.N - gj0 : 0;  // 0: a padding row
#pragma unroll 1
          for (int c8 = 0; c8 < 2; ++c8, rp += 64 * ld) {
            if (half * 2 + c8 >= f.nb) break;  // columns the tile did not multiply
            uint32_t r[64];  // two loads in flight per wait
            ptx::tmem_ld_32x32(tmem + lane_addr + buf * OZ_BN + half * 128 + c8 * 64, r);
            ptx::tmem_ld_32x32(tmem + lane_addr + buf * OZ_BN + half * 128 + c8 * 64 + 32, r + 32);
            ptx::tmem_ld_wait();
            // residue bytes: the residue rr < 256 is the low byte of the bits
            // of rr + 2^23.  Two columns per paired FP32 instruction: q and
            // r = RN(q (-m) + x), then 2^23 + r and 2^23 + m + r (both exact
            // integers below 2^24), the second kept where r < 0 (a float
            // compare, so that r = -0 keeps the first)
            const unsigned long long inv2 = f32x2(invf, invf), negm2 = f32x2(-mf, -mf),
                                     rnd2 = f32x2(12582912.0f, 12582912.0f),
                                     off2 = f32x2(8388608.0f, 8388608.0f),
                                     offm2 = f32x2(8388608.0f + mf, 8388608.0f + mf);
#pragma unroll
            for (int e = 0; e < 64; e += 2) {
              const unsigned long long x = f32x2(__uint_as_float(r[e]), __uint_as_float(r[e + 1]));
              const unsigned long long q = sub_x2(add_x2(mul_x2(x, inv2), rnd2), rnd2);
              const unsigned long long rr = fma_x2(q, negm2, x);
              const unsigned long long a = add_x2(rr, off2), b = add_x2(rr, offm2);
              r[e] = __uint_as_float((uint32_t)rr) < 0.0f ? (uint32_t)b : (uint32_t)a;
              r[e + 1] = __uint_as_float((uint32_t)(rr >> 32)) < 0.0f ? (uint32_t)(b >> 32)
                                                                      : (uint32_t)(a >> 32);
            }
            const int nc = ncol - c8 * 64;
            if (nc >= 64) {  // the common case: no per-column test
#pragma unroll
              for (int e = 0; e < 64; ++e) rp[e * ld] = (uint8_t)r[e];
            } else {
#pragma unroll
              for (int e = 0; e < 64; ++e)
                if (e < nc) rp[e * ld] = (uint8_t)r[e];
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) release_acc<PAIR>(&sm.tempty[buf]);
          continue;
        }
        if (kind == OZ_CRT) {
          // residue group of several chunks (one pair: the group's modulus):
          // every chunk is reduced to |r| <= m/2 + 2 and summed on the FP32
          // pipe, two columns per instruction; the sum is an exact integer
          // (below 2^24 for any inner dimension under 10^8) and is reduced
          // once more to the residue byte.  (As int32 sums -- conversions on
          // the XU pipe, an integer remainder at the end -- the epilogue of
          // two chunks outlasted their MMAs now and then: the product of
          // 1225^3 took 109 us, now 88; 2048^3 288, now 279.)
          const int ncb = (f.nb * 64 - half * 128) >> 5;  // column blocks multiplied
          const float mf = (float)args.moduli[g];
          const float invf = __frcp_rn(mf);
          const unsigned long long inv2 = f32x2(invf, invf), negm2 = f32x2(-mf, -mf),
                                   rnd2 = f32x2(12582912.0f, 12582912.0f);
          auto reduce = [&](unsigned long long x) {
            return fma_x2(sub_x2(add_x2(mul_x2(x, inv2), rnd2), rnd2), negm2, x);
          };
          unsigned long long S[64];
#pragma unroll
          for (int e = 0; e < 64; ++e) S[e] = 0;
          for (int idx = 0; idx < nchunks; ++idx, ++acc) {
            const int buf = acc & 1;
            const uint32_t par = (acc >> 1) & 1;
            if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.tfull[buf], par, lim)) {
              if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 3);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              if (c4 < ncb) {
                uint32_t r[32];
                ptx::tmem_ld_32x32(tmem + lane_addr + buf * OZ_BN + half * 128 + c4 * 32, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                  S[c4 * 16 + e] = add_x2(
                      S[c4 * 16 + e], reduce(f32x2(__uint_as_float(r[2 * e]),
                                                   __uint_as_float(r[2 * e + 1]))));
              }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) release_acc<PAIR>(&sm.tempty[buf]);
          }
          if (!ok) break;
          uint8_t* rp = f.res + (size_t)args.gres[g] * f.Np * f.Mp + (size_t)gj0 * f.Mp + gi;
          const size_t ld = (size_t)f.Mp;
          const int ncol = gi < f.M ? f.N - gj0 : 0;  // 0: a padding row
          const unsigned long long off2 = f32x2(8388608.0f, 8388608.0f),
                                   offm2 = f32x2(8388608.0f + mf, 8388608.0f + mf);
#pragma unroll
          for (int e = 0; e < 64; ++e) {
            const unsigned long long rr = reduce(S[e]);
            const unsigned long long a = add_x2(rr, off2), b = add_x2(rr, offm2);
            const uint32_t r0 = __uint_as_float((uint32_t)rr) < 0.0f ? (uint32_t)b : (uint32_t)a;
            const uint32_t r1 = __uint_as_float((uint32_t)(rr >> 32)) < 0.0f
                                    ? (uint32_t)(b >> 32)
                                    : (uint32_t)(a >> 32);
            if (2 * e < ncol) rp[(2 * e) * ld] = (uint8_t)r0;
            if (2 * e + 1 < ncol) rp[(2 * e + 1) * ld] = (uint8_t)r1;
          }
          continue;
        }
        if constexpr (PAIR || GROUP) continue;  // (no other kinds there)
        // OZ_MID: the chunks of a digit group as int32 sums, folded into W
        const int t = args.pl.gt[g];
        const int sh = 8 * (args.t_ref - t);
        const int npg = args.pl.gstart[g + 1] - args.pl.gstart[g];
        const int total = npg * nchunks;
        int c[128];
#pragma unroll
        for (int e = 0; e < 128; ++e) c[e] = 0;
        int cnt = 0;
        for (int idx = 0; idx < total; ++idx, ++acc) {
          const int buf = acc & 1;
          const uint32_t par = (acc >> 1) & 1;
          if (*(volatile int*)&sm.abort || !ptx::mbar_wait(&sm.tfull[buf], par, lim)) {
            if (!*(volatile int*)&sm.abort) raise_timeout(&sm, args.flag, 3);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            uint32_t r[32];
            ptx::tmem_ld_32x32(tmem + lane_addr + buf * OZ_BN + half * 128 + c4 * 32, r);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) c[c4 * 32 + e] += __float2int_rn(__uint_as_float(r[e]));
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) release_acc<PAIR>(&sm.tempty[buf]);
          ++cnt;
          const bool last_of_group = idx == total - 1;
          if (cnt == OZ_FOLD_CHUNKS || last_of_group) {
            // fold into W (global, column-major, ld = Mp); the first fold of
            // a tile stores, later folds add
#pragma unroll
            for (int e = 0; e < 128; ++e) {
              long long* wp = args.W + (size_t)(gj0 + e) * args.Mp + gi;
              const long long v = shift_t(c[e], sh);
              *wp = have_w ? *wp + v : v;
              c[e] = 0;
            }
            have_w = true;
            cnt = 0;
          }
        }
      }
      if (!ok) break;
      if constexpr (PAIR || GROUP) continue;
      if (!mid) continue;  // CRT residues / radius folds: combined later
      // ------------------------------------------------------ final epilogue
      const int Ei = (gi < args.M) ? args.Erow[(size_t)args.erow_stride * gi] : OZ_ZERO_EXP;
      double dlt = 0.0;
      if (args.mode == OZ_MID && gi < args.M) dlt = __dmul_ru((double)args.delta[gi], 0.515625);
      if (gi < args.M) {
        for (int e = 0; e < 128; ++e) {
          const int gj = gj0 + e;
          if (gj >= args.N) break;
          const long long v = args.W[(size_t)gj * args.Mp + gi];
          const int Fj = args.Fcol[(size_t)args.fcol_stride * gj];
          const bool zero = (Ei == OZ_ZERO_EXP) || (Fj == OZ_ZERO_EXP);
          const int ex = Ei + Fj - 8 * args.t_ref;
          double* Tp = args.T + (size_t)gj * args.Mp + gi;
          {
            double mlo = 0.0, mup = 0.0, tr = 0.0;
            if (!zero) {
              mlo = scale_dir(__ll2double_rd(v), ex, false);
              mup = scale_dir(__ll2double_ru(v + args.R), ex, true);
              const double bh = __dmul_ru(args.beta[gj], 0.5);
              const double x = __fma_ru(dlt, pow2_ru(Fj - 8), bh);
              tr = scale_dir(x, Ei - 8 * args.s, true);
            }
            const double err = __dadd_ru(tr, *Tp);
            double lo = __dsub_rd(mlo, err), up = __dadd_ru(mup, err);
            if (nonfinite) lo = up = __longlong_as_double(0x7ff8000000000000LL);
            double* cp = args.C + 2 * ((size_t)gi + (size_t)gj * args.ldc);
            cp[0] = lo;
            cp[1] = up;
          }
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {
    // no CTA leaves while its peer may still signal it (the issuer's last
    // arrival on the other CTA is that on mma_done)
    if (rank == 1 && threadIdx.x == 32) ptx::mbar_wait(&sm.mma_done, 0, lim);
    __syncwarp();
    ptx::cluster_sync();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (PAIR)
      ptx::tmem_dealloc_pair(tmem, TMEM_COLS);
    else
      ptx::tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Map of operand planes, read in boxes of box_rows lines x 64 k: planes of
// whole lines (the slice form), or tiled ones (oz_tile_off: 64 entries wide,
// a box one contiguous run).
int make_tmap(CUtensorMap* m, const void* base, int Kp, int rows, int planes, int box_rows,
              bool tiled, size_t pstride = 0) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return VCPCU_ERR_CUDA;
  }
  const cuuint64_t width = tiled ? OZ_BK : Kp;
  cuuint64_t dims[3] = {width, (cuuint64_t)rows * (tiled ? Kp / OZ_BK : 1), (cuuint64_t)planes};
  cuuint64_t strides[2] = {width * 2,
                           (cuuint64_t)(pstride ? pstride : (size_t)Kp * rows) * 2};
  cuuint32_t box[3] = {(cuuint32_t)OZ_BK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return VCPCU_ERR_CUDA;
  }
  return VCPCU_OK;
}

int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// CTA pairs for products of several chunks that fill the device: their gain is
// in the loads of a long inner dimension (single CTAs -> pairs, the GEMM alone:
// 2048^3 279 -> 263 us, 4096^3 1869 -> 1800, 1225x1225x12544 649 -> 599).
//   One chunk: within 2 % of each other, either way round (4096x4096x1024 508
// and 512 us).  Below one item per SM the pair's start-up shows (256x256x4096
// 97 and 102 us).  An odd last row block costs half a pair: not where that
// adds more than a tenth of the rounds.
//   From about 2^42 multiply-adds (4 ms) the power limit sets the clock, and
// single CTAs do more work at it; whole products in a sustained loop, single
// CTAs and pairs: 8192x8192x2048 4836 and 4654 us, 3000x3000x16384 5855 and
// 5780, 6000^3 7130 and 7208, 8192^3 16598 and 17175.
bool use_pairs(int tiles_m, int tiles_n, int Kp, const OzPairList& pl) {
  if (tiles_m < 2 || Kp <= OZ_CHUNK) return false;
  const long sms = num_sms(), pairs = sms / 2;
  const long tiles = (long)tiles_m * tiles_n, items = tiles * pl.ngroups;
  if (items < sms || pairs < 1) return false;
  if ((double)tiles * OZ_BM * OZ_BN * Kp * pl.npairs > 0x1p42) return false;
  const long one = (items + sms - 1) / sms;
  const long two = ((long)((tiles_m + 1) / 2) * tiles_n * pl.ngroups + pairs - 1) / pairs;
  return 10 * two <= 11 * one;
}

// The radius products and the residue GEMMs in one launch: the A planes are
// [residues (mpl) | |mA| + rA digits (sr) | rA digits (sr)] at one plane
// stride, the B planes [residues | rB digits | |mB| digits]; the groups of
// radius product 1, product 2 (each skipped for a point factor, point_mask
// as OzPlan's) and the moduli, each tagged with its kind.
void all_groups(const OzPairList& rad, const OzPairList& crt, int mpl, int sr, int point_mask,
                OzGemmArgs& a) {
  OzPairList& m = a.pl;
  int ng = 0, np = 0;
  auto add = [&](const OzPairList& src, int offA, int offB, int kind) {
    for (int g = 0; g < src.ngroups; ++g) {
      m.gstart[ng] = (int16_t)np;
      m.gt[ng] = src.gt[g];
      a.gkind[ng] = (int8_t)kind;
      a.gres[ng] = (int8_t)(kind == OZ_CRT ? g : 0);
      if (kind == OZ_CRT) a.moduli[ng] = OZ_MODULI[g];
      for (int q = src.gstart[g]; q < src.gstart[g + 1]; ++q, ++np) {
        m.pa[np] = (int8_t)(src.pa[q] + offA);
        m.pb[np] = (int8_t)(src.pb[q] + offB);
        m.pt[np] = src.pt[q];
      }
      ++ng;
    }
  };
  if (!(point_mask & 2)) add(rad, mpl, mpl, OZ_RAD_SET);
  if (!(point_mask & 1)) add(rad, mpl + sr, mpl + sr, OZ_RAD_ADD);
  add(crt, 0, 0, OZ_CRT);
  m.gstart[ng] = (int16_t)np;
  m.ngroups = ng;
  m.npairs = np;
}

}  // namespace

size_t oz_dyn_smem() { return (size_t)OZ_STAGES * STAGE_BYTES + 1024; }

// The dynamic shared-memory opt-in of the slice GEMM is a property of the
// device context: set it once per device ordinal (under a lock, since host
// threads may start products concurrently).
static int oz_gemm_smem_optin() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  VCPCU_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("slice GEMM: device ordinal %d out of range", dev);
    return VCPCU_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (!done[dev]) {
    VCPCU_CUDA_TRY(cudaFuncSetAttribute(oz_slice_gemm_kernel<false, false>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)oz_dyn_smem()));
    VCPCU_CUDA_TRY(cudaFuncSetAttribute(oz_slice_gemm_kernel<true, false>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)oz_dyn_smem()));
    VCPCU_CUDA_TRY(cudaFuncSetAttribute(oz_slice_gemm_kernel<false, true>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)oz_dyn_smem()));
    done[dev] = true;
  }
  return VCPCU_OK;
}

int oz_run_gemm(const OzPlan& plan, int mode, const OzWorkspace& ws, double* C, long ldc,
                cudaStream_t st, bool chained) {
  const OzProblem& pb = plan.pb;
  if (int e = oz_gemm_smem_optin()) return e;
  OzGemmArgs a;
  memset(&a, 0, sizeof(a));
  int st_;
  const bool mid = mode == OZ_MID;
  const uint16_t* ap;
  const uint16_t* bp;
  int apl, bpl;
  if (mid) {
    ap = ws.a_mid; bp = ws.b_mid; apl = pb.mplanes; bpl = pb.mplanes;
    a.Erow = ws.E3 + 0; a.Fcol = ws.F2 + 0;
    a.pl = plan.mid; a.t_ref = plan.t_ref_mid; a.R = plan.R_mid;
  } else if (mode == OZ_RAD_SET) {  // (|mA| + rA) * rB
    ap = ws.a_p; bp = ws.b_r; apl = pb.sr; bpl = pb.sr;
    a.Erow = ws.E3 + 1; a.Fcol = ws.F2 + 1;
    a.pl = plan.rad; a.t_ref = plan.t_ref_rad; a.R = plan.R_rad;
  } else if (mode == OZ_RAD_ADD) {  // rA * |mB|
    ap = ws.a_r; bp = ws.b_s; apl = pb.sr; bpl = pb.sr;
    a.Erow = ws.E3 + 2; a.Fcol = ws.F2 + 0;
    a.pl = plan.rad; a.t_ref = plan.t_ref_rad; a.R = plan.R_rad;
  } else if (mode == OZ_ALL) {
    ap = ws.a_mid; bp = ws.b_mid;
    apl = bpl = pb.mplanes + 2 * pb.sr;
    a.Erow = ws.E3 + 0; a.Fcol = ws.F2 + 0;
    a.t_ref = plan.t_ref_rad; a.R = plan.R_rad;
    a.res = ws.res;
    all_groups(plan.rad, plan.crt, pb.mplanes, pb.sr, plan.point_mask, a);
  } else {  // OZ_CRT: residue products, one modulus per group
    ap = ws.a_mid; bp = ws.b_mid; apl = pb.L; bpl = pb.L;
    a.Erow = ws.E3 + 0; a.Fcol = ws.F2 + 0;
    a.pl = plan.crt; a.t_ref = 0; a.R = 0;
    a.res = ws.res;
    for (int l = 0; l < pb.L; ++l) a.moduli[l] = OZ_MODULI[l];
  }
  if (mode != OZ_ALL)
    for (int g = 0; g < a.pl.ngroups; ++g) {
      a.gkind[g] = (int8_t)mode;
      a.gres[g] = (int8_t)g;
    }
  a.tiled = mode == OZ_ALL || mode == OZ_CRT;
  if ((st_ = make_tmap(&a.tmA, ap, pb.Kp, pb.Mp, apl, OZ_BM, a.tiled, ws.a_pstride))) return st_;
  a.tiles_m = pb.Mp / OZ_BM;
  a.tiles_n = pb.Np / OZ_BN;
  const bool pair = !mid && use_pairs(a.tiles_m, a.tiles_n, pb.Kp, a.pl);
  if ((st_ = make_tmap(&a.tmB, bp, pb.Kp, pb.Np, bpl, pair ? OZ_BN / 2 : OZ_BN, a.tiled,
                       ws.b_pstride)))
    return st_;
  a.M = pb.M; a.N = pb.N; a.Mp = pb.Mp; a.Np = pb.Np; a.Kp = pb.Kp;
  a.mode = mode;
  a.s = pb.s;
  a.erow_stride = 3;
  a.fcol_stride = 2;
  a.delta = ws.delta;
  a.beta = ws.beta;
  a.W = ws.W;
  a.T = ws.T;
  a.P = ws.P;
  a.slot_add = plan.rad_slots;
  a.C = C;
  a.ldc = ldc;
  a.flag = ws.flag;
  a.timeout_cycles = 4000000000LL;  // about 2 s at 2 GHz
  if (pair) {
    const int nitems = (a.tiles_m + 1) / 2 * a.tiles_n * a.pl.ngroups;
    const int pairs = nitems < num_sms() / 2 ? nitems : num_sms() / 2;
    VCPCU_CUDA_TRY(launch_dep(chained, 2, oz_slice_gemm_kernel<true, false>, dim3(2 * pairs),
                              dim3(NTHREADS), oz_dyn_smem(), st, a));
    VCPCU_LAUNCH_CHECK("oz_slice_gemm_kernel");
    return VCPCU_OK;
  }
  const int ntiles = a.tiles_m * a.tiles_n;
  const int nitems = mode == OZ_MID ? ntiles : ntiles * a.pl.ngroups;
  const int grid = nitems < num_sms() ? nitems : num_sms();
  VCPCU_CUDA_TRY(launch_dep(chained, 1, oz_slice_gemm_kernel<false, false>, dim3(grid),
                            dim3(NTHREADS), oz_dyn_smem(), st, a));
  VCPCU_LAUNCH_CHECK("oz_slice_gemm_kernel");
  return VCPCU_OK;
}

// One launch of the slice GEMM over all problems of a bucket: the radius
// products and the residue GEMMs.  `shape` supplies the pair lists (radius
// digit pairs, Lmax moduli) and the fold count.
int oz_grun_gemm(const OzGBucket& b, const OzPlan& shape, int nitems, cudaStream_t st) {
  if (nitems <= 0) return VCPCU_OK;
  if (int e = oz_gemm_smem_optin()) return e;
  OzGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.t_ref = shape.t_ref_rad;
  a.res = b.res;
  all_groups(shape.rad, shape.crt, b.Lmax, 2, 0, a);
  a.tiled = 1;
  int st_;
  if ((st_ = make_tmap(&a.tmA, b.planesA, OZ_BK, b.Arows, b.Lmax + 4, OZ_BM, true))) return st_;
  if ((st_ = make_tmap(&a.tmB, b.planesB, OZ_BK, b.Brows, b.Lmax + 4, 64, true))) return st_;
  a.Kp = OZ_BK;  // (each item has its problem's)
  a.mode = OZ_ALL;
  a.P = b.P;
  a.slot_add = shape.rad_slots;
  a.flag = b.flag;  // problem 0's status words take the (global) timeout bit
  a.timeout_cycles = 4000000000LL;  // about 2 s at 2 GHz
  a.gp = b.probs;
  a.gitem = b.item;
  a.gprob = b.prob_item;
  a.gnitems = nitems;
  const int grid = nitems < num_sms() ? nitems : num_sms();
  oz_slice_gemm_kernel<false, true><<<grid, NTHREADS, oz_dyn_smem(), st>>>(a);
  VCPCU_LAUNCH_CHECK("oz_slice_gemm_kernel");
  return VCPCU_OK;
}

}  // namespace vcpcu
