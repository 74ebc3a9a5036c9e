// Products of residue planes on the int8 tensor cores (see crt.cuh).
#include "crt_dev.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace sfq {
namespace crt {
using namespace tc;

namespace {

constexpr int BM = 128;       // MMA M: accumulator rows = TMEM lanes
constexpr int BN = 256;       // widest tile: one of two accumulator buffers of 256 columns
constexpr int BK = 128;       // K slice: one 128-byte swizzle row
constexpr int KSTEP = 32;     // K of one kind::i8 MMA
constexpr int STAGES = 4;
// warps: 0 TMA producer, 1 TMEM owner + MMA issuer, 2-17 epilogue (four per TMEM lane quarter: the reduction
// of a tile with short K is what bounds it, and two warps a scheduler left half of its issue slots idle)
constexpr int kThreads = 576;
constexpr int kEpiThreads = 512;
constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK, STAGE = A_BYTES + B_BYTES;
constexpr int BAR_OFF = STAGES * STAGE;
constexpr int SMEM = BAR_OFF + (2 * STAGES + 5) * 8 + 16 + 1024;
static_assert(SMEM <= 232448, "shared memory budget");
constexpr unsigned long long kWaitNs = 2000000000ull;  // limit of one wait: 2 s without progress
__device__ unsigned long long g_expiries;               // calls in which a bounded wait expired

// A launch gave up: the call's flag (its FP64 product then replaces the result) and one count for the call
__device__ __forceinline__ void report_expiry(int* expired) {
  if (atomicExch(expired, 1) == 0) atomicAdd(&g_expiries, 1ull);
}
// the self-test's hold: before its at-th slice the producer waits for *hold, which nothing sets, and gives up
__device__ __noinline__ void held_back(const int* hold, unsigned long long limit_ns, volatile int* abort) {
  const unsigned long long deadline = gtimer() + limit_ns;
  while (*reinterpret_cast<const volatile int*>(hold) == 0 && gtimer() < deadline) {
  }
  *abort = 1;
}

struct Maps {
  CUtensorMap a, b;
};
struct KP {
  int M, N, K, parts, segs, bn;
  int MT, NT, KT;  // tiles along M and N; K slices per segment
  long tiles;
  long a_off[2][2], b_off[2];
  uint8_t* C;
  long ldc, c_plane;
  int wide;        // reduce_kind of the K sums
  Redo redo;
  int least, wmod; // magnitudes that pass; walker of a row: m % wmod
  unsigned long long wait_ns;
  const int* hold;
  uint32_t hold_at;
};

__device__ __forceinline__ uint32_t idesc_i8(uint32_t n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (uint32_t(BM >> 4) << 24);
}
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// 32 consecutive accumulator columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  // the wait names the registers so that nothing reads them before it
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// 32 int32 sums -> their residues mod p as bytes (0 .. p: p, where a byte holds it, for 0 now and then).
// kind 0: |sum| <= 2^24, q = mulhi(sum, ceil(2^32 / p)) is floor(sum / p) or, for a negative multiple of p, one
// less; 1: |sum| <= 2^27; 2: |sum| < 3 2^29, folded at 16 bits first
struct Mod {
  uint32_t p, m39, big, r16;
  int m32;
};
__device__ __forceinline__ Mod mod_of(int i, int kind) {
  Mod m;
  m.p = c_crt.mod[i];
  m.m39 = c_crt.m39[i];
  m.m32 = c_crt.m32[i];
  m.big = kind == 2 ? c_crt.big30[i] : c_crt.big27[i];
  m.r16 = c_crt.r16[i];
  return m;
}
template <int KIND>
__device__ __forceinline__ void reduce32_k(const uint32_t* v, uint32_t* w, const Mod& m) {
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint32_t r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (KIND == 0) {
        r[j] = v[4 * g + j] - uint32_t(__mulhi(int(v[4 * g + j]), m.m32)) * m.p;
      } else {
        uint32_t u = v[4 * g + j] + m.big;  // congruent and nonnegative
        if (KIND == 2) u = (u >> 16) * m.r16 + (u & 0xffffu);
        r[j] = u - (__umulhi(u, m.m39) >> 7) * m.p;
      }
    }
    w[g] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
  }
}
__device__ __forceinline__ void reduce32(const uint32_t* v, uint32_t* w, const Mod& m, int kind) {
  if (kind == 0) reduce32_k<0>(v, w, m);
  else if (kind == 1) reduce32_k<1>(v, w, m);
  else reduce32_k<2>(v, w, m);
}
// A warp's 32 rows x 64 columns of accumulators at taddr -> bytes of C.  Each lane reduces its own row; four
// lanes then trade 16-byte pieces so that a store instruction writes 64-byte pieces of eight rows (a lane's own
// 16 bytes a row took 32 cache lines an instruction, and the stores bounded the tiles with short K).
// rows[i]: C's row of the group's lane i at this block's first column, null where there is none; left: bytes
// of the row from there on, a multiple of 16.
__device__ __forceinline__ void drain64(uint32_t taddr, const Mod& m, int kind, uint8_t* const* rows, int left, int lane) {
  uint32_t w[16];
  {
    uint32_t v[32];
    tmem_ld32(taddr, v);
    reduce32(v, w, m, kind);
  }
  if (left > 32) {  // the same for the whole warp
    uint32_t v[32];
    tmem_ld32(taddr + 32, v);
    reduce32(v, w + 8, m, kind);
  }
  // 4 x 4 transpose of the pieces: after it piece i of this lane is piece (lane & 3) of the group's row i
  const bool b1 = lane & 1, b2 = lane & 2;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // pieces 2 h and 2 h + 1 with lane ^ 1
      uint32_t &lo = w[8 * h + i], &hi = w[8 * h + 4 + i];
      const uint32_t x = __shfl_xor_sync(0xffffffffu, b1 ? lo : hi, 1);
      if (b1) lo = x;
      else hi = x;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // pieces h and h + 2 with lane ^ 2
      uint32_t &lo = w[4 * h + i], &hi = w[8 + 4 * h + i];
      const uint32_t x = __shfl_xor_sync(0xffffffffu, b2 ? lo : hi, 2);
      if (b2) lo = x;
      else hi = x;
    }
  }
  const int at = 16 * (lane & 3);
  if (at < left) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (rows[i]) *reinterpret_cast<uint4*>(rows[i] + at) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
}
// A warp's 32 rows x n <= 64 columns of the magnitudes' product at taddr: the walker of a row with a sum below `least`
// is asked for again
__device__ __forceinline__ void check64(uint32_t taddr, int n, int least, bool live_row, const Redo& redo, int w) {
  int lowest = least;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (32 * h >= n) break;  // the same for the whole warp
    uint32_t v[32];
    tmem_ld32(taddr + 32 * h, v);
    if (32 * h + 32 <= n) {
#pragma unroll
      for (int j = 0; j < 32; ++j) lowest = min(lowest, int(v[j]));
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) lowest = 32 * h + j < n ? min(lowest, int(v[j])) : lowest;
    }
  }
  if (lowest < least && live_row) redo.ask(w);
}
inline int reduce_kind(long K) { return K <= 1024 ? 0 : K <= 8192 ? 1 : 2; }

struct Tile {
  int mt, part, nt, p;
};
// tiles in the order (modulus, column tile, part, row tile): the row tiles that share a B
// tile run side by side, so a B operand larger than L2 is read from memory once
__device__ __forceinline__ Tile decode(const KP& k, long t) {
  Tile c;
  c.mt = int(t % k.MT);
  t /= k.MT;
  c.part = int(t % k.parts);
  t /= k.parts;
  c.nt = int(t % k.NT);
  c.p = int(t / k.NT);
  return c;
}

// One tile of one modulus: 128 x bn x K int8 products with exact int32 accumulation in tensor memory,
// reduced mod p and stored as bytes (the sixteenth plane's, the magnitudes, compared and not stored).  Bound by the tensor pipe where K is long and by operand
// traffic out of L2 (a 128 x 256 tile takes 48 KB per 128-element K slice of 512 MMA cycles); the two
// 256-column accumulators let a tile's reduction run under the next tile's MMAs.
__global__ void __launch_bounds__(kThreads, 1) crt_gemm_kernel(const __grid_constant__ Maps maps,
                                                               const __grid_constant__ KP k) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;   // [2]
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiThreads);
    }
    mbar_init(done, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      uint32_t it = 0;
      bool stop = false;
      const uint32_t bytes = uint32_t(A_BYTES + k.bn * BK);
      for (long t = blockIdx.x; t < k.tiles && !stop; t += gridDim.x) {
        const Tile c = decode(k, t);
        for (int sg = 0; sg < k.segs && !stop; ++sg) {
          const int ra = int(k.a_off[c.part][sg]) + c.mt * BM;
          const int rb = int(k.b_off[sg]) + c.nt * k.bn;
          const int kend = k.hold ? min(k.KT, int(k.hold_at - it)) : k.KT;
          for (int kt = 0; kt < kend; ++kt, ++it) {
            const int s = int(it % STAGES);
            if (!mbar_wait_abort(&empty[s], ((it / STAGES) & 1) ^ 1, k.wait_ns, s_abort)) {
              stop = true;
              break;
            }
            unsigned char* stg = smem + s * STAGE;
            mbar_expect_tx(&full[s], bytes);
            tma_load_3d(stg, &maps.a, &full[s], kt * BK, ra, c.p);
            tma_load_3d(stg + A_BYTES, &maps.b, &full[s], kt * BK, rb, c.p);
          }
          if (kend < k.KT && !stop) {
            held_back(k.hold, k.wait_ns, s_abort);
            stop = true;
          }
        }
      }
      // every issued stage must have landed before the CTA may exit
      for (uint32_t j = (it > uint32_t(STAGES) ? it - STAGES : 0u); j < it; ++j)
        mbar_wait_for(&full[j % STAGES], (j / STAGES) & 1, kWaitNs);
    }
  } else if (warp == 1) {
    if (elect_one()) {  // MMA issuer
      // The issue loop is short on purpose: an MMA of 128 x 256 x 32 takes 128 cycles of the tensor pipe,
      // and one issued through a loop of descriptor arithmetic and operand masks took 220 (two fifths of
      // the pipe's rate, whatever the operands' traffic).
      const uint32_t idesc = idesc_i8(uint32_t(k.bn));
      const uint64_t ad0 = smem_desc(smem), bd0 = smem_desc(smem + A_BYTES);
      const int tail = k.K - (k.KT - 1) * BK;             // K of the last slice
      const int ntail = (tail + KSTEP - 1) / KSTEP;       // its MMA steps that are not all zeros
      const int slices = k.segs * k.KT;
      uint32_t s = 0, ph = 0, n = 0;
      bool stop = false;
      for (long t = blockIdx.x; t < k.tiles && !stop; t += gridDim.x, ++n) {
        const uint32_t b = n & 1;
        if (!mbar_wait_abort(&acc_empty[b], ((n >> 1) & 1) ^ 1, k.wait_ns, s_abort)) break;
        fence_after();
        const uint32_t d = tmem + b * BN;
        int left = k.KT;
        for (int i = 0; i < slices; ++i) {
          if (!mbar_wait_abort(&full[s], ph, k.wait_ns, s_abort)) {
            stop = true;
            break;
          }
          fence_after();
          const uint64_t ad = ad0 + uint64_t(s * (STAGE >> 4)), bd = bd0 + uint64_t(s * (STAGE >> 4));
          if (--left) {
#pragma unroll
            for (int kk = 0; kk < BK / KSTEP; ++kk)
              umma_i8(d, ad + 2 * kk, bd + 2 * kk, idesc, kk > 0 ? 1u : uint32_t(i));
          } else {  // the last slice of a segment: all-zero steps skipped
            left = k.KT;
            for (int kk = 0; kk < ntail; ++kk) umma_i8(d, ad + 2 * kk, bd + 2 * kk, idesc, uint32_t(kk | i));
          }
          umma_commit(&empty[s]);
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!stop) umma_commit(&acc_full[b]);
      }
      // every MMA issued has completed before the tensor memory may be released
      umma_commit(done);
      mbar_wait_for(done, 0, kWaitNs);
    }
    __syncwarp();
  } else {  // epilogue warps -> TMEM lane quarters 2,3,0,1 (a warp reaches only its quarter)
    const int q = warp & 3;
    uint32_t n = 0;
    for (long t = blockIdx.x; t < k.tiles; t += gridDim.x, ++n) {
      const uint32_t b = n & 1;
      const bool ok = mbar_wait_for(&acc_full[b], (n >> 1) & 1, k.wait_ns);
      const bool go = __all_sync(0xffffffffu, ok) && !__any_sync(0xffffffffu, *s_abort != 0);
      if (!go) {
        *s_abort = 1;
        break;
      }
      fence_after();
      const Tile c = decode(k, t);
      const Mod md = mod_of(c.p, k.wide);
      uint8_t* out = k.C + c.p * k.c_plane + (long)c.part * k.M * k.ldc;
      const uint32_t taddr = tmem + (uint32_t(q * 32) << 16) + b * BN;
      const int n0 = c.nt * k.bn, mg = c.mt * BM + q * 32 + (lane & ~3);
      const int cc = 64 * ((warp - 2) >> 2);  // the quarter's four warps take 64 columns each
      const int left = min(k.bn - cc, int(k.ldc) - n0 - cc);
      if (c.p == NMOD) {
        const int m = c.mt * BM + q * 32 + lane;
        check64(taddr + uint32_t(cc), min(k.bn - cc, k.N - n0 - cc), k.least, m < k.M, k.redo, m % k.wmod);
      } else if (left > 0) {
        uint8_t* rows[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) rows[i] = mg + i < k.M ? out + (mg + i) * k.ldc + n0 + cc : nullptr;
        drain64(taddr + uint32_t(cc), md, k.wide, rows, left, lane);
      }
      fence_before();
      mbar_arrive(&acc_empty[b]);
    }
  }
  fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort) report_expiry(k.redo.call + 1);
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ---- per-walker products ---------------------------------------------------------------------
// C[w] (2 N x cols) = [re; im] rows of walker w's operand times shared or per-walker rows, for every
// modulus.  One work unit is a walker (or a range of its electrons, or of the columns), one modulus: the
// walker's residues (blocks -im, re, im; or re, im) stay in shared memory while the other operand's rows
// stream past them.  The one-tile-at-a-time kernel above loads both operands of every 128 x 208 tile, 341 KB at 400
// orbitals, this one a third of it.  Per-walker operands larger than L2 together come from memory (the Taylor term at
// M = 400, N = 100: DRAM 58 % busy, L2 42 %, tensor pipe 34 %); with short K and a shared operand the producer thread's
// issue loop and the stores of the residues bound it (the energy at M = 200: 0.68 ms a launch of 128 walkers and 150
// vectors, 1.44 GB of residues written; a test of two more words per slice in that loop cost 7 %).
constexpr int RBK = 64;        // K slice: one 64-byte swizzle row
constexpr int RMAXKT = 64;     // K slices at most
constexpr int RMAXST = 8;
constexpr int RBAR = (2 * RMAXST + 2 * RMAXKT + 5) * 8 + 16;
constexpr int RSMEM = 232448 - 1024 - RBAR;  // operand bytes

struct RMaps {
  CUtensorMap a, b, b_last;
};
struct RKP {
  int K, KT, segs, nblk, batch;
  int N, Np, EC;            // electrons of a walker, padded rows of a block in shared memory, chunks of electrons
  int MT;                   // 128-row tiles of the 2 Np rows
  int cols, bn, bn_last, NT, CC, tpc;  // columns, tile width, tiles, column chunks of tpc tiles
  int stages, res_slice, stage;        // bytes of a resident slice and of a stage
  long units;
  long a_blk, b_bs, b_off1;            // A rows: blk * a_blk + w N + a; B rows: w * b_bs + seg * b_off1 + col
  uint8_t* C;
  long ldc, c_plane, c_part;           // C row (c, w, a): c * c_part + w N + a
  int wide;
  Redo redo;
  int least;                           // magnitudes that pass
  unsigned long long wait_ns;
  const int* hold;
  uint32_t hold_at;
};
struct RUnit {
  int p, w, e0, t0, t1;
};
__device__ __forceinline__ RUnit unit_of(const RKP& k, long u) {
  RUnit r;
  const int cc = int(u % k.CC);
  u /= k.CC;
  r.e0 = int(u % k.EC) * k.Np;
  u /= k.EC;
  r.w = int(u % k.batch);
  r.p = int(u / k.batch);
  r.t0 = cc * k.tpc;
  r.t1 = min(k.NT, r.t0 + k.tpc);
  return r;
}
// K-major tile of 64-byte rows, 64-byte swizzle, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t smem_desc64(uint32_t addr) {
  uint64_t d = 0;
  d |= (addr & 0x3FFFFull) >> 4;
  d |= uint64_t(1) << 16;
  d |= uint64_t(512 >> 4) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(4) << 61;
  return d;
}

// CHECK: the magnitudes' product
template <int SEGS, int MT, bool CHECK>
__global__ void __launch_bounds__(kThreads, 1) crt_walker_kernel(const __grid_constant__ RMaps maps,
                                                                 const __grid_constant__ RKP k) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + RSMEM);
  uint64_t* empty = full + RMAXST;
  uint64_t* rfull = empty + RMAXST;
  uint64_t* rempty = rfull + RMAXKT;
  uint64_t* acc_full = rempty + RMAXKT;  // [2]
  uint64_t* acc_empty = acc_full + 2;    // [2]
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // nothing to do where the FP64 product computes all walkers (flags of launches before this one)
  if (CHECK && k.redo.none_left(k.batch)) return;
  if (!CHECK) {
    if (blockIdx.x == 0 && threadIdx.x == 0) k.redo.settle();
    if (k.redo.all_asked(k.batch)) return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < k.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < k.KT; ++s) {
      mbar_init(&rfull[s], 1);
      mbar_init(&rempty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiThreads);
    }
    mbar_init(done, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  unsigned char* stages0 = smem + k.KT * k.res_slice;
  const int blk_bytes = k.Np * RBK;

  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      uint32_t it = 0, un = 0, s = 0, ph = 0;
      const uint32_t nst = uint32_t(k.stages);
      uint32_t rows_un = 0;  // where it gave up: units whose rows were all issued, and the slices issued of the next one's
      int rows_kt = 0;
      bool stop = false;
      for (long u = blockIdx.x; u < k.units && !stop; u += gridDim.x, ++un) {
        const RUnit c = unit_of(k, u);
        for (int t = c.t0; t < c.t1 && !stop; ++t) {
          const bool last = t == k.NT - 1;
          const uint32_t bytes = uint32_t(k.segs * (last ? k.bn_last : k.bn) * RBK);
          const int rb = int(c.w * k.b_bs) + t * k.bn;
          // (the loop over slices bounds the tiles with short K: bookkeeping for a stop stays out of it)
          const int kend = k.hold ? min(k.KT, int(k.hold_at - it)) : k.KT;
          auto give_up = [&](int issued) {
            stop = true;
            rows_un = un + (t > c.t0 || issued == k.KT ? 1u : 0u);
            rows_kt = t > c.t0 || issued == k.KT ? 0 : issued;
          };
          for (int kt = 0; kt < kend; ++kt, ++it) {
            if (t == c.t0) {  // the unit's own rows, slice by slice as the last unit's are done with
              if (!mbar_wait_abort(&rempty[kt], (un & 1) ^ 1, k.wait_ns, s_abort)) {
                give_up(kt);
                break;
              }
              mbar_expect_tx(&rfull[kt], uint32_t(k.nblk * blk_bytes));
              unsigned char* dst = smem + kt * k.res_slice;
              for (int j = 0; j < k.nblk; ++j) {
                // in shared memory: -im, re, im (three blocks) or re, im; in the planes: re, im, -im
                const int blk = k.nblk == 3 ? (j + 2) % 3 : j;
                tma_load_3d(dst + j * blk_bytes, &maps.a, &rfull[kt], kt * RBK,
                            int(blk * k.a_blk) + c.w * k.N + c.e0, CHECK ? NMOD : c.p);
              }
            }
            if (!mbar_wait_abort(&empty[s], ph ^ 1, k.wait_ns, s_abort)) {
              give_up(kt + 1);
              break;
            }
            unsigned char* stg = stages0 + s * k.stage;
            mbar_expect_tx(&full[s], bytes);
            for (int sg = 0; sg < k.segs; ++sg)
              tma_load_3d(stg + sg * k.bn * RBK, last ? &maps.b_last : &maps.b, &full[s], kt * RBK,
                          rb + int(sg * k.b_off1), CHECK ? NMOD : c.p);
            if (++s == nst) {
              s = 0;
              ph ^= 1;
            }
          }
          if (kend < k.KT && !stop) {
            held_back(k.hold, k.wait_ns, s_abort);
            give_up(kend);
          }
        }
      }
      if (!stop) rows_un = un;
      // every issued copy must have landed before the CTA may exit
      for (uint32_t j = (it > uint32_t(k.stages) ? it - k.stages : 0u); j < it; ++j)
        mbar_wait_for(&full[j % k.stages], (j / k.stages) & 1, kWaitNs);
      // (a slice of rows that an MMA took has landed; one issued by a unit that was given up may not have)
      for (int kt = 0; kt < k.KT; ++kt) {
        const uint32_t issued = rows_un + (kt < rows_kt ? 1u : 0u);
        if (issued) mbar_wait_for(&rfull[kt], (issued - 1) & 1, kWaitNs);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {  // MMA issuer
      const uint32_t id_full = idesc_i8(uint32_t(k.bn)), id_last = idesc_i8(uint32_t(k.bn_last));
      // segment 0 reads the rows [re; im] of a resident slice, segment 1 the rows [-im; re] (its first)
      const uint64_t ra0 = smem_desc64(su32(smem) + (SEGS == 2 ? uint32_t(blk_bytes) : 0u));
      const uint64_t ra1 = smem_desc64(su32(smem));
      const uint64_t bd0 = smem_desc64(su32(stages0));
      const uint32_t rstep = uint32_t(k.res_slice) >> 4, sstep = uint32_t(k.stage) >> 4,
                     seg1 = uint32_t(k.bn * RBK) >> 4;
      const bool half_tail = k.K - (k.KT - 1) * RBK <= KSTEP;  // the last slice has one MMA step
      const uint32_t nst = uint32_t(k.stages);
      uint32_t s = 0, ph = 0, n = 0, un = 0;
      bool stop = false;
      for (long u = blockIdx.x; u < k.units && !stop; u += gridDim.x, ++un) {
        const RUnit c = unit_of(k, u);
        for (int t = c.t0; t < c.t1; ++t, ++n) {
          const uint32_t b = n & 1;
          if (!mbar_wait_abort(&acc_empty[b], ((n >> 1) & 1) ^ 1, k.wait_ns, s_abort)) {
            stop = true;
            break;
          }
          fence_after();
          const uint32_t d = tmem + b * BN;
          const uint32_t idesc = t == k.NT - 1 ? id_last : id_full;
          const bool first = t == c.t0, last = t == c.t1 - 1;
          for (int kt = 0; kt < k.KT; ++kt) {
            if ((first && !mbar_wait_abort(&rfull[kt], un & 1, k.wait_ns, s_abort)) ||
                !mbar_wait_abort(&full[s], ph, k.wait_ns, s_abort)) {
              stop = true;
              break;
            }
            fence_after();
            const uint64_t r0 = ra0 + uint64_t(kt * rstep), r1 = ra1 + uint64_t(kt * rstep);
            const uint64_t bd = bd0 + uint64_t(s * sstep);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              if (kk == 1 && half_tail && kt == k.KT - 1) break;
#pragma unroll
              for (int m = 0; m < MT; ++m)
                umma_i8(d + uint32_t(m * 128), r0 + uint64_t(2 * kk + m * (BM * RBK >> 4)), bd + 2 * kk, idesc,
                        kk > 0 ? 1u : uint32_t(kt));
              if (SEGS == 2) {
#pragma unroll
                for (int m = 0; m < MT; ++m)
                  umma_i8(d + uint32_t(m * 128), r1 + uint64_t(2 * kk + m * (BM * RBK >> 4)), bd + seg1 + 2 * kk, idesc,
                          1u);
              }
            }
            umma_commit(&empty[s]);
            if (last) umma_commit(&rempty[kt]);
            if (++s == nst) {
              s = 0;
              ph ^= 1;
            }
          }
          if (stop) break;
          umma_commit(&acc_full[b]);
        }
      }
      // every MMA issued has completed before the tensor memory may be released
      umma_commit(done);
      mbar_wait_for(done, 0, kWaitNs);
    }
    __syncwarp();
  } else {  // epilogue warps: a TMEM lane quarter, a row tile and 64 columns
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int mt = MT == 2 ? (h & 1) : 0;
    const int rg = mt * BM + q * 32 + (lane & ~3);  // the lane group's first row of [re; im], Np each (Np % 8 == 0)
    const int part = rg >= k.Np ? 1 : 0, ag = rg - part * k.Np;
    const int cc = 64 * (MT == 2 ? h >> 1 : h);
    uint32_t n = 0;
    bool stop = false;
    for (long u = blockIdx.x; u < k.units && !stop; u += gridDim.x) {
      const RUnit c = unit_of(k, u);
      const Mod md = mod_of(c.p, k.wide);
      uint8_t* row = k.C + c.p * k.c_plane + (part * k.c_part + (long)c.w * k.N + c.e0 + ag) * k.ldc;
      const int nrow = rg < 2 * k.Np ? k.N - c.e0 - ag : 0;  // rows of the group that exist (4 or more: all)
      for (int t = c.t0; t < c.t1; ++t, ++n) {
        const uint32_t b = n & 1;
        const bool ok = mbar_wait_for(&acc_full[b], (n >> 1) & 1, k.wait_ns);
        const bool go = __all_sync(0xffffffffu, ok) && !__any_sync(0xffffffffu, *s_abort != 0);
        if (!go) {
          *s_abort = 1;
          stop = true;
          break;
        }
        fence_after();
        const uint32_t taddr = tmem + (uint32_t(q * 32) << 16) + b * BN + uint32_t(mt * 128);
        const int bn = t == k.NT - 1 ? k.bn_last : k.bn, n0 = t * k.bn;
        const int left = min(bn - cc, int(k.ldc) - n0 - cc);
        if (CHECK) {
          const int r = rg + (lane & 3), a = ag + (lane & 3);  // this lane's own row
          check64(taddr + uint32_t(cc), min(bn - cc, k.cols - n0 - cc), k.least, r < 2 * k.Np && c.e0 + a < k.N,
                  k.redo, c.w);
        } else if (left > 0) {
          uint8_t* rows[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) rows[i] = i < nrow ? row + i * k.ldc + n0 + cc : nullptr;
          drain64(taddr + uint32_t(cc), md, k.wide, rows, left, lane);
        }
        fence_before();
        mbar_arrive(&acc_empty[b]);
      }
    }
  }
  fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort) report_expiry(k.redo.call + 1);
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

int make_map(CUtensorMap* m, const Planes& o, long K, int box_rows, int bk = BK) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return record_error(SFQ_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(o.rows), cuuint64_t(kPlanes)};
  cuuint64_t strides[2] = {cuuint64_t(o.ld), cuuint64_t(o.plane)};
  cuuint32_t box[3] = {cuuint32_t(bk), cuuint32_t(box_rows), 1};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, o.q, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   bk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return record_error(SFQ_ERR_CUDA, "crt gemm: cuTensorMapEncodeTiled failed (%d)", int(r));
  return SFQ_OK;
}

}  // namespace

int gemm(const Gemm& g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return record_error(SFQ_ERR_SHAPE, "crt gemm: empty product");
  if ((long)g.K * g.segs > kMaxK) return record_error(SFQ_ERR_SHAPE, "crt gemm: K of %ld too long", (long)g.K * g.segs);
  if (g.parts < 1 || g.parts > 2 || g.segs < 1 || g.segs > 2 || g.wmod < 1 || !g.redo.call || !g.redo.row)
    return record_error(SFQ_ERR_ARG, "crt gemm: %d parts of %d segments, walkers %d", g.parts, g.segs, g.wmod);
  KP k{};
  k.M = g.M; k.N = g.N; k.K = g.K; k.parts = g.parts; k.segs = g.segs;
  k.MT = (g.M + BM - 1) / BM;
  // equal column tiles of at most 256, a multiple of 16 wide: the count that leaves the least to the last wave,
  // a tile costing its columns plus about 64 for its share of the other operand (2400 columns against 512
  // rows: 12 tiles of 208 in five waves against 10 of 240 in five)
  double best = 0.0;
  const int nt0 = (g.N + BN - 1) / BN;
  for (int nt = nt0; nt < nt0 + 6; ++nt) {
    const int bn = ((g.N + nt - 1) / nt + 15) / 16 * 16, tiles = (g.N + bn - 1) / bn;
    const long waves = ((long)k.MT * g.parts * tiles * kPlanes + sm_count() - 1) / sm_count();
    const double cost = double(waves) * (bn + 64);
    if (nt == nt0 || cost < 0.98 * best) {
      best = cost;
      k.bn = bn;
      k.NT = tiles;
    }
  }
  k.KT = (g.K + BK - 1) / BK;
  k.tiles = (long)k.MT * k.parts * k.NT * (g.check ? kPlanes : NMOD);
  for (int p = 0; p < 2; ++p)
    for (int s = 0; s < 2; ++s) k.a_off[p][s] = g.a_off[p][s];
  k.b_off[0] = g.b_off[0]; k.b_off[1] = g.b_off[1];
  k.C = g.C; k.ldc = g.ldc; k.c_plane = g.c_plane;
  k.wide = reduce_kind((long)g.K * g.segs);
  k.redo = g.redo;
  k.least = mag_least(g.K, g.segs); k.wmod = g.wmod;
  k.wait_ns = g.wait_ns ? g.wait_ns : kWaitNs;
  k.hold = g.hold; k.hold_at = g.hold_at;
  Maps maps;
  int rc;
  if ((rc = make_map(&maps.a, g.A, g.K, BM)) || (rc = make_map(&maps.b, g.B, g.K, k.bn))) return rc;
  SFQ_CUDA_TRY(cudaFuncSetAttribute(crt_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
  const long grid = k.tiles < sm_count() ? k.tiles : sm_count();
  crt_gemm_kernel<<<unsigned(grid), kThreads, SMEM, st>>>(maps, k);
  SFQ_LAUNCHED();
  return SFQ_OK;
}

namespace {
// the layout of a per-walker product, false where a walker's rows do not fit in shared memory
bool plan_walker(const WalkerGemm& g, RKP* out) {
  RKP k{};
  k.K = g.K; k.KT = (g.K + RBK - 1) / RBK;
  k.segs = g.segs; k.nblk = g.segs == 2 ? 3 : 2; k.batch = g.batch; k.N = g.N;
  if (k.KT > RMAXKT || g.N <= 0) return false;
  // electrons per unit: all of them, or equal chunks of at most 128, while the rows leave room for four
  // stages of the stream
  const int minst = 4;
  for (k.EC = 1;; ++k.EC) {
    k.Np = ((g.N + k.EC - 1) / k.EC + 7) / 8 * 8;
    if (k.Np < 8 || k.EC > 64) return false;
    if (k.Np > 128) continue;
    k.MT = 2 * k.Np > 128 ? 2 : 1;
    const int most = k.MT == 2 ? 128 : 256;
    k.NT = (g.cols + most - 1) / most;
    k.bn = ((g.cols + k.NT - 1) / k.NT + 15) / 16 * 16;
    k.NT = (g.cols + k.bn - 1) / k.bn;
    k.bn_last = (g.cols - (k.NT - 1) * k.bn + 15) / 16 * 16;
    k.res_slice = k.nblk * k.Np * RBK;
    k.stage = k.segs * k.bn * RBK;
    const long room = (long)RSMEM - (long)k.KT * k.res_slice;
    // (a tile's 128 rows may reach past the last slice's rows, into the stages: at most 16 KB)
    if (room >= std::max<long>((long)minst * k.stage, 16384)) {
      k.stages = int(std::min<long>(RMAXST, room / k.stage));
      break;
    }
    if (k.Np <= 8) return false;
  }
  k.EC = (g.N + k.Np - 1) / k.Np;
  k.cols = g.cols;
  k.a_blk = g.a_blk; k.b_bs = g.b_bs; k.b_off1 = g.b_off1;
  k.C = g.C; k.ldc = g.ldc; k.c_plane = g.c_plane; k.c_part = g.c_part;
  k.wide = reduce_kind((long)g.K * g.segs);
  k.redo = g.redo;
  k.least = mag_least(g.K, g.segs);
  k.wait_ns = g.wait_ns ? g.wait_ns : kWaitNs;
  k.hold = g.hold; k.hold_at = g.hold_at;
  *out = k;
  return true;
}
}  // namespace

bool walker_gemm_fits(int N, int cols, int K, int segs) {
  WalkerGemm g;
  g.N = N; g.cols = cols; g.K = K; g.segs = segs; g.batch = 1;
  RKP k;
  return plan_walker(g, &k);
}

int walker_gemm(const WalkerGemm& g, cudaStream_t st) {
  if (g.N <= 0 || g.cols <= 0 || g.batch <= 0 || g.K <= 0 || g.segs < 1 || g.segs > 2 || !g.redo.call || !g.redo.row)
    return record_error(SFQ_ERR_SHAPE, "crt walker gemm: empty product");
  RKP k;
  if (!plan_walker(g, &k)) return record_error(SFQ_ERR_SHAPE, "crt walker gemm: N=%d K=%d do not fit", g.N, g.K);
  RMaps maps;
  int rc;
  if ((rc = make_map(&maps.a, g.A, g.K, k.Np, RBK)) || (rc = make_map(&maps.b, g.B, g.K, k.bn, RBK)) ||
      (rc = make_map(&maps.b_last, g.B, g.K, k.bn_last, RBK)))
    return rc;
  constexpr int smem = RSMEM + RBAR + 1024;
  static_assert(smem <= 232448, "shared memory budget");
  for (int pass = g.check ? 0 : 1; pass < 2; ++pass) {  // the magnitudes, then the moduli of the walkers that passed
    // column chunks: whole rows of tiles per unit, split where there are too few walkers to fill the SMs
    auto kern = pass == 0 ? (k.segs == 2 ? (k.MT == 2 ? crt_walker_kernel<2, 2, true> : crt_walker_kernel<2, 1, true>)
                                         : (k.MT == 2 ? crt_walker_kernel<1, 2, true> : crt_walker_kernel<1, 1, true>))
                          : (k.segs == 2 ? (k.MT == 2 ? crt_walker_kernel<2, 2, false> : crt_walker_kernel<2, 1, false>)
                                         : (k.MT == 2 ? crt_walker_kernel<1, 2, false> : crt_walker_kernel<1, 1, false>));
    SFQ_MAX_SMEM(kern, smem);
    const long base = (pass == 0 ? 1L : NMOD) * g.batch * k.EC;
    const long cc = std::max<long>(1, std::min<long>((4L * sm_count() + base - 1) / base, k.NT));
    k.tpc = int((k.NT + cc - 1) / cc);
    k.CC = (k.NT + k.tpc - 1) / k.tpc;
    k.units = base * k.CC;
    const long grid = k.units < sm_count() ? k.units : sm_count();
    kern<<<unsigned(grid), kThreads, smem, st>>>(maps, k);
    SFQ_LAUNCHED();
  }
  return SFQ_OK;
}

int expiries(unsigned long long* n) {
  SFQ_CUDA_TRY(cudaMemcpyFromSymbol(n, g_expiries, sizeof(*n)));
  return SFQ_OK;
}

}  // namespace crt
}  // namespace sfq
