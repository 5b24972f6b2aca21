// FP64 trailing update on the integer tensor pipe by residues (see ozaki_update.h).
//
//   F[J1:m, J1:m] -= X X^T,   X = F[J1:m, J0:J1]  (K = J1 - J0 <= kOzK)
//
// The method is the Ozaki scheme II (Ozaki, Uchino and Imamura 2025).  Row a of X is
// scaled by 2^s_a and rounded to integers q, with s_a the largest shift that keeps the
// row's 2-norm at or below 2^62.18.  With P the product of the 16 coprime moduli below
// (P = 2^125.38), |Q_a . Q_b| <= |Q_a| |Q_b| < P / 2, so the integer product is fixed by
// its residues.  Those are exact: each modulus takes one 8-bit product of the rows'
// symmetric residues (|r| <= 128, sums of 512 products below 2^23 in int32).  The
// Chinese remainder theorem gives
//   Q_a . Q_b / P = sum_l acc_l T_l  (mod 1),   T_l = ((P / p_l)^-1 mod p_l) / p_l,
// which the epilogue sums in 64-bit fixed point (and a float below it) straight from the int32 accumulators
// (no reduction modulo p_l: an accumulator only matters modulo p_l).  The sum errs by at
// most 2^-60.8 P (the float's roundings with all 16 accumulators at their largest 8.6 units
// of 2^-64, the T_l, kept to 2^-88, 0.4) and by 2^-68 P for accumulators of usual size.  The
// rounding of a row to integers errs by at most 2^-62 of the row's norm per entry, 2^-57.6 of
// it over 512 entries, where a row of doubles is known to 2^-53.  What remains is one FP64
// rounding of the product and one of the subtraction.
//
// Against digit splitting (eight 7-bit digits, 36 products of one output tile), which
// this replaces, the tensor pipe does 16 products instead of 36, and because the
// moduli are independent one accumulator is alive at a time, so a tile can be 256 x 96
// per CTA pair instead of 128 x 64 per CTA.
//
// k_oz_residues writes the residues of every row; k_oz_update multiplies them.  Per
// cluster of two CTAs one 256 x 96 output tile: UMMA M = 256, N = 96, K = 32
// (tcgen05.mma.cta_group::2 kind::i8, K-major operands, 128-byte swizzle), every CTA
// holding its 128 rows' operand, half of the columns' and its 128 x 96 accumulator, so
// the pair brings the columns' operand into shared memory once.  Warp 0 streams pairs
// of 128-byte K blocks of both operands through four stages with TMA (this GPU's own
// residue buffer only, no multicast; with one K block a stage the loads' issue, 550
// cycles a stage, was the bound); warp 1 of the first CTA issues the MMAs, one accumulator per
// modulus, five of them in flight in tensor memory; warp 2 decodes the tile list ahead
// of everybody; warps 4-11 of both CTAs add each accumulator to their sums (48 columns of one row per thread: 144 registers,
// which is why the two epilogue warpgroups take registers from the first, and why a
// tile has 96 columns: with 128 the sums alone are 192 and the loop spills).  The sums of
// a modulus run while the next ones multiply, and the read-modify-write of a finished
// tile while the next tile's first moduli multiply.
//
// Bound and times (one front, K = 512, alone): the tensor pipe needs 768 cycles a
// modulus and tile but shared memory 1,400 (per 128-byte K block 22 KB written and 24 KB read,
// 128 bytes a cycle); a modulus takes 1,500 cycles, its sums 1,150 on
// the 32-bit integer pipe beside it.  r = 7,488 rows: 330 us where the digit kernel took
// 582 (1,520 against 1,840 TOP/s, of less than half the products); r = 4,928: 164 and 272;
// r = 2,368: 50 and 82.  The backward error of dense solves whose updates all take this
// path is 0.4 to 0.65 of the digit kernel's (rms 5.9e-18 to 9.6e-18 componentwise).
//
// Every mbarrier wait is bounded by time; a CTA that gives up records err[2], waits
// for its loads and MMAs (bounded) and frees its tensor memory.
#include "ozaki_update.h"

#include <algorithm>
#include <string>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "symbolic.h"

namespace tdem {
namespace {

constexpr int NM = kOzModuli;
constexpr int OM = 128;                  // tile rows of one CTA (the pair: UMMA M = 256)
constexpr int ON = kOzTileCols;          // tile columns of the pair (UMMA N)
constexpr int OKB = 128;                 // bytes of K per swizzled row (one K block)
constexpr int KBS = 2;                   // K blocks per stage
constexpr int A_BYTES = OM * OKB;        // 16 KB, per K block
constexpr int B_BYTES = ON / 2 * OKB;    // 6 KB: the CTA's half of the columns
constexpr int STAGE_BYTES = KBS * (A_BYTES + B_BYTES);
constexpr int NST = 4;                   // stages
constexpr int NACC = 5;                  // accumulators in tensor memory
constexpr int NTHR = 384;                // load, MMA, tile-list and idle warp; eight epilogue warps
constexpr int EPI_WARPS = 8;
constexpr int EC = ON / 2;               // columns per epilogue thread
constexpr int ACC_COLS = ON;             // tensor-memory columns from one accumulator to the next
constexpr int TMEM_COLS = 512;           // allocated (a power of two)
static_assert(NACC * ACC_COLS <= TMEM_COLS, "accumulators");
constexpr int NSLOT = 3;                 // tiles decoded ahead
constexpr int NBAR = 2 * NST + 2 * NACC + 2 * NSLOT + 1;
// One decoded tile: what the roles need of it (see oz_tile) and the front's offsets.
struct TileSlot {
  int64_t lo, uo;
  int m, k, nkb, r0, c0, arow, brow, live;
  double ra[OM], rb[ON];  // the rows' and columns' powers of two (their product includes 2^125)
};
constexpr size_t SMEM_BYTES =
    1024 /* alignment */ + (size_t)NST * STAGE_BYTES + NSLOT * sizeof(TileSlot) + 8 * NBAR + 32;
constexpr int RW = 8;                   // columns read and written at a time
constexpr long long kWaitCycles = 4000000000ll;  // about two seconds
// Registers: the block is launched with 384 x 168; the first warpgroup gives its
// share back down to 40 and the two epilogue warpgroups take 232 each.
constexpr int kRegsFew = 40, kRegsMany = 232;
static_assert(128 * kRegsFew + 256 * kRegsMany <= 384 * 168, "register split");
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");

// instruction descriptor: D S32, A and B signed 8-bit, both K-major, M = 256, N = 96
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ON >> 3) << 17) |
                            ((uint32_t)((2 * OM) >> 4) << 24);

typedef unsigned __int128 u128;

constexpr int kModuli[NM] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};

// What the kernels need of the moduli.
struct OzTable {
  // residues of 256^i, i = 0..3 and 4..7, as packed signed bytes
  uint32_t c_lo[NM] = {}, c_hi[NM] = {};
  int p[NM] = {};
  float inv_p[NM] = {};
  int t1[NM] = {}, t2[NM] = {};  // T_l = t2 2^-32 + t1 2^-64 + t0 2^-64
  float t0[NM] = {};
  double ph = 0, pl = 0, ph32 = 0;  // P 2^(-32 - 125) = ph + pl, ph32 = ph 2^-32
};

constexpr int sym_mod(int64_t v, int p) {
  int r = (int)(v % p);
  if (r < 0) r += p;
  return 2 * r > p - 1 + (p & 1) ? r - p : r;  // odd p: [-(p - 1) / 2, (p - 1) / 2]; even: [-p / 2, p / 2)
}

constexpr double pow2(int n) {
  double v = 1.0;
  for (; n > 0; --n) v *= 2.0;
  for (; n < 0; ++n) v *= 0.5;
  return v;
}

constexpr OzTable make_table() {
  OzTable z;
  u128 P = 1;
  for (int l = 0; l < NM; ++l) P *= (u128)kModuli[l];
  for (int l = 0; l < NM; ++l) {
    const int p = kModuli[l];
    z.p[l] = p;
    z.inv_p[l] = 1.0f / (float)p;
    int64_t pw = 1;
    for (int i = 0; i < 8; ++i) {
      const uint32_t b = (uint32_t)sym_mod(pw, p) & 0xFFu;
      if (i < 4) z.c_lo[l] |= b << (8 * i);
      else z.c_hi[l] |= b << (8 * (i - 4));
      pw = pw * 256 % p;
    }
    int rest = 1, inv = 1;  // the other moduli's product modulo p, and its inverse
    for (int j = 0; j < NM; ++j)
      if (j != l) rest = rest * (kModuli[j] % p) % p;
    while (rest * inv % p != 1) ++inv;
    // 2^96 T_l; limbs of 2^31 or more are taken less 2^32, which the next makes up for
    const u128 t = (((u128)inv << 96) + (u128)(p / 2)) / (u128)p;
    const int64_t w0 = (int)(uint32_t)t;
    const uint64_t w1 = (uint64_t)(uint32_t)(t >> 32) + ((uint32_t)t >> 31);
    const uint64_t w2 = (uint64_t)(uint32_t)(t >> 64) + (w1 >> 31);
    z.t0[l] = (float)((double)w0 * pow2(-32));
    z.t1[l] = (int)(uint32_t)w1;
    z.t2[l] = (int)(uint32_t)w2;
  }
  const u128 hi = P >> 73, rem = P - (hi << 73);
  z.ph = (double)(uint64_t)hi * pow2(73 - 32 - 125);
  z.pl = (double)(uint64_t)(rem >> 20) * pow2(20 - 32 - 125);
  z.ph32 = z.ph * pow2(-32);
  return z;
}

__constant__ OzTable c_oz = make_table();

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor of a K-major operand with 128-byte swizzle at addr
// (1024-byte aligned): stride byte offset 1024 (8-row groups), version 1, layout
// SWIZZLE_128B.  The 32-byte K steps inside the 128-byte rows add 2 to the start field.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(16 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// address of this CTA's shared-memory location in the pair's CTA `rank`
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// (no cluster-scope release here and no acquire in the waits: what the barriers order
// is tensor memory, through the tcgen05 fences; a cluster-scope release is a memory
// fence that waits for the warp's global stores, and cost half the kernel's time)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void next_slot(int& sl, uint32_t& parity) {
  if (++sl == NSLOT) {
    sl = 0;
    parity ^= 1;
  }
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  do {
    if (mbar_try(bar, parity)) return true;
  } while (clock64() - t0 < kWaitCycles);
  return false;
}
// 4D tiled TMA load of the box at row x, K block y, modulus z into this CTA's dst,
// completing on bar, which may be the peer's
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
      "l"(map), "r"(bar), "r"(0), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accum) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p; }" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(kIdesc), "r"(accum)
      : "memory");
}
// the MMAs issued so far arrive at bar (the same location in both CTAs) when done
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
// one lane of the converged warp.  Loads, MMAs and commits are issued by warps that run
// their loops whole, under this predicate: the compiler then keeps their operands in
// uniform registers.  From a branch on the lane index a load cost 200 cycles to issue
// and a stage of four MMAs 620, more than twice its 256 cycles on the tensor pipe.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 16 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld(uint32_t (&a)[16], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]), "=r"(a[8]),
        "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15])
      : "r"(addr));
}
// the loads have landed: the registers are tied to the wait, so that no use of them
// moves above it
__device__ __forceinline__ void tmem_wait(uint32_t (&a)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
               :
               : "memory");
}

// One more modulus' term of the sum, modulo 1: s (at weight 2^-64) += a (t2 2^32 + t1),
// f (at weight 2^-64) += a t0, for t = t2 2^-32 + t1 2^-64 + t0 2^-64 with signed limbs
// t2, t1 and |t0| <= 1/2; |a| <= 2^23.  The integer part wraps where the sum does, so
// no carries leave it, and what lies below it only needs single precision.  8 issue
// cycles a warp, where 96-bit sums with carrying 32-bit multiply-adds took 60, with
// 64-bit products and carrying adds 45, and with the high half of a t0 as an integer
// product 23 (a high product alone is 6, a 64-bit add 8, a wide multiply-add 3).
__device__ __forceinline__ void add_term(unsigned long long& s, float& f, int a, int t2, int t1, float t0) {
  asm("{ .reg .u32 lo, hi;\n\t"
      "mad.wide.s32 %0, %2, %4, %0;\n\t"
      "mov.b64 {lo, hi}, %0;\n\t"
      "mad.lo.s32 hi, %2, %3, hi;\n\t"
      "mov.b64 %0, {lo, hi};\n\t"
      "fma.rn.f32 %1, %6, %5, %1; }"
      : "+l"(s), "+f"(f)
      : "r"(a), "r"(t2), "r"(t1), "f"(t0), "f"((float)a));
}

// 2^n for -1022 <= n <= 1023
__device__ __forceinline__ double pow2d(int n) { return __longlong_as_double((long long)(n + 1023) << 52); }

// The rounded products of EC columns subtracted from one row of the trailing matrix:
// column x of the tile at p + x ld (x < kx) or q + x ldq, for x <= last, times the row's
// and the column's power of two.  WHOLE: every column, all at p.
//
// Every 32-bit integer instruction is two issue cycles a warp here, and with the index
// arithmetic left to the compiler (per column: two predicates, a pointer selected twice,
// two 64-bit products, 64-bit shifts into the conversions and a scaling by exponent bits)
// this step took 160 of them, 21,000 cycles a tile; as a reduction at L2 it was bound by
// the rate of those, 112 a cycle over the chip.  RW columns are read ahead of the RW
// being written.
template <bool WHOLE, int EC>
__device__ __forceinline__ void write_columns(const unsigned long long (&sum)[EC], const float (&low)[EC], double* p,
                                              int ld, double* q, int ldq, int kx, int last, double ra,
                                              const double* rb) {
  // (a column's address is one wide multiply-add; kept as running pointers it is two)
  auto at = [&](int x) { return WHOLE || x < kx ? p + (int64_t)x * ld : q + (int64_t)x * ldq; };
  double old[2][RW];
  auto load = [&](int h, double (&o)[RW]) {
#pragma unroll
    for (int i = 0; i < RW; ++i) o[i] = WHOLE || RW * h + i <= last ? *at(RW * h + i) : 0.0;
  };
  load(0, old[0]);
#pragma unroll
  for (int h = 0; h < EC / RW; ++h) {
    if (h + 1 < EC / RW) load(h + 1, old[(h + 1) & 1]);
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      const int x = RW * h + i;
      // the sum as a signed fraction of 2^64: both words by the exponent trick (the bits
      // of 2^52 with a word below them are 2^52 plus the word), and the float below them
      const uint32_t s1 = (uint32_t)(sum[x] >> 32), s0 = (uint32_t)sum[x];
      const double hi = __hiloint2double(0x43300000, (int)(s1 ^ 0x80000000u)) - 0x1.000008p52;  // 2^52 + 2^31
      const double lw = (__hiloint2double(0x43300000, (int)s0) - 0x1p52) + (double)low[x];
      const double v = fma(c_oz.ph, hi, fma(c_oz.pl, hi, c_oz.ph32 * lw));
      if (WHOLE || x <= last) *at(x) = old[h & 1][i] - v * ra * rb[x];
    }
  }
}

__device__ __forceinline__ int find_task(const int64_t* __restrict__ prefix, int count, int64_t b) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Residues of rows [row0, row0 + 64) of the panel of one front (64 rows per CTA,
// 256 threads): pass 1 finds each row's shift, pass 2 stages 64 x 64 blocks of the
// panel (coalesced along the rows) and writes 16 residues per thread and modulus as
// one 16-byte store; columns in [K, roundup(K, 128)) get zeros.
//
// An integer q (|q| <= 2^62.2) is taken as eight signed base-256 digits (adding 128 to
// every byte and flipping its top bit back gives the balanced digits), so q mod p is
// two dp4a with the residues of 256^i, |t| <= 2^17, and one rounded division done in
// single precision: t is exact there, the quotient's fraction is at least 1 / (2 p) =
// 2^-9 away from a half for odd p and its error below 2^-13, so the rounding always
// gives the symmetric residue (p = 256: t is the lowest digit itself).
__global__ void __launch_bounds__(256) k_oz_residues(const double* __restrict__ L, const int64_t* __restrict__ l_off,
                                                     const int* __restrict__ fm, const int* __restrict__ fk,
                                                     const int* __restrict__ fronts,
                                                     const int64_t* __restrict__ prefix,
                                                     const int64_t* __restrict__ aux, int count, int j0,
                                                     int8_t* __restrict__ residues, int* __restrict__ exps,
                                                     int64_t nrows_buf) {
  __shared__ double T[64][65];  // [column][row]
  __shared__ double red[4][64], red2[4][64];
  __shared__ int shift[64];
  const int idx = find_task(prefix, count, blockIdx.x);
  const int s = fronts[idx];
  const int m = fm[s], k = fk[s];
  const int J0 = (j0 / kOuter) * kOuter, J1 = min(k, J0 + kOuter), K = J1 - J0;
  const int row0 = J1 + (int)(blockIdx.x - prefix[idx]) * 64;
  const int nrows = min(64, m - row0);
  const int64_t out0 = aux[idx] + (row0 - J1);
  const double* F = L + l_off[s];
  const int t = threadIdx.x, i = t & 63, g = t >> 6;
  double mx = 0.0, sq = 0.0;
  if (i < nrows)
    for (int kk = g; kk < K; kk += 4) {
      const double v = F[(row0 + i) + (int64_t)(J0 + kk) * m];
      mx = fmax(mx, fabs(v));
      sq = fma(v, v, sq);
    }
  red[g][i] = mx;
  red2[g][i] = sq;
  __syncthreads();
  if (t < 64) {
    mx = fmax(fmax(red[0][t], red[1][t]), fmax(red[2][t], red[3][t]));
    int sh = 0;
    if (mx > 0.0) {
      int e;
      if (mx > 0x1p-400 && mx < 0x1p400) {
        const double f = frexp(sqrt(red2[0][t] + red2[1][t] + red2[2][t] + red2[3][t]), &e);  // 0.5 <= f < 1
        sh = 62 - e + (f < 0.565 ? 1 : 0);  // 0.565 2^63 < 2^62.18
      } else {  // the squares may leave the range: |row| <= sqrt(512) max < 2^(e + 5)
        frexp(mx, &e);
        sh = 57 - e;
      }
      // rows below 2^-738 keep 2^-800 as their unit; none is above 2^512 (its square is
      // part of a diagonal entry).  The powers of two then scale without rounding.
      sh = max(-500, min(800, sh));
    }
    shift[t] = sh;
    if (t < nrows) exps[out0 + t] = -sh;
  }
  __syncthreads();
  const int rr = t >> 2, seg = t & 3;
  const int Kp = (K + OKB - 1) / OKB * OKB;
  const double sc = pow2d(shift[rr]);
  for (int kc = 0; kc < Kp; kc += 64) {
#pragma unroll 4
    for (int j = 0; j < 16; ++j) {
      const int kk = kc + g + 4 * j;
      T[g + 4 * j][i] = (i < nrows && kk < K) ? F[(row0 + i) + (int64_t)(J0 + kk) * m] : 0.0;
    }
    __syncthreads();
    uint32_t lo[16], hi[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const unsigned long long v =
          (unsigned long long)__double2ll_rn(T[16 * seg + q][rr] * sc) + 0x8080808080808080ull;
      lo[q] = (uint32_t)v ^ 0x80808080u;
      hi[q] = (uint32_t)(v >> 32) ^ 0x80808080u;
    }
#pragma unroll 1
    for (int l = 0; l < NM; ++l) {
      const int cl = (int)c_oz.c_lo[l], ch = (int)c_oz.c_hi[l], p = c_oz.p[l];
      const float ip = c_oz.inv_p[l];
      uint32_t w[4];
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        uint32_t r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int d = __dp4a((int)hi[4 * q4 + q], ch, __dp4a((int)lo[4 * q4 + q], cl, 0));
          const float f = __int_as_float(0x4B400000 + d) - 12582912.0f;
          const int n = __float_as_int(fmaf(f, ip, 12582912.0f)) - 0x4B400000;
          r[q] = (uint32_t)(d - n * p);
        }
        w[q4] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
      }
      if (rr < nrows)
        *reinterpret_cast<int4*>(residues + ((int64_t)l * nrows_buf + out0 + rr) * kOzK + kc + 16 * seg) =
            make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]);
    }
    __syncthreads();
  }
}

// Tile `id` of the task list for the pair's CTA of this rank: its front and coordinates
// (order: oz_tiles; the 74 tiles in flight then share about nine row tiles and eight
// column tiles, whose residues stay in L2).  live: the CTA's 128 rows reach the lower
// triangle of the front.
struct OzTile {
  int s, m, k, J1, nkb, r0, c0, arow, brow;
  bool live;
};

__device__ __forceinline__ OzTile oz_tile(const int* __restrict__ fm, const int* __restrict__ fk,
                                          const int* __restrict__ fronts, const int64_t* __restrict__ prefix,
                                          const int64_t* __restrict__ aux, int count, int j0, int64_t id, int rank) {
  OzTile z;
  const int idx = find_task(prefix, count, id);
  z.s = fronts[idx];
  z.m = fm[z.s];
  z.k = fk[z.s];
  const int J0 = (j0 / kOuter) * kOuter;
  z.J1 = min(z.k, J0 + kOuter);
  z.nkb = (z.J1 - J0 + OKB - 1) / OKB;
  const int r = z.m - z.J1, cols = (r + ON - 1) / ON;
  int t = (int)(id - prefix[idx]), below = (r + 255) / 256, cb = 0, w, n0, n1;
  for (;; cb += kOzSuper, below -= 3) {
    w = min(kOzSuper, cols - cb);
    n0 = min(3, w);
    n1 = below > 1 ? min(6, w) : 0;
    const int all = n0 + n1 + (below > 2 ? (below - 2) * w : 0);
    if (t < all) break;
    t -= all;
  }
  int rp = 0;
  if (t >= n0 + n1) {
    t -= n0 + n1;
    rp = 2 + t / w;
    t %= w;
  } else if (t >= n0) {
    t -= n0;
    rp = 1;
  }
  const int ro = (3 * (cb / kOzSuper) + rp) * 256 + rank * OM, co = (cb + t) * ON;
  z.live = ro < r && ro + OM > co;
  z.r0 = z.J1 + ro;
  z.c0 = z.J1 + co;
  z.arow = (int)aux[idx] + ro;
  z.brow = (int)aux[idx] + co;
  return z;
}

// Persistent: pair b takes the tiles b, b + pairs, ... of the list (all roles of both
// CTAs walk the same sequence).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHR, 1)
k_oz_update(double* __restrict__ L, double* __restrict__ U, const int64_t* __restrict__ l_off,
            const int64_t* __restrict__ u_off, const int* __restrict__ fm, const int* __restrict__ fk,
            const int* __restrict__ fronts, const int64_t* __restrict__ prefix, const int64_t* __restrict__ aux,
            int count, int64_t ntiles, int j0, const int* __restrict__ exps, int64_t nrows_buf, int* err,
            const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  // 1024-byte aligned operand area (swizzle atoms are 1024 bytes; the same offset in
  // both CTAs, whose shared-memory windows are laid out alike)
  const uint32_t raw = smem_u32(sm_raw);
  unsigned char* ops = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  // full[NST] and free[NACC] are waited on in the first CTA only
  TileSlot* slots = reinterpret_cast<TileSlot*>(ops + NST * STAGE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(slots + NSLOT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBAR);
  int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * NST, acc0 = empty0 + 8 * NST, free0 = acc0 + 8 * NACC,
                 tile0 = free0 + 8 * NACC, taken0 = tile0 + 8 * NSLOT, done_bar = taken0 + 8 * NSLOT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int64_t first = blockIdx.x >> 1, stride = gridDim.x >> 1;

  if (tid == 0) {
    for (int q = 0; q < NST; ++q) {
      mbar_init(full0 + 8 * q, 1);   // the first CTA's expect_tx arrival (+ both CTAs' bytes)
      mbar_init(empty0 + 8 * q, 1);  // one tcgen05.commit frees the stage in both CTAs
    }
    for (int q = 0; q < NACC; ++q) {
      mbar_init(acc0 + 8 * q, 1);                  // the commit after a modulus' last MMA
      mbar_init(free0 + 8 * q, 2 * EPI_WARPS);     // every epilogue warp of both CTAs, after its reads
    }
    for (int q = 0; q < NSLOT; ++q) {
      mbar_init(tile0 + 8 * q, 1);                                  // the decoding warp
      mbar_init(taken0 + 8 * q, EPI_WARPS + 1 + (rank == 0 ? 1 : 0));  // every warp that reads the slot
    }
    mbar_init(done_bar, 1);
    *s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // the peer's barriers and tensor memory are ready
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsFew));
    if (warp == 0) {
      // producer: K block kb of modulus l of the tile's rows (A) and half its columns (B)
      const uint32_t lead_full0 = peer_addr(full0, 0);
      int st = 0, sl = 0;
      uint32_t ph = 1, tph = 0;  // the first pass over the stages finds them free
      bool stop = false;
      for (int64_t id = first; id < ntiles && !stop; id += stride) {
        if (!mbar_wait(tile0 + 8 * sl, tph)) {
          stop = true;
          break;
        }
        const int nkb = slots[sl].nkb, arow = slots[sl].arow, brow = slots[sl].brow + (int)rank * (ON / 2);
        __syncwarp();
        if (lane == 0) mbar_arrive(taken0 + 8 * sl);
        next_slot(sl, tph);
        for (int l = 0; l < NM && !stop; ++l) {
          for (int kb = 0; kb < nkb; kb += KBS) {
            if (!mbar_wait(empty0 + 8 * st, ph)) {
              stop = true;
              break;
            }
            const uint32_t a = smem_u32(ops) + st * STAGE_BYTES;
            if (elect_one()) {
              if (rank == 0) mbar_expect_tx(full0 + 8 * st, 2u * STAGE_BYTES);
              tma_load(a, &tmA, lead_full0 + 8 * st, arow, kb, l);
              tma_load(a + KBS * A_BYTES, &tmB, lead_full0 + 8 * st, brow, kb, l);
            }
            __syncwarp();
            if (++st == NST) {
              st = 0;
              ph ^= 1;
            }
          }
        }
      }
      if (stop && lane == 0) atomicExch(s_fail, 1);
    } else if (warp == 1 && rank == 0) {
      // MMA issuer: one accumulator per modulus
      int st = 0, bu = 0, sl = 0;
      uint32_t ph = 0, fph = 1, tph = 0;
      bool stop = false;
      for (int64_t id = first; id < ntiles && !stop; id += stride) {
        if (!mbar_wait(tile0 + 8 * sl, tph)) {
          stop = true;
          break;
        }
        const int nkb = slots[sl].nkb;
        __syncwarp();
        if (lane == 0) mbar_arrive(taken0 + 8 * sl);
        next_slot(sl, tph);
        for (int l = 0; l < NM && !stop; ++l) {
          // the epilogues have read this accumulator's previous modulus
          if (!mbar_wait(free0 + 8 * bu, fph)) {
            stop = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int kb = 0; kb < nkb; kb += KBS) {
            if (!mbar_wait(full0 + 8 * st, ph)) {
              stop = true;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = sdesc(smem_u32(ops) + st * STAGE_BYTES);
            const uint64_t db = sdesc(smem_u32(ops) + st * STAGE_BYTES + KBS * A_BYTES);
            if (elect_one()) {
#pragma unroll
              for (int b = 0; b < KBS; ++b)
                if (kb + b < nkb) {
#pragma unroll
                  for (int ks = 0; ks < OKB / 32; ++ks)
                    mma_i8(tmem + (uint32_t)(ACC_COLS * bu), da + ((b * A_BYTES) >> 4) + 2 * ks,
                           db + ((b * B_BYTES) >> 4) + 2 * ks, (kb + b + ks > 0) ? 1u : 0u);
                }
              mma_commit(empty0 + 8 * st);
              if (kb + KBS >= nkb) mma_commit(acc0 + 8 * bu);
            }
            __syncwarp();
            if (++st == NST) {
              st = 0;
              ph ^= 1;
            }
          }
          if (++bu == NACC) {
            bu = 0;
            fph ^= 1;
          }
        }
      }
      if (stop && lane == 0) atomicExch(s_fail, 1);
      // every MMA issued: arrives once they have completed
      if (elect_one()) mma_commit(done_bar);
      __syncwarp();
    } else if (warp == 2) {
      // tile list: decodes up to NSLOT tiles ahead (half a dozen dependent loads each)
      int sl = 0;
      uint32_t eph = 1;
      for (int64_t id = first; id < ntiles; id += stride) {
        const OzTile z = oz_tile(fm, fk, fronts, prefix, aux, count, j0, id, (int)rank);
        if (!mbar_wait(taken0 + 8 * sl, eph) || *(volatile int*)s_fail) break;
        TileSlot& t = slots[sl];
        for (int q = lane; q < OM; q += 32) {
          t.ra[q] = pow2d(62 + (z.arow + q < nrows_buf ? exps[z.arow + q] : 0));
          if (q < ON) t.rb[q] = pow2d(63 + (z.brow + q < nrows_buf ? exps[z.brow + q] : 0));
        }
        if (lane == 0) {
          t.lo = l_off[z.s];
          t.uo = u_off[z.s];
          t.m = z.m;
          t.k = z.k;
          t.nkb = z.nkb;
          t.r0 = z.r0;
          t.c0 = z.c0;
          t.arow = z.arow;
          t.brow = z.brow;
          t.live = z.live ? 1 : 0;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(tile0 + 8 * sl);
        next_slot(sl, eph);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMany));
    // epilogue: row 32 (warp % 4) + lane of the CTA's tile (its tensor-memory lanes),
    // columns [cb, cb + EC)
    const int sub = warp & 3, rl = 32 * sub + lane, cb = EC * ((warp - 4) >> 2);
    const uint32_t lead_free0 = peer_addr(free0, 0);
    const uint32_t taddr = tmem + ((uint32_t)(32 * sub) << 16) + (uint32_t)cb;
    int bu = 0, sl = 0;
    uint32_t par = 0, tph = 0;
    bool ok = true;
    for (int64_t id = first; id < ntiles && ok; id += stride) {
      ok = mbar_wait(tile0 + 8 * sl, tph);
      if (!__all_sync(0xffffffffu, ok)) break;
      const bool live = slots[sl].live != 0;
      unsigned long long sum[EC];
      float low[EC];
#pragma unroll
      for (int c = 0; c < EC; ++c) {
        sum[c] = 0;
        low[c] = 0.0f;
      }
#pragma unroll 1
      for (int l = 0; l < NM; ++l) {
        const int t2 = c_oz.t2[l], t1 = c_oz.t1[l];
        const float t0 = c_oz.t0[l];
        // one lane polls where the accumulator is not there yet (256 threads polling
        // would take issue slots from the MMA and load warps), then all see it
        const uint32_t bar = acc0 + 8 * bu;
        if (!__all_sync(0xffffffffu, mbar_try(bar, par))) {
          if (lane == 0) ok = mbar_wait(bar, par) && !*(volatile int*)s_fail;
          __syncwarp();
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0 && mbar_wait(bar, par);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (live) {
          const uint32_t acc = taddr + (uint32_t)(ACC_COLS * bu);
          // 16 columns at a time, the next 16 on their way meanwhile (with 8 the loads'
          // latency, about 200 cycles, shows: 1,750 cycles a modulus)
          uint32_t x[2][16];
          tmem_ld(x[0], acc);
#pragma unroll
          for (int h = 0; h < EC / 16; ++h) {
            tmem_wait(x[h & 1]);
            if (h + 1 < EC / 16) tmem_ld(x[(h + 1) & 1], acc + 16 * (h + 1));
#pragma unroll
            for (int q = 0; q < 16; ++q)
              add_term(sum[16 * h + q], low[16 * h + q], (int)x[h & 1][q], t2, t1, t0);
          }
        }
        // the accumulator is free for a later modulus
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_free0 + 8 * bu);
        if (++bu == NACC) {
          bu = 0;
          par ^= 1;
        }
      }
      if (ok && live) {
        const TileSlot& t = slots[sl];
        const int m = t.m, k = t.k, r = t.r0 + rl, c0 = t.c0 + cb;
        const double ra = t.ra[rl];
        const double* rb = t.rb + cb;
        // columns c0 + x of row r for x < last; those at or right of column k in the
        // update block
        const int last = r < m ? r - c0 : -1;
        double* pl = L + t.lo + r + (int64_t)c0 * m;
        double* pu = U + t.uo + (r - k) + (int64_t)(c0 - k) * (m - k);
        if (t.r0 >= c0 + EC && t.r0 + OM <= m && (c0 + EC <= k || c0 >= k)) {
          // no edge, no diagonal, one array
          write_columns<true>(sum, low, c0 < k ? pl : pu, c0 < k ? m : m - k, pu, 0, EC, EC, ra, rb);
        } else {
          write_columns<false>(sum, low, pl, m, pu, m - k, k - c0, last, ra, rb);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(taken0 + 8 * sl);
      next_slot(sl, tph);
    }
  }
  __syncwarp();
  __syncthreads();
  const bool good = mbar_wait(done_bar, 0u) && *(volatile int*)s_fail == 0;
  __syncwarp();
  cluster_sync();  // both CTAs have stopped issuing loads, MMAs and remote arrivals
  if (!good && tid == 0) {
    atomicExch(err + 2, 1);
    // loads that no MMA waited for may still be on their way into shared memory (a
    // stage whose other half was never issued cannot complete): a millisecond covers them
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace

std::string ozaki_setup(OzakiBuffers& ob) {
  static_assert(sizeof(CUtensorMap) <= sizeof(ob.map_a), "tensor map storage");
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
  if (e != cudaSuccess || !fn || q != cudaDriverEntryPointSuccess)
    return "cuTensorMapEncodeTiled not available from the driver";
  auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
  // K as blocks of 128 bytes outside the rows, so that one box holds whole K blocks
  const cuuint64_t dims[4] = {OKB, (cuuint64_t)ob.rows, kOzK / OKB, (cuuint64_t)NM};
  const cuuint64_t strides[3] = {(cuuint64_t)kOzK, OKB, (cuuint64_t)kOzK * (cuuint64_t)ob.rows};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const cuuint32_t box_a[4] = {OKB, OM, KBS, 1}, box_b[4] = {OKB, ON / 2, KBS, 1};
  CUresult r = encode(reinterpret_cast<CUtensorMap*>(ob.map_a), CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, ob.residues, dims,
                      strides, box_a, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled (128-row residue boxes) failed: " + std::to_string((int)r);
  r = encode(reinterpret_cast<CUtensorMap*>(ob.map_b), CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, ob.residues, dims, strides,
             box_b, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled (48-row residue boxes) failed: " + std::to_string((int)r);
  e = cudaFuncSetAttribute(k_oz_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
  if (e != cudaSuccess) return std::string("cudaFuncSetAttribute(k_oz_update): ") + cudaGetErrorString(e);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&ob.sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                 cudaSuccess)
    return "cannot read the SM count";
  return "";
}

void launch_ozaki_residues(const double* L, const int64_t* l_off, const int* m, const int* k, const int* fronts,
                           const int64_t* prefix, const int64_t* aux, int count, int64_t ctas, int j0,
                           const OzakiBuffers& ob, cudaStream_t s) {
  k_oz_residues<<<(unsigned)ctas, 256, 0, s>>>(L, l_off, m, k, fronts, prefix, aux, count, j0, ob.residues, ob.exps,
                                               ob.rows);
}

void launch_ozaki_update(double* L, double* U, const int64_t* l_off, const int64_t* u_off, const int* m,
                         const int* k, const int* fronts, const int64_t* prefix, const int64_t* aux, int count,
                         int64_t tiles, int j0, const OzakiBuffers& ob, int* err, cudaStream_t s) {
  const int64_t pairs = std::min<int64_t>(tiles, std::max(1, (ob.sms > 0 ? ob.sms : 148) / 2));
  k_oz_update<<<(unsigned)(2 * pairs), NTHR, SMEM_BYTES, s>>>(
      L, U, l_off, u_off, m, k, fronts, prefix, aux, count, tiles, j0, ob.exps, ob.rows, err,
      *reinterpret_cast<const CUtensorMap*>(ob.map_a), *reinterpret_cast<const CUtensorMap*>(ob.map_b));
}

}  // namespace tdem
