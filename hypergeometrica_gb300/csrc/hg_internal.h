// hg_internal.h -- structures shared by the kernels and the host driver.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "hg_common.cuh"

namespace hg {

// Device twiddle tables of one prime.
struct NttTables {
  const ulonglong2 *sub_fwd;  // (w_4096^e, Shoup companion), e < 2048: sub-transform twiddles, any R <= 4096
  const ulonglong2 *sub_inv;  // (w_4096^-e, companion)
  const uint64_t *hi_fwd;     // w_{2^30}^(e * 2^15), e < 2^15, Montgomery form
  const uint64_t *lo_fwd;     // w_{2^30}^e,          e < 2^15, Montgomery form
  const uint64_t *hi_inv;
  const uint64_t *lo_inv;
  // Sub-transform tables of every block size R = 2^T, T = 1..12, in the
  // contiguous pass's padded order: entry tw_pos(e) of the table of T is
  // (w_R^e, companion), e < R / 2.  The forward table of T starts at entry
  // tw_base(T), its inverse kTwInverse entries later.
  const ulonglong2 *swz;
};

// Padded position of entry e of a contiguous pass's twiddle table: one gap
// entry after every 8, 64 and 512, so that 8 lanes reading 16-byte entries
// at a power-of-two stride of up to 2^8 entries hit 8 different bank quads.
// Additive over disjoint bits (tw_pos(a | b) = tw_pos(a) + tw_pos(b) when
// a & b = 0), so a thread's part and a register's compile-time part of an
// index combine by an addition the load instruction's offset absorbs.  The
// 12-bit middle kernel ran 1.2% faster than with an XOR swizzle of the same
// bank property (no gaps, but an XOR per load), and spilled less.
__host__ __device__ __forceinline__ constexpr uint32_t tw_pos(uint32_t e) {
  return e + (e >> 3) + (e >> 6) + (e >> 9);
}

// First entry of the padded table of block size 2^T (T = 1..13; 13 gives
// the entries of all forward tables).
__host__ __device__ __forceinline__ constexpr uint32_t tw_base(int T) {
  uint32_t b = 0;
  for (int t = 1; t < T; ++t) b += tw_pos((1u << (t - 1)) - 1u) + 1u;
  return b;
}

constexpr uint32_t kTwInverse = tw_base(kTileBits + 1);  // entries in all forward tables

// Shared-memory word of position x of a contiguous pass's block: bits 4..7
// XORed into bits 0..3, so that 16 lanes reading 8-byte words at a
// power-of-two stride of up to 128 positions hit 16 different bank pairs.
// Not padded: a gap word per 16 takes three middle-kernel CTAs past the
// 196 KB shared-memory carveout, which leaves the SM 28 KB of L1 for the
// twiddle tables instead of 60 KB (measured 2.3% slower).
__host__ __device__ __forceinline__ constexpr uint32_t data_swz(uint32_t x) { return x ^ ((x >> 4) & 15u); }

__host__ __device__ __forceinline__ const ulonglong2 *swz_table(const NttTables &t, int T, bool inverse) {
  return t.swz + (inverse ? kTwInverse : 0u) + tw_base(T);
}

// One product of a batch, as the kernels read it.  y == nullptr squares x.
struct ProductDesc {
  const uint64_t *x, *y;
  uint64_t nx, ny;
  uint64_t *out;
  uint64_t nout;
};

// One NTT pass over the residue arrays of nprod products x nops operands x
// nprimes primes.  The N residues of an array form blocks of M = R*S; the
// pass performs the reference's radix-2 stages subn = M .. 2S, i.e. an
// R-point transform down each of the S columns of every block, followed
// (forward) or preceded (inverse) by the twiddle w_M^(s * bitrev(r)).
// Product k's arrays start at data[op] + k * ws_stride; prime i's at a
// further (i - prime_lo) * prime_stride.
struct PassArgs {
  uint64_t *data[2];           // residues per operand
  const uint64_t *limbs[2];    // single product: this pass reads and reduces limbs
  uint64_t nlimbs[2];
  const ProductDesc *batch;    // batch: operands of product k are batch[k].x / .y
  uint64_t chunk;              // single product cut into chunks: product k reads
                               // operand 0's limbs [k * chunk, (k + 1) * chunk)
  int read_limbs;              // batch: this pass reads and reduces limbs
  // The operands' coefficients are digits of 80 bits (5 limbs hold 4) instead
  // of limbs; a pass that reads limbs then forms them.
  int dig80;
  int nops;                    // operands handled by this launch
  int logN;
  int logR;                    // log2 rows (transform points) of this pass
  int logS;                    // log2 stride; 0 = contiguous pass
  int logT;                    // log2 residues per tile
  // Residues of each array: 2^logN, or fewer in a truncated transform
  // (krows rows of the outer pass, see hg_ntt_strided.cu).
  uint64_t points;
  int krows;                   // strided passes: rows of a block that are kept (R unless truncated)
  int prime_lo, nprimes;
  uint64_t prime_stride;       // words between the arrays of consecutive primes
  uint64_t nprod;              // products in the launch
  uint64_t ws_stride;          // words between consecutive products' arrays
  uint64_t tiles;              // tiles per (product, operand, prime) in this launch
  uint64_t tile_lo;            // strided passes: the launch covers tiles [tile_lo, tile_lo + tiles)
  PrimeConst pc[kPrimes];
  NttTables tb[kPrimes];
  // Strided passes: the inter-pass twiddles w_M^(+-s * bitrev r) of this
  // (M, R, direction), Montgomery form, [prime][r][s] with M words per prime
  // (all primes of the scheme), or null to form them from tb.
  const uint64_t *ptw;
  // Spectrum entry point: the transform's last inverse pass (strided or
  // contiguous) multiplies every residue by this Montgomery-form factor, which
  // leaves it in [0, p); 0 elsewhere (one prime per launch).
  uint64_t scale;
  int *err;                    // device error word (a tile copy that did not land)
};

// Limbs a pass reads for (product, operand), or nullptr when it reads residues.
__host__ __device__ __forceinline__ const uint64_t *pass_limbs(const PassArgs &P, uint64_t prod, int op,
                                                               uint64_t &nl) {
  if (P.batch) {
    if (!P.read_limbs) return nullptr;
    const ProductDesc &d = P.batch[prod];
    nl = op ? d.ny : d.nx;
    return op ? d.y : d.x;
  }
  nl = P.nlimbs[op];
  if (P.chunk && op == 0 && P.limbs[0]) {
    const uint64_t o = prod * P.chunk;
    nl = nl > o ? (nl - o < P.chunk ? nl - o : P.chunk) : 0;
    return P.limbs[0] + o;
  }
  return P.limbs[op];
}

// Constants of the Garner reconstruction for one transform length.
// Each constant is a (value, Shoup companion) pair.  The residues are
// N c 2^-64 mod p_j for the coefficient c (the inverse transform is
// unscaled, the pointwise product Montgomery), unless `prescaled`: then the
// product's last inverse pass read an inter-pass table multiplied by
// N^-1 2^64 mod p_j, and the residues are c mod p_j (in [0, 2p_j)).
struct CrtConst {
  PrimeConst pc[kPrimes];
  ulonglong2 k0;            // N^-1 2^64                                         mod p0
  ulonglong2 k1a, k1b;      // N^-1 2^64 p0^-1, p0^-1                            mod p1
  ulonglong2 k2a, k2b, k2c; // N^-1 2^64 (p0p1)^-1, (p0p1)^-1, p1^-1            mod p2
  uint64_t p01_lo, p01_hi;  // p0 * p1
  uint32_t prescaled;
  uint32_t pad;
};

// Carry launch state: the finished-tile count and the tiles' published aggregates.
struct ScanState {
  unsigned *done;              // 0 before and after every launch (launches sharing it are ordered)
  unsigned long long *flags;   // one word per tile
  uint32_t epoch;              // distinguishes launches sharing `flags`
  int *err;                    // device error word
};

// Whether a truncated transform's outer pass of 2^logR rows can keep k
// sixteenths of them (16: all): its last round holds the top four row bits of
// a 4- or 8-bit pass in registers, three of a 7-bit one, two of a 6-bit one.
__host__ __device__ __forceinline__ constexpr bool truncation_ok(int logR, int k) {
  return k == 16 || (k >= 9 && k < 16 &&
                     (logR == 4 || logR == 8 || (logR == 7 && k % 2 == 0) || (logR == 6 && k == 12)));
}

// The 80-bit digit at bit 80 j of a vector from the three 32-bit words that hold
// it: word (5 j) / 2 and the next two, from bit 16 (odd j) or bit 0 (even j).
// Byte permutes instead of 64-bit shifts by a variable: 2^24 x 2^24 limbs 4583
// -> 4545 us, 2^24 x 2^16 1692 -> 1669.
__device__ __forceinline__ uint64_t digit80_words(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t odd,
                                                  const PrimeConst &pc) {
  const uint32_t sel = odd ? 0x5432u : 0x3210u;
  const uint64_t lo = __byte_perm(w0, w1, sel) | (static_cast<uint64_t>(__byte_perm(w1, w2, sel)) << 32);
  return reduce80(lo, __byte_perm(w2, 0u, odd ? 0x4432u : 0x4410u), pc);
}

// The same digit from its two 64-bit words, (5 j) / 4 and the next, for loads
// from global memory (selecting three words first and permuting was no faster).
__device__ __forceinline__ uint64_t digit80(uint64_t a, uint64_t b, uint32_t j, const PrimeConst &pc) {
  const uint32_t s = (j & 3u) << 4;  // bits of `a` below the digit
  return reduce80((a >> s) | ((b << 1) << (63 - s)), static_cast<uint32_t>(b >> s) & 0xffffu, pc);
}

// Coefficient j of an operand of nl limbs modulo p: limb j, or 80-bit digit j.
template <bool D80>
__device__ __forceinline__ uint64_t coefficient(const uint64_t *limbs, uint64_t nl, uint64_t j, const PrimeConst &pc) {
  if constexpr (D80) {
    const uint64_t w = (5 * j) >> 2;
    if (w >= nl) return 0;
    return digit80(limbs[w], w + 1 < nl ? limbs[w + 1] : 0, static_cast<uint32_t>(j), pc);
  } else {
    return j < nl ? reduce64(limbs[j], pc.p) : 0;
  }
}

// ---- dependent launches ----------------------------------------------------
//
// A product is a chain of kernels, each reading what the one before wrote.
// They are launched with programmatic stream serialization: a kernel is
// launched while the one before drains, sets up (barriers, twiddle tables)
// and waits in pdl_wait, which returns once the kernels before have completed
// and their writes are visible.  Every kernel launched by launch_dep calls
// pdl_wait before its first access to memory that another kernel writes or
// reads, and reads such memory (residues, spectra, operands) by plain, .cg or
// volatile loads: the read-only path (__ldg) is for memory that nothing writes
// while the kernel is resident, which here leaves the twiddle tables, and a
// load in asm that is not volatile may be moved above the wait.  A product of 2^13 points 31.8 -> 23.2 us, of 2^16 points 37.0 ->
// 28.0, a 2^20-limb square 261 -> 244, 2^24 x 2^24 limbs 5528 -> 5508, the
// 4096-pair batch 3545 -> 3438.  No kernel triggers its successor early
// (griddepcontrol.launch_dependents): CTAs that become resident beside a
// running kernel are spread badly over the SMs (2^16 points 43.6 us, 2^24 x
// 2^24 limbs 5650).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... K, class... A>
cudaError_t launch_dep(void (*kernel)(K...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const A &...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// Kernel launchers.
// Strided pass (hg_ntt_strided.cu): 4 <= logR <= 8, logT = 12.
cudaError_t launch_ntt_strided(const PassArgs &a, bool inverse, cudaStream_t st);
// Contiguous pass (hg_ntt_contig.cu), mode: 0 forward, 1 inverse, 2 product
// of operands 0 and 1, 3 square of operand 0, 4 product of operand 0 with a
// finished spectrum at data[1] that every product of the launch shares;
// logR == logT <= 12.
constexpr int kContigFwd = 0, kContigInv = 1, kContigMul = 2, kContigSqr = 3, kContigMulSpec = 4;
cudaError_t launch_ntt_contig(const PassArgs &a, int mode, cudaStream_t st);
cudaError_t launch_crt_carry(const uint64_t *res, uint64_t n, bool dig80, const CrtConst &cc, uint64_t *out, uint64_t nout,
                             const ScanState &ss, cudaStream_t st, uint64_t *tiles_used);
// Reconstruction + carry for nprod products of n residues per prime that
// start ws_stride words apart at res.
cudaError_t launch_crt_carry_batch(const uint64_t *res, uint64_t ws_stride, uint64_t n, bool dig80, const CrtConst &cc,
                                   const ProductDesc *batch, uint64_t nprod, const ScanState &ss, cudaStream_t st);
// Reconstruction + carry of a product computed in chunks: chunk k's
// residues ([3][2^logN], unscaled inverse) start k * ws_stride words past
// res and hold the product of limbs [k * chunk, (k + 1) * chunk) of the long
// operand with the short one; position i of the result sums chunk i / chunk
// at i % chunk and the chunk before it at i % chunk + chunk.  Writes
// out[0, nproc).  n residues per prime hold a chunk's product of at most
// 2 chunk coefficients; chunk (in coefficients) is a multiple of 8.
cudaError_t launch_crt_carry_chunks(const uint64_t *res, uint64_t ws_stride, uint64_t n, bool dig80, uint64_t chunk,
                                    uint64_t nchunks, const CrtConst &cc, uint64_t *out, uint64_t nproc,
                                    const ScanState &ss, cudaStream_t st, uint64_t *tiles_used);
// An operand of a signed sum: n limbs, `shift` whole limbs up.
struct SumOperand {
  const uint64_t *p;
  uint64_t n, shift;
  __host__ __device__ __forceinline__ uint64_t end() const { return n ? n + shift : 0; }
  __device__ __forceinline__ uint64_t at(uint64_t i) const { return i - shift < n ? p[i - shift] : 0; }  // i < shift wraps
};

// Search words of a long sum, in device memory: -1, -1 and 0 before and after
// every sum (sums that share them are ordered).
struct SumWords {
  long long top_diff;  // highest limb where the operands differ
  long long top_out;   // highest nonzero limb of the result
  unsigned done;
};
// sa |a| + sb |b| into out[0, n + 1) (n = the longer operand's end; out[0, n)
// when the signs differ) over the whole GPU, with the carry scan of the products;
// result = (sign, size).
cudaError_t launch_large_sum(const SumOperand &a, int64_t sa, const SumOperand &b, int64_t sb, uint64_t *out,
                             SumWords *words, int64_t *result, const ScanState &ss, cudaStream_t st);
// Zero out[N, nout) of every product (out[0, nout) when N == 0), N the
// residues per prime.
cudaError_t launch_zero_tails(const ProductDesc *batch, uint64_t nprod, uint64_t N, cudaStream_t st);
// Schoolboy products of up to kSchoolMax limbs read every operand limb once.
constexpr uint32_t kSchoolMax = 1024;
cudaError_t launch_schoolboy_carry(const uint64_t *x, uint64_t nx, const uint64_t *y, uint64_t ny, uint64_t *out,
                                   uint64_t nout, const ScanState &ss, cudaStream_t st, uint64_t *tiles_used);
cudaError_t launch_digit_carry(const uint64_t *x, uint64_t nx, uint64_t d, uint64_t *out, uint64_t nout,
                               const ScanState &ss, cudaStream_t st, uint64_t *tiles_used);
// Fill out[j * M + r * S + s] = w_M^(+-s * bitrev_R(r)) (Montgomery form) for
// the primes j = 0 .. nprimes - 1 of tb, M = 2^logM, R = 2^logR, S = M / R.
cudaError_t launch_pass_twiddles(uint64_t *out, int logM, int logR, bool inverse, const NttTables *tb,
                                 const PrimeConst *pc, int nprimes, cudaStream_t st, const uint64_t *scale = nullptr);

// Coefficients of the smallest tile of a carry (short launches).
constexpr uint64_t kCarryMinTile = 1024;
// Tiles per product that a carry over nprod products of n coefficients uses,
// and whether it is one launch (short) or two.
uint64_t carry_tiles(uint64_t n, uint64_t nprod = 1);
bool carry_short(uint64_t n, uint64_t nprod = 1);
// Coefficients that n limbs hold, and limbs that n coefficients (a multiple of 4) fill.
__host__ __device__ __forceinline__ constexpr uint64_t coefs_of(uint64_t n, bool dig80) {
  return dig80 ? n - n / 5 : n;  // ceil(4 n / 5)
}
__host__ __device__ __forceinline__ constexpr uint64_t limbs_of(uint64_t n, bool dig80) {
  return dig80 ? n + n / 4 : n;
}

#if HG_CHECKED
// The fault word of each translation unit with kernels (checked builds),
// read and cleared: 0, a DevErr code, or -1 when the read failed.
int checked_fault_strided();
int checked_fault_contig();
int checked_fault_crt();
int checked_fault_persist();
int checked_fault_peak();
int checked_fault_sum();
int checked_fault_series();
#endif

// ---- one persistent launch for a batch (hg_persist.cu) --------------------
//
// A phase is one launch of the per-pass schedule; each of its items covers
// `per` consecutive units (CTAs of that launch).  Items of a phase with
// dep >= 0 start once phase dep has counted all its items done.
enum PersistKind : int {
  kPhaseZero = 0,     // out[n, nout) of products batch[0, count) (all of out when n == 0)
  kPhaseStrided = 1,  // sel = logR | inverse << 4
  kPhaseContig = 2,   // sel = T | mode << 4 (kContigMul or kContigSqr); item = by * gx + bx
  kPhaseTiny = 3,     // sel = mode; 256 (product, prime) pairs per item
  kPhaseCarry = 4,    // one carry tile of the persistent kernel per item
  kPhaseFix = 5,      // eight carry tiles per item, one per warp
};

struct PersistPhase {
  int kind, sel, dep, pad;
  uint64_t first, count, gx;
  uint64_t units, per;  // the launch's CTAs (warps for kPhaseFix, 256-pair groups for kPhaseTiny); per item
  PassArgs a;
  // reconstruction, carry and zeroing
  const uint64_t *res;
  uint64_t n, ws_stride, tpp, tiles;
  CrtConst cc;
  const ProductDesc *batch;
  ScanState ss;
};

constexpr int kPersistMaxPhases = 512;
constexpr size_t kPersistSmemBytes = 2 * (size_t(1) << kTileBits) * sizeof(uint64_t);

// The work counter, the abort word and one completion count per phase.
struct PersistState {
  unsigned long long next;
  unsigned abort, pad;
  unsigned done[1];
};
__host__ __device__ constexpr size_t persist_state_bytes(int nphases) {
  return sizeof(PersistState) + sizeof(unsigned) * static_cast<size_t>(nphases);
}

// CTAs of the persistent grid (SMs x resident CTAs per SM), 0 if unavailable.
int persist_grid();
// Carry tiles of the persistent kernel over n positions.
uint64_t persist_carry_tiles(uint64_t n);
// Clear the state and launch; phases and state are device memory.
cudaError_t launch_persist(const PersistPhase *phases, int nphases, uint64_t total, PersistState *state, int *err,
                           cudaStream_t st);

}  // namespace hg
