// Mixed-precision Lloyd step on the sm_103a tensor cores (tcgen05 + TMEM).
//
// The assignment needs, for each sample x and centroid c_j, the reference's
// pseudo-distance D_j = half_norm[j] - x.c_j (src/device_functions.hpp:
// 106-162).  Here the score s_j = sigma^2 (x.c_j - hn_j) is produced entirely
// by the tensor cores: the contraction over the features runs with fp16 (or
// bf16) operands and fp32 accumulation, and one more K=16 MMA per chunk adds
// -hn_j, split into three 16-bit parts against constant columns
// (-2^10, -1, -2^-10), so TMEM holds finished scores.  For every sample the
// epilogue finds the best score M and an exact bound on the runner-up R
// without sorting (see "runner-up" below).  A sample whose margin M - R
// exceeds twice its error bound E_i is certified: no rounding of the
// operands, of the tensor-core accumulation or of the reference's own fp32
// evaluation can change its winner, so its label equals the reference's.
// Every other sample is re-evaluated in exact fp32 reference arithmetic over
// the few centroids that can still win (recheck kernel), so labels never
// drift from the plain form.
//
// Error bound (unscaled units; operands scaled by a global power of two
// sigma and rounded to 16 bits: sigma x + dX_i and sigma c_j + dC_j, where the
// rounding errors dX_i, dC_j are exact in fp32 and measured, subnormals
// included; u = 2^-11 for fp16, 2^-8 for bf16; d features):
//   E_i = ||x_i|| alpha + ||dX_i|| / sigma beta1 + beta0
//   alpha = dCmax + 2^-16 (Cmax + dCmax) + (d + 4) 2^-23 Cmax
//   beta1 = (Cmax + dCmax)(1 + 2^-16)
//   beta0 = Hmax (u^3 + 2^-16 + 2^-23) + hfloor
// with Cmax = max_j ||c_j||, dCmax = max_j ||dC_j|| / sigma, Hmax = max_j
// |hn_j|.  By Cauchy-Schwarz |(sigma x + dX).(sigma c + dC) - sigma^2 x.c| <=
// ||dX|| (||sigma c|| + ||dC||) + ||sigma x|| ||dC||: the measured rounding
// errors (about 0.4 u ||.|| for random data) replace the worst case u ||.||
// of each operand.  The bound also covers the three-part split of the half
// norms (u^3, plus subnormal parts hfloor), tensor-core fp32 accumulation
// (<= 2^-17 relative to the sum of magnitudes, allowing truncation), and the
// reference's sequential fp32 dot (d 2^-24) and final subtraction; for bf16,
// whose subnormal inputs the tensor cores may flush, 2^-126 sqrt(d) (1 + u)
// is added to alpha and that times Cmax to beta0.  All norms are rounded up.
// sigma keeps |x sigma| <= 2^14 and sigma^2 * hn <= 2^25 so every 16-bit part
// is finite.
//
// Runner-up without sorting: per sample, P1[s] = max over 32-column
// sub-chunk s and P2[t] = max over columns j = t (mod 32).  Two distinct
// columns in the same sub-chunk lie in different classes, so
//   runner-up = max(second largest P1, second largest P2),
// and the winner is (argmax P1) * 32 + argmax P2 whenever the maximum is
// unique (otherwise the margin is zero and the sample is rechecked).  P1 comes
// with the scores (tcgen05.ld.red returns the maximum of the columns it loads),
// which leaves half a three-input max per score for P2.  Padding columns score
// -inf (their half norm), so no score needs a test against k.  A pass without
// sums over 4M x 64: 560 -> 454 us at k = 1024, 443 -> 211 us at k = 64.
//
// Kernel roles (one CTA of 320 threads per SM, persistent over 128-sample
// tiles, 168 registers per thread at most):
//   warp 0      bulk copies: the centroid image once, X tiles into a 2-4 stage ring
//   warp 1      TMEM allocation; one thread issues tcgen05.mma (M=128, N=256,
//               K=16) into two 256-column TMEM accumulators
//   warps 2-9   epilogue: tcgen05.ld of scores, P1/P2, certification, labels (two
//               threads per row; tiles of one chunk: two groups, a thread per row)
// The recheck kernel labels the samples that were not certified; the cluster
// sums are a pass of their own over the labels (sum_sorted_kernel).
// A pass without sums over 4M x 64 (before, two warps that added the sums ran
// beside the epilogue): 454 -> 416 us at k = 1024, 217 -> 177 us at k = 256, 211 -> 159 us at k = 64
// (146 and 145 with the two groups).
//
// Every wait is bounded.  A wait that runs out raises the CTA's error flag;
// the other roles see it and stop, the producer and the MMA issuer then wait
// (ignoring the flag) for the copies and tensor-core operations they already
// issued, TMEM is freed, and the fit's loop state records the error and stops
// the loop, so the host gets KMC_ERR_DEVICE_TIMEOUT and the context stays
// usable.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "km_batch.cuh"
#include "km_dist.cuh"
#include "km_fit.cuh"
#include "km_mixed.cuh"
#include "km_step.cuh"

namespace kmc {

namespace {

using namespace tc;

constexpr int kTileM = 128;
constexpr int kChunkN = 256;
constexpr uint32_t kNormRowBytes = 32;  // K=16 block holding the half-norm parts
constexpr int kEpiWarps = 8;
constexpr int kThreadsMixed = 32 * (2 + kEpiWarps);
constexpr uint32_t kTileBytes = kTileM * 128;  // one 64-wide K block of a tile
constexpr size_t kSmemLimit = 232448;

struct MixedConsts {
    float s2;       // sigma^2 (scores in TMEM are sigma^2 (x.c - hn))
    float alpha;    // E_i = nx_i * alpha + ndx_i * beta1 + beta0
    float beta1;
    float beta0;
    float sigma;
    unsigned int xmax_bits;  // max |x| (fp32 bits)
    int overflow;            // an operand left the 16-bit range this pass
    unsigned int wmax_bits;  // max |w| (fp32 bits; fixed-point sums only)
    int fx_shift;            // w x and w are summed as the integers w x 2^fx_shift, w 2^fx_shift
    int fx_ok;               // the fixed-point sums may be used (finite bounds)
    // per pass, cleared by the preparation's last CTA
    int acc_dirty;                  // fixed-point fits: a term went to the float64 copies
    unsigned prep_ticket;
    unsigned hmax_bits;             // max |hn_j| (fp32 bits)
    unsigned long long c2max_bits;  // max ||c_j||^2, max of its operands' rounding
    unsigned long long dc2max_bits; // errors' squared norms, scaled (fp64 bits)
};

// Order-independent totals of the fixed-point sums (d <= 32): element e
// (cluster-major [k][d4] sums, then the k sizes) of copy c is sum[c stride + e];
// CTA b adds into copy b mod copies, which spreads the contention, and the
// scale keeps every copy below 2^61.  The copies are added as integers too, so
// every order gives the same bits.  xq: the packed terms ([n][d4 + 4]); null
// when not in use.
struct FxAcc {
    const int *xq;
    unsigned long long *sum;
    int64_t stride;  // elements per copy
    int copies;
    int *dirty;      // set when a term went to the float64 copies instead
};

struct MixedArgs {
    const uint8_t *ximg;
    const uint8_t *cimg;
    const float *nx;
    const float *ndx;   // ||operand rounding error of x_i|| / sigma, rounded up
    const MixedConsts *consts;
    void *labels;
    uint4 *cand;
    int *flagged;
    int *n_flagged;
    int *err_global;
    const LoopState *guard;
    int64_t n;
    int label64;
    int stages;        // depth of the X-tile ring
    long long wait_limit;  // SM clocks after which a wait gives up
    int stall;         // test of the timeout path: the epilogue first waits on a
                       // barrier that nothing completes
    LoopState *state;  // receives the error bit and stops the loop (nullable)
    // Column passes (n_clusters beyond what one launch holds in shared
    // memory): this launch covers columns col0 .. col0 + NCH*256 - 1 of a
    // global centroid image of k_img rows.  With column passes it writes, per
    // sample, its best score of the pass (pmax) and full candidate masks of
    // the pass (cand) instead of labels; a combine kernel decides.
    int64_t k_img, col0;
    float *pmax;
    int last_k;  // 16-feature steps of the last feature block (the rest is zero)
};

struct SmemLayout {
    size_t c, hnb, aon, x, xch, bar, total;
};

// c:    centroid image, NKB blocks of k_pad x 128 bytes (128-byte swizzle)
// hnb:  half-norm parts, k_pad x 32 bytes (32-byte swizzle); c and hnb are
//       one contiguous copy of the global centroid image
// aon:  constant A block (128 x 32 bytes): columns 0..2 = -2^10, -1, -2^-10
// x:    X-tile ring (stages x NKB x 16 KB)
// xch:  per-row maxima of the two column halves (two tiles in flight)
__host__ __device__ inline SmemLayout smem_layout(int nkb, int64_t k_pad, int stages) {
    SmemLayout L;
    size_t off = 0;
    L.c = off;
    off += (size_t)nkb * k_pad * 128;
    L.hnb = off;
    off += (size_t)k_pad * kNormRowBytes;
    off = (off + 1023) & ~size_t(1023);
    L.aon = off;
    off += (size_t)kTileM * kNormRowBytes;
    off = (off + 1023) & ~size_t(1023);
    L.x = off;
    off += (size_t)stages * nkb * kTileBytes;
    L.xch = off;
    off += sizeof(float) * 2 * 2 * kTileM;
    L.bar = off;
    off += 8 * 15 + 8;
    L.total = off + 1024;  // slack for aligning the dynamic shared memory base
    return L;
}

// Bytes of the global centroid image (128-byte-swizzled blocks + norm parts).
__host__ __device__ inline size_t cimg_bytes(int nkb, int64_t k_pad) {
    return (size_t)nkb * k_pad * 128 + (size_t)k_pad * kNormRowBytes;
}

__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ float u2f(uint32_t v) { return __uint_as_float(v); }

// tcgen05.ld writes its registers asynchronously; after tcgen05.wait::ld the
// empty asm statements (ordered after the wait like every volatile asm) make
// each later use of the registers depend on the wait.
__device__ __forceinline__ void tmem_ld_wait_regs(uint32_t (&r0)[32], uint32_t (&r1)[32],
                                                  uint32_t (&r2)[32], uint32_t (&r3)[32],
                                                  uint32_t (&m)[4]) {
    tmem_ld_wait();
#pragma unroll
    for (int t = 0; t < 4; ++t) asm volatile("" : "+r"(m[t]));
#pragma unroll
    for (int t = 0; t < 32; ++t)
        asm volatile("" : "+r"(r0[t]), "+r"(r1[t]), "+r"(r2[t]), "+r"(r3[t]));
}

// The test v >= thr as a fused multiply-add with saturation, which runs on
// the FMA pipe instead of the ALU pipe the compares and selects use.  thrp is
// the float just below thr and K = 2 / ulp(thrp), a power of two: for every
// float v > thrp (equivalently v >= thr), v - thrp >= ulp(thrp) / 2 (v lies
// in thrp's binade or above, or at most one binade below it, where floats are
// spaced ulp(thrp) / 2), so the exact K (v - thrp) is >= 1 and saturates to
// exactly 1; for v <= thrp it is <= 0 and saturates to 0 (a NaN score also
// gives 0, as a NaN compare is false).  thrp K is exact.  Products that
// overflow give +-inf, which saturate to the right side as well.  Thresholds
// whose neighbour's exponent is too small for K to be finite (|thr| below
// about 2^-88), zero, infinite or NaN thresholds take the compare path.
struct HotTest {
    float K, nK;
    bool ok;
    __device__ __forceinline__ float hot(float v) const { return __saturatef(fmaf(v, K, nK)); }
};

__device__ __forceinline__ HotTest hot_test(float thr) {
    HotTest h;
    const uint32_t b = __float_as_uint(thr);
    const uint32_t e = (b >> 23) & 0xffu;
    h.ok = e >= 40u && e < 255u;
    // the float just below thr (|thr| >= 2^-87 here, so it is normal)
    const uint32_t pb = (b & 0x80000000u) ? b + 1u : b - 1u;
    const uint32_t ep = (pb >> 23) & 0xffu;
    h.K = __uint_as_float(h.ok ? (278u - ep) << 23 : 0x3f800000u);  // 2^(151 - ep)
    h.nK = -__uint_as_float(pb) * h.K;
    return h;
}

// OR over the 64 epilogue threads of TMEM lane quadrant q (the two warps that
// scan the two column halves of the same rows), named barrier 8 + q.  Only
// these two warps exchange data, so the other quadrants are not held back.
__device__ __forceinline__ bool pair_any(bool v, int q) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.red.or.pred q, %2, 64, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(8 + q)
        : "memory");
    return r != 0;
}

// 2^e as a float (e in [-126, 127]).
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }

// Packed fixed-point term of a float v = +-m 2^(E - 150) (E its exponent
// field, m its 24-bit mantissa) at scale 2^s, emin = 150 - s: when
// 0 <= E - emin <= 30, v 2^s = +-m 2^(E - emin) is an integer, stored as
// (+-m) << 6 | (E - emin) << 1; zero is 0; every other v (below the scale's
// resolution, denormal, infinite, NaN; the field 255 lies more than 30 above
// any emin <= 224) is the flag 1, which adds nothing.
__host__ __device__ inline int pack_fixed(float v, int emin) {
    uint32_t b;
    memcpy(&b, &v, 4);
    if ((b & 0x7fffffffu) == 0u) return 0;
    const uint32_t sh = (uint32_t)((int)((b >> 23) & 0xffu) - emin);
    if (sh > 30u) return 1;
    const int m = (int)((b & 0x7fffffu) | 0x800000u);
    const int ms = (b >> 31) ? -m : m;
    return (int)(((uint32_t)ms << 6) | (sh << 1));
}

template <int BF16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    if (BF16) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    } else {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    }
}

// Constant columns of the half-norm block: the score receives
// -(c0 h0 + c1 h1 + c2 h2) with (h0, h1, h2) the 16-bit parts of sigma^2 hn.
__host__ __device__ constexpr float norm_coef(int bf16, int part) {
    return bf16 ? -1.f : (part == 0 ? -1024.f : (part == 1 ? -1.f : -0x1p-10f));
}

template <int BF16, int NKB, int NCH, bool MULTI>
__global__ void __launch_bounds__(kThreadsMixed, 1) mixed_assign_kernel(MixedArgs a) {
    wait_for_previous();
    if (a.guard != nullptr && *reinterpret_cast<const volatile int *>(&a.guard->done)) return;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // the swizzles are functions of absolute shared-memory address bits, so
    // every operand image starts on a 1024-byte boundary
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int64_t k_pad = (int64_t)NCH * kChunkN;
    const int stages = a.stages;
    const SmemLayout L = smem_layout(NKB, k_pad, stages);
    uint8_t *cimg_s = smem + L.c;
    uint8_t *aon_s = smem + L.aon;
    uint8_t *xring = smem + L.x;
    float *xch = reinterpret_cast<float *>(smem + L.xch);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar);
    uint64_t *full = bars, *empty = bars + 4, *tfull = bars + 8, *tempty = bars + 10;
    uint64_t *cbar = bars + 12, *tdone = bars + 13;
    uint64_t *never = bars + 14;  // completed by no role (timeout test only)
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 15);
    volatile int *err = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n = a.n;
    const long long lim = a.wait_limit;
    const int64_t ntiles = ceil_div<int64_t>(n, kTileM);
    const uint32_t cbytes = (uint32_t)cimg_bytes(NKB, k_pad);

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            // one chunk: an accumulator belongs to a group of four warps
            mbar_init(&tempty[b], NCH == 1 ? 16 * kEpiWarps : 32 * kEpiWarps);
        }
        mbar_init(cbar, 1);
        mbar_init(tdone, 1);
        mbar_init(never, 1);
        *err = 0;
        fence_barrier_init();
    }
    // constant A block of the half-norm MMA: row r = (c0, c1, c2, 0, ..., 0)
    for (int t = threadIdx.x; t < 2 * kTileM; t += blockDim.x) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if ((t & 1) == 0) {
            v.x = pack2<BF16>(norm_coef(BF16, 0), norm_coef(BF16, 1));
            v.y = pack2<BF16>(norm_coef(BF16, 2), 0.f);
        }
        *reinterpret_cast<uint4 *>(aon_s + sw32_offset((uint32_t)(t >> 1), (uint32_t)(t & 1) * 8)) = v;
    }
    fence_proxy_async();  // generic-proxy writes -> tensor-core operand reads
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const MixedConsts cst = *a.consts;

    if (warp == 0) {
        // ------------------------------ producer ------------------------------
        if (lane == 0) {
            mbar_arrive_expect_tx(cbar, cbytes);
            // rows col0 .. col0 + k_pad - 1 of every feature block and of the
            // half-norm block of the global image
            for (int kb = 0; kb <= NKB; ++kb) {
                const uint32_t row = kb < NKB ? 128u : kNormRowBytes;
                const uint32_t bytes = (uint32_t)k_pad * row;
                const uint8_t *src = a.cimg + (size_t)kb * a.k_img * 128 + (size_t)a.col0 * row;
                uint8_t *dst = cimg_s + (size_t)kb * k_pad * 128;
                for (uint32_t off = 0; off < bytes; off += 32768u)
                    bulk_g2s(dst + off, src + off, min(32768u, bytes - off), cbar);
            }
            int s = 0;
            uint32_t ph = 0, issued = 0u, last_ph = 0u;
            for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                if (!mbar_wait(&empty[s], ph ^ 1u, err, lim)) break;
                mbar_arrive_expect_tx(&full[s], NKB * kTileBytes);
                bulk_g2s(xring + (size_t)s * NKB * kTileBytes,
                         a.ximg + (size_t)tile * NKB * kTileBytes, NKB * kTileBytes, &full[s]);
                issued |= 1u << s;
                last_ph = (last_ph & ~(1u << s)) | (ph << s);
                if (++s == stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // never leave a copy in flight into this CTA's shared memory: the
            // centroid image and the last copy into each ring stage (a stage
            // holds at most one copy in flight) are waited for even after an
            // error
            mbar_wait_drain(cbar, 0, err);
            for (int q = 0; q < stages; ++q)
                if ((issued >> q) & 1u) mbar_wait_drain(&full[q], (last_ph >> q) & 1u, err);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ----------------------------
        if (lane == 0) {
            const uint32_t idesc = idesc_f16(BF16, kTileM, kChunkN);
            const uint32_t cbase = smem_u32(cimg_s);
            const uint32_t hbase = cbase + (uint32_t)(NKB * k_pad * 128);
            const uint64_t adesc_norm = desc_sw32(smem_u32(aon_s));
            const int last_k = a.last_k;
            bool ok = mbar_wait(cbar, 0, err, lim);
            int s = 0;
            uint32_t ph = 0, cnt = 0;
            for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
                if (!mbar_wait(&full[s], ph, err, lim)) break;
                tc_fence_after();
                const uint32_t xbase = smem_u32(xring + (size_t)s * NKB * kTileBytes);
                for (int c = 0; c < NCH; ++c) {
                    const uint32_t b = cnt & 1u, bph = (cnt >> 1) & 1u;
                    if (!mbar_wait(&tempty[b], bph ^ 1u, err, lim)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t dt = tmem + b * kChunkN;
#pragma unroll
                    for (int kb = 0; kb < NKB; ++kb)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            // steps of padding would add zeros (2M x 32, k = 1000:
                            // 216 -> 200 us; 4M x 16, 100: 153 -> 144)
                            if (kb == NKB - 1 && kk > 0 && kk >= last_k) continue;
                            const uint64_t ad = desc_sw128(xbase + kb * kTileBytes + kk * 32);
                            const uint64_t bd = desc_sw128(cbase + (uint32_t)(kb * k_pad * 128) +
                                                           (uint32_t)(c * kChunkN * 128) + kk * 32);
                            mma_f16(dt, ad, bd, idesc, (kb | kk) != 0 ? 1u : 0u);
                        }
                    // - sigma^2 hn_j for the 256 columns of this chunk
                    mma_f16(dt, adesc_norm,
                            desc_sw32(hbase + (uint32_t)(c * kChunkN) * kNormRowBytes), idesc, 1u);
                    mma_commit(&tfull[b]);
                    ++cnt;
                }
                mma_commit(&empty[s]);
                if (++s == stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // all issued MMAs must have finished before TMEM is released,
            // error or not
            mma_commit(tdone);
            mbar_wait_drain(tdone, 0, err);
        }
        __syncwarp();
    } else if constexpr (NCH == 1) {
        // ---------------------- epilogue, one chunk per tile -------------------
        // Two groups of four warps take tiles in turn, each with an accumulator
        // of its own; a thread scans a whole row, so nothing is exchanged, and
        // one group's loads and masks run beside the other's (a chunk's chain of
        // load, exchange, masks and labels bounded the tile: 4M x 64, k = 64
        // 159 -> 144 us, k = 256 177 -> 153; 16 and 100 163 -> 153).  With more chunks the scans are as
        // long as the tensor cores' work and two accumulators per tile hide
        // more.
        constexpr int kSub = 8;
        const int ew = warp - 2, g = ew >> 2;
        const int q = warp & 3;   // TMEM lane quadrant accessible to this warp
        const int row = 32 * q + lane;
        const uint32_t cb = tmem + ((uint32_t)(32 * q) << 16) + g * kChunkN;
        // test of the timeout path: this wait runs out after `lim` clocks
        if (a.stall) mbar_wait(never, 0, err, lim);
        const int64_t step = 2 * (int64_t)gridDim.x;
        // per-sample norms of the next tile are loaded one tile ahead
        float nx_next = 0.f, dx_next = 0.f;
        auto load_norms = [&](int64_t tile) {
            const int64_t i = tile * kTileM + row;
            if (i < n) {
                nx_next = a.nx[i];
                dx_next = a.ndx[i];
            }
        };
        const int64_t first = blockIdx.x + (int64_t)g * gridDim.x;
        load_norms(first);
        uint32_t phase = 0;
        for (int64_t tile = first; tile < ntiles; tile += step, phase ^= 1u) {
            const int64_t i = tile * kTileM + row;
            const float e = fmaf(nx_next, cst.alpha, fmaf(dx_next, cst.beta1, cst.beta0));
            const float E2 = i < n ? 2.f * e * 1.000001f : 0.f;
            load_norms(tile + step);
            const bool bad = !mbar_wait(&tfull[g], phase, err, lim);
            // tcgen05.ld is warp-collective: re-converge after the wait
            if (__any_sync(0xffffffffu, bad || *err != 0)) break;
            tc_fence_after();
            float P2[32], P1[kSub];
            {
                uint32_t ra[32], rb[32], rc[32], rd[32], m[4];
                tmem_ld32_max(cb, ra, m[0]);
                tmem_ld32_max(cb + 32, rb, m[1]);
                tmem_ld32_max(cb + 64, rc, m[2]);
                tmem_ld32_max(cb + 96, rd, m[3]);
                tmem_ld_wait_regs(ra, rb, rc, rd, m);
#pragma unroll
                for (int t = 0; t < 32; ++t)
                    P2[t] = max3f(fmaxf(u2f(ra[t]), u2f(rb[t])), u2f(rc[t]), u2f(rd[t]));
#pragma unroll
                for (int t = 0; t < 4; ++t) P1[t] = u2f(m[t]);
                // the loads below reuse the registers: finish every read first
#pragma unroll
                for (int t = 0; t < 32; ++t) asm volatile("" : "+f"(P2[t]));
                tmem_ld32_max(cb + 128, ra, m[0]);
                tmem_ld32_max(cb + 160, rb, m[1]);
                tmem_ld32_max(cb + 192, rc, m[2]);
                tmem_ld32_max(cb + 224, rd, m[3]);
                tmem_ld_wait_regs(ra, rb, rc, rd, m);
                tc_fence_before();
                mbar_arrive(&tempty[g]);  // the accumulator may be overwritten now
#pragma unroll
                for (int t = 0; t < 32; ++t)
                    P2[t] = max3f(max3f(P2[t], u2f(ra[t]), u2f(rb[t])), u2f(rc[t]), u2f(rd[t]));
#pragma unroll
                for (int t = 0; t < 4; ++t) P1[4 + t] = u2f(m[t]);
            }
            float M = -pos_inf<float>();
#pragma unroll
            for (int t = 0; t < kSub; ++t) M = fmaxf(M, P1[t]);
            // as in the other form: columns that reach thr can win; two distinct
            // ones differ in their sub-chunk or in their class
            const float thr = M - E2;
            uint32_t hot1 = 0u, hot2 = 0u;
            const HotTest ht = hot_test(thr);
            if (ht.ok) {
                float l1 = 0.f, l2 = 0.f, h2 = 0.f;
#pragma unroll
                for (int t = 0; t < kSub; ++t) l1 = fmaf(ht.hot(P1[t]), (float)(1u << t), l1);
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    l2 = fmaf(ht.hot(P2[t]), (float)(1u << t), l2);
                    h2 = fmaf(ht.hot(P2[16 + t]), (float)(1u << t), h2);
                }
                hot1 = __float2uint_rz(l1);
                hot2 = __float2uint_rz(l2) | (__float2uint_rz(h2) << 16);
            } else {
#pragma unroll
                for (int t = 0; t < kSub; ++t) hot1 |= (P1[t] >= thr) ? (1u << t) : 0u;
#pragma unroll
                for (int t = 0; t < 32; ++t) hot2 |= (P2[t] >= thr) ? (1u << t) : 0u;
            }
            if (!(thr == thr)) {  // cannot happen with finite operands; recheck all
                hot1 = 0xffu;
                hot2 = ~0u;
            }
            if (i >= n) continue;
            const bool sure = __popc(hot1) == 1 && __popc(hot2) == 1;
            if (MULTI || !sure) {
                // by column halves, the classes of a row in both
                const uint32_t lo = hot1 & 15u, hi = hot1 >> 4;
                a.cand[i] = make_uint4(lo, hi, lo ? hot2 : 0u, hi ? hot2 : 0u);
            }
            if (MULTI) {
                a.pmax[i] = M;  // decided by the combine
            } else if (sure) {
                const int code = (__ffs(hot1) - 1) * 32 + __ffs(hot2) - 1;
                if (a.label64)
                    reinterpret_cast<int64_t *>(a.labels)[i] = code;
                else
                    reinterpret_cast<int32_t *>(a.labels)[i] = code;
            } else {
                const int pos = atomicAdd(a.n_flagged, 1);
                if (pos >= 0 && pos < n) a.flagged[pos] = (int)i;
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        // Thread (row, h) scans columns h*128 .. h*128+127 of every chunk for
        // tile row `row`: P2[t] = max over its columns j = t (mod 32), P1[s] =
        // max over its 32-column sub-chunk s (4 per chunk).
        constexpr int kSub = 4 * NCH;
        constexpr uint32_t kAll1 = (kSub == 32) ? ~0u : ((1u << kSub) - 1u);
        const int ew = warp - 2;
        const int q = warp & 3;   // TMEM lane quadrant accessible to this warp
        const int h = ew >> 2;    // column half of each 256-wide chunk
        const int row = 32 * q + lane;
        const uint32_t lane_addr = (uint32_t)(32 * q) << 16;
        uint32_t cnt = 0;
        int tl = 0;
        // test of the timeout path: this wait runs out after `lim` clocks
        if (a.stall) mbar_wait(never, 0, err, lim);
        // per-sample norms of the next tile are loaded one tile ahead
        float nx_next = 0.f, dx_next = 0.f;
        {
            const int64_t i0 = (int64_t)blockIdx.x * kTileM + row;
            if (i0 < n) {
                nx_next = a.nx[i0];
                dx_next = a.ndx[i0];
            }
        }
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++tl) {
            const int64_t i = tile * kTileM + row;
            float E2 = 0.f;
            if (i < n) {
                const float e = fmaf(nx_next, cst.alpha, fmaf(dx_next, cst.beta1, cst.beta0));
                E2 = 2.f * e * 1.000001f;
            }
            {
                const int64_t inext = (tile + gridDim.x) * kTileM + row;
                if (inext < n) {
                    nx_next = a.nx[inext];
                    dx_next = a.ndx[inext];
                }
            }
            float P2[32], P1[kSub];
            float Mh = -pos_inf<float>();
#pragma unroll
            for (int t = 0; t < 32; ++t) P2[t] = -pos_inf<float>();
            bool bad = false;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const uint32_t b = cnt & 1u, bph = (cnt >> 1) & 1u;
                if (!mbar_wait(&tfull[b], bph, err, lim)) bad = true;
                // tcgen05.ld is warp-collective: re-converge after the spin-wait
                if (__any_sync(0xffffffffu, bad)) {
                    bad = true;
                    break;
                }
                tc_fence_after();
                const uint32_t cb = tmem + lane_addr + b * kChunkN + h * 128;
                // all 128 columns into registers, so that the accumulator is free
                // again before they are looked at
                uint32_t ra[32], rb[32], rc[32], rd[32], m[4];
                tmem_ld32_max(cb, ra, m[0]);
                tmem_ld32_max(cb + 32, rb, m[1]);
                tmem_ld32_max(cb + 64, rc, m[2]);
                tmem_ld32_max(cb + 96, rd, m[3]);
                tmem_ld_wait_regs(ra, rb, rc, rd, m);
                tc_fence_before();
                mbar_arrive(&tempty[b]);  // the accumulator may be overwritten now
#pragma unroll
                for (int t = 0; t < 32; ++t)
                    P2[t] = max3f(max3f(P2[t], u2f(ra[t]), u2f(rb[t])), u2f(rc[t]), u2f(rd[t]));
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    P1[4 * c + t] = u2f(m[t]);
                    Mh = fmaxf(Mh, u2f(m[t]));
                }
                ++cnt;
            }

            // best score of this half, exchanged with the other half
            float *xb = xch + (size_t)(tl & 1) * (2 * kTileM);
            xb[h * kTileM + row] = Mh;
            // one pair barrier per tile: publishes the exchange and agrees on errors
            if (pair_any(bad || *err != 0, q)) break;
            const float Mo = xb[(h ^ 1) * kTileM + row];
            // Columns whose score reaches thr = M - E2 can hold the reference's
            // winner (every score is within E2 / 2 of its exact value).  The
            // winner is certified when exactly one column can: no column of
            // the other half reaches thr, and exactly one sub-chunk and one
            // class of the winning half do (two distinct columns of one
            // sub-chunk lie in distinct classes).
            const float thr = fmaxf(Mh, Mo) - E2;
            // exactly one of the pair wins, whatever the maxima (a NaN loses
            // every comparison: the first half then wins)
            const bool win = (Mh > Mo) || (h == 0 && !(Mo > Mh));
            uint32_t hot1 = 0u, hot2 = 0u;
            const HotTest ht = hot_test(thr);
            if (ht.ok) {
                // the masks on the FMA pipe: 0 / 1 per maximum, summed as
                // exact powers of two in two 16-bit float halves
                float l1 = 0.f, l2 = 0.f, h2 = 0.f;
#pragma unroll
                for (int t = 0; t < kSub; ++t) {
                    const float m = P1[t];
                    l1 = fmaf(ht.hot(m), (float)(1u << t), l1);
                }
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    l2 = fmaf(ht.hot(P2[t]), (float)(1u << t), l2);
                    h2 = fmaf(ht.hot(P2[16 + t]), (float)(1u << t), h2);
                }
                hot1 = __float2uint_rz(l1);
                hot2 = __float2uint_rz(l2) | (__float2uint_rz(h2) << 16);
            } else {
#pragma unroll
                for (int t = 0; t < kSub; ++t) {
                    const float m = P1[t];
                    hot1 |= (m >= thr) ? (1u << t) : 0u;
                }
#pragma unroll
                for (int t = 0; t < 32; ++t) hot2 |= (P2[t] >= thr) ? (1u << t) : 0u;
            }
            bool loser_hot = fminf(Mh, Mo) >= thr;
            if (!(thr == thr)) {  // cannot happen with finite operands; recheck all
                hot1 = kAll1;
                hot2 = ~0u;
                loser_hot = true;
            }
            if (MULTI && i < n) {
                // column pass: the pass's best score and both halves' masks
                // (single bits for a unique winner), decided by the combine
                uint32_t *cw = reinterpret_cast<uint32_t *>(a.cand + i);
                if (win) {
                    cw[h] = hot1;
                    cw[2 + h] = hot2;
                    if (!loser_hot) {
                        cw[h ^ 1] = 0u;
                        cw[2 + (h ^ 1)] = 0u;
                    }
                    a.pmax[i] = fmaxf(Mh, Mo);
                } else if (loser_hot) {
                    cw[h] = hot1;
                    cw[2 + h] = hot2;
                }
            } else if (i < n) {
                uint32_t *cw = reinterpret_cast<uint32_t *>(a.cand + i);
                if (win) {
                    if (!loser_hot && __popc(hot1) == 1 && __popc(hot2) == 1) {
                        const int sc = __ffs(hot1) - 1, t = __ffs(hot2) - 1;
                        const int code = (sc >> 2) * kChunkN + h * 128 + (sc & 3) * 32 + t;
                        if (a.label64)
                            reinterpret_cast<int64_t *>(a.labels)[i] = code;
                        else
                            reinterpret_cast<int32_t *>(a.labels)[i] = code;
                    } else {
                        cw[h] = hot1;
                        cw[2 + h] = hot2;
                        if (!loser_hot) {
                            cw[h ^ 1] = 0u;
                            cw[2 + (h ^ 1)] = 0u;
                        }
                        const int pos = atomicAdd(a.n_flagged, 1);
                        if (pos >= 0 && pos < n) a.flagged[pos] = (int)i;
                    }
                } else if (loser_hot) {
                    cw[h] = hot1;
                    cw[2 + h] = hot2;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && *err) {
        atomicExch(a.err_global, 1);
        if (a.state != nullptr) {
            // the remaining kernels of the iteration and the host loop stop
            atomicOr(&a.state->err, 1u);
            atomicExch(&a.state->done, 1);
        }
    }
}

// ---------------------------------------------------------------------------
// preparation kernels
// ---------------------------------------------------------------------------
// max |X[e]| (NaNs lose).  One atomic per CTA: one per warp of 4096 CTAs took 27
// us whatever the size (1M floats now 3 us; 640M floats 440 -> 367 us, 7.0 TB/s).
constexpr int kAbsmaxThreads = 256;
__global__ void __launch_bounds__(kAbsmaxThreads)
    absmax_kernel(const float *X, int64_t count, unsigned int *out_bits) {
    __shared__ float red[kAbsmaxThreads / 32];
    constexpr int kBatch = 4;
    const int64_t tid = blockIdx.x * (int64_t)kAbsmaxThreads + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kAbsmaxThreads;
    float m = 0.f;
    // whole float4s from the first 16-byte boundary on, the rest one by one
    const int64_t head = min(count, (int64_t)((16u - ((uint32_t)reinterpret_cast<uintptr_t>(X) & 15u)) & 15u) / 4);
    const int64_t vecs = (count - head) / 4;
    const float4 *V = reinterpret_cast<const float4 *>(X + head);
    for (int64_t e = tid; e < vecs; e += kBatch * step) {
        float4 v[kBatch];
#pragma unroll
        for (int t = 0; t < kBatch; ++t) v[t] = load_f4_if(V + e + t * step, e + t * step < vecs);
#pragma unroll
        for (int t = 0; t < kBatch; ++t)
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v[t].x), fabsf(v[t].y)), fmaxf(fabsf(v[t].z), fabsf(v[t].w))));
    }
    if (tid < head) m = fmaxf(m, fabsf(X[tid]));
    const int64_t rest = head + 4 * vecs + tid;
    if (rest < count) m = fmaxf(m, fabsf(X[rest]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < kAbsmaxThreads / 32; ++q) m = fmaxf(m, red[q]);
        atomicMax(out_bits, __float_as_uint(m));
    }
}

// fp16 operands: sigma is the largest power of two in [2^-60, 2^60] with
// max|x| sigma <= 2^14 and sigma^2 d max|x|^2 / 2 <= 2^25, so that every
// scaled sample, every scaled centroid inside the data's range and the
// largest part of sigma^2 hn stay finite in fp16 with room to spare.  bf16
// shares fp32's exponent range and is never scaled.
__global__ void sigma_kernel(MixedConsts *c, int bf16, int64_t d) {
    const double xmax = (double)__uint_as_float(c->xmax_bits);

    double sigma = 1.0;
    if (!bf16 && xmax > 0.0 && xmax < 1e300) {
        const double hx = 0.5 * (double)d * xmax * xmax;
        auto fits = [&](double s) { return xmax * s <= 0x1p14 && s * s * hx <= 0x1p25; };
        while (sigma < 0x1p60 && fits(sigma * 2.0)) sigma *= 2.0;
        while (sigma > 0x1p-60 && !fits(sigma)) sigma *= 0.5;
    }
    c->sigma = (float)sigma;
    c->s2 = (float)(sigma * sigma);
    c->overflow = 0;
}

// Shift of the fixed-point cluster sums: a copy adds up at most `rows` (>= 128)
// values w x per feature (|w x| <= max|x| max|w|) and `rows` weights, so with
// bound = rows max(max|x| max|w|, max|w|) < 2^e the shift 61 - e keeps every
// sum below 2^61 and every term below 2^54 (all-zero data gives 0).
__global__ void fixed_scale_kernel(MixedConsts *c, double rows) {
    const double xm = (double)__uint_as_float(c->xmax_bits);
    const double wm = (double)__uint_as_float(c->wmax_bits);
    auto shift_for = [](double bound) {
        int sh = 0;
        if (bound > 0.0 && bound < 1e300) {
            int e = 0;
            frexp(bound, &e);
            sh = min(100, 61 - e);
        }
        return sh;
    };
    const int sx = shift_for(rows * fmax(xm * wm, wm));
    // products w x that may overflow fp32, and scales whose resolution field
    // 150 - shift would come within 30 of the infinity / NaN field, keep the
    // float64 reductions
    c->fx_ok = (xm * wm < 1e37 && sx >= -70) ? 1 : 0;
    c->fx_shift = sx;
}

// Round to the 16-bit operand type and back (exact in fp32).
template <int BF16>
__device__ __forceinline__ float round16(float v) {
    if (BF16) return __bfloat162float(__float2bfloat16_rn(v));
    return __half2float(__float2half_rn(v));
}

// One-time conversion of X.  A CTA takes one 128-sample tile at a time (the image
// holds K blocks of 64 features, zero-padded, for every 128-sample
// tile): the tile's features are staged in shared memory (coalesced reads of
// each feature's 128 samples from a feature-major X, or of each sample's d
// features from a row-major one), then written out as the 128-byte-swizzled
// K-major image of (x * sigma) and the row-major fp32 copy of x (features
// d..d4-1 zero), both as contiguous 16-byte chunks, and per sample ||x|| and
// the norm of the image's rounding error ||round16(x sigma) - x sigma|| /
// sigma, both rounded up; with xq also the packed fixed-point terms (w x_j
// rounded as the reference forms it, then w, 0, 0, 0).
// Bound by memory.  10M x 64: 1.41 -> 1.29 ms (the norms had a loop of their own in
// half of the threads); 1M x 16 with packed terms, which had a kernel of their
// own: 139 -> 89 us.
constexpr int kXImageThreads = 256;
constexpr int kXsPitch = kTileM + 1;  // floats per staged feature (bank offset)

__host__ __device__ inline size_t x_image_smem(int nkb) {
    return sizeof(float) * (size_t)nkb * 64 * kXsPitch;
}

template <int BF16>
__global__ void __launch_bounds__(kXImageThreads) x_image_kernel(
    const float *X, int64_t n, int64_t d, int64_t d4, int nkb, int64_t ntiles,
    const MixedConsts *c, uint8_t *img, float *xrow, float *nx, float *ndx, int rowmajor,
    const float *w, int *xq) {
    extern __shared__ float xs[];  // [feature][kXsPitch]
    constexpr int kBatch = 8;
    constexpr int kRows = 4;  // rows of a thread in each feature block
    static_assert(kRows * kXImageThreads == kTileM * 8, "eight lanes per row");
    const float sigma = c->sigma;
    const int F = nkb * 64, tid = threadIdx.x;
    const int g4 = (int)(d4 / 4), emin = 150 - c->fx_shift;
    // the padding features stay zero
    for (int e = (int)d * kXsPitch + tid; e < F * kXsPitch; e += kXImageThreads) xs[e] = 0.f;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t i0 = tile * kTileM;
        const int rows_here = (n - i0 < (int64_t)kTileM) ? (int)(n - i0) : kTileM;
        const int total = (int)d * kTileM;
        for (int e0 = tid; e0 < total; e0 += kBatch * kXImageThreads) {
            float v[kBatch];
            int o[kBatch];
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                const int e = e0 + t * kXImageThreads;
                int f, r;
                if (rowmajor) {
                    r = e / (int)d;
                    f = e - r * (int)d;
                } else {
                    f = e >> 7;
                    r = e & (kTileM - 1);
                }
                o[t] = e < total ? f * kXsPitch + r : -1;
                const float *src = rowmajor ? X + (i0 + r) * d + f : X + (int64_t)f * n + i0 + r;
                v[t] = load_f_if(src, e < total && r < rows_here);
            }
#pragma unroll
            for (int t = 0; t < kBatch; ++t)
                if (o[t] >= 0) xs[o[t]] = v[t];
        }
        __syncthreads();
        // image: 16-byte chunk q of feature block kb holds row r, features
        // 8 ch .. 8 ch + 7 with ch = (q mod 8) xor (r mod 8) (128-byte swizzle);
        // the eight lanes of a row also sum its squares.  (An upper bound of
        // the norms needs no order: see below.)
        float s2[kRows] = {0.f, 0.f, 0.f, 0.f}, sd[kRows] = {0.f, 0.f, 0.f, 0.f};
        for (int kb = 0; kb < nkb; ++kb) {
#pragma unroll
            for (int t = 0; t < kRows; ++t) {
                const int qq = tid + t * kXImageThreads;
                const int r = (qq >> 6) * 8 + ((qq >> 3) & 7);
                const int ch = (qq & 7) ^ (r & 7);
                const float *src = xs + (kb * 64 + ch * 8) * kXsPitch + r;
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float x = src[e * kXsPitch];
                    s2[t] = __fmaf_rn(x, x, s2[t]);
                    v[e] = x * sigma;
                    const float dv = round16<BF16>(v[e]) - v[e];  // exact
                    sd[t] = __fmaf_rn(dv, dv, sd[t]);
                }
                uint4 pk;
                pk.x = pack2<BF16>(v[0], v[1]);
                pk.y = pack2<BF16>(v[2], v[3]);
                pk.z = pack2<BF16>(v[4], v[5]);
                pk.w = pack2<BF16>(v[6], v[7]);
                *reinterpret_cast<uint4 *>(img + ((size_t)tile * nkb + kb) * kTileBytes +
                                           (size_t)qq * 16) = pk;
            }
        }
#pragma unroll
        for (int t = 0; t < kRows; ++t) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                s2[t] += __shfl_xor_sync(0xffffffffu, s2[t], o);
                sd[t] += __shfl_xor_sync(0xffffffffu, sd[t], o);
            }
            const int qq = tid + t * kXImageThreads;
            const int r = (qq >> 6) * 8 + ((qq >> 3) & 7);
            if ((tid & 7) == 0 && r < rows_here) {
                // A float32 sum of m non-negative terms, in any order, is at
                // least (1 - 2^-24)^m times the exact sum (each term passes at
                // most m roundings); m <= 256 here, so the factor 1 + (m + 2)
                // 2^-23 applied with upward rounding (and an upward square
                // root) gives upper bounds of both norms (1 / sigma is a power
                // of two).
                const float grow = 1.f + (float)(nkb * 64 + 2) * 0x1p-23f;
                nx[i0 + r] = __fsqrt_ru(__fmul_ru(s2[t], grow));
                ndx[i0 + r] = __fmul_ru(__fsqrt_ru(__fmul_ru(sd[t], grow)), 1.f / sigma);
            }
        }
        // row-major fp32 rows: the tile's block of xrow is contiguous
        for (int e = tid; e < rows_here * g4; e += kXImageThreads) {
            const int r = e / g4, g = e - r * g4;
            const float *src = xs + (4 * g) * kXsPitch + r;
            reinterpret_cast<float4 *>(xrow + i0 * d4)[e] =
                make_float4(src[0], src[kXsPitch], src[2 * kXsPitch], src[3 * kXsPitch]);
        }
        if (xq != nullptr) {
            for (int e = tid; e < rows_here * (g4 + 1); e += kXImageThreads) {
                const int r = e / (g4 + 1), g = e - r * (g4 + 1);
                const float wi = w[i0 + r];
                const float *src = xs + (4 * g) * kXsPitch + r;
                int4 q = make_int4(pack_fixed(wi, emin), 0, 0, 0);
                if (g < g4)
                    q = make_int4(pack_fixed(__fmul_rn(src[0], wi), emin),
                                  pack_fixed(__fmul_rn(src[kXsPitch], wi), emin),
                                  pack_fixed(__fmul_rn(src[2 * kXsPitch], wi), emin),
                                  pack_fixed(__fmul_rn(src[3 * kXsPitch], wi), emin));
                reinterpret_cast<int4 *>(xq + i0 * (d4 + 4))[e] = q;
            }
        }
        __syncthreads();
    }
}

// Largest finite operand value: fp16 65504, bf16 (1 - 2^-8) 2^128.
template <int BF16>
__device__ __forceinline__ float max16() {
    return BF16 ? 3.3895313892515355e38f : 65504.f;
}

// Preparation of a pass: half norms (sequential fma over the features, as the
// reference's), the centroid image (rows j < k_pad, zero padding) with its
// half-norm block, the row-major fp32 centroids, the constants of the error
// bound, and a cleared recheck count.  Row j of the half-norm block holds
// (h0, h1, h2) with
//   c0 h0 + c1 h1 + c2 h2 = -sigma^2 hn_j   (c = norm_coef)
// up to sigma^2 |hn_j| u^3 (u = 2^-11 fp16, 2^-8 bf16; plus 2^-35 for fp16
// subnormal parts): h0 is the rounded leading part and each following part
// the rounded remainder, formed exactly in fp64.  A value that would leave the
// operand range is clamped and raises consts->overflow, which disables
// certification for the pass (every sample is then re-evaluated exactly).
//
// One launch instead of five (half norms, image, bound constants and two
// resets: 27 us at k = 1024, all latency): a CTA takes the 8 rows of one
// swizzle atom, G = 8 nkb (rounded up to a power of two) lanes per row, lane
// qc of a row its features 8 qc .. 8 qc + 7; the float64 operations (2 per
// clock and SM) are kept to the squared norms, the square roots to the last
// CTA, which turns the maxima over all rows into the bound's constants.
constexpr int kPrepRows = 8;

template <int BF16>
__global__ void __launch_bounds__(256) mixed_prep_kernel(
    const float *C, int64_t d, int64_t k, int64_t k_pad, int nkb, MixedConsts *c, uint8_t *img,
    float *hn, float *ct, int64_t d4, int *n_flagged, const LoopState *guard) {
    wait_for_previous();
    allow_next();
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    __shared__ float cs[64 * 4 * (kPrepRows + 1)];
    __shared__ double q_sh[2][kPrepRows];
    __shared__ float h_sh[kPrepRows];
    const int tid = threadIdx.x, G = (int)blockDim.x / kPrepRows;
    const int64_t j0 = (int64_t)blockIdx.x * kPrepRows;
    const float sigma = c->sigma;
    const double s2 = (double)sigma * (double)sigma;
    const float lim = max16<BF16>();
    bool ovf = false;
    if (blockIdx.x == 0 && tid == 0) *n_flagged = 0;
    for (int e = tid; e < nkb * 64 * kPrepRows; e += (int)blockDim.x) {
        const int f = e / kPrepRows, r = e % kPrepRows;
        cs[f * (kPrepRows + 1) + r] = (f < d && j0 + r < k) ? C[f * k + j0 + r] : 0.f;
    }
    __syncthreads();
    const int r = tid / G, qc = tid % G, kb = qc >> 3, ch = qc & 7;
    const int64_t j = j0 + r;
    const int f0 = qc * 8;
    double q2 = 0.0, qd = 0.0;
    if (kb < nkb) {
        float v[8], xr[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float x = cs[(f0 + e) * (kPrepRows + 1) + r];
            q2 += (double)x * (double)x;
            float sv = x * sigma;
            if (!(fabsf(sv) <= lim)) {
                ovf = true;
                sv = (sv > 0.f) ? lim : ((sv < 0.f) ? -lim : 0.f);
            }
            const double dv = (double)(round16<BF16>(sv) - sv);  // exact in fp32
            qd += dv * dv;
            v[e] = sv;
            xr[e] = x;
        }
        // d4 is a multiple of 4 and f0 of 8: whole float4 stores
        float4 *cdst = reinterpret_cast<float4 *>(ct + j * d4 + f0);
        if (f0 < d4) cdst[0] = make_float4(xr[0], xr[1], xr[2], xr[3]);
        if (f0 + 4 < d4) cdst[1] = make_float4(xr[4], xr[5], xr[6], xr[7]);
        uint4 pk;
        pk.x = pack2<BF16>(v[0], v[1]);
        pk.y = pack2<BF16>(v[2], v[3]);
        pk.z = pack2<BF16>(v[4], v[5]);
        pk.w = pack2<BF16>(v[6], v[7]);
        *reinterpret_cast<uint4 *>(img + (size_t)kb * k_pad * 128 +
                                   sw128_offset((uint32_t)j, (uint32_t)ch * 8)) = pk;
    }
    // the row's squared norms over its G lanes
    for (int o = G >> 1; o > 0; o >>= 1) {
        q2 += __shfl_xor_sync(0xffffffffu, q2, o);
        qd += __shfl_xor_sync(0xffffffffu, qd, o);
    }
    if (qc == 0) {
        // padding rows score -inf (c0 < 0), so they never win
        float h = 0.f, h0 = pos_inf<float>(), h1 = 0.f, h2 = 0.f;
        if (j < k) {
#pragma unroll 8
            for (int f = 0; f < (int)d; ++f) {
                const float x = cs[f * (kPrepRows + 1) + r];
                h = __fmaf_rn(x, x, h);
            }
            h = h / 2.f;
            hn[j] = h;
            const double H = (double)h * s2;
            // the coefficients are powers of two: exact reciprocals
            const double c0 = -(double)norm_coef(BF16, 0), c1 = -(double)norm_coef(BF16, 1),
                         c2 = -(double)norm_coef(BF16, 2);
            h0 = round16<BF16>((float)(H * (1.0 / c0)));
            if (!(fabsf(h0) <= lim)) {
                ovf = true;
                h0 = (H > 0.0) ? lim : -lim;
            }
            const double r1 = H - c0 * (double)h0;
            h1 = round16<BF16>((float)(r1 * (1.0 / c1)));
            const double r2 = r1 - c1 * (double)h1;
            h2 = round16<BF16>((float)(r2 * (1.0 / c2)));
            if (!(fabsf(h1) <= lim) || !(fabsf(h2) <= lim)) {
                ovf = true;
                h1 = 0.f;
                h2 = 0.f;
            }
        }
        uint8_t *nb = img + (size_t)nkb * k_pad * 128;
        uint4 p0 = make_uint4(pack2<BF16>(h0, h1), pack2<BF16>(h2, 0.f), 0u, 0u);
        *reinterpret_cast<uint4 *>(nb + sw32_offset((uint32_t)j, 0)) = p0;
        *reinterpret_cast<uint4 *>(nb + sw32_offset((uint32_t)j, 8)) = make_uint4(0u, 0u, 0u, 0u);
        // NaN norms never raise a maximum
        q_sh[0][r] = q2 == q2 ? q2 : 0.0;
        q_sh[1][r] = qd == qd ? qd : 0.0;
        h_sh[r] = h == h ? fabsf(h) : 0.f;
    }
    if (ovf) atomicOr(&c->overflow, 1);
    __syncthreads();
    if (tid == 0) {
        double m2 = 0.0, md = 0.0;
        float mh = 0.f;
        for (int q = 0; q < kPrepRows; ++q) {
            m2 = fmax(m2, q_sh[0][q]);
            md = fmax(md, q_sh[1][q]);
            mh = fmaxf(mh, h_sh[q]);
        }
        // non-negative: ordered like their bits
        atomicMax(&c->c2max_bits, (unsigned long long)__double_as_longlong(m2));
        atomicMax(&c->dc2max_bits, (unsigned long long)__double_as_longlong(md));
        atomicMax(&c->hmax_bits, __float_as_uint(mh));
    }
    if (!last_cta(&c->prep_ticket) || tid != 0) return;
    volatile MixedConsts *vc = c;
    const double u = BF16 ? 0x1p-8 : 0x1p-11;
    const double m2 = __longlong_as_double((long long)vc->c2max_bits);
    const double md = __longlong_as_double((long long)vc->dc2max_bits);
    const double mh = (double)__uint_as_float(vc->hmax_bits);
    const int over = vc->overflow;
    const double cmax = (double)__double2float_ru(sqrt(m2) * (1.0 + 1e-12));
    const double dcmax = (double)__double2float_ru(sqrt(md) / (double)sigma * (1.0 + 1e-12));
    // bf16 subnormal inputs may be flushed by the tensor cores (fp16
    // subnormals are part of the measured rounding errors)
    const double flush = BF16 ? 0x1p-126 * sqrt((double)d) * (1 + u) : 0.0;
    const double alpha =
        dcmax + 0x1p-16 * (cmax + dcmax) + (double)(d + 4) * 0x1p-23 * cmax + flush;
    const double beta1 = (cmax + dcmax) * (1 + 0x1p-16);
    const double hfloor = (BF16 ? 0x1p-126 : 0x1p-34) / s2;
    const double beta0 = mh * (u * u * u + 0x1p-16 + 0x1p-23) + hfloor + flush * cmax;
    c->alpha = __double2float_ru(alpha * s2 * (1 + 1e-6));
    c->beta1 = __double2float_ru(beta1 * s2 * (1 + 1e-6));
    c->beta0 =
        over ? pos_inf<float>() : __double2float_ru(beta0 * s2 * (1 + 1e-6) + 1e-37);
    c->overflow = 0;
    c->acc_dirty = 0;
    c->c2max_bits = 0ull;
    c->dc2max_bits = 0ull;
    c->hmax_bits = 0u;
    c->prep_ticket = 0u;
}

// Exact fp32 re-evaluation of samples whose margin did not certify them: the
// reference's arithmetic (sequential fma dot over f = 0..d-1, hn - dot,
// strict < with the lowest index on ties) over the candidate set (hot
// sub-chunks x hot classes of each column half).  A warp takes its share of the
// flagged samples, up to 32 at a time, and spreads their (sample, candidate) pairs evenly over its lanes,
// so one sample with many candidates does not hold its warp back; each pair's
// result goes into the sample's 64-bit (distance, index) key with a
// shared-memory atomic minimum, which is exactly the lexicographic minimum a
// strict-< scan in ascending index finds.  The sample's features come from the
// row-major fp32 copy of X (cached in L1 across its candidates) and the
// centroids from their transposed fp32 copy (one contiguous row each).  All latency:
// 35,000 samples (300,007 x 100, k = 500, bf16) spread over all warps instead of 32
// to a warp take 11 us instead of 38 (4M x 64, k = 256: 23 -> 10).
constexpr int kRecheckThreads = 256;

// Order-preserving map of a float to an unsigned key (NaN never compared).
__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Candidates of a flagged sample: per column pass p (cand[p * n + i], columns
// offset by p * pass_cols; one pass unless n_clusters needed several), hot
// sub-chunks x hot classes of each column half.
__device__ __forceinline__ int pass_count(const uint4 &m) {
    return __popc(m.x) * __popc(m.z) + __popc(m.y) * __popc(m.w);
}

__global__ void __launch_bounds__(kRecheckThreads) recheck_kernel(
    const float *xrow, const float *ct, const float *hn, const uint4 *cand, const int *flagged,
    const int *n_flagged, int64_t n, int64_t d, int64_t k, int64_t d4, void *labels, int label64,
    const LoopState *guard, int passes, int64_t pass_cols, long long *stats) {
    wait_for_previous();
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the fit's statistics: samples rechecked in this pass, and in total
        stats[0] = *n_flagged;
        stats[1] += *n_flagged;
    }
    constexpr int kWarps = kRecheckThreads / 32;
    __shared__ unsigned long long key_s[kWarps][32];
    __shared__ int incl_s[kWarps][32];
    __shared__ int row_s[kWarps][32];
    __shared__ uint4 cm_s[kWarps][32];
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const int64_t nf = (int64_t)*n_flagged;
    const int64_t total = nf < n ? nf : n;
    const int64_t g4 = d4 / 4;
    const unsigned long long kNone = ((unsigned long long)order_key(pos_inf<float>()) << 32);
    // samples of a warp at a time: 32, fewer where that leaves warps idle
    const int64_t warps = (int64_t)gridDim.x * kWarps;
    const int per = (int)(total >= 32 * warps ? 32 : (total + warps - 1) / warps);
    const int64_t wstride = warps * per;
    for (int64_t base = ((int64_t)blockIdx.x * kWarps + wq) * per; base < total; base += wstride) {
        const int64_t e = lane < per ? base + lane : total;
        int64_t i = -1;
        uint4 cm = make_uint4(0u, 0u, 0u, 0u);
        int cnt = 0;
        if (e < total) {
            i = flagged[e];
            if (i >= 0 && i < n) {
                cm = cand[i];
                cnt = pass_count(cm);
                for (int p = 1; p < passes; ++p) cnt += pass_count(cand[(int64_t)p * n + i]);
            } else {
                i = -1;
            }
        }
        // candidates of this lane's sample: per column half, hot sub-chunks x hot classes
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int tot = __shfl_sync(0xffffffffu, incl, 31);
        key_s[wq][lane] = kNone;
        incl_s[wq][lane] = incl;
        row_s[wq][lane] = (int)i;
        cm_s[wq][lane] = cm;
        __syncwarp();
        for (int pr = lane; pr < tot; pr += 32) {
            // owner: the first lane whose inclusive count exceeds pr
            int lo = 0, hi = 31;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (incl_s[wq][mid] > pr) hi = mid; else lo = mid + 1;
            }
            const int owner = lo;
            int r = pr - (owner ? incl_s[wq][owner - 1] : 0);
            const int64_t oi = row_s[wq][owner];
            uint4 om = cm_s[wq][owner];
            int64_t jbase = 0;
            for (int p = 1; p < passes && r >= pass_count(om); ++p) {
                r -= pass_count(om);
                om = cand[(int64_t)p * n + oi];
                jbase += pass_cols;
            }
            const int oc0 = __popc(om.x) * __popc(om.z);
            int h = 0;
            uint32_t m1 = om.x, m2 = om.z;
            if (r >= oc0) {
                h = 1;
                r -= oc0;
                m1 = om.y;
                m2 = om.w;
            }
            // the (r / n2)-th hot sub-chunk and the (r % n2)-th hot class
            const int n2 = __popc(m2);
            for (int q = r / n2; q > 0; --q) m1 &= m1 - 1u;
            for (int q = r % n2; q > 0; --q) m2 &= m2 - 1u;
            const int sc = __ffs(m1) - 1, t = __ffs(m2) - 1;
            const int64_t j = jbase + (int64_t)(sc >> 2) * kChunkN + h * 128 + (sc & 3) * 32 + t;
            if (j >= k) continue;
            const float4 *xr = reinterpret_cast<const float4 *>(xrow + oi * d4);
            const float4 *cr = reinterpret_cast<const float4 *>(ct + j * d4);
            float dot = 0.f;
            // unrolled so that a candidate's row loads are in flight
            // before its fma chain needs them
#pragma unroll 8
            for (int64_t g = 0; g < g4; ++g) {
                const float4 xv = __ldg(xr + g), cv = __ldg(cr + g);
                dot = __fmaf_rn(xv.x, cv.x, dot);
                if (4 * g + 1 < d) dot = __fmaf_rn(xv.y, cv.y, dot);
                if (4 * g + 2 < d) dot = __fmaf_rn(xv.z, cv.z, dot);
                if (4 * g + 3 < d) dot = __fmaf_rn(xv.w, cv.w, dot);
            }
            const float D = hn[j] - dot;
            if (D == D)
                atomicMin(&key_s[wq][owner],
                          ((unsigned long long)order_key(D) << 32) | (unsigned long long)j);
        }
        __syncwarp();
        if (i >= 0) {
            const int bj = (int)(key_s[wq][lane] & 0xffffffffull);
            if (label64)
                reinterpret_cast<int64_t *>(labels)[i] = bj;
            else
                reinterpret_cast<int32_t *>(labels)[i] = bj;
        }
        __syncwarp();  // this batch's keys and masks are read before the next batch
    }
}

// After the column passes of one assignment: per sample the best score M
// over the passes and thr = M - E2 (the bound the passes used).  Every
// score within E2 / 2 of its exact value, a pass whose best score is below
// thr holds no candidate; the pass masks were made against the pass's own
// best score minus E2, which is at most thr, so a hot pass's masks hold a
// superset of its candidates.  The sample is certified when exactly one pass
// reaches thr and that pass has a unique winner (single bits in one half,
// nothing in the other): its label is written.  Otherwise the masks of the
// passes below thr are cleared and the sample goes to the recheck list.
__global__ void __launch_bounds__(256) combine_kernel(
    const float *pmax, uint4 *cand, int passes, int64_t pass_cols, const float *nx,
    const float *ndx, const MixedConsts *consts, void *labels, int label64, int *flagged,
    int *n_flagged, int64_t n, int64_t k, const LoopState *guard) {
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    const MixedConsts cst = *consts;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float e = fmaf(nx[i], cst.alpha, fmaf(ndx[i], cst.beta1, cst.beta0));
        const float E2 = 2.f * e * 1.000001f;
        int64_t label = -1;
        float M = -pos_inf<float>();
        bool nan = false;
        for (int p = 0; p < passes; ++p) {
            const float v = pmax[(int64_t)p * n + i];
            nan |= !(v == v);
            M = fmaxf(M, v);
        }
        const float thr = M - E2;
        nan |= !(thr == thr);
        int hot = 0, ph = -1;
        for (int p = 0; p < passes; ++p)
            if (nan || pmax[(int64_t)p * n + i] >= thr) {
                ++hot;
                ph = p;
            }
        if (!nan && hot == 1) {
            const uint4 m = cand[(int64_t)ph * n + i];
            const bool a0 = (m.x | m.z) != 0u, a1 = (m.y | m.w) != 0u;
            if (a0 != a1) {
                const int h = a1 ? 1 : 0;
                const uint32_t h1 = h ? m.y : m.x, h2 = h ? m.w : m.z;
                if (__popc(h1) == 1 && __popc(h2) == 1) {
                    const int sc = __ffs(h1) - 1, t = __ffs(h2) - 1;
                    label = (int64_t)ph * pass_cols + (int64_t)(sc >> 2) * kChunkN + h * 128 +
                            (sc & 3) * 32 + t;
                    if (label >= k) label = -1;
                }
            }
        }
        if (label >= 0) {
            if (label64)
                reinterpret_cast<int64_t *>(labels)[i] = label;
            else
                reinterpret_cast<int32_t *>(labels)[i] = (int32_t)label;
        } else {
            if (!nan)
                for (int p = 0; p < passes; ++p)
                    if (!(pmax[(int64_t)p * n + i] >= thr))
                        cand[(int64_t)p * n + i] = make_uint4(0u, 0u, 0u, 0u);
            const int pos = atomicAdd(n_flagged, 1);
            if (pos >= 0 && pos < n) flagged[pos] = (int)i;
        }
    }
}

// ---------------------------------------------------------------------------
// Cluster sums of an iteration, from the labels that the kernels above wrote.
//
// Their own pass over the samples: inside the assignment kernel, few warps had
// to load each tile's rows, wait for its labels and reduce them, and those
// chains, not the tensor cores, set its pace (4M x 64, k = 64: 665 us with the
// sums, 167 us without).  Here every SM is full of warps that do nothing else.
// A warp takes 32 samples; their rows are one contiguous run of the row-major
// copy, which its lanes walk together, so that a load or reduction touches one
// or a few rows.  The reductions' rate bounds it (26 clocks per warp and SM of
// red.v4.f32, 13 of red.u64).
// ---------------------------------------------------------------------------
constexpr int kSumThreads = 256;

template <typename I>
__device__ __forceinline__ int label_of(const I *labels, int64_t i, int64_t n, int64_t k) {
    if (i >= n) return -1;
    const I c = labels[i];
    return c >= 0 && c < k ? (int)c : -1;
}

// Beyond 32 features: float32 sums in copies of [k_pad][d4] and k_pad sizes
// (CTA b adds into copy b mod n_copies).
template <typename I>
__global__ void __launch_bounds__(kSumThreads) sum_rows_kernel(
    const float *xrow, const float *w, const I *labels, int64_t n, int64_t d4, int64_t k,
    int64_t k_pad, float *sums, int n_copies, const LoopState *guard) {
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    constexpr int kBatch = 4;
    const int lane = threadIdx.x & 31, g4 = (int)(d4 / 4);
    const int step_r = 32 / g4, step_m = 32 % g4;
    sums += (int64_t)(blockIdx.x % (unsigned)n_copies) * (k_pad * d4 + k_pad);
    for (int64_t base = (int64_t)blockIdx.x * kSumThreads + (threadIdx.x & ~31); base < n;
         base += (int64_t)gridDim.x * kSumThreads) {
        const int c = label_of(labels, base + lane, n, k);
        const float wv = base + lane < n ? w[base + lane] : 0.f;
        const float4 *src = reinterpret_cast<const float4 *>(xrow) + base * g4 + lane;
        int r = lane / g4, m = lane - r * g4;
        for (int t0 = 0; t0 < g4; t0 += kBatch) {
            float4 v[kBatch];
            float wr[kBatch];
            int64_t e[kBatch];
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                // r < 32 while t0 + t < g4
                const int cr = __shfl_sync(0xffffffffu, c, r & 31);
                wr[t] = __shfl_sync(0xffffffffu, wv, r & 31);
                e[t] = cr >= 0 && t0 + t < g4 ? (int64_t)cr * g4 + m : -1;
                v[t] = load_f4_if(src + 32 * (t0 + t), e[t] >= 0);
                r += step_r;
                m += step_m;
                if (m >= g4) {
                    m -= g4;
                    ++r;
                }
            }
#pragma unroll
            for (int t = 0; t < kBatch; ++t)
                if (e[t] >= 0)
                    atomicAdd(reinterpret_cast<float4 *>(sums) + e[t],
                              make_float4(__fmul_rn(v[t].x, wr[t]), __fmul_rn(v[t].y, wr[t]),
                                          __fmul_rn(v[t].z, wr[t]), __fmul_rn(v[t].w, wr[t])));
        }
        if (c >= 0) atomicAdd(sums + k_pad * d4 + c, wv);
    }
}

// Columns 4 l .. 4 l + 3 of sample i (label c) into the float64 copies, out of
// line: those whose packed terms are flagged (packed null: all of them).
__device__ __noinline__ void add_columns_f64(const float *xrow, const float *w, const int *packed,
                                             int64_t i, int c, int l, int64_t d4, int64_t k_pad,
                                             double *acc, int *dirty) {
    const float wv = w[i];
    *reinterpret_cast<volatile int *>(dirty) = 1;
    for (int64_t j = 4 * l; j < 4 * l + 4 && j <= d4; ++j) {
        if (packed != nullptr && packed[j] != 1) continue;
        const float v = j < d4 ? __fmul_rn(xrow[i * d4 + j], wv) : wv;
        atomicAdd(j < d4 ? acc + c * d4 + j : acc + k_pad * d4 + c, (double)v);
    }
}

// Up to 32 features: the packed terms (w x_j, then w) into the integer copies,
// one 64-bit reduction per term that is not zero; F terms of a lane in flight.
// No float64 instruction on the main path: on this part even a predicated-off
// float64 conversion costs the issue slots of a whole row.
template <typename I, int F>
__global__ void __launch_bounds__(kSumThreads) sum_terms_kernel(
    const float *xrow, const float *w, const I *labels, int64_t n, int64_t d4, int64_t k,
    int64_t k_pad, FxAcc fx, double *acc, int n_copies, const MixedConsts *consts,
    const LoopState *guard) {
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    const int lane = threadIdx.x & 31, w1 = (int)d4 + 1, ds = (int)d4 + 4;
    const int step_r = 32 / w1, step_m = 32 % w1;
    const bool fx_ok = consts->fx_ok;
    unsigned long long *sum = fx.sum + (int64_t)(blockIdx.x % (unsigned)fx.copies) * fx.stride;
    acc += (int64_t)(blockIdx.x % (unsigned)n_copies) * (k_pad * d4 + k_pad);
    for (int64_t base = (int64_t)blockIdx.x * kSumThreads + (threadIdx.x & ~31); base < n;
         base += (int64_t)gridDim.x * kSumThreads) {
        const int c = label_of(labels, base + lane, n, k);
        if (!fx_ok) {
            for (int l = 0; c >= 0 && l <= (int)d4 / 4; ++l)
                add_columns_f64(xrow, w, nullptr, base + lane, c, l, d4, k_pad, acc, fx.dirty);
            continue;
        }
        const int *src = fx.xq + base * ds;
        int r = lane / w1, m = lane - r * w1, flags = 0;
        for (int t0 = 0; t0 < w1; t0 += F) {
            int v[F];
            int64_t e[F];
#pragma unroll
            for (int t = 0; t < F; ++t) {
                // r < 32 while t0 + t < w1
                const int cr = __shfl_sync(0xffffffffu, c, r & 31);
                const bool in = cr >= 0 && t0 + t < w1;
                e[t] = m < (int)d4 ? cr * d4 + m : k * d4 + cr;
                v[t] = load_i_if(src + r * ds + m, in);
                r += step_r;
                m += step_m;
                if (m >= w1) {
                    m -= w1;
                    ++r;
                }
            }
#pragma unroll
            for (int t = 0; t < F; ++t) {
                flags |= v[t];
                // not zero, not flagged
                if ((unsigned)v[t] > 1u)
                    atomicAdd(sum + e[t], (unsigned long long)((long long)(v[t] >> 6) *
                                                               (1 << ((v[t] >> 1) & 31))));
            }
        }
        if (__any_sync(0xffffffffu, (flags & 1) != 0))
            for (int l = 0; c >= 0 && l <= (int)d4 / 4; ++l)
                add_columns_f64(xrow, w, src + lane * ds, base + lane, c, l, d4, k_pad, acc, fx.dirty);
    }
}

// Up to kSortClusters clusters: a CTA sorts a tile of samples by label first
// (counting sort in shared memory), then groups of lanes walk runs of the sorted
// samples, one lane per 16 bytes of a row, sum equal labels in registers and
// reduce once per run of a label.  F = 0: float32 rows and weights, four rows of
// a group in flight; F = 2, 4: packed terms, F rows in flight.
// 4M samples, direct kernel -> sorted: 64 features, k = 64: 299 -> 172 us (5.9
// TB/s), k = 1024: 285 -> 194; packed, 16 features, k = 100: 199 -> 113; 32 and
// 256: 350 -> 195 (2M, 32 and 1000: 195 -> 160).  The larger the tile, the fewer
// runs: k = 1024 takes 219 us with 2048 samples.  Bound by memory for few
// clusters, by the runs' reductions for many; with more clusters than
// kSortClusters most runs are single samples and the sort only costs.
constexpr int kSortTile = 4096, kSortClusters = 2048;
constexpr int kSortCtas = 4;  // resident per SM (64 registers)

// Shared memory of a CTA.  All of it is dynamic: beside the 1024-byte aligned
// image of the assignment kernel, a static array would take 1 KB.
constexpr size_t kSortRowBytes = sizeof(int2) + sizeof(float);
constexpr size_t sort_smem(int tile, int64_t k) {
    return kSortRowBytes * (size_t)tile + sizeof(int) * (size_t)(k + 1 + kSumThreads / 32);
}
// The most rows of a tile, so that kSortCtas CTAs fit an SM (228 KB, 1 KB of a
// CTA reserved): 4096 up to 2031 clusters, 4064 beyond.
constexpr size_t kSortSmem = 228 * 1024 / kSortCtas - 1024;
constexpr int sort_rows(int64_t k) {
    const int64_t fit = (int64_t)((kSortSmem - sort_smem(0, k)) / kSortRowBytes) / 32 * 32;
    return fit < kSortTile ? (int)fit : kSortTile;
}
static_assert(sort_rows(1) == kSortTile && sort_rows(2031) == kSortTile &&
                  sort_rows(kSortClusters) == 4064 &&
                  sort_smem(sort_rows(kSortClusters), kSortClusters) <= kSortSmem,
              "tiles of the sorted sums");

template <typename I, int F>
__global__ void __launch_bounds__(kSumThreads, kSortCtas) sum_sorted_kernel(
    const float *xrow, const float *w, const I *labels, int64_t n, int64_t d4, int64_t k,
    int64_t k_pad, int tile_rows, float *sums, FxAcc fx, double *acc, int n_copies,
    const MixedConsts *consts, const LoopState *guard) {
    wait_for_previous();
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    constexpr bool FX = F != 0;
    constexpr int kPer = kSortTile / kSumThreads, kWarps = kSumThreads / 32, kBatch = FX ? F : 4;
    extern __shared__ __align__(16) uint8_t sort_raw[];
    int2 *key = reinterpret_cast<int2 *>(sort_raw);  // (label, row of the tile) by label
    float *ws = reinterpret_cast<float *>(key + tile_rows);  // weights, same order
    int *hist = reinterpret_cast<int *>(ws + tile_rows);     // counts, then first positions
    int *warp_sum = hist + k + 1;
    const int tid = threadIdx.x, lane = tid & 31, wq = tid >> 5;
    const int vecs = FX ? (int)d4 / 4 + 1 : (int)d4 / 4;  // 16-byte vectors of a row
    unsigned long long *isum = nullptr;
    if (FX) {
        isum = fx.sum + (int64_t)(blockIdx.x % (unsigned)fx.copies) * fx.stride;
        acc += (int64_t)(blockIdx.x % (unsigned)n_copies) * (k_pad * d4 + k_pad);
    } else {
        sums += (int64_t)(blockIdx.x % (unsigned)n_copies) * (k_pad * d4 + k_pad);
    }
    const bool fx_ok = !FX || consts->fx_ok;
    for (int64_t i0 = (int64_t)blockIdx.x * tile_rows; i0 < n; i0 += (int64_t)gridDim.x * tile_rows) {
        const int rows = (int)(n - i0 < tile_rows ? n - i0 : tile_rows);
        __syncthreads();  // every read of the previous tile's order
        for (int64_t j = tid; j <= k; j += kSumThreads) hist[j] = 0;
        int c[kPer], rank[kPer];
#pragma unroll
        for (int t = 0; t < kPer; ++t)
            c[t] = tid + kSumThreads * t < rows ? label_of(labels, i0 + tid + kSumThreads * t, n, k) : -1;
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kPer; ++t)
            if (c[t] >= 0) rank[t] = atomicAdd(hist + c[t], 1);
        __syncthreads();
        // exclusive sums of the counts, a run of them per thread
        const int per = ((int)k + kSumThreads) / kSumThreads, j0 = tid * per;
        int total = 0;
        for (int j = j0; j < j0 + per && j <= k; ++j) total += hist[j];
        int incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_sum[wq] = incl;
        __syncthreads();
        int first = incl - total;
        for (int q = 0; q < wq; ++q) first += warp_sum[q];
        for (int j = j0; j < j0 + per && j <= k; ++j) {
            const int v = hist[j];
            hist[j] = first;
            first += v;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kPer; ++t)
            if (c[t] >= 0) {
                const int row = tid + kSumThreads * t, pos = hist[c[t]] + rank[t];
                key[pos] = make_int2(c[t], row);
                ws[pos] = FX ? 0.f : w[i0 + row];
            }
        __syncthreads();
        const int valid = hist[k];  // samples with a label (all of them)
        for (int v0 = 0; v0 < vecs; v0 += 32) {
            const int L = vecs - v0 < 32 ? vecs - v0 : 32, per_warp = 32 / L;
            const int grp = lane / L, l = v0 + lane - grp * L;
            if (grp >= per_warp) continue;
            const int groups = kWarps * per_warp, id = wq * per_warp + grp;
            const int a = valid * id / groups, b = valid * (id + 1) / groups;
            int cur = -1;
            float4 fs = make_float4(0.f, 0.f, 0.f, 0.f);
            float fw = 0.f;
            long long qs[4] = {0, 0, 0, 0};
            auto flush = [&]() {
                if (cur < 0) return;
                if constexpr (FX) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int64_t j = 4 * l + q;
                        if (j <= d4 && qs[q] != 0)
                            atomicAdd(isum + (j < d4 ? cur * d4 + j : k * d4 + cur),
                                      (unsigned long long)qs[q]);
                        qs[q] = 0;
                    }
                } else {
                    atomicAdd(reinterpret_cast<float4 *>(sums + cur * d4) + l, fs);
                    if (l == 0) atomicAdd(sums + k_pad * d4 + cur, fw);
                    fs = make_float4(0.f, 0.f, 0.f, 0.f);
                    fw = 0.f;
                }
            };
            for (int p0 = a; p0 < b; p0 += kBatch) {
                int2 kk[kBatch];
                float4 x[kBatch];
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const bool in = p0 + t < b;
                    kk[t] = key[in ? p0 + t : a];
                    const float *src = FX ? reinterpret_cast<const float *>(fx.xq) + (i0 + kk[t].y) * (d4 + 4)
                                          : xrow + (i0 + kk[t].y) * d4;
                    x[t] = load_f4_if(reinterpret_cast<const float4 *>(src) + l, in);
                    if (!in) kk[t].x = -1;
                }
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    if (kk[t].x < 0) continue;
                    if (kk[t].x != cur) {
                        flush();
                        cur = kk[t].x;
                    }
                    if constexpr (FX) {
                        const int v[4] = {__float_as_int(x[t].x), __float_as_int(x[t].y),
                                          __float_as_int(x[t].z), __float_as_int(x[t].w)};
                        if (!fx_ok || ((v[0] | v[1] | v[2] | v[3]) & 1))
                            add_columns_f64(xrow, w,
                                            fx_ok ? fx.xq + (i0 + kk[t].y) * (d4 + 4) : nullptr,
                                            i0 + kk[t].y, cur, l, d4, k_pad, acc, fx.dirty);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            qs[q] += (long long)(v[q] >> 6) * (1 << ((v[q] >> 1) & 31));
                    } else {
                        const float wv = ws[p0 + t];
                        fs.x += __fmul_rn(x[t].x, wv);
                        fs.y += __fmul_rn(x[t].y, wv);
                        fs.z += __fmul_rn(x[t].z, wv);
                        fs.w += __fmul_rn(x[t].w, wv);
                        fw += wv;
                    }
                }
            }
            flush();
        }
    }
}

// The sums of an iteration (km_step.cuh): the fixed-point totals (exact to one
// rounding), then the cluster-major float copies ([copy][k_pad d4 + k_pad]),
// each copy zeroed once read.  With fixed-point totals the float64 copies hold
// anything only when a kernel set acc_dirty.
template <typename A>
struct MixedSums {
    A *copies;
    int n_copies;
    int64_t k, k_pad, d4;
    FxAcc fx;
    MixedConsts *consts;
    struct Part {
        double v;
        long long hi;
        unsigned long long lo;
    };
    // cluster-major, the sizes last
    __device__ __forceinline__ void at(int64_t e, int64_t d, int64_t *f, int64_t *j) const {
        if (e < k * d) {
            // a 64-bit division is a hundred instructions
            *j = e <= 0xffffffffll ? (int64_t)((uint32_t)e / (uint32_t)d) : e / d;
            *f = e - *j * d;
        } else {
            *f = d;
            *j = e - k * d;
        }
    }
    __device__ __forceinline__ Part load(int64_t f, int64_t j, int64_t d, int g, int groups) const {
        Part p = zero();
        const bool use_fx = fx.sum != nullptr && consts->fx_ok;
        if (use_fx) {
            const int64_t e = f < d ? j * d4 + f : k * d4 + j;
            for (int c = g; c < fx.copies; c += 8 * groups) {
                unsigned long long l[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    l[u] = c + u * groups < fx.copies ? fx.sum[(c + u * groups) * fx.stride + e] : 0ull;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (c + u * groups < fx.copies) fx.sum[(c + u * groups) * fx.stride + e] = 0ull;
                    // copies below 2^61 in two parts: no overflow for any count
                    p.hi += (long long)l[u] >> 32;
                    p.lo += l[u] & 0xffffffffull;
                }
            }
        }
        if (!use_fx || consts->acc_dirty) {
            A *q = copies + (f < d ? j * d4 + f : k_pad * d4 + j);
            const int64_t stride = k_pad * d4 + k_pad;
            for (int c = g; c < n_copies; c += 8 * groups) {
                A v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    v[u] = c + u * groups < n_copies ? q[(c + u * groups) * stride] : A(0);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (c + u * groups < n_copies) q[(c + u * groups) * stride] = A(0);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (c + u * groups < n_copies) p.v += (double)v[u];
            }
        }
        return p;
    }
    static __device__ __forceinline__ Part zero() { return Part{0.0, 0, 0ull}; }
    static __device__ __forceinline__ void add(Part &a, const Part &b) {
        a.v += b.v;
        a.hi += b.hi;
        a.lo += b.lo;
    }
    __device__ __forceinline__ double value(const Part &p) const {
        if (fx.sum == nullptr || !consts->fx_ok) return p.v;
        return ((double)p.hi * 4294967296.0 + (double)p.lo) *
                   (1.0 / (double)pow2f(consts->fx_shift)) + p.v;
    }
};

using MixedKernel = void (*)(MixedArgs);

// The widest pass each feature-block count takes (shared memory); column
// passes always use it, so only those shapes have a multi-pass kernel.
constexpr int max_chunks(int nkb) { return nkb == 1 ? 4 : (nkb == 2 ? 2 : 1); }

template <int BF16, int NKB>
MixedKernel pick_chunks(int nch, bool multi) {
    constexpr int W = max_chunks(NKB);
    if (multi) return nch == W ? mixed_assign_kernel<BF16, NKB, W, true> : nullptr;
    switch (nch) {
        case 1: return mixed_assign_kernel<BF16, NKB, 1, false>;
        case 2: return W >= 2 ? mixed_assign_kernel<BF16, NKB, (W >= 2 ? 2 : 1), false> : nullptr;
        case 3: return W >= 3 ? mixed_assign_kernel<BF16, NKB, (W >= 3 ? 3 : 1), false> : nullptr;
        case 4: return W >= 4 ? mixed_assign_kernel<BF16, NKB, (W >= 4 ? 4 : 1), false> : nullptr;
        default: return nullptr;
    }
}

// Kernel for (operand type, 64-feature blocks, 256-column chunks per pass,
// column passes or one).
MixedKernel pick_kernel(int bf16, int nkb, int nch, bool multi = false) {
    switch (nkb) {
        case 1: return bf16 ? pick_chunks<1, 1>(nch, multi) : pick_chunks<0, 1>(nch, multi);
        case 2: return bf16 ? pick_chunks<1, 2>(nch, multi) : pick_chunks<0, 2>(nch, multi);
        case 3: return bf16 ? pick_chunks<1, 3>(nch, multi) : pick_chunks<0, 3>(nch, multi);
        case 4: return bf16 ? pick_chunks<1, 4>(nch, multi) : pick_chunks<0, 4>(nch, multi);
        default: return nullptr;
    }
}

// Up to 4 feature blocks (d <= 256) fit next to one 256-column chunk.
constexpr int kMaxFeatureBlocks = 4;

// Column chunks per pass and X-ring depth for nkb feature blocks: the widest
// pass (no wider than needed for kp columns)
// that fits shared memory with a ring of at least two stages, else one stage.
bool pass_plan(int nkb, int64_t kp, int *nch_out, int *stages_out) {
    const int want = (int)std::min<int64_t>(max_chunks(nkb), kp / kChunkN);
    for (int nch = want; nch >= 1; --nch) {
        if (pick_kernel(0, nkb, nch) == nullptr) continue;
        for (int st = 4; st >= 1; --st)
            if (smem_layout(nkb, (int64_t)nch * kChunkN, st).total <= kSmemLimit) {
                if (st == 1 && nch > 1) break;  // a narrower pass keeps a two-stage ring
                *nch_out = nch;
                *stages_out = st;
                return true;
            }
    }
    return false;
}

// Four float4s per thread and round, at most eight CTAs per SM.
unsigned absmax_grid(int64_t count) {
    return (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(ceil_div<int64_t>(count, 16 * kAbsmaxThreads), (int64_t)num_sms() * 8));
}

unsigned grid1d(int64_t work, int block, int cap = 8192) {
    int64_t g = ceil_div<int64_t>(work, block);
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

}  // namespace

// ---------------------------------------------------------------------------
// Mixed-form variant choice.  A variant forced process-wide (a test hook) or
// for the fits the autotuner creates on this thread overrides the tuner.
std::atomic<int> g_force_mixed_variant{-1};
thread_local int tl_force_mixed_variant = -1;
// Fits created while this is set use a cached choice or the default, never
// time variants (the request server: no measurement on a request's path).
thread_local bool tl_mixed_lookup_only = false;

int forced_variant() {
    const int g = g_force_mixed_variant.load();
    return g >= 0 ? g : tl_force_mixed_variant;
}

int64_t pow2_at_least(int64_t v) {
    int64_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

template <typename I>
int make_mixed_fit_impl(const FitParams<float, I> &p, int form, std::unique_ptr<FitBase> *out);

// Times each candidate variant on a synthetic fit (Gaussian blobs of d
// features, k clusters) for four iterations after one warm-up, and keeps the
// fastest per (d, k, form, size class) in memory (the file's reader takes tile
// widths only, so every process times these anew).  Fits of at least 32 tiles per SM
// ("large") are timed with 48 tiles per SM, smaller ones with 8.  KMC_TUNE=0 keeps
// the default (the first candidate).
int tune_mixed_variant(int64_t d, int64_t k, int form, bool large, const std::vector<int> &cand,
                       cudaStream_t s, int *code) {
    Range range("kmc.tune_mixed_variant");
    *code = cand.front();
    if (const char *e = std::getenv("KMC_TUNE"))
        if (e[0] == '0') return KMC_OK;
    const char *tag = form == KMC_FORM_MIXED_BF16 ? (large ? "mixed-bf16-large" : "mixed-bf16")
                                                  : (large ? "mixed-fp16-large" : "mixed-fp16");
    int cached = -1;
    if (tune_lookup(d, k, tag, &cached) &&
        std::find(cand.begin(), cand.end(), cached) != cand.end()) {
        *code = cached;
        return KMC_OK;
    }
    if (tl_mixed_lookup_only) return KMC_OK;
    const int64_t n = (int64_t)num_sms() * kTileM * (large ? 48 : 8);
    Scratch mem;
    const size_t oX = 0, oC0 = oX + align256(sizeof(float) * n * d);
    const size_t oC = oC0 + align256(sizeof(float) * d * k), oCn = oC + align256(sizeof(float) * d * k);
    const size_t ow = oCn + align256(sizeof(float) * d * k), ol = ow + align256(sizeof(float) * n);
    const size_t oi = ol + align256(sizeof(int32_t) * n);
    KMC_TRY(mem.alloc(oi + align256(sizeof(int32_t) * k), s));
    char *b = mem.as<char>();
    float *X = reinterpret_cast<float *>(b + oX), *C0 = reinterpret_cast<float *>(b + oC0);
    float *C = reinterpret_cast<float *>(b + oC), *Cn = reinterpret_cast<float *>(b + oCn);
    float *w = reinterpret_cast<float *>(b + ow);
    int32_t *lab = reinterpret_cast<int32_t *>(b + ol), *idx = reinterpret_cast<int32_t *>(b + oi);
    KMC_TRY(launch_blobs(X, n, d, k, -10.f, 10.f, 1.f, 1.f, 77, s));
    KMC_TRY(launch_fill<float>(w, 1.f, n, s));
    std::vector<int32_t> rows;
    seeded_rows(n, k, 78, &rows);
    KMC_CUDA_TRY(cudaMemcpyAsync(idx, rows.data(), sizeof(int32_t) * k, cudaMemcpyHostToDevice, s));
    KMC_TRY(launch_gather_rows(X, n, d, idx, k, C0, s));
    KMC_CUDA_TRY(cudaStreamSynchronize(s));  // rows (host vector) copied
    cudaEvent_t e0, e1;
    KMC_CUDA_TRY(cudaEventCreate(&e0));
    KMC_CUDA_TRY(cudaEventCreate(&e1));
    float best_ms = 0.f;
    int best = -1;
    for (int c : cand) {
        FitParams<float, int32_t> q;
        q.X = X;
        q.w = w;
        q.centroids = C;
        q.new_centroids = Cn;
        q.labels = lab;
        q.n = n;
        q.d = d;
        q.k = k;
        q.tol = 0.0;
        q.max_iter = 1000;
        q.stream = s;
        if (cudaMemcpyAsync(C, C0, sizeof(float) * d * k, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
            continue;
        tl_force_mixed_variant = c;
        std::unique_ptr<FitBase> fit;
        int rc = make_mixed_fit_impl<int32_t>(q, form, &fit);
        tl_force_mixed_variant = -1;
        if (rc != KMC_OK) continue;
        float ms = 0.f;
        rc = fit->enqueue_iteration(true);
        if (rc == KMC_OK) rc = cudaEventRecord(e0, s) == cudaSuccess ? KMC_OK : KMC_ERR_CUDA;
        for (int it = 0; it < 4 && rc == KMC_OK; ++it) rc = fit->enqueue_iteration(true);
        if (rc == KMC_OK) rc = cudaEventRecord(e1, s) == cudaSuccess ? KMC_OK : KMC_ERR_CUDA;
        if (rc == KMC_OK) rc = cudaEventSynchronize(e1) == cudaSuccess ? KMC_OK : KMC_ERR_CUDA;
        if (rc == KMC_OK) rc = cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess ? KMC_OK : KMC_ERR_CUDA;
        if (rc == KMC_OK && (best < 0 || ms < best_ms)) {
            best_ms = ms;
            best = c;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    KMC_CUDA_TRY(cudaStreamSynchronize(s));
    if (best >= 0) {
        tune_record(d, k, tag, best);
        *code = best;
    }
    return KMC_OK;
}

template <typename I>
struct MixedFit : PlainFit<float, I> {
    using Base = PlainFit<float, I>;
    int bf16 = 0;
    int nkb = 1;
    int acc_f64 = 0;
    int stages = 2;
    int64_t k_pad = 0, d4 = 0, ntiles = 0;
    Scratch mws;
    uint8_t *ximg = nullptr, *cimg = nullptr;
    float *nx = nullptr, *ndx = nullptr, *ct = nullptr, *xrow = nullptr;
    float *sums32 = nullptr;
    double *acc64 = nullptr;
    int n_copies = 1;  // private copies of the cluster sums
    MixedConsts *consts = nullptr;
    uint4 *cand = nullptr;
    int *flagged = nullptr, *n_flagged = nullptr, *err_dev = nullptr;
    long long *stats = nullptr;  // [0] last pass, [1] total
    int stall_once = 0;

    int set_wait_limit(long long clocks, int stall) override {
        stall_once = stall != 0;
        return Base::set_wait_limit(clocks, stall);
    }

    // The one-time conversion reads X in either layout; afterwards every
    // kernel reads the row-major fp32 copy.
    bool reads_rowmajor() const override { return true; }
    bool uses_private_copies() const override { return false; }
    void x_view(const float **x, int64_t *fs, int64_t *ss) const override {
        *x = xrow;
        *fs = 1;
        *ss = d4;
    }

    int nch = 1;     // 256-column chunks per pass
    int passes = 1;  // column passes per assignment (n_clusters beyond one pass)
    float *pmax = nullptr;
    int variant = 0;  // 10 stages + packed rows in flight per lane of the sums (0: no such sums)
    int *xq = nullptr;  // [n][d4 + 4] packed fixed-point terms
    unsigned long long *fxsum = nullptr;  // their integer totals
    // Up to 32 features (fits with weights): packed terms, integer totals
    bool fx_on = false;
    FxAcc fx_acc() const {
        return fx_on ? FxAcc{xq, fxsum, this->prm.k * d4 + this->prm.k, n_copies, &consts->acc_dirty}
                     : FxAcc{nullptr, nullptr, 0, 1, &consts->acc_dirty};
    }

    static bool supported(int64_t d, int64_t k) {
        const int nk = (int)ceil_div<int64_t>(std::max<int64_t>(d, 1), 64);
        if (nk > kMaxFeatureBlocks || k < 1) return false;
        const int64_t kp = ceil_div<int64_t>(k, kChunkN) * kChunkN;
        int c = 0, st = 0;
        return pass_plan(nk, kp, &c, &st);
    }

    int init_mixed(int form) {
        const FitParams<float, I> &p = this->prm;
        cudaStream_t s = p.stream;
        bf16 = (form == KMC_FORM_MIXED_BF16) ? 1 : 0;
        nkb = (int)ceil_div<int64_t>(std::max<int64_t>(p.d, 1), 64);
        d4 = ceil_div<int64_t>(std::max<int64_t>(p.d, 1), 4) * 4;
        ntiles = ceil_div<int64_t>(p.n, kTileM);
        if (!pass_plan(nkb, ceil_div<int64_t>(p.k, kChunkN) * kChunkN, &nch, &stages)) {
            set_error("mixed form: operands do not fit in shared memory");
            return KMC_ERR_UNSUPPORTED;
        }
        // the centroid image has whole passes of rows (zero padding)
        passes = (int)ceil_div<int64_t>(p.k, (int64_t)nch * kChunkN);
        k_pad = (int64_t)passes * nch * kChunkN;
        // Cluster sums: up to 32 features, exact integer sums of packed terms
        // (float64 for terms that do not fit; they keep the trajectory on the
        // float64 reference's), beyond that float32 four-wide reductions.
        acc_f64 = d4 <= 32 ? 1 : 0;
        // Ring depth and, for the integer sums, the rows (or terms) a lane has
        // in flight: a variant code 10 stages + f (f = 4 or 2; 0: other sums).
        // The autotuner times the variants that fit on a synthetic fit once
        // per (d, power-of-two bucket of k, form, size class) and keeps the
        // fastest; the deepest ring with f = 2 is the default when tuning is
        // off.
        {
            std::vector<int> cand;
            const int64_t kb = std::min<int64_t>(k_pad, std::max<int64_t>(pow2_at_least(p.k), 1));
            const bool fx_shape = acc_f64 && p.w != nullptr;
            for (int st = stages; st >= std::min(stages, 2); --st)
                if (fx_shape) {
                    cand.push_back(10 * st + 2);
                    cand.push_back(10 * st + 4);
                } else {
                    cand.push_back(10 * st);
                }
            if (cand.empty()) cand.push_back(10 * stages);
            int code = cand.front();
            const int forced = forced_variant();
            if (forced >= 0) {
                if (std::find(cand.begin(), cand.end(), forced) == cand.end()) {
                    set_error("mixed form: variant %d does not fit this shape", forced);
                    return KMC_ERR_INVALID_ARGUMENT;
                }
                code = forced;
            } else if (cand.size() > 1) {
                // a measurement that cannot run (out of memory, say) leaves the
                // default: tuning never fails a fit
                const bool large = ntiles >= 32 * (int64_t)num_sms();
                if (tune_mixed_variant(p.d, kb, form, large, cand, s, &code) != KMC_OK)
                    code = cand.front();
            }
            variant = code;
            stages = code / 10;
        }
        size_t off = 0;
        auto take = [&](size_t bytes) {
            size_t o = off;
            off += align256(bytes);
            return o;
        };
        const size_t o_x = take((size_t)std::max<int64_t>(ntiles, 1) * nkb * kTileBytes);
        const size_t o_c = take(cimg_bytes(nkb, k_pad));
        const size_t o_ct = take(sizeof(float) * k_pad * d4);
        const size_t o_nx = take(sizeof(float) * p.n);
        const size_t o_ndx = take(sizeof(float) * p.n);
        // Private copies of the sums, CTA b of their kernel into copy b mod
        // n_copies: with few clusters their few addresses would serialise the
        // reductions of all SMs (4M x 64 alone: k = 100 and 1 copy 502 us, 16
        // copies 260, 152 copies 231; k = 1024 and 1 copy 272, 4 copies 227).
        // Every iteration reads and clears every copy, so there are 4096 / k of
        // them (at least 4, of the integer sums 16, since the rows that a copy
        // adds up cost the scale bits), at most one per SM and per eight tiles.
        {
            const int64_t most = std::min<int64_t>(ntiles / 8, num_sms());
            const int64_t want = std::max<int64_t>(4096 / p.k, acc_f64 ? 16 : 4);
            n_copies = (int)std::max<int64_t>(1, std::min(most, want));
        }
        const int64_t csz = (int64_t)n_copies * (k_pad * d4 + k_pad);
        const size_t o_s32 = take(acc_f64 ? 16 : sizeof(float) * csz);
        const size_t o_a64 = take(acc_f64 ? sizeof(double) * csz : 16);
        const size_t o_xf = take(sizeof(float) * std::max<int64_t>(p.n, 1) * d4);
        fx_on = acc_f64 && p.w != nullptr;
        const size_t o_xq = take(fx_on ? sizeof(int) * std::max<int64_t>(p.n, 1) * (d4 + 4) : 16);
        const size_t o_fx = take(fx_on ? sizeof(long long) * (size_t)n_copies * (size_t)(p.k * d4 + p.k)
                                       : 16);
        const size_t o_cst = take(sizeof(MixedConsts));
        // candidate masks (and best scores) of every column pass
        const size_t o_cand = take(sizeof(uint4) * (size_t)p.n * passes);
        const size_t o_pmax = take(passes > 1 ? sizeof(float) * (size_t)p.n * passes : 16);
        const size_t o_flg = take(sizeof(int) * p.n);
        const size_t o_cnt = take(sizeof(int) * 4);
        const size_t o_st = take(sizeof(long long) * 2);
        KMC_TRY(mws.alloc(off, s));
        char *b = mws.as<char>();
        ximg = reinterpret_cast<uint8_t *>(b + o_x);
        cimg = reinterpret_cast<uint8_t *>(b + o_c);
        ct = reinterpret_cast<float *>(b + o_ct);
        nx = reinterpret_cast<float *>(b + o_nx);
        ndx = reinterpret_cast<float *>(b + o_ndx);
        sums32 = reinterpret_cast<float *>(b + o_s32);
        acc64 = reinterpret_cast<double *>(b + o_a64);
        xrow = reinterpret_cast<float *>(b + o_xf);
        xq = reinterpret_cast<int *>(b + o_xq);
        fxsum = reinterpret_cast<unsigned long long *>(b + o_fx);
        consts = reinterpret_cast<MixedConsts *>(b + o_cst);
        cand = reinterpret_cast<uint4 *>(b + o_cand);
        pmax = reinterpret_cast<float *>(b + o_pmax);
        flagged = reinterpret_cast<int *>(b + o_flg);
        n_flagged = reinterpret_cast<int *>(b + o_cnt);
        err_dev = n_flagged + 1;
        stats = reinterpret_cast<long long *>(b + o_st);
        KMC_CUDA_TRY(cudaMemsetAsync(consts, 0, sizeof(MixedConsts), s));
        if (p.w != nullptr) {
            // the sums start at zero; each iteration's end leaves them so
            KMC_CUDA_TRY(cudaMemsetAsync(b + o_s32, 0, o_xf - o_s32, s));
            KMC_CUDA_TRY(cudaMemsetAsync(b + o_fx, 0, o_cst - o_fx, s));
        }
        KMC_CUDA_TRY(cudaMemsetAsync(n_flagged, 0, sizeof(int) * 4, s));
        KMC_CUDA_TRY(cudaMemsetAsync(stats, 0, sizeof(long long) * 2, s));
        // one-time conversion of X (charged to the fit, reported separately)
        absmax_kernel<<<absmax_grid(p.n * p.d), kAbsmaxThreads, 0, s>>>(p.X, p.n * p.d,
                                                                       &consts->xmax_bits);
        KMC_TRY(check_launch("absmax"));
        sigma_kernel<<<1, 1, 0, s>>>(consts, bf16, p.d);
        KMC_TRY(check_launch("sigma"));
        if (fx_on) {
            absmax_kernel<<<absmax_grid(p.n), kAbsmaxThreads, 0, s>>>(p.w, p.n, &consts->wmax_bits);
            KMC_TRY(check_launch("absmax_w"));
            // rows that one copy of the sums adds up at most
            const int64_t g = sum_grid(), tile = sum_tile();
            const int64_t cta = ceil_div<int64_t>(p.n, g * tile) * tile;
            const double rows = (double)std::max<int64_t>(kTileM, std::min(p.n, ceil_div<int64_t>(g, n_copies) * cta));
            fixed_scale_kernel<<<1, 1, 0, s>>>(consts, rows);
            KMC_TRY(check_launch("fixed_scale"));
            this->launches += 2;
        }
        {
            auto xk = bf16 ? x_image_kernel<1> : x_image_kernel<0>;
            const size_t xsm = x_image_smem(nkb);
            if (xsm > 48 * 1024) KMC_TRY(allow_smem(xk, x_image_smem(kMaxFeatureBlocks)));
            const int64_t xg = std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)num_sms() * 8));
            xk<<<(unsigned)xg, kXImageThreads, xsm, s>>>(p.X, p.n, p.d, d4, nkb, ntiles, consts,
                                                         ximg, xrow, nx, ndx, p.x_rowmajor, p.w,
                                                         fx_on ? xq : nullptr);
        }
        KMC_TRY(check_launch("x_image"));
        this->launches += 3;
        return KMC_OK;
    }

    // the preparation is part of the assignment pass
    int begin_step(int64_t *n_launches) override {
        *n_launches = 0;
        return KMC_OK;
    }
    const float *c_rows(int64_t *stride) const override {
        *stride = d4;
        return ct;
    }

    int centroid_prep(const float *cur, const LoopState *guard) {
        const FitParams<float, I> &p = this->prm;
        const int lanes = nkb <= 1 ? 8 : (nkb == 2 ? 16 : 32);
        auto kern = bf16 ? mixed_prep_kernel<1> : mixed_prep_kernel<0>;
        return launch_chained("mixed_prep", kern, dim3((unsigned)(k_pad / kPrepRows)),
                              dim3((unsigned)(lanes * kPrepRows)), 0, p.stream, cur, p.d, p.k, k_pad,
                              nkb, consts, cimg, this->hn, ct, d4, n_flagged, guard);
    }

    // enough CTAs for every sample flagged (8 warps of 32 per CTA round), at
    // most 8 per SM
    int64_t recheck_grid() const {
        return std::max<int64_t>(1, std::min<int64_t>((int64_t)num_sms() * 8,
                                                      ceil_div<int64_t>(this->prm.n, kRecheckThreads)));
    }

    int assign_pass(const float *cur, const LoopState *guard) {
        const FitParams<float, I> &p = this->prm;
        cudaStream_t s = p.stream;
        KMC_TRY(centroid_prep(cur, guard));
        MixedArgs a;
        a.ximg = ximg;
        a.cimg = cimg;
        a.nx = nx;
        a.ndx = ndx;
        a.consts = consts;
        a.labels = p.labels;
        a.flagged = flagged;
        a.n_flagged = n_flagged;
        a.err_global = err_dev;
        a.guard = guard;
        a.n = p.n;
        a.label64 = sizeof(I) == 8 ? 1 : 0;
        a.stages = stages;
        a.wait_limit = this->wait_limit;
        a.stall = stall_once;
        a.state = this->state;
        stall_once = 0;
        const int64_t pass_cols = (int64_t)nch * kChunkN;
        a.k_img = k_pad;
        a.last_k = (int)ceil_div<int64_t>(std::max<int64_t>(p.d, 1) - 64 * (nkb - 1), 16);
        const bool multi = passes > 1;
        const SmemLayout L = smem_layout(nkb, pass_cols, stages);
        auto kern = pick_kernel(bf16, nkb, nch, multi);
        if (kern == nullptr) {
            set_error("mixed form: no kernel for %d feature blocks and %d chunks", nkb, nch);
            return KMC_ERR_UNSUPPORTED;
        }
        KMC_TRY(allow_smem(kern, kSmemLimit));
        const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(ntiles, num_sms()));
        if (p.n > 0) {
            for (int ps = 0; ps < passes; ++ps) {
                a.col0 = (int64_t)ps * pass_cols;
                a.cand = cand + (int64_t)ps * p.n;
                a.pmax = pmax + (multi ? (int64_t)ps * p.n : 0);
                KMC_TRY(launch_chained("mixed_assign", kern, dim3((unsigned)grid), dim3(kThreadsMixed),
                                       L.total, s, a));
                a.stall = 0;
            }
            if (multi) {
                combine_kernel<<<grid1d(p.n, 256, num_sms() * 8), 256, 0, s>>>(
                    pmax, cand, passes, pass_cols, nx, ndx, consts, p.labels, a.label64, flagged,
                    n_flagged, p.n, p.k, guard);
                KMC_TRY(check_launch("mixed_combine"));
            }
        }
        return launch_chained("mixed_recheck", recheck_kernel, dim3((unsigned)recheck_grid()),
                              dim3(kRecheckThreads), 0, s, xrow, ct, this->hn, cand, flagged,
                              n_flagged, p.n, p.d, p.k, d4, p.labels, a.label64, guard, passes,
                              pass_cols, stats);
    }

    // The sums' kernel: CTAs, samples of a CTA's tile, rounds of tiles.  The
    // sorted one has all of its CTAs resident (kSortCtas per SM, whose shared
    // memory sort_rows keeps within an SM's) and gives them equal rounds; the
    // direct ones, beyond kSortClusters, take 256 samples at a time.
    bool sums_sorted() const { return this->prm.k <= kSortClusters; }
    int64_t sum_grid() const {
        const int64_t n = std::max<int64_t>(this->prm.n, 1);
        const int64_t most = (int64_t)num_sms() * (sums_sorted() ? kSortCtas : 8);
        return std::min(most, ceil_div<int64_t>(n, kSumThreads));
    }
    int sum_tile() const {
        if (!sums_sorted()) return kSumThreads;
        const int64_t n = std::max<int64_t>(this->prm.n, 1), g = sum_grid();
        const int64_t rounds = ceil_div<int64_t>(n, g * sort_rows(this->prm.k));
        return (int)(ceil_div<int64_t>(n, g * rounds * 32) * 32);
    }

    int sum_pass(const LoopState *guard) {
        const FitParams<float, I> &p = this->prm;
        if (sums_sorted()) {
            const int tile = sum_tile();
            auto kern = !acc_f64 ? sum_sorted_kernel<I, 0>
                                 : (variant % 10 == 2 ? sum_sorted_kernel<I, 2> : sum_sorted_kernel<I, 4>);
            const size_t smem = sort_smem(tile, p.k);
            if (smem > 48 * 1024) KMC_TRY(allow_smem(kern, kSortSmem));
            return launch_chained("mixed_sums", kern, dim3((unsigned)sum_grid()), dim3(kSumThreads), smem,
                                  p.stream, xrow, p.w, p.labels, p.n, d4, p.k, k_pad, tile, sums32,
                                  fx_acc(), acc64, n_copies, consts, guard);
        }
        const unsigned grid = (unsigned)sum_grid();
        if (acc_f64) {
            auto kern = variant % 10 == 2 ? sum_terms_kernel<I, 2> : sum_terms_kernel<I, 4>;
            kern<<<grid, kSumThreads, 0, p.stream>>>(xrow, p.w, p.labels, p.n, d4, p.k, k_pad, fx_acc(),
                                                     acc64, n_copies, consts, guard);
        } else {
            sum_rows_kernel<I><<<grid, kSumThreads, 0, p.stream>>>(xrow, p.w, p.labels, p.n, d4, p.k,
                                                                   k_pad, sums32, n_copies, guard);
        }
        return check_launch("mixed_sums");
    }

    int step_assign_and_accumulate(const float *cur, int64_t *n_launches) override {
        *n_launches = 4 + (passes > 1 ? passes : 0);
        KMC_TRY(assign_pass(cur, this->state));
        return sum_pass(this->state);
    }

    int finish_step(int64_t *n_launches) override {
        const FitParams<float, I> &p = this->prm;
        if (acc_f64) {
            const MixedSums<double> src{acc64, n_copies, p.k, k_pad, d4, fx_acc(), consts};
            return launch_reduce_and_finish<float>(src, n_copies, this->finish_args(), n_launches,
                                                   p.stream);
        }
        const MixedSums<float> src{sums32, n_copies, p.k, k_pad, d4,
                                   FxAcc{nullptr, nullptr, 0, 1, nullptr}, consts};
        return launch_reduce_and_finish<float>(src, n_copies, this->finish_args(), n_launches,
                                               p.stream);
    }

    int final_assignment() override { return assign_pass(this->prm.centroids, nullptr); }

    int counters(int64_t *last, int64_t *total, int *device_error) override {
        long long h[2] = {0, 0};
        int e = 0;
        KMC_CUDA_TRY(cudaMemcpyAsync(h, stats, sizeof(h), cudaMemcpyDeviceToHost,
                                     this->prm.stream));
        KMC_CUDA_TRY(cudaMemcpyAsync(&e, err_dev, sizeof(int), cudaMemcpyDeviceToHost,
                                     this->prm.stream));
        KMC_CUDA_TRY(cudaStreamSynchronize(this->prm.stream));
        int reloc = 0;  // a relocation's wait
        KMC_TRY(Base::counters(nullptr, nullptr, &reloc));
        if (last) *last = h[0];
        if (total) *total = h[1];
        if (device_error) *device_error = e != 0 || reloc != 0;
        return KMC_OK;
    }
};

template <typename I>
int make_mixed_fit_impl(const FitParams<float, I> &p, int form, std::unique_ptr<FitBase> *out) {
    if (!MixedFit<I>::supported(p.d, p.k)) {
        set_error("mixed form supports n_features <= %d (got d=%lld, k=%lld)",
                  64 * kMaxFeatureBlocks, (long long)p.d, (long long)p.k);
        return KMC_ERR_UNSUPPORTED;
    }
    auto f = std::make_unique<MixedFit<I>>();
    KMC_TRY(f->init(p));
    KMC_TRY(f->init_mixed(form));
    *out = std::move(f);
    return KMC_OK;
}

template <typename T, typename I>
int make_mixed_fit(const FitParams<T, I> &p, int form, std::unique_ptr<FitBase> *out) {
    if constexpr (!std::is_same<T, float>::value) {
        set_error("the mixed tensor-core form needs float32 data");
        return KMC_ERR_UNSUPPORTED;
    } else {
        return make_mixed_fit_impl<I>(p, form, out);
    }
}

void mixed_tuning_lookup_only(bool on) { tl_mixed_lookup_only = on; }

int force_mixed_variant(int code) {
    KMC_CHECK_ARG(code == -1 || (code >= 10 && code <= 44), "variant must be -1 or 10 s + f");
    g_force_mixed_variant.store(code);
    return KMC_OK;
}

int mixed_variant_of(FitBase *fit, int *code) {
    auto *m32 = dynamic_cast<MixedFit<int32_t> *>(fit);
    auto *m64 = dynamic_cast<MixedFit<int64_t> *>(fit);
    *code = m32 ? m32->variant : (m64 ? m64->variant : -1);
    return KMC_OK;
}

bool mixed_fit_supported(int64_t d, int64_t k) { return MixedFit<int32_t>::supported(d, k); }

int pack_fixed_term(float v, int shift) { return pack_fixed(v, 150 - shift); }

template int make_mixed_fit<float, int32_t>(const FitParams<float, int32_t> &, int,
                                            std::unique_ptr<FitBase> *);
template int make_mixed_fit<float, int64_t>(const FitParams<float, int64_t> &, int,
                                            std::unique_ptr<FitBase> *);
template int make_mixed_fit<double, int32_t>(const FitParams<double, int32_t> &, int,
                                             std::unique_ptr<FitBase> *);
template int make_mixed_fit<double, int64_t>(const FitParams<double, int64_t> &, int,
                                             std::unique_ptr<FitBase> *);

}  // namespace kmc
