// Local dV sandwich of the plain (FP64) form on the tensor cores.
//
//   g[nu][m][n] = (1/M) sum_{s,r} a(nu m; s r) conj(psi_kq,n,s(r)),
//   a(nu m; s r) = sum_s' dV_nu^{s s'}(r) psi_k,m,s'(r)
// (the real-space sandwich, see sandwich.cu) with every product of the sum
// exact: a, formed in FP64, and psi_kq are taken to 63-bit fixed point under a
// power-of-two scale per (mode, band) row and per band, cut into seven signed
// base-512 digits, and the digit products are formed by f16 MMAs, whose FP32
// accumulators hold integers below 2^24 exactly (the error-free matrix product
// of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012, on a fixed
// digit grid).  Digits i of a and j of psi go into the accumulator of level
// i + j, weight 512^-(i+j); the 28 products with i + j <= 6 are formed, the rest
// lie below 2^-63 of the scales' product.  Every 32 points the levels are
// drained: 0 to 3 into 64-bit integers (exact), 4 to 6 -- 2^-36 and less of the
// leading level -- into an FP32 sum.
//
// The scales are those of the CTA's K chunk, from exponents kept per four points
// of psi and of dV: a band's from its largest |psi|, a row's from the largest
// |dV| |psi| at the same four points (not the product of the two maxima, which a
// dV on one atom and a psi on another never reach).  An element about 2^6 below its
// row's largest in the chunk is cut off at one FP64 rounding of its own; what is
// smaller loses more, but below the rounding that the transforms of psi and dV leave
// at every point.  (Measured against scales from the two maxima: error 8.4e-16 ->
// 5.3e-16 on the 4-atom cell with its dV on one atom, 3.1e-8 -> 1.5e-8 where the bands
// lie elsewhere and the elements are 1e-10 of max |dV|; the time: at the prologue.)
//
// What bounds it: the FP64 products a (four operations an element; GB300 issues
// about two per cycle and SM), then the integer work of the digits; the MMAs take
// a third of that time.  The SIMT kernel that this replaces did the whole
// contraction on the FP64 pipe (8 nb flops per element instead of 6).
// Measured, SIMT -> this: 64 pairs of 384 rows x 32 bands x 27,648 points, 176 ->
// 11.3 ms; 64 pairs of 48 x 8 x 5,832, 12.6 -> 0.36 ms; error against 64 bits
// (norm) 5.5e-15 -> 1.9e-15 and 3.4e-15 -> 0.86e-15.  (With 16 warps instead of 32:
// 12.5 and 0.41 ms; the FP64 pipe is busy 45 % of the time, the rest is latency
// between the barriers.  Forming part of the next stage's products between the digit
// stores: no change; two rows at a time in straight-line code: 3 % slower.)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lelph_common.cuh"
#include "lelph_internal.h"
#include "tc_operands.cuh"

#define OZ_S 7        // digits
#define OZ_THREADS 1024
#define OZ_WARPS (OZ_THREADS / 32)
#define OZ_ROWS 128   // (mode, band of k) rows of a tile
#define OZ_BANDS 32   // bands of k+q of a tile
#define OZ_PTS 32     // grid points of a stage (one 128-byte K atom of (re, im) digits)
#define OZ_RPW (OZ_ROWS / OZ_WARPS)
#define OZ_BPW (OZ_BANDS / OZ_WARPS)
#define OZ_SUM 60000   // stages that the 64-bit sums hold (a stage adds less than 2^47 + 2^41)
#define OZ_COLS (2 * OZ_BANDS / (OZ_WARPS / 4))  // accumulator columns of a thread (its row of the tile)

// (One 24-byte record a row: with the exponent in an array of its own the compiler ordered
// the loads of two components, nmag 4, so that the kernel took 16 % longer.)
struct OzRow
{
    const double2* psi;  // component 0 of the row's band of k (null: no such row)
    const double2* dv;   // component 0 of its mode's window
    int e;               // exponent of the row's scale
};
struct OzSmem
{
    OzRow row[OZ_ROWS];
    const double2* bpsi[OZ_BANDS];
    int be[OZ_BANDS];                           // exponents of the bands' scales
    int badrow[OZ_ROWS], badband[OZ_BANDS];  // met an infinity or a NaN
    uint64_t bar;
    uint32_t tmem;
};

// |x| 2^e < 1 as a signed 63-bit fixed-point number (units of 2^-62), truncated
__device__ __forceinline__ long long oz_fixed(double x, int e, bool& bad)
{
    const long long b = __double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    bad |= ex == 0x7ff;
    const unsigned long long m = (((unsigned long long)b << 10) & 0x3ffffffffffffc00ull) | (1ull << 62);
    const int d = 1023 - ex - e;  // m = 2^62 1.f, x 2^e 2^62 = m 2^-d
    const long long v = (ex == 0 || d > 62) ? 0 : (long long)(m >> (d < 1 ? 1 : d));
    return b < 0 ? -v : v;
}

// sum_j 256 512^j: t = v + OZ_BIAS has the digits + 256 as plain base-512 digits
#define OZ_BIAS 0x4020100804020100ull

__device__ __forceinline__ uint32_t oz_digits(unsigned long long tr, unsigned long long ti, int j)
{
    // 0x6400 | u is the half 1024 + u for u < 1024; minus 1280: u - 256, exact
    const uint32_t u = ((uint32_t)(tr >> (9 * j)) & 511u) | (((uint32_t)(ti >> (9 * j)) & 511u) << 16) | 0x64006400u;
    const __half2 h = __hadd2(*reinterpret_cast<const __half2*>(&u), __floats2half2_rn(-1280.f, -1280.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

#define OZ_NO_EXP (-16384)  // four points without a normal finite number
#define OZ_NO_EXP2 0xc000c000u  // two of them

// Limits below the suspend hint of mbar_wait_bounded poll instead: a suspended wait sleeps
// past them, and the MMAs of a stage (a microsecond) then always complete first.
__device__ __forceinline__ bool oz_wait(uint64_t* bar, uint32_t parity, unsigned long long limit_ns)
{
    if (limit_ns >= 20000ull) return mbar_wait_bounded(bar, parity, limit_ns);
    const unsigned long long t0 = gtimer_ns();
    while (!mbar_test_wait(bar, parity))
        if (gtimer_ns() - t0 > limit_ns) return false;
    return true;
}

// One CTA: one (pair, spin), 128 rows x up to 32 bands, one K chunk of the stages
// stage0 .. nstage_total - 1; add: to what an earlier launch left in out.
// grid: (mode-row tiles x band tiles, pair * nspin, K chunks)
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_local_oz(const PairInfo* __restrict__ pairs, const double2* __restrict__ psi, const short* __restrict__ epsi,
               const double2* __restrict__ dV, const short* __restrict__ edv, GeomDev gd, int ntn, int stage0,
               int nstage_total, int stages_per_chunk, int add, double scale, long long chunk_stride, double* __restrict__ out,
               unsigned* __restrict__ status, unsigned long long wait_ns)
{
    extern __shared__ __align__(1024) uint8_t smraw[];
    uint8_t* sm = smraw + ((1024u - (smem_u32(smraw) & 1023u)) & 1023u);
    const int nb = gd.nbnds, nrows = gd.nmodes * nb;
    const int mt = blockIdx.x / ntn, nt = blockIdx.x - mt * ntn;
    const int zp = blockIdx.y;
    const int pair = zp / gd.nspin, spin = zp - pair * gd.nspin;
    const PairInfo P = pairs[pair];
    const int n0 = nt * OZ_BANDS, nbt = min(OZ_BANDS, nb - n0);
    const int nbp = (nbt + 7) / 8 * 8, NT = 2 * nbp;
    const long long M = lelph_grid_points(gd);
    const long long Ktot = (long long)gd.nspinor * M;
    uint8_t* sA = sm;                                  // [digit][128 rows][128 bytes], swizzled
    uint8_t* sB = sA + OZ_S * OZ_ROWS * 128;           // [digit][NT rows][128 bytes]
    OzSmem& ss = *reinterpret_cast<OzSmem*>(sB + OZ_S * 2 * OZ_BANDS * 128);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    for (int r = threadIdx.x; r < OZ_ROWS; r += OZ_THREADS)
    {
        const int R = mt * OZ_ROWS + r;
        const double2 *rp = nullptr, *rd = nullptr;
        if (R < nrows)
        {
            const int nu = R / nb, m = R - nu * nb;
            rp = psi + (((size_t)P.kbz_k * gd.nspin + spin) * nb + m) * gd.nspinor * M;
            rd = dV + ((size_t)P.dvslot * gd.nmodes + nu) * gd.nmag * M + (gd.nmag == 2 ? (size_t)spin * M : 0);
        }
        ss.row[r].psi = rp;
        ss.row[r].dv = rd;  // (e comes from the warp that finds it, below)
        ss.badrow[r] = 0;
    }
    for (int b = threadIdx.x; b < OZ_BANDS; b += OZ_THREADS)
    {
        const size_t idx = ((size_t)P.kbz_kq * gd.nspin + spin) * nb + n0 + b;
        ss.bpsi[b] = b < nbt ? psi + idx * gd.nspinor * M : nullptr;
        ss.badband[b] = 0;
    }
    const int st0 = stage0 + blockIdx.z * stages_per_chunk;
    const int nst = min(stages_per_chunk, nstage_total - st0);
    // scales of the chunk: eight exponents (32 points) a 16-byte word, eight lanes a row or band,
    // four words in flight.  What they cost: 50 (pair, spin)s of 27 rows x 3 bands x 4,608 points
    // 211 -> 213 us, 27 pairs of 240 x 20 x 11,664 1278 -> 1296 (a warp a row 1308), 125 of 72 x 12
    // with nmag 4 3082 -> 3134, 64 of 384 x 32 x 27,648 within 0.4 %.  (The tensor memory is
    // allocated after them: before, its wait for the last CTA's added 3 us.)
    {
        const long long k0 = (long long)st0 * OZ_PTS, k1 = min(Ktot, k0 + (long long)nst * OZ_PTS);
        const unsigned wpc = (unsigned)((M + 31) / 32);  // words of a component
        const int lo = (int)(k0 >= M ? 1 : 0), hi = (int)(k1 > M ? 1 : 0);
        const int nrt = min(OZ_ROWS, nrows - mt * OZ_ROWS), total = nrt + nbt;
        const int nc = gd.nmag == 4 ? 2 : 1;
        for (int i0 = 4 * warp; i0 < total; i0 += 4 * OZ_WARPS)
        {
            const int i = i0 + (lane >> 3);
            const bool row = i < nrt;
            unsigned mx = 0x80008000u;
            if (i < total)
            {
                const int R = mt * OZ_ROWS + i, nu = row ? R / nb : 0, band = row ? R - nu * nb : n0 + i - nrt;
                const uint4* p = reinterpret_cast<const uint4*>(epsi) +
                                 (size_t)(((row ? P.kbz_k : P.kbz_kq) * gd.nspin + spin) * nb + band) * (gd.nspinor * wpc);
                const uint4* d = reinterpret_cast<const uint4*>(edv) +
                                 (size_t)(P.dvslot * gd.nmodes + nu) * (gd.nmag * wpc) + (gd.nmag == 2 ? spin * wpc : 0u);
                for (int s = lo; s <= hi; ++s)
                {
                    const unsigned w0 = s == lo ? (unsigned)((k0 - s * M) >> 5) : 0u;
                    const unsigned w1 = s == hi ? (unsigned)((k1 - s * M + 31) >> 5) : wpc;
                    for (int c = 0; c < (row ? nc : 1); ++c)
                    {
                        const uint4* pc = p + (row && nc == 2 ? c : s) * wpc;
                        const uint4* dc = d + (nc == 2 ? (2 * s + c) * wpc : 0u);
                        for (unsigned w = w0 + (lane & 7); w < w1; w += 32)
                        {
                            uint4 x[4], y[4];  // four words of each in flight
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                            {
                                const bool in = w + 8 * u < w1;
                                x[u] = in ? pc[w + 8 * u] : make_uint4(OZ_NO_EXP2, OZ_NO_EXP2, OZ_NO_EXP2, OZ_NO_EXP2);
                                y[u] = in && row ? dc[w + 8 * u] : make_uint4(0u, 0u, 0u, 0u);
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                            {
                                mx = __viaddmax_s16x2(x[u].x, y[u].x, mx);
                                mx = __viaddmax_s16x2(x[u].y, y[u].y, mx);
                                mx = __viaddmax_s16x2(x[u].z, y[u].z, mx);
                                mx = __viaddmax_s16x2(x[u].w, y[u].w, mx);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) mx = __vmaxs2(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const int m = max((int)(short)(mx & 0xffffu), (int)(short)(mx >> 16));
            // |re|, |im| < 2^(E+1) of either factor: |dV psi| < 2^(Ed+Ep+3), a sum of two (nmag 4)
            // twice that; scaled below 1/2
            const int e = m < OZ_NO_EXP / 2 ? 0 : -(m + (!row ? 2 : 3 + nc));
            if ((lane & 7) == 0 && i < total) (row ? ss.row[i].e : ss.be[i - nrt]) = e;
        }
    }
    if (threadIdx.x == 0)
    {
        mbar_init(&ss.bar, 1);
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&ss.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ss.tmem;

    long long ar[OZ_RPW], ai[OZ_RPW], br[OZ_BPW], bi[OZ_BPW];
    // fixed-point values of stage st: this lane's point of the warp's rows and bands
    auto form = [&](int st) {
        const long long kc = (long long)(st0 + st) * OZ_PTS + lane;
        const bool in = kc < Ktot;
        const int s = kc >= M ? 1 : 0;
        const long long r = kc - s * M;
#pragma unroll
        for (int i = 0; i < OZ_RPW; ++i)
        {
            const OzRow w = ss.row[warp + i * OZ_WARPS];
            ar[i] = ai[i] = 0;
            if (w.psi && in)
            {
                double2 a;
                if (gd.nmag == 4)
                {
                    const double2* d = w.dv + 2 * s * M + r;
                    a = cadd(cmul(d[0], w.psi[r]), cmul(d[M], w.psi[M + r]));
                }
                else
                    a = cmul(w.dv[r], w.psi[kc]);
                bool bad = false;
                ar[i] = oz_fixed(a.x, w.e, bad);
                ai[i] = oz_fixed(a.y, w.e, bad);
                if (bad) ss.badrow[warp + i * OZ_WARPS] = 1;
            }
        }
#pragma unroll
        for (int i = 0; i < OZ_BPW; ++i)
        {
            const int b = warp + i * OZ_WARPS;
            const double2* p = ss.bpsi[b];
            br[i] = bi[i] = 0;
            if (p && in)
            {
                const double2 v = p[kc];
                bool bad = false;
                br[i] = oz_fixed(v.x, ss.be[b], bad);
                bi[i] = oz_fixed(v.y, ss.be[b], bad);
                if (bad) ss.badband[b] = 1;
            }
        }
    };
    // digits to shared memory: row r of digit d, the lane's (re, im) word in the swizzled 16-byte chunks
    auto store = [&]() {
        const uint32_t wofs = (uint32_t)(lane & 3) * 4;
#pragma unroll
        for (int i = 0; i < OZ_RPW; ++i)
        {
            const int r = warp + i * OZ_WARPS;
            if (mt * OZ_ROWS + r >= nrows) break;
            uint8_t* p = sA + tc_swz128(r, lane >> 2) + wofs;
            const unsigned long long tr = (unsigned long long)ar[i] + OZ_BIAS, ti = (unsigned long long)ai[i] + OZ_BIAS;
#pragma unroll
            for (int d = 0; d < OZ_S; ++d)
                *reinterpret_cast<uint32_t*>(p + d * (OZ_ROWS * 128)) = oz_digits(tr, ti, OZ_S - 1 - d);
        }
#pragma unroll
        for (int i = 0; i < OZ_BPW; ++i)
        {
            const int b = warp + i * OZ_WARPS;
            if (b >= nbt) break;
            // row b: (Re, Im); row nbp + b: (-Im, Re)
            uint8_t* p = sB + tc_swz128(b, lane >> 2) + wofs;
            uint8_t* q = sB + tc_swz128(nbp + b, lane >> 2) + wofs;
            const unsigned long long tr = (unsigned long long)br[i] + OZ_BIAS, ti = (unsigned long long)bi[i] + OZ_BIAS;
#pragma unroll
            for (int d = 0; d < OZ_S; ++d)
            {
                const uint32_t w = oz_digits(tr, ti, OZ_S - 1 - d);
                *reinterpret_cast<uint32_t*>(p + d * (NT * 128)) = w;
                *reinterpret_cast<uint32_t*>(q + d * (NT * 128)) = __byte_perm(w, 0, 0x1032) ^ 0x00008000u;
            }
        }
    };
    // this thread's OZ_COLS columns of its row: levels 0..3 exactly, 4..6 in FP32
    const int cg = warp >> 2;
    const bool mine = cg * OZ_COLS < NT;
    long long H[OZ_COLS];
    float L[OZ_COLS];
#pragma unroll
    for (int c = 0; c < OZ_COLS; ++c)
    {
        H[c] = 0;
        L[c] = 0.f;
    }
    auto drain = [&]() {
        if (mine)
        {
            const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(cg * OZ_COLS);
            float v[OZ_COLS];
#pragma unroll
            for (int l = 0; l < 4; ++l)
            {
                tmem_ld8(ta + (uint32_t)(l * NT), v);
#pragma unroll
                for (int c = 0; c < OZ_COLS; ++c)
                    H[c] += (long long)__float2int_rn(v[c]) * (long long)(1 << (27 - 9 * l));
            }
#pragma unroll
            for (int l = 4; l < OZ_S; ++l)
            {
                tmem_ld8(ta + (uint32_t)(l * NT), v);
                const float w = l == 4 ? 1.f : (l == 5 ? 0x1p-9f : 0x1p-18f);
#pragma unroll
                for (int c = 0; c < OZ_COLS; ++c) L[c] = fmaf(v[c], w, L[c]);
            }
        }
        tc_fence_before();
    };

    form(0);
    bool ok = true;
    int last = nst - 1;  // last stage issued
    for (int st = 0; st < nst; ++st)
    {
        if (st > 0)
        {
            // the MMAs of the previous stage: accumulators complete, operand tiles free
            ok = oz_wait(&ss.bar, (uint32_t)(st - 1) & 1u, wait_ns);
            if (__syncthreads_or(!ok))
            {
                ok = false;
                last = st - 1;
                break;
            }
            tc_fence_after();
            drain();
        }
        store();
        fence_proxy_async_smem();
        __syncthreads();
        if (threadIdx.x == 0)
        {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int d = 0; d < OZ_S; ++d)
                {
                    // digit d of a against digits 0 .. 6 - d of psi: levels d .. 6
                    const uint64_t ad = umma_desc_sw128(a0 + (uint32_t)(d * OZ_ROWS * 128) + 32u * k);
                    const uint32_t en = (k == 0 && d == 0) ? 0u : 1u;
                    const int nn = (OZ_S - d) * NT;
                    for (int c = 0; c < nn; c += 256)
                        umma_f16(tmem + (uint32_t)(d * NT + c), ad,
                                 umma_desc_sw128(b0 + (uint32_t)(c * 128) + 32u * k),
                                 umma_idesc_f16(0u, 128u, (uint32_t)min(256, nn - c)), en);
                }
            umma_commit(&ss.bar);
        }
        if (st + 1 < nst) form(st + 1);
    }
    if (ok)
    {
        ok = oz_wait(&ss.bar, (uint32_t)(nst - 1) & 1u, wait_ns);
        ok = !__syncthreads_or(!ok);
    }
    if (ok)
    {
        tc_fence_after();
        drain();
        const int r = (warp & 3) * 32 + lane, R = mt * OZ_ROWS + r;
        if (mine && R < nrows)
        {
            const bool bad = ss.badrow[r] != 0;
            double* o = out + (size_t)blockIdx.z * chunk_stride + 2 * ((size_t)zp * nrows + R) * nb;
#pragma unroll
            for (int c = 0; c < OZ_COLS; ++c)
            {
                const int col = cg * OZ_COLS + c, im = col >= nbp, b = im ? col - nbp : col;
                if (b >= nbt) continue;
                // (H 2^27 + L 2^18) units of 2^(54 - 124) of the two scales' product
                double v = fma((double)H[c], 0x1p27, (double)L[c] * 0x1p18);
                v = scalbn(v, -70 - ss.row[r].e - ss.be[b]) * scale;
                if (add) v += o[2 * (n0 + b) + im];
                o[2 * (n0 + b) + im] = (bad || ss.badband[b]) ? __longlong_as_double(0x7ff8000000000000ll) : v;
            }
        }
    }
    else
    {
        // a wait ran out: let the MMAs in flight finish before the tensor memory is released
        if (threadIdx.x == 0) atomicOr(status, LELPH_DEV_ERR_TIMEOUT);
        mbar_wait_bounded(&ss.bar, (uint32_t)last & 1u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
    {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// Exponents of every four points of each row (component) of M complex numbers:
// E of the largest |finite re or im| in [2^E, 2^(E+1)), OZ_NO_EXP where there is
// none.  Infinities and NaN do not count: the products that they enter are marked
// as such, and the row's other products keep a scale that holds them.  A row takes
// M rounded up to 32 points.  The exponent fields alone are compared (integer
// instructions: no FP64 work); reading the numbers bounds it.
__global__ void __launch_bounds__(256) k_oz_exponents(const double2* __restrict__ x, long long nrows, long long M,
                                                      short* __restrict__ e)
{
    const long long per = (M + 31) / 32, ng = nrows * per;
    const int lane = threadIdx.x & 31;
    for (long long g = blockIdx.x * 8ll + (threadIdx.x >> 5); g < ng; g += gridDim.x * 8ll)
    {
        const long long row = g / per, r = (g - row * per) * 32 + lane;
        unsigned m = 0;
        if (r < M)
        {
            const double2 v = x[row * M + r];
            const unsigned a = (unsigned)__double2hiint(v.x) & 0x7fffffffu, b = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
            if (a < 0x7ff00000u) m = a;
            if (b < 0x7ff00000u) m = max(m, b);
        }
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
        if ((lane & 3) == 0) e[g * 8 + (lane >> 2)] = (short)(m >> 20 ? (int)(m >> 20) - 1023 : OZ_NO_EXP);
    }
}

size_t lelph_oz_exponent_bytes(long long nrows, long long M) { return sizeof(short) * 8 * (size_t)nrows * ((M + 31) / 32); }

void lelph_launch_oz_exponents(const double2* x, long long nrows, long long M, short* e, cudaStream_t st)
{
    const long long blocks = (nrows * ((M + 31) / 32) + 7) / 8;
    if (blocks > 0) k_oz_exponents<<<(unsigned)std::min<long long>(blocks, 152 * 64), 256, 0, st>>>(x, nrows, M, e);
}

// K chunks of a launch: enough CTAs for about sixteen rounds over the chip (the
// last, partly filled round then costs a few percent) in chunks of at least 24
// stages (prologue and drain), within the partial-sum space.
int lelph_local_fp64_chunks(int npairs, const GeomDev& g, size_t part_bytes)
{
    const long long nst = (g.nspinor * lelph_grid_points(g) + OZ_PTS - 1) / OZ_PTS;
    const long long nrows = (long long)g.nmodes * g.nbnds;
    const long long units = (long long)npairs * g.nspin * ((nrows + OZ_ROWS - 1) / OZ_ROWS) *
                            ((g.nbnds + OZ_BANDS - 1) / OZ_BANDS);
    const size_t one = sizeof(double2) * (size_t)npairs * g.nspin * nrows * g.nbnds;
    long long n = std::min<long long>((16 * 152 + units - 1) / units, nst / 24);
    n = std::min<long long>(n, (long long)(part_bytes / std::max<size_t>(1, one)));
    return (int)std::max<long long>(1, std::min<long long>(n, 1024));
}

int lelph_launch_local_fp64(const PairInfo* pairs, int npairs, const double2* psi, const short* epsi, const double2* dV,
                            const short* edv, const GeomDev& g, int nchunks, double2* part, double2* glocal,
                            unsigned* status, unsigned long long wait_ns, cudaStream_t st)
{
    if (wait_ns == 0) wait_ns = LELPH_WAIT_LIMIT_NS;
    const long long nst = (g.nspinor * lelph_grid_points(g) + OZ_PTS - 1) / OZ_PTS;
    const int nrows = g.nmodes * g.nbnds;
    const int ntm = (nrows + OZ_ROWS - 1) / OZ_ROWS, ntn = (g.nbnds + OZ_BANDS - 1) / OZ_BANDS;
    const int smem = OZ_S * (OZ_ROWS + 2 * OZ_BANDS) * 128 + (int)sizeof(OzSmem) + 1024;
    if (lelph_smem_opt_in<k_local_oz>(smem, smem) != cudaSuccess) return -1;
    const double invM = 1.0 / (double)lelph_grid_points(g);
    const long long nel = (long long)npairs * g.nspin * nrows * g.nbnds;
    // chunks of more than OZ_SUM stages go in several launches, each adding to the last one's
    // sums; grid.y is limited to 65535 (pair, spin)s a launch
    const long long pass = std::min<long long>(nst, (long long)nchunks * OZ_SUM);
    const int per = (int)((pass + nchunks - 1) / nchunks);
    nchunks = (int)((pass + per - 1) / per);
    int launches = 0;
    for (long long s0 = 0; s0 < nst; s0 += pass)
        for (int z0 = 0; z0 < npairs * g.nspin; z0 += 65535 / g.nspin * g.nspin, ++launches)
        {
            const int nz = std::min(npairs * g.nspin - z0, 65535 / g.nspin * g.nspin);
            const int se = (int)std::min(nst, s0 + pass);
            const dim3 grid((unsigned)(ntm * ntn), (unsigned)nz, (unsigned)((se - s0 + per - 1) / per));
            double2* o = (nchunks > 1 ? part : glocal) + (size_t)z0 * nrows * g.nbnds;
            k_local_oz<<<grid, OZ_THREADS, smem, st>>>(pairs + z0 / g.nspin, psi, epsi, dV, edv, g, ntn, (int)s0, se, per,
                                                       s0 > 0, nchunks > 1 ? 1.0 : invM, 2 * nel, (double*)o, status,
                                                       wait_ns);
        }
    if (nchunks > 1) lelph_launch_gs_reduce(1, part, nel, nchunks, invM, glocal, st);
    return launches - 1 + (nchunks > 1 ? 1 : 0);
}
