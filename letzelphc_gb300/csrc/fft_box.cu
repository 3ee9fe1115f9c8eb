// Wavefunction boxes of the mixed form, one CTA per box: sphere coefficients in,
// tensor-core operands out, the 3-D inverse FFT in shared memory between them.
//
// For grids whose copies fit in shared memory with every length at most 32 (the
// interleaved grids of cells with up to about 30^3 points a copy).  Each thread
// transforms whole lines in registers, in place: z lines of the sphere's
// columns, y lines of its x planes (unoccupied columns read as zero), x lines,
// whose results go straight to the split k+q rows and the FP32 psi rows.  What
// bounds it is writing those (24 bytes a point); the multi-pass form
// (fft_gather.cu: scatter into cleared boxes, z, y and x passes over HBM) moved
// every box four more times.
// Measured for 512 k x 32 bands x 2 copies of 24^3: scatter 1.7 + z, y 3.8 + x pass
// 2.1 ms -> 1.2 (unfolding, FP64 pipe) + 2.8 ms (10.9 GB written: 58 % of the
// measured copy bandwidth); 432 k x 13 bands of 20^3: 0.81 -> 0.37 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fft_smem.cuh"
#include "lelph_common.cuh"
#include "lelph_internal.h"

#define FB_THREADS 256
#define FB_SMEM_LIMIT (226 * 1024)

// ------------------------------------------------------ line FFT in registers

template <int M, int L>
__device__ __forceinline__ float2 fb_twiddle(float2 x)
{
    constexpr int m = M % L;
    if constexpr (m == 0) return x;
    constexpr float c = (float)ct_trig(m, L, false), s = (float)ct_trig(m, L, true);
    return make_float2(x.x * c - x.y * s, x.x * s + x.y * c);
}

__host__ __device__ constexpr int fb_radix(int L)
{
    return L % 4 == 0 ? 4 : L % 5 == 0 ? 5 : L % 3 == 0 ? 3 : 2;
}

template <int N2, int K1, int R1, int R2, int L>
__device__ __forceinline__ void fb_twiddles(float2* t)
{
    if constexpr (N2 < R2)
    {
        t[K1 * R2 + N2] = fb_twiddle<N2 * K1, L>(t[K1 * R2 + N2]);
        if constexpr (K1 + 1 < R1) fb_twiddles<N2, K1 + 1, R1, R2, L>(t);
        else fb_twiddles<N2 + 1, 0, R1, R2, L>(t);
    }
}

// unnormalised inverse DFT (e^{+2 pi i n k / L}) of v[0 .. L)
template <int L>
__device__ __forceinline__ void fb_line(float2* v)
{
    constexpr int R1 = fb_radix(L), R2 = L / R1;
    if constexpr (R2 == 1)
        dft_base<float2, float, L>(v, 1);
    else
    {
        float2 t[L];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2)
        {
            float2 u[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) u[n1] = v[R2 * n1 + n2];
            dft_base<float2, float, R1>(u, 1);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) t[k1 * R2 + n2] = u[k1];
        }
        fb_twiddles<1, 1, R1, R2, L>(t);
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1)
        {
            fb_line<R2>(t + k1 * R2);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k1 * R2 + k2];
        }
    }
}

#define FB_SIZES(X) X(12) X(15) X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32)

static bool fb_length(int L)
{
    switch (L)
    {
#define FB_CASE(N) case N:
        FB_SIZES(FB_CASE)
#undef FB_CASE
        return true;
    default: return false;
    }
}

// Box in shared memory: element (x, y, z) at z SZ + x SX + y, SX and SZ odd, so
// that consecutive threads' lines (columns along y; rows (z, x); points along z)
// fall into distinct banks in all three passes.
struct FbLayout
{
    int SX, SZ;
    size_t bytes;
};
__host__ __device__ inline FbLayout fb_layout(const GeomDev& g)
{
    FbLayout L;
    L.SX = g.Ny | 1;
    L.SZ = (g.Nx * L.SX) | 1;
    L.bytes = sizeof(float2) * (size_t)g.Nz * L.SZ + 40 * sizeof(unsigned);
    return L;
}

bool lelph_box_fft_supported(const GeomDev& g)
{
    return fb_length(g.Nx) && fb_length(g.Ny) && fb_length(g.Nz) && fb_layout(g).bytes <= FB_SMEM_LIMIT &&
           g.nspinor * lelph_grid_points(g) < (1ll << 31);
}

// position in the shared box of every plane wave of every k, and the occupancy of the box
__global__ void __launch_bounds__(256) k_box_pos(const KPointSym* __restrict__ ks, const int* __restrict__ miller,
                                                 const long long* __restrict__ pw_off, const int* __restrict__ npw_arr,
                                                 const long long* __restrict__ chat_off, int nsets, GeomDev gd,
                                                 int* __restrict__ pos, BoxMask mk)
{
    const int k = blockIdx.y;
    const KPointSym s = ks[k];
    const int npw = npw_arr[s.ik];
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= npw) return;
    const int* n = miller + 3 * (pw_off[s.ik] + g);
    const int N[3] = {gd.Nx, gd.Ny, gd.Nz};
    int i[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
        i[r] = (s.W[3 * r] * n[0] + s.W[3 * r + 1] * n[1] + s.W[3 * r + 2] * n[2]) % N[r];
        if (i[r] < 0) i[r] += N[r];
    }
    const FbLayout L = fb_layout(gd);
    pos[chat_off[k] / nsets + g] = i[2] * L.SZ + i[0] * L.SX + i[1];
    mk.col[((size_t)k * gd.Nx + i[0]) * gd.Ny + i[1]] = 1;
    mk.xpl[(size_t)k * gd.Nx + i[0]] = 1;
}

template <int BF16>
__device__ __forceinline__ void fb_split(float a, float b, uint32_t& hi, uint32_t& lo)
{
    if (BF16)
    {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        float2 hf = __bfloat1622float2(h);
        __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
        hi = *reinterpret_cast<uint32_t*>(&h);
        lo = *reinterpret_cast<uint32_t*>(&l);
    }
    else
    {
        __half2 h = __floats2half2_rn(a, b);
        float2 hf = __half22float2(h);
        __half2 l = __floats2half2_rn(a - hf.x, b - hf.y);
        hi = *reinterpret_cast<uint32_t*>(&h);
        lo = *reinterpret_cast<uint32_t*>(&l);
    }
}

// one box per CTA: box = ((k nsets + set) nsub + copy); coef[copy]: the unfolded
// coefficients times the copy's shift phase, (k, set, plane wave) at chat_off
template <int BF16>
__global__ void __launch_bounds__(FB_THREADS, 2)
    k_box_fft_split(const float2* __restrict__ coef0, const float2* __restrict__ coefs, long long copy_stride,
                    const KPointSym* __restrict__ ks, const int* __restrict__ npw_arr,
                    const long long* __restrict__ chat_off, const int* __restrict__ pos, const int* __restrict__ collist,
                    const int* __restrict__ colcnt, const uint8_t* __restrict__ colmask, GeomDev gd,
                    const float* __restrict__ band_scale, uint16_t* __restrict__ Bsplit, float2* __restrict__ psi32)
{
    extern __shared__ __align__(16) unsigned char fbsm[];
    const FbLayout L = fb_layout(gd);
    float2* sm = reinterpret_cast<float2*>(fbsm);
    unsigned* ymask = reinterpret_cast<unsigned*>(sm + (size_t)gd.Nz * L.SZ);  // [x]: occupied y of the plane
    unsigned* xany = ymask + 32;                                              // occupied x
    const int nsets = gd.nspin * gd.nbnds * gd.nspinor;
    int t = blockIdx.x;
    const int cpy = t % gd.nsub;
    t /= gd.nsub;
    const int set = t % nsets, k = t / nsets;
    const int npw = npw_arr[ks[k].ik];
    const int ncol = gd.Nx * gd.Ny, cnt = colcnt[k];
    const int* cl = collist + (size_t)k * ncol;
    // occupancy as bit masks (lengths are at most 32)
    if (threadIdx.x < 32)
    {
        unsigned m = 0;
        if ((int)threadIdx.x < gd.Nx)
            for (int y = 0; y < gd.Ny; ++y)
                m |= (unsigned)(colmask[((size_t)k * gd.Nx + threadIdx.x) * gd.Ny + y] != 0) << y;
        ymask[threadIdx.x] = m;
        const unsigned b = __ballot_sync(0xffffffffu, m != 0);
        if (threadIdx.x == 0) *xany = b;
    }
    // the sphere's columns: zeros, then the coefficients
    for (int e = threadIdx.x; e < cnt * gd.Nz; e += FB_THREADS)
    {
        const int z = e / cnt, c = cl[e - z * cnt];
        const int x = c / gd.Ny;
        sm[z * L.SZ + x * L.SX + (c - x * gd.Ny)] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    const long long kbase = chat_off[k];
    const float2* c = (cpy == 0 ? coef0 : coefs + (cpy - 1) * copy_stride) + kbase + (size_t)set * npw;
    const int* pk = pos + kbase / nsets;
    for (int g = threadIdx.x; g < npw; g += FB_THREADS) sm[pk[g]] = c[g];
    __syncthreads();
    // z lines of the columns
    switch (gd.Nz)
    {
#define FB_CASE(N)                                                              \
    case N:                                                                     \
        for (int i = threadIdx.x; i < cnt; i += FB_THREADS)                     \
        {                                                                       \
            const int x = cl[i] / gd.Ny, y = cl[i] - x * gd.Ny;                 \
            float2* p = sm + x * L.SX + y;                                      \
            float2 v[N];                                                        \
            _Pragma("unroll") for (int z = 0; z < N; ++z) v[z] = p[z * L.SZ];   \
            fb_line<N>(v);                                                      \
            _Pragma("unroll") for (int z = 0; z < N; ++z) p[z * L.SZ] = v[z];   \
        }                                                                       \
        break;
        FB_SIZES(FB_CASE)
#undef FB_CASE
    default: break;
    }
    __syncthreads();
    // y lines of the occupied planes
    const unsigned xa = *xany;
    switch (gd.Ny)
    {
#define FB_CASE(N)                                                                                          \
    case N:                                                                                                 \
        for (int i = threadIdx.x; i < gd.Nz * gd.Nx; i += FB_THREADS)                                       \
        {                                                                                                   \
            const int z = i / gd.Nx, x = i - z * gd.Nx;                                                     \
            if (!((xa >> x) & 1u)) continue;                                                                \
            const unsigned ym = ymask[x];                                                                   \
            float2* p = sm + z * L.SZ + x * L.SX;                                                           \
            float2 v[N];                                                                                    \
            _Pragma("unroll") for (int y = 0; y < N; ++y) v[y] = (ym >> y) & 1u ? p[y] : make_float2(0.f, 0.f); \
            fb_line<N>(v);                                                                                  \
            _Pragma("unroll") for (int y = 0; y < N; ++y) p[y] = v[y];                                      \
        }                                                                                                   \
        break;
        FB_SIZES(FB_CASE)
#undef FB_CASE
    default: break;
    }
    __syncthreads();
    // x lines, and the operands: (Re, Im) and (-Im, Re) rows split into (hi, lo), FP32 rows
    const int sp = set % gd.nspinor, band = set / gd.nspinor % gd.nbnds, spin = set / gd.nspinor / gd.nbnds;
    const float sc = band_scale[((size_t)k * gd.nspin + spin) * gd.nbnds + band];
    const int inner = gd.Ny * gd.Nz;
    const long long Ns = (long long)gd.Nx * inner, M = gd.nsub * Ns;
    const int NT = 2 * gd.nbp;
    const size_t nkb = (size_t)gd.nspinor * M / 32, npb = (size_t)gd.nspinor * M / 16;
    const size_t kg = (size_t)k * gd.nspin + spin;
    uint32_t* const Bhi = reinterpret_cast<uint32_t*>(Bsplit) + kg * 2 * nkb * NT * 32 + (size_t)band * 32;
    uint32_t* const Blo = Bhi + nkb * NT * 32;
    const uint32_t rot = (uint32_t)gd.nbp * 32;
    float2* const P = psi32 + kg * npb * gd.nbp * 16 + (size_t)band * 16;
    const uint32_t kc0 = (uint32_t)(sp * M + cpy * Ns);
    switch (gd.Nx)
    {
#define FB_CASE(N)                                                                                          \
    case N:                                                                                                 \
        for (int i = threadIdx.x; i < inner; i += FB_THREADS)                                               \
        {                                                                                                   \
            const int y = i / gd.Nz, z = i - y * gd.Nz;                                                     \
            const float2* p = sm + z * L.SZ + y;                                                            \
            float2 v[N];                                                                                    \
            _Pragma("unroll") for (int x = 0; x < N; ++x) v[x] =                                            \
                (xa >> x) & 1u ? p[x * L.SX] : make_float2(0.f, 0.f);                                       \
            fb_line<N>(v);                                                                                  \
            _Pragma("unroll") for (int x = 0; x < N; ++x)                                                   \
            {                                                                                               \
                const float2 w = make_float2(v[x].x * sc, v[x].y * sc);                                     \
                const uint32_t kc = kc0 + (uint32_t)(x * inner + i);                                        \
                uint32_t h0, l0, h1, l1;                                                                    \
                fb_split<BF16>(w.x, w.y, h0, l0);                                                           \
                fb_split<BF16>(-w.y, w.x, h1, l1);                                                          \
                const size_t off = (size_t)(kc >> 5) * (uint32_t)(NT * 32) + (kc & 31u);                     \
                Bhi[off] = h0;                                                                              \
                Blo[off] = l0;                                                                              \
                Bhi[off + rot] = h1;                                                                        \
                Blo[off + rot] = l1;                                                                        \
                P[(size_t)(kc >> 4) * (uint32_t)(gd.nbp * 16) + (kc & 15u)] = w;                             \
            }                                                                                               \
        }                                                                                                   \
        break;
        FB_SIZES(FB_CASE)
#undef FB_CASE
    default: break;
    }
}

void lelph_launch_box_pos(const KPointSym* ks, int nk, const int* miller, const long long* pw_off, const int* npw,
                          int npw_max, const long long* chat_off, const GeomDev& g, int* pos, const BoxMask& mk,
                          cudaStream_t st)
{
    const dim3 grid((unsigned)((npw_max + 255) / 256), (unsigned)nk);
    k_box_pos<<<grid, 256, 0, st>>>(ks, miller, pw_off, npw, chat_off, g.nspin * g.nbnds * g.nspinor, g, pos, mk);
}

int lelph_launch_box_fft_split(const float2* coef0, const float2* coefs, long long copy_stride, const KPointSym* ks,
                               int nk, const int* npw, const long long* chat_off, const int* pos, const int* collist,
                               const int* colcnt, const uint8_t* colmask, const GeomDev& g, const float* band_scale,
                               int ab_bf16, uint16_t* Bsplit, float2* psi32, cudaStream_t st)
{
    const size_t smem = fb_layout(g).bytes;
    auto k = ab_bf16 ? k_box_fft_split<1> : k_box_fft_split<0>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM_LIMIT) != cudaSuccess) return -1;
    const long long nbox = (long long)nk * g.nspin * g.nbnds * g.nspinor * g.nsub;
    if (nbox > 0x7fffffffll) return -1;
    k<<<(unsigned)nbox, FB_THREADS, smem, st>>>(coef0, coefs, copy_stride, ks, npw, chat_off, pos, collist, colcnt,
                                                colmask, g, band_scale, Bsplit, psi32);
    return 0;
}
