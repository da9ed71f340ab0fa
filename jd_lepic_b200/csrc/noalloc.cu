// noalloc.cu -- charge deposition that allocates no device memory.
//
// Some hosts cannot call cudaMalloc: an application whose whole device memory is reserved up
// front and handed out by its own allocator (or by another framework's caching allocator), or
// code on a path where the implicit device synchronisation of an allocation is not allowed.
// Such a caller owns its particle arrays, its node-factor grid and its output grid already;
// this entry point needs no other memory of its own.  The temporary integer accumulator lives
// in the file-scope device array below, of fixed size, which every GPU that loads the library
// holds until the process exits.
//
// The deposit is the same integer CIC as the fused push kernel (push.cu): per-particle weights
// are exact products of the fixed-point cell offsets, rounded to 2^-44, summed in uint64, and
// scaled once to np = kq * (k1 * acc * 2^-44); the result is bit-identical to the context path.
// A position outside the box (X >= nx << shift or Y >= ny << shift) is skipped, so no write
// can land outside the (nx+3)(ny+3) nodes of the accumulator.
// Compiled with -fmad=false like the other FP64 grid kernels.
#include <algorithm>
#include <mutex>
#include "lepic_internal.cuh"

#define LEPIC_NOALLOC_MAX_NODES (1 << 20)  // (nx+3)*(ny+3) limit: 8 MiB of uint64

static __device__ __align__(256) unsigned long long g_noalloc_acc[LEPIC_NOALLOC_MAX_NODES];

// Host code must not use g_noalloc_acc directly (it names a host-side shadow, not device
// memory): its device address is looked up once per device and cached here, with the
// device's SM count for the launch shape.
static unsigned long long *g_noalloc_ptr[64];
static int g_noalloc_sms[64];
static std::mutex g_noalloc_mu;

__global__ void k_na_zero(unsigned long long *acc, long long nn) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nn; t += (long long)gridDim.x * blockDim.x)
        acc[t] = 0ull;
}

// Each thread walks `per` consecutive slots and keeps a run of particles in one cell as its
// moments (count, sum fx, sum fy, sum fx fy), which give the sum of the particles' rounded weights
// exactly, so that one run costs four atomics instead of four per particle.  Without rounding
// (sh <= 0) the products are only shifted up.  With it each weight is (v + h) >> sh, h = 2^(sh-1),
// and a run's sum is (sum v + n h - sum of the bits cut off) >> sh: the cell size 2^S being a
// multiple of 2^sh, the four products are +-fx fy modulo 2^sh, so r = (fx fy + h) mod 2^sh gives
// the bits cut off for two of the nodes and 2^sh - r (0 for r = 0) for the other two.
struct NaRun {
    int cx, cy;                 // its cell; cx < 0: none
    uint32_t n, sx, sy;         // n: count (bits 0..7), nonzero remainders (8..15), their sum (16..)
    uint64_t sxy;
};

__device__ __forceinline__ void na_add(const NaRun &r, int S, int sh, int W, unsigned long long *acc) {
    const uint64_t n = r.n & 255u, ax = (uint64_t)r.sx << S, ay = (uint64_t)r.sy << S;
    uint64_t w0 = (n << (2 * S)) - ax - ay + r.sxy, w1 = ax - r.sxy, w2 = r.sxy, w3 = ay - r.sxy;
    if (sh > 0) {
        const int nh = (int)n << (sh - 1), cut = (int)(r.n >> 16), cut2 = ((int)((r.n >> 8) & 255u) << sh) - cut;
        const uint64_t p = (uint64_t)(long long)(nh - cut), q = (uint64_t)(long long)(nh - cut2);
        w0 = (w0 + p) >> sh; w2 = (w2 + p) >> sh;
        w1 = (w1 + q) >> sh; w3 = (w3 + q) >> sh;
    } else {
        w0 <<= -sh; w1 <<= -sh; w2 <<= -sh; w3 <<= -sh;
    }
    // cx <= nx-1 and cy <= ny-1, so the four nodes (cx+1..cx+2, cy+1..cy+2) are inside
    unsigned long long *q = acc + ((long long)r.cx + 1) + ((long long)r.cy + 1) * W;
    if (w0) atomicAdd(q, (unsigned long long)w0);
    if (w1) atomicAdd(q + 1, (unsigned long long)w1);
    if (w2) atomicAdd(q + W + 1, (unsigned long long)w2);
    if (w3) atomicAdd(q + W, (unsigned long long)w3);
}

#define NA_PER_MAX 32   // slots per thread at most (the run's packed counts hold up to 255)

// VEC: X, Y and VX are 16-byte aligned, four slots per load; else one slot at a time.  `per` is a
// multiple of 4.
template <bool VEC>
__global__ void __launch_bounds__(256) k_na_deposit(const uint32_t *X, const uint32_t *Y, const float *VX, long long n,
                                                    int per, int S, int nx, int ny, unsigned long long *acc) {
    const uint32_t mask = (1u << S) - 1u;
    const int sh = 2 * S - LEPIC_DEP_SHIFT;
    const uint32_t rh = sh > 0 ? 1u << (sh - 1) : 0u, rm = sh > 0 ? (1u << sh) - 1u : 0u;
    const int W = nx + 3;
    for (long long i0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * per; i0 < n;
         i0 += (long long)gridDim.x * blockDim.x * per) {
        NaRun r;
        r.cx = -1; r.cy = 0; r.n = r.sx = r.sy = 0u; r.sxy = 0ull;
        const long long i1 = min(i0 + per, n);
        for (long long i = i0; i < i1; i += 4) {
            uint32_t xs[4], ys[4];
            float vs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (VEC && i + 4 <= n) {
                const uint4 x = *reinterpret_cast<const uint4 *>(X + i), y = *reinterpret_cast<const uint4 *>(Y + i);
                xs[0] = x.x; xs[1] = x.y; xs[2] = x.z; xs[3] = x.w;
                ys[0] = y.x; ys[1] = y.y; ys[2] = y.z; ys[3] = y.w;
                if (VX) {
                    const float4 v = *reinterpret_cast<const float4 *>(VX + i);
                    vs[0] = v.x; vs[1] = v.y; vs[2] = v.z; vs[3] = v.w;
                }
            } else {
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const bool in = i + p < n;
                    xs[p] = in ? X[i + p] : 0u;
                    ys[p] = in ? Y[i + p] : 0u;
                    if (!in) vs[p] = __int_as_float(HOLE_NAN);
                    else if (VX) vs[p] = VX[i + p];
                }
            }
#pragma unroll
            for (int p = 0; p < 4; p++) {
                if (isnan(vs[p])) continue; // a hole left by a lost particle, or past the end
                const uint32_t cx = xs[p] >> S, cy = ys[p] >> S;
                if (cx >= (uint32_t)nx || cy >= (uint32_t)ny) continue; // outside the box: not deposited
                const uint32_t fx = xs[p] & mask, fy = ys[p] & mask;
                const uint64_t fxy = (uint64_t)fx * fy;
                const uint32_t rem = ((uint32_t)fxy + rh) & rm;
                const uint32_t one = (rem << 16) + (rem ? 257u : 1u);
                if ((int)cx != r.cx || (int)cy != r.cy) {
                    if (r.cx >= 0) na_add(r, S, sh, W, acc);
                    r.cx = (int)cx; r.cy = (int)cy;
                    r.n = one; r.sx = fx; r.sy = fy; r.sxy = fxy;
                } else {
                    r.n += one; r.sx += fx; r.sy += fy; r.sxy += fxy;
                }
            }
        }
        if (r.cx >= 0) na_add(r, S, sh, W, acc);
    }
}

__global__ void k_na_finish(const unsigned long long *acc, const double *kq, double k1, long long nn, double *out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nn; t += (long long)gridDim.x * blockDim.x) {
        double w = (double)acc[t] * 5.684341886080802e-14; // 2^-44
        out[t] = kq[t] * (k1 * w);
    }
}

extern "C" int lepic_gpu_deposit_noalloc(const uint32_t *X, const uint32_t *Y, const float *VX, int64_t n,
                                         int32_t nx, int32_t ny, int32_t shift, double k1, const double *kq,
                                         double *np_out, void *stream) {
    if (n < 0 || nx < 1 || ny < 1 || shift < 1 || shift > 24 || !kq || !np_out || (n > 0 && (!X || !Y)))
        return LEPIC_EINVAL;
    if ((long long)nx << shift > (1ll << 32) || (long long)ny << shift > (1ll << 32)) return LEPIC_EINVAL;
    const long long nn = (long long)(nx + 3) * (ny + 3);
    if (nn > LEPIC_NOALLOC_MAX_NODES) return LEPIC_ECAPACITY; // larger than the static scratch
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LEPIC_ECUDA;
    unsigned long long *acc;
    int sms;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void *p = nullptr;
            int m = 0;
            if (cudaGetSymbolAddress(&p, g_noalloc_acc) != cudaSuccess || !p) return LEPIC_ECUDA;
            if (cudaDeviceGetAttribute(&m, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || m < 1)
                return LEPIC_ECUDA;
            g_noalloc_sms[dev] = m;
            g_noalloc_ptr[dev] = (unsigned long long *)p;
        }
        acc = g_noalloc_ptr[dev];
        sms = g_noalloc_sms[dev];
    }
    // an error left pending by earlier work of the caller is reported here and not cleared;
    // nothing is enqueued then
    if (cudaPeekAtLastError() != cudaSuccess) return LEPIC_ECUDA;
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = 4 * sms;
    k_na_zero<<<grid, 256, 0, st>>>(acc, nn); // the array keeps the previous call's sums
    if (n > 0) {
        // slots per thread: as many as still fill the GPU with threads, so that sorted arrays come
        // in long runs (1e7 sorted particles on 511 x 300: 362 us
        // with four atomics per particle, 59 us so, 2 TB/s of the 12 B per particle)
        const long long threads = (long long)sms * 2048;
        const int per = (int)std::min<long long>(NA_PER_MAX, std::max<long long>(4, (n / threads + 3) / 4 * 4));
        const int blocks = (int)std::min<long long>(16ll * sms, (n + 256ll * per - 1) / (256ll * per));
        const bool vec = (((uintptr_t)X | (uintptr_t)Y | (uintptr_t)VX) & 15) == 0;
        if (vec) k_na_deposit<true><<<blocks, 256, 0, st>>>(X, Y, VX, n, per, shift, nx, ny, acc);
        else k_na_deposit<false><<<blocks, 256, 0, st>>>(X, Y, VX, n, per, shift, nx, ny, acc);
    }
    k_na_finish<<<grid, 256, 0, st>>>(acc, kq, k1, nn, np_out);
    return cudaGetLastError() == cudaSuccess ? LEPIC_OK : LEPIC_ECUDA;
}
