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

// A warp takes 32 Q consecutive slots at a time, Q per lane, and keeps a run of particles in one
// cell as its moments (count, sum fx, sum fy, sum fx fy), which give the sum of the particles'
// rounded weights exactly, so that one run costs four atomics instead of four per particle: each
// lane's own runs first, then its last one joined with the neighbours' where they are in the same
// cell.  Sorted arrays come in long runs; arrays in random order come in runs of one, skip the
// joining and are bound by their atomics.  Every load of a warp covers whole lines whatever the
// arrays' alignment.  1e7 particles on 511 x 300: in cell order 353 us with four atomics per
// particle, 58 so (2 TB/s of their 12 B); in random order 232 and 222.  (A thread that walked 32
// slots of its own read lines 128 bytes apart: 71 us in order, 259 in random order, 138 and 306
// where the arrays are not 16-byte aligned.)
// Without rounding (sh <= 0) the products are only shifted up.  With it each weight is (v + h) >> sh,
// h = 2^(sh-1), and a run's sum is (sum v + n h - sum of the bits cut off) >> sh: the cell size 2^S
// being a multiple of 2^sh, the four products are +-fx fy modulo 2^sh, so r = (fx fy + h) mod 2^sh
// gives the bits cut off for two of the nodes and 2^sh - r (0 for r = 0) for the other two.
struct NaRun {
    int node;                   // its cell's first node; < 0: none
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
    unsigned long long *q = acc + r.node;
    if (w0) atomicAdd(q, (unsigned long long)w0);
    if (w1) atomicAdd(q + 1, (unsigned long long)w1);
    if (w2) atomicAdd(q + W + 1, (unsigned long long)w2);
    if (w3) atomicAdd(q + W, (unsigned long long)w3);
}

// A run of 128 slots at most fits: its packed counts hold up to 255, its sums of offsets below
// 2^24 stay below 2^31.  Up to NA_SMALL slots a lane takes one of them: with four too few warps are in
// flight (2e5 in random order on 511 x 300: 21.5 us against 19.5, as many in order 17.4 both);
// beyond it the longer runs pay (1e6 in order 23.5 us with one, 21.4 with four).
#define NA_SMALL (1ll << 19)

// Q: slots per lane (1 or 4)
template <int Q>
__global__ void __launch_bounds__(256) k_na_deposit(const uint32_t *X, const uint32_t *Y, const float *VX, long long n,
                                                    int S, int nx, int ny, unsigned long long *acc) {
    const unsigned full = 0xffffffffu;
    const uint32_t mask = (1u << S) - 1u;
    const int sh = 2 * S - LEPIC_DEP_SHIFT;
    const uint32_t rh = sh > 0 ? 1u << (sh - 1) : 0u, rm = sh > 0 ? (1u << sh) - 1u : 0u;
    const int W = nx + 3, lane = threadIdx.x & 31;
    const long long w0 = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long base = w0 * (32 * Q); base < n; base += nw * (32 * Q)) {   // the same for a whole warp
        const long long i = base + Q * lane;
        uint32_t xs[Q], ys[Q];
        float vs[Q];
#pragma unroll
        for (int p = 0; p < Q; p++) {
            const bool in = i + p < n;
            xs[p] = in ? X[i + p] : 0u;
            ys[p] = in ? Y[i + p] : 0u;
            vs[p] = !in ? __int_as_float(HOLE_NAN) : (VX ? VX[i + p] : 0.0f);
        }
        NaRun r;
        r.node = -1; r.n = r.sx = r.sy = 0u; r.sxy = 0ull;
#pragma unroll
        for (int p = 0; p < Q; p++) {
            if (isnan(vs[p])) continue; // a hole left by a lost particle, or past the end
            const uint32_t cx = xs[p] >> S, cy = ys[p] >> S;
            if (cx >= (uint32_t)nx || cy >= (uint32_t)ny) continue; // outside the box: not deposited
            const uint32_t fx = xs[p] & mask, fy = ys[p] & mask;
            const uint64_t fxy = (uint64_t)fx * fy;
            const uint32_t rem = ((uint32_t)fxy + rh) & rm;
            const uint32_t one = (rem << 16) + (rem ? 257u : 1u);
            const int node = (int)cx + 1 + ((int)cy + 1) * W;
            if (node != r.node) {
                if (r.node >= 0) na_add(r, S, sh, W, acc);
                r.node = node;
                r.n = one; r.sx = fx; r.sy = fy; r.sxy = fxy;
            } else {
                r.n += one; r.sx += fx; r.sy += fy; r.sxy += fxy;
            }
        }
        // the lanes' last runs: a segment is a run of lanes in one cell, summed into its last lane
        const int before = __shfl_up_sync(full, r.node, 1);
        const unsigned heads = __ballot_sync(full, lane == 0 || before != r.node);
        const int start = 31 - __clz(heads & (full >> (31 - lane)));
        for (int o = 1; o < 32; o <<= 1) {
            const bool take = lane - o >= start;
            if (!__any_sync(full, take)) break;      // no segment is longer than o lanes
            const uint32_t n2 = __shfl_up_sync(full, r.n, o), x2 = __shfl_up_sync(full, r.sx, o), y2 = __shfl_up_sync(full, r.sy, o);
            const uint64_t xy2 = __shfl_up_sync(full, r.sxy, o);
            if (take) { r.n += n2; r.sx += x2; r.sy += y2; r.sxy += xy2; }
        }
        const bool last = lane == 31 || ((heads >> (lane + 1)) & 1u);
        if (r.node >= 0 && last) na_add(r, S, sh, W, acc);
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
        const int q = n <= NA_SMALL ? 1 : 4;
        const int blocks = (int)std::min<long long>(16ll * sms, (n + 256 * q - 1) / (256 * q));
        if (q == 1) k_na_deposit<1><<<blocks, 256, 0, st>>>(X, Y, VX, n, shift, nx, ny, acc);
        else k_na_deposit<4><<<blocks, 256, 0, st>>>(X, Y, VX, n, shift, nx, ny, acc);
    }
    k_na_finish<<<grid, 256, 0, st>>>(acc, kq, k1, nn, np_out);
    return cudaGetLastError() == cudaSuccess ? LEPIC_OK : LEPIC_ECUDA;
}
