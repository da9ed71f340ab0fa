// backup.cu -- the particle backup of main.f90:1102-1139 and its reader restart.f90:48-149,
// streamed between the device's structure-of-arrays particles and the reference's file.
//
// File: Fortran unformatted sequential records (4-byte little-endian length markers before
// and after each record), as the reference's compilers write them:
//   (time, gtype, Pabs_cor)                      real(8), integer(4), real(8)
//   np_tot(1:ntype, 1:nproc)                     integer(4)
//   vxp(1:6, 1:np_tot(ptype,iproc)) per iproc, ptype (iproc outer)   real(8)
// A record longer than 2^31 - 9 bytes is split into subrecords: the leading marker of every
// subrecord but the last is negative, the trailing marker of every subrecord but the first
// (the convention of the Intel and GNU Fortran runtimes).
//
// Device side: live particles are packed in slot order (holes skipped) into FP64 vxp(6, n)
// chunks -- a count of live particles per 1024-slot block, its prefix sum on the host, one
// packing kernel per chunk -- copied to pinned host buffers (two, alternating, so that the
// next chunk is packed and copied while the host writes the previous one).  z is not kept on
// the device and is written as 0.  Reading unpacks FP64 chunks into the fixed-point and FP32
// arrays after the occupied slots, then deposits every species (restart_OMP).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>
#include <vector>
#include <sys/mman.h>
#include "lepic_internal.cuh"

#define BK_BLOCK 1024                 // slots per counting block
#define BK_CHUNK (1ll << 22)          // slots per packing chunk (a multiple of BK_BLOCK)
static const long long kMaxSub = 2147483639ll;  // the runtimes' largest subrecord

// live particles per BK_BLOCK slots
__global__ void k_live_counts(const float *VX, long long n, int *counts) {
    __shared__ int s;
    if (threadIdx.x == 0) s = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * BK_BLOCK;
    int c = 0;
    for (int t = threadIdx.x; t < BK_BLOCK; t += blockDim.x) {
        const long long i = base + t;
        if (i < n && !isnan(VX[i])) c++;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s, c);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = s;
}

// packs the live particles of blocks [b0, b0 + nb) into out (vxp(6, .) from offset
// off[b] - off[b0] of block b), in slot order
__global__ void __launch_bounds__(BK_BLOCK) k_pack(const uint32_t *X, const uint32_t *Y, const float *VX,
                                                  const float *VY, const float *VZ, const float *Z, long long n,
                                                  long long b0, const long long *off, double ux, double uy,
                                                  double *out) {
    __shared__ int wsum[BK_BLOCK / 32];
    const long long b = b0 + blockIdx.x;
    const long long i = b * BK_BLOCK + threadIdx.x;
    const float vx = i < n ? VX[i] : __int_as_float(HOLE_NAN);
    const bool live = !isnan(vx);
    const unsigned m = __ballot_sync(0xffffffffu, live);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) wsum[w] = __popc(m);
    __syncthreads();
    int pre = 0;
    for (int k = 0; k < w; k++) pre += wsum[k];
    if (!live) return;
    const long long o = off[b] - off[b0] + pre + __popc(m & ((1u << lane) - 1u));
    double *p = out + 6 * o;
    p[0] = (double)X[i] * ux;   // as lepic_gpu_get_particles
    p[1] = (double)Y[i] * uy;
    p[2] = Z ? (double)Z[i] : 0.0;   // z: the 3rd dimension's, else 0
    p[3] = vx;
    p[4] = VY[i];
    p[5] = VZ[i];
}

// unpacks n FP64 particles into the slots from dst (as lepic_gpu_put_particles); a particle
// outside the box raises LERR_RANGE and becomes a hole
__global__ void k_unpack(const double *in, long long n, long long dst, double sx, double sy, long long xl,
                         long long yl, uint32_t *X, uint32_t *Y, float *VX, float *VY, float *VZ, float *Z,
                         DevCounters *cnt) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const double *p = in + 6 * k;
        const long long xi = llrint(p[0] * sx), yi = llrint(p[1] * sy);
        const long long s = dst + k;
        if (!(xi >= 0 && xi < xl && yi >= 0 && yi < yl) || !(p[3] == p[3])) {
            set_err(cnt, LERR_RANGE, 800);
            X[s] = 0; Y[s] = 0; VX[s] = __int_as_float(HOLE_NAN); VY[s] = 0.f; VZ[s] = 0.f;
            continue;
        }
        X[s] = (uint32_t)xi; Y[s] = (uint32_t)yi;
        VX[s] = (float)p[3]; VY[s] = (float)p[4]; VZ[s] = (float)p[5];
        if (Z) Z[s] = (float)p[2];
    }
}

// ---------------------------------------------------------------------------------------
// Particles to and from the host's FP64 vxp(6, n): the records cross in chunks, converted to and
// from the device's arrays on the device.  The device side of a chunk is the sort's scratch (keys
// and perm, free between sorts).
//  * From IO_LANED particles on, up to IO_LANES host threads take chunks in turn, each through two
//    pinned buffers of its own: one thread's copy, and its page faults on a new array, are slower
//    than the bus.  Put / get of 1.3 M particles: 2.9 / 2.7 ms, 5.8 into a new array; straight
//    from and to the caller's array 4.9 / 3.6 and 14.  A context's first such call pays for the
//    pinned memory, about 1 ms per MB (6.3 MB; with 12.6 MB steady times were the same), which a
//    smaller number of particles does not earn back: 2^19 cross in 1.6 / 1.8 ms without.
//  * Fewer cross straight from and to the caller's array, in chunks of up to IO_CHUNK particles taken
//    by keys and perm in turn, which hold that many even where the species are smaller (a full
//    species of 20000 in chunks of a third of the scratch: put 0.19, get 0.61 ms; so 0.11, 0.14).
//    The driver is slow to copy into pages that do not exist yet, so they are made before
//    (20000 particles into a new array 1.0 -> 0.43 ms, 300000 7.5 -> 3.6).
// (Converted by one host thread between plain copies, put + sort + deposit + get of 2 x 1.3 M
// particles took 66 ms; so 18.7 ms, most of it the page faults of the new host arrays.)
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23        // Linux 5.14; older headers do not name it
#endif
#define IO_CHUNK (1ll << 17)          // particles per direct chunk at most (a multiple of BK_BLOCK): 6.3 MB
#define IO_LANED (1ll << 20)
#define IO_LANES 4
#define IO_LANE_CHUNK (16ll * BK_BLOCK)   // particles per pinned buffer: 786 kB
struct IoStage {
    double *h = nullptr;
    cudaEvent_t ev[IO_LANES][2] = {};
};

void io_free(lepic_ctx *c) {
    IoStage *S = (IoStage *)c->io;
    if (!S) return;
    if (S->h) cudaFreeHost(S->h);
    for (auto &e : S->ev)
        for (auto &v : e)
            if (v) cudaEventDestroy(v);
    delete S;
    c->io = nullptr;
}

// the context's pinned buffers, kept until it is destroyed; null when they cannot be had (the
// caller's array is then used directly)
static IoStage *io_stage(lepic_ctx *c) {
    if (c->io) return (IoStage *)c->io;
    IoStage *S = new (std::nothrow) IoStage;
    if (!S) return nullptr;
    c->io = S;
    bool ok = cudaMallocHost((void **)&S->h, 48 * IO_LANE_CHUNK * 2 * IO_LANES) == cudaSuccess;
    for (auto &e : S->ev)
        for (auto &v : e) ok = ok && cudaEventCreateWithFlags(&v, cudaEventDisableTiming) == cudaSuccess;
    if (ok) return S;
    cudaGetLastError();
    io_free(c);
    return nullptr;
}

// A get's block offsets and counts lie at the start of keys: bytes for nb blocks
static long long io_offsets(long long nb) { return (8 * (nb + 1) + 4 * nb + 255) / 256 * 256; }

// ints that keys and perm need to stage a species of `cap` slots
long long io_scratch(long long cap) {
    const long long nb = div_up(cap, BK_BLOCK);
    return std::max(cap, (48 * std::min(IO_CHUNK, nb * BK_BLOCK) + io_offsets(nb)) / 4);
}

// particles per direct chunk, a multiple of BK_BLOCK, behind `used` bytes of the scratch
static long long io_chunk(const lepic_ctx *c, long long used) {
    return std::min(IO_CHUNK, (4 * c->scratch_cap - used) / 48 / BK_BLOCK * BK_BLOCK);
}

// A call's chunks, dispensed to a few host threads (this one among them; only this one when no
// more can be started).  lane(t, next) works on as lane t, taking chunk numbers from next until
// they run out, and returns the first error it meets.
template <class Lane>
static cudaError_t io_run(lepic_ctx *c, Lane lane) {
    std::atomic<long long> next(0);
    cudaError_t err[IO_LANES] = {};
    std::thread pool[IO_LANES];
    const int nt = (int)std::min((unsigned)IO_LANES, std::max(1u, std::thread::hardware_concurrency()));
    try {
        for (int t = 1; t < nt; t++)
            pool[t] = std::thread([&, t] {
                err[t] = cudaSetDevice(c->dev);
                if (err[t] == cudaSuccess) err[t] = lane(t, next);
            });
    } catch (...) { }                 // no more threads: those that run take all chunks
    err[0] = lane(0, next);
    for (auto &t : pool)
        if (t.joinable()) t.join();
    for (cudaError_t e : err)
        if (e != cudaSuccess) {
            cudaStreamSynchronize(c->stream);      // nothing of the call is left in flight
            return e;
        }
    return cudaSuccess;
}

// makes the pages of an output that is about to be written (the contents stay), a few threads
// together when it is large
static void io_touch(lepic_ctx *c, double *out, size_t bytes) {
    const uintptr_t kPage = 4096, kPart = 1 << 20;
    const uintptr_t o = (uintptr_t)out / kPage * kPage, end = (uintptr_t)out + bytes;
    auto touch = [](uintptr_t p, uintptr_t e) {
        if (p >= e || madvise((void *)p, e - p, MADV_POPULATE_WRITE) == 0) return;
        for (; p < e; p += kPage) __atomic_fetch_add((char *)p, 0, __ATOMIC_RELAXED);   // a system that does not have it
    };
    if (bytes < 4 * kPart) { touch(o, end); return; }
    io_run(c, [&](int, std::atomic<long long> &next) {
        for (uintptr_t p; (p = o + kPart * (uintptr_t)next++) < end;) touch(p, std::min(end, p + kPart));
        return cudaSuccess;
    });
}

// n host particles into slots dst ..; one outside the box (or at no number) sets *bad
__global__ void k_put(const double *in, long long n, long long dst, double sx, double sy, long long xl, long long yl,
                      uint32_t *X, uint32_t *Y, float *VX, float *VY, float *VZ, float *Z, int *bad) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const double2 *p = reinterpret_cast<const double2 *>(in + 6 * k);
        const double2 xy = p[0], zu = p[1], vw = p[2];
        const long long xi = llround(xy.x * sx), yi = llround(xy.y * sy), s = dst + k;
        if (!(xi >= 0 && xi < xl && yi >= 0 && yi < yl)) *bad = 1;
        X[s] = (uint32_t)xi; Y[s] = (uint32_t)yi;
        VX[s] = isnan(zu.y) ? __int_as_float(HOLE_NAN) : (float)zu.y;
        VY[s] = (float)vw.x; VZ[s] = (float)vw.y;
        if (Z) Z[s] = (float)zu.x;
    }
}

// the end of a put whose particles were all inside the box: the n slots into the species' own
// arrays, and its counts
struct PutArrays {
    uint32_t *X, *Y;
    float *VX, *VY, *VZ, *Z;
};
__global__ void k_put_commit(const int *bad, PutArrays from, PutArrays to, long long n, DevCounters *cnt, int sp) {
    if (*bad) return;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        to.X[k] = from.X[k]; to.Y[k] = from.Y[k];
        to.VX[k] = from.VX[k]; to.VY[k] = from.VY[k]; to.VZ[k] = from.VZ[k];
        if (to.Z) to.Z[k] = from.Z[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        cnt->n_slots[sp] = n;
        cnt->n_alive[sp] = n;
        cnt->n_sorted[sp] = 0;
        cnt->n_items[sp] = 0;
    }
}

// Replaces a species' particles.  They go to the buffer that is not in use and are copied to the one
// in use when all of them have been found inside the box: a refused call leaves the species as
// it was, and pointers to its arrays show the new particles (the copy is 40 B per particle at the
// device's rate, a thousandth of the way across the bus).
int particles_put(lepic_ctx *c, int sp, const double *vxp, long long n) {
    SpeciesBuf &B = c->sp[sp];
    if (n < 0 || n > B.cap) { c->last_err = "particle count exceeds capacity"; return LEPIC_ECAPACITY; }
    const lepic_config &g = c->cfg;
    IoStage *S = n >= IO_LANED ? io_stage(c) : nullptr;
    const double sx = (double)(1u << c->S) / g.dx, sy = (double)(1u << c->S) / g.dy;
    const long long xl = (long long)g.nx << c->S, yl = (long long)g.ny << c->S;
    double *const d[2] = {(double *)c->keys, (double *)c->perm};
    int *const bad = c->blocksums;                   // scratch of the sort's scan
    const int cur = B.cur, o = 1 - cur;
    LCUDA(cudaMemsetAsync(bad, 0, sizeof(int), c->stream));
    auto convert = [&](const double *in, long long k, long long m) {
        k_put<<<(int)std::min<long long>(div_up(m, 256), c->num_sms * 8), 256, 0, c->stream>>>(
            in, m, k, sx, sy, xl, yl, B.X[o], B.Y[o], B.VX[o], B.VY[o], B.VZ[o], B.Z[o], bad);
        return cudaGetLastError();
    };
    if (S) {
        const cudaError_t er = io_run(c, [&](int t, std::atomic<long long> &next) {
            cudaError_t e = cudaSuccess;
            for (int i = 0; e == cudaSuccess; i++) {
                const long long k = IO_LANE_CHUNK * next++, m = std::min(IO_LANE_CHUNK, n - k);
                if (m <= 0) break;
                const int b = i & 1;
                double *const h = S->h + 6 * IO_LANE_CHUNK * (2 * t + b), *const q = d[b] + 6 * IO_LANE_CHUNK * t;
                if (i >= 2) e = cudaEventSynchronize(S->ev[t][b]);   // the buffer's last chunk has left it
                if (e != cudaSuccess) break;
                std::memcpy(h, vxp + 6 * k, 48 * (size_t)m);
                e = cudaMemcpyAsync(q, h, 48 * (size_t)m, cudaMemcpyHostToDevice, c->stream);
                if (e == cudaSuccess) e = cudaEventRecord(S->ev[t][b], c->stream);
                if (e == cudaSuccess) e = convert(q, k, m);
            }
            return e;
        });
        LCUDA(er);
    } else {
        const long long chunk = io_chunk(c, 0);
        int b = 0;
        for (long long k = 0; k < n; k += chunk, b ^= 1) {
            const long long m = std::min(chunk, n - k);
            LCUDA(cudaMemcpyAsync(d[b], vxp + 6 * k, 48 * (size_t)m, cudaMemcpyHostToDevice, c->stream));
            LCUDA(convert(d[b], k, m));
        }
    }
    const PutArrays from = {B.X[o], B.Y[o], B.VX[o], B.VY[o], B.VZ[o], B.Z[o]};
    const PutArrays to = {B.X[cur], B.Y[cur], B.VX[cur], B.VY[cur], B.VZ[cur], B.Z[cur]};
    k_put_commit<<<(int)std::min<long long>(div_up(n, 256) + 1, c->num_sms * 8), 256, 0, c->stream>>>(bad, from, to, n,
                                                                                                  c->dcnt, sp);
    LCUDA(cudaGetLastError());
    int hbad = 0;
    LCUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    LCUDA(cudaStreamSynchronize(c->stream));
    if (hbad) { c->last_err = "particle outside the box"; return LEPIC_EINVAL; }
    B.ordered = false;
    return LEPIC_OK;
}

// The live particles of a species in slot order (at most cap of them); n_out: how many there are
int particles_get(lepic_ctx *c, int sp, double *vxp, long long cap, long long *n_out) {
    int r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    SpeciesBuf &B = c->sp[sp];
    const lepic_config &g = c->cfg;
    const long long ns = c->hcnt->n_slots[sp], nb = div_up(ns, BK_BLOCK);
    if (n_out) *n_out = 0;
    if (ns == 0) return LEPIC_OK;
    // the scratch: block offsets and counts at the start of keys, chunks behind them and in perm
    const long long used = io_offsets(nb);
    long long *const d_off = (long long *)c->keys;
    int *const d_cnt = (int *)(d_off + nb + 1);
    double *const d[2] = {(double *)((char *)c->keys + used), (double *)c->perm};
    std::vector<int> cnt((size_t)nb);
    std::vector<long long> off((size_t)nb + 1, 0);
    k_live_counts<<<(unsigned)nb, 256, 0, c->stream>>>(B.VX[B.cur], ns, d_cnt);
    LCUDA(cudaGetLastError());
    LCUDA(cudaMemcpyAsync(cnt.data(), d_cnt, sizeof(int) * nb, cudaMemcpyDeviceToHost, c->stream));
    LCUDA(cudaStreamSynchronize(c->stream));
    for (long long b = 0; b < nb; b++) off[b + 1] = off[b] + cnt[b];
    const long long total = off[nb];
    if (n_out) *n_out = total;
    if (vxp) {
        IoStage *S = total >= IO_LANED ? io_stage(c) : nullptr;
        LCUDA(cudaMemcpyAsync(d_off, off.data(), sizeof(long long) * (nb + 1), cudaMemcpyHostToDevice, c->stream));
        const double ux = g.dx * std::ldexp(1.0, -c->S), uy = g.dy * std::ldexp(1.0, -c->S);
        // blocks b0 .. b0 + bn packed into q and copied to h; how many particles, up to cap
        auto fetch = [&](long long b0, long long bn, double *q, double *h, long long &len) {
            k_pack<<<(unsigned)bn, BK_BLOCK, 0, c->stream>>>(B.X[B.cur], B.Y[B.cur], B.VX[B.cur], B.VY[B.cur], B.VZ[B.cur],
                                                             B.Z[B.cur], ns, b0, d_off, ux, uy, q);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
            len = std::min(off[b0 + bn], cap) - off[b0];
            return cudaMemcpyAsync(h, q, 48 * (size_t)len, cudaMemcpyDeviceToHost, c->stream);
        };
        if (S) {
            const cudaError_t er = io_run(c, [&](int t, std::atomic<long long> &next) {
                const long long per = IO_LANE_CHUNK / BK_BLOCK;
                long long at[2] = {0, 0}, len[2] = {0, 0};   // where a buffer's particles go, and how many
                auto buf = [&](int b) { return S->h + 6 * IO_LANE_CHUNK * (2 * t + b); };
                auto finish = [&](int b) {
                    if (!len[b]) return cudaSuccess;
                    const cudaError_t e = cudaEventSynchronize(S->ev[t][b]);
                    if (e == cudaSuccess) std::memcpy(vxp + 6 * at[b], buf(b), 48 * (size_t)len[b]);
                    len[b] = 0;
                    return e;
                };
                cudaError_t e = cudaSuccess;
                int b = 0;
                for (; e == cudaSuccess; b ^= 1) {
                    const long long b0 = per * next++;
                    if (b0 >= nb || off[b0] >= cap) break;
                    at[b] = off[b0];
                    e = fetch(b0, std::min(per, nb - b0), d[b] + 6 * IO_LANE_CHUNK * t, buf(b), len[b]);
                    if (e == cudaSuccess) e = cudaEventRecord(S->ev[t][b], c->stream);
                    if (e == cudaSuccess) e = finish(b ^ 1);   // the chunk before, while this one is on its way
                }
                return e == cudaSuccess ? finish(b ^ 1) : e;
            });
            LCUDA(er);
        } else {
            io_touch(c, vxp, 48 * (size_t)std::min(total, std::max(cap, 0ll)));
            const long long per = io_chunk(c, used) / BK_BLOCK;
            int b = 0;
            for (long long b0 = 0; b0 < nb && off[b0] < cap; b0 += per, b ^= 1) {
                long long len = 0;
                LCUDA(fetch(b0, std::min(per, nb - b0), d[b], vxp + 6 * off[b0], len));
            }
            LCUDA(cudaStreamSynchronize(c->stream));
        }
    }
    if (vxp && total > cap) { c->last_err = "output capacity too small"; return LEPIC_ECAPACITY; }
    return LEPIC_OK;
}

// ---------------------------------------------------------------------------------------
// Fortran sequential records with subrecords
struct RecWriter {
    FILE *f = nullptr;
    long long left = 0, sub_left = 0;   // bytes of the record / of the current subrecord
    bool first = true, ok = true;
    long long max_sub = kMaxSub;
    void marker(long long v) {
        const int32_t m = (int32_t)v;
        ok = ok && fwrite(&m, 4, 1, f) == 1;
    }
    void begin(long long len) {
        left = len;
        first = true;
        if (len == 0) {  // an empty record: both markers at once
            marker(0);
            marker(0);
            sub_left = 0;
            return;
        }
        open_sub();
    }
    void open_sub() {
        sub_left = std::min(left, max_sub);
        marker(sub_left < left ? -sub_left : sub_left);   // negative: more subrecords follow
    }
    void write(const void *p, long long nbytes) {
        const char *c = (const char *)p;
        while (nbytes > 0 && ok) {
            const long long k = std::min(nbytes, sub_left);
            ok = ok && fwrite(c, 1, (size_t)k, f) == (size_t)k;
            c += k; nbytes -= k; sub_left -= k;
            if (sub_left == 0) close_sub();
        }
    }
    void close_sub() {
        const long long len = std::min(left, max_sub);
        marker(first ? len : -len);                       // negative: continues a subrecord
        left -= len;
        first = false;
        if (left > 0) open_sub();
    }
    void end() {
        if (left == 0 && sub_left == 0) return;
        ok = false;  // wrote fewer bytes than announced
    }
};

struct RecReader {
    FILE *f = nullptr;
    long long sub_left = 0;
    bool last = true, ok = true;
    bool marker(int32_t *m) { return fread(m, 4, 1, f) == 1; }
    // starts a record: sub_left is the first subrecord's length, last whether it is the only one
    bool begin() {
        int32_t m;
        if (!marker(&m)) return ok = false;
        sub_left = std::llabs((long long)m);
        last = m >= 0;
        return true;
    }
    // reads nbytes of the record's data, across subrecords
    bool read(void *p, long long nbytes) {
        char *c = (char *)p;
        while (nbytes > 0) {
            if (sub_left == 0) {
                if (last) return ok = false;  // past the end of the record
                int32_t t, h;
                if (!marker(&t) || !marker(&h)) return ok = false;
                sub_left = std::llabs((long long)h);
                last = h >= 0;
            }
            const long long k = std::min(nbytes, sub_left);
            if (fread(c, 1, (size_t)k, f) != (size_t)k) return ok = false;
            c += k; nbytes -= k; sub_left -= k;
        }
        return true;
    }
    // the record must end here
    bool end() {
        if (sub_left != 0 || !last) return ok = false;
        int32_t t;
        return ok = ok && marker(&t);
    }
};

// a smaller subrecord limit (lepic_options::fortran_max_subrecord) exercises the
// multi-subrecord layout with small files
static long long max_subrecord(const lepic_ctx *c) {
    const long long v = c->opt.fortran_max_subrecord;
    return (v >= 8 && v <= kMaxSub) ? v : kMaxSub;
}

// ---------------------------------------------------------------------------------------
extern "C" int lepic_gpu_write_backup(lepic_ctx *c, const char *path, double time, int32_t gtype, double Pabs_cor) {
    if (!c || !path) return LEPIC_EINVAL;
    if (const int rm = materialize_all(c)) return rm;   // records of a pending sort moved first
    int r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    const lepic_config &g = c->cfg;
    // live particles per species and block
    std::vector<std::vector<long long>> offs(g.ntype);
    std::vector<int32_t> np_tot(g.ntype);
    long long max_blocks = 1;
    for (int s = 0; s < g.ntype; s++) max_blocks = std::max<long long>(max_blocks, div_up(c->hcnt->n_slots[s], BK_BLOCK));
    int *d_counts = nullptr;
    long long *d_off = nullptr;
    double *d_out = nullptr;
    double *h_buf[2] = {nullptr, nullptr};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    FILE *f = nullptr;
    auto cleanup = [&]() {
        if (d_counts) cudaFree(d_counts);
        if (d_off) cudaFree(d_off);
        if (d_out) cudaFree(d_out);
        for (int k = 0; k < 2; k++) {
            if (h_buf[k]) cudaFreeHost(h_buf[k]);
            if (ev[k]) cudaEventDestroy(ev[k]);
        }
        if (f) fclose(f);
    };
#define BK_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t _e = (call);                                                                   \
        if (_e != cudaSuccess) {                                                                   \
            c->last_err = std::string(#call) + ": " + cudaGetErrorString(_e);                     \
            cleanup();                                                                             \
            return LEPIC_ECUDA;                                                                    \
        }                                                                                          \
    } while (0)
    BK_CUDA(cudaMalloc((void **)&d_counts, sizeof(int) * max_blocks));
    BK_CUDA(cudaMalloc((void **)&d_off, sizeof(long long) * (max_blocks + 1)));
    BK_CUDA(cudaMalloc((void **)&d_out, sizeof(double) * 6 * BK_CHUNK));
    for (int k = 0; k < 2; k++) {
        BK_CUDA(cudaMallocHost((void **)&h_buf[k], sizeof(double) * 6 * BK_CHUNK));
        BK_CUDA(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming));
    }
    for (int s = 0; s < g.ntype; s++) {
        const long long n = c->hcnt->n_slots[s];
        const long long nb = div_up(n, BK_BLOCK);
        SpeciesBuf &B = c->sp[s];
        std::vector<int> cnt(nb);
        if (nb > 0) {
            k_live_counts<<<(unsigned)nb, 256, 0, c->stream>>>(B.VX[B.cur], n, d_counts);
            BK_CUDA(cudaGetLastError());
            BK_CUDA(cudaMemcpyAsync(cnt.data(), d_counts, sizeof(int) * nb, cudaMemcpyDeviceToHost, c->stream));
            BK_CUDA(cudaStreamSynchronize(c->stream));
        }
        offs[s].assign(nb + 1, 0);
        for (long long b = 0; b < nb; b++) offs[s][b + 1] = offs[s][b] + cnt[b];
        if (offs[s][nb] > 2147483647ll) { c->last_err = "np_tot beyond integer(4)"; cleanup(); return LEPIC_ECAPACITY; }
        np_tot[s] = (int32_t)offs[s][nb];
    }
    f = fopen(path, "wb");
    if (!f) { c->last_err = std::string("cannot open ") + path; cleanup(); return LEPIC_EINVAL; }
    RecWriter w;
    w.f = f;
    w.max_sub = max_subrecord(c);
    w.begin(8 + 4 + 8);
    w.write(&time, 8); w.write(&gtype, 4); w.write(&Pabs_cor, 8);
    w.end();
    w.begin(4ll * g.ntype);
    w.write(np_tot.data(), 4ll * g.ntype);
    w.end();
    const double ux = g.dx * std::ldexp(1.0, -c->S), uy = g.dy * std::ldexp(1.0, -c->S);
    for (int s = 0; s < g.ntype && w.ok; s++) {
        SpeciesBuf &B = c->sp[s];
        const long long n = c->hcnt->n_slots[s];
        const long long nb = (long long)offs[s].size() - 1;
        w.begin(48ll * np_tot[s]);
        if (nb > 0) BK_CUDA(cudaMemcpyAsync(d_off, offs[s].data(), sizeof(long long) * (nb + 1), cudaMemcpyHostToDevice,
                                            c->stream));
        const long long blocks_per_chunk = BK_CHUNK / BK_BLOCK;
        long long pend_bytes[2] = {0, 0};
        int pend = -1;   // buffer waiting to be written
        int k = 0;
        for (long long b0 = 0; b0 < nb; b0 += blocks_per_chunk, k ^= 1) {
            const long long bn = std::min(blocks_per_chunk, nb - b0);
            const long long cnt = offs[s][b0 + bn] - offs[s][b0];
            k_pack<<<(unsigned)bn, BK_BLOCK, 0, c->stream>>>(B.X[B.cur], B.Y[B.cur], B.VX[B.cur], B.VY[B.cur],
                                                             B.VZ[B.cur], B.Z[B.cur], n, b0, d_off, ux, uy,
                                                             d_out);
            BK_CUDA(cudaGetLastError());
            if (pend == k) {  // the buffer this chunk goes to is still being written: finish it
                w.write(h_buf[k], pend_bytes[k]);
                pend = -1;
            }
            BK_CUDA(cudaMemcpyAsync(h_buf[k], d_out, sizeof(double) * 6 * cnt, cudaMemcpyDeviceToHost, c->stream));
            BK_CUDA(cudaEventRecord(ev[k], c->stream));
            if (pend == (k ^ 1)) {  // write the previous chunk while this one is copied
                w.write(h_buf[k ^ 1], pend_bytes[k ^ 1]);
                pend = -1;
            }
            BK_CUDA(cudaEventSynchronize(ev[k]));
            pend_bytes[k] = 48 * cnt;
            pend = k;
        }
        if (pend >= 0) w.write(h_buf[pend], pend_bytes[pend]);
        w.end();
    }
    const bool ok = w.ok;
    if (fclose(f) != 0 || !ok) {
        f = nullptr;
        c->last_err = std::string("write failed: ") + path;
        cleanup();
        return LEPIC_EINVAL;
    }
    f = nullptr;
    cleanup();
    return LEPIC_OK;
#undef BK_CUDA
}

extern "C" int lepic_gpu_read_backup(lepic_ctx *c, const char *path, double *time, int32_t *gtype, double *Pabs_cor) {
    if (!c || !path) return LEPIC_EINVAL;
    if (const int rm = materialize_all(c)) return rm;   // records of a pending sort moved first
    int r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    const lepic_config &g = c->cfg;
    FILE *f = fopen(path, "rb");
    if (!f) { c->last_err = std::string("cannot open ") + path; return LEPIC_EINVAL; }
    RecReader rd;
    rd.f = f;
    double t = 0.0, pc = 0.0;
    int32_t gt = 0;
    bool ok = rd.begin() && rd.read(&t, 8) && rd.read(&gt, 4) && rd.read(&pc, 8) && rd.end();
    // np_tot(1:ntype, 1:nproc): nproc from the record length (single subrecord)
    std::vector<int32_t> np;
    if (ok) {
        ok = rd.begin() && rd.last && rd.sub_left % (4ll * g.ntype) == 0;
        if (ok) {
            np.resize((size_t)(rd.sub_left / 4));
            ok = rd.read(np.data(), rd.sub_left) && rd.end();
        }
    }
    if (!ok) { fclose(f); c->last_err = "backup header unreadable"; return LEPIC_EINVAL; }
    const int nproc = (int)(np.size() / g.ntype);
    std::vector<long long> want(g.ntype, 0), alive0(g.ntype);
    for (int s = 0; s < g.ntype; s++) alive0[s] = c->hcnt->n_alive[s];
    for (int p = 0; p < nproc; p++)
        for (int s = 0; s < g.ntype; s++) {
            if (np[(size_t)p * g.ntype + s] < 0) ok = false;
            want[s] += np[(size_t)p * g.ntype + s];
        }
    for (int s = 0; s < g.ntype && ok; s++)
        if (c->hcnt->n_slots[s] + want[s] > c->sp[s].cap) {
            fclose(f);
            c->last_err = "backup exceeds the particle capacity (restart.f90:117-121)";
            return LEPIC_ECAPACITY;
        }
    double *d_in = nullptr, *h_in = nullptr;
    if (cudaMalloc((void **)&d_in, sizeof(double) * 6 * BK_CHUNK) != cudaSuccess ||
        cudaMallocHost((void **)&h_in, sizeof(double) * 6 * BK_CHUNK) != cudaSuccess) {
        if (d_in) cudaFree(d_in);
        fclose(f);
        c->last_err = "read_backup: allocation failed";
        return LEPIC_ENOMEM;
    }
    const double sx = (double)(1u << c->S) / g.dx, sy = (double)(1u << c->S) / g.dy;
    const long long xl = (long long)g.nx << c->S, yl = (long long)g.ny << c->S;
    for (int p = 0; p < nproc && ok; p++)
        for (int s = 0; s < g.ntype && ok; s++) {
            const long long n = np[(size_t)p * g.ntype + s];
            SpeciesBuf &B = c->sp[s];
            const long long base = c->hcnt->n_slots[s];
            ok = rd.begin();
            for (long long k0 = 0; k0 < n && ok; k0 += BK_CHUNK) {
                const long long m = std::min(BK_CHUNK, n - k0);
                ok = rd.read(h_in, 48 * m);
                if (!ok) break;
                if (cudaMemcpyAsync(d_in, h_in, 48 * m, cudaMemcpyHostToDevice, c->stream) != cudaSuccess) { ok = false; break; }
                k_unpack<<<(unsigned)std::min<long long>(div_up(m, 256), (long long)c->num_sms * 8), 256, 0, c->stream>>>(
                    d_in, m, base + k0, sx, sy, xl, yl, B.X[B.cur], B.Y[B.cur], B.VX[B.cur], B.VY[B.cur], B.VZ[B.cur],
                    B.Z[B.cur], c->dcnt);
                if (cudaStreamSynchronize(c->stream) != cudaSuccess) { ok = false; break; }
            }
            ok = ok && rd.end();
            c->hcnt->n_slots[s] = base + n;   // host mirror until the counters are written below
        }
    cudaFree(d_in);
    cudaFreeHost(h_in);
    fclose(f);
    if (!ok) { c->last_err = std::string("backup unreadable: ") + path; return LEPIC_EINVAL; }
    for (int s = 0; s < g.ntype; s++) {
        long long v = c->hcnt->n_slots[s], a = alive0[s] + want[s], zero = 0;
        LCUDA(cudaMemcpy(&c->dcnt->n_slots[s], &v, sizeof(v), cudaMemcpyHostToDevice));
        LCUDA(cudaMemcpy(&c->dcnt->n_alive[s], &a, sizeof(a), cudaMemcpyHostToDevice));
        LCUDA(cudaMemcpy(&c->dcnt->n_sorted[s], &zero, sizeof(zero), cudaMemcpyHostToDevice));
        int zi = 0;
        LCUDA(cudaMemcpy(&c->dcnt->n_items[s], &zi, sizeof(int), cudaMemcpyHostToDevice));
        c->sp[s].ordered = false;
    }
    if (time) *time = t;
    if (gtype) *gtype = gt;
    if (Pabs_cor) *Pabs_cor = pc;
    r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    return lepic_gpu_charge_deposition(c);  // restart_OMP: np of the loaded particles
}

// ---------------------------------------------------------------------------------------
// restart.f90:115-129: |np_dup| - 1 copies of every slot appended after the occupied slots
// (copy i of slot k at i * n + k).  A copied hole stays a plain hole (a loss record is tallied
// once, from the original).
__global__ void k_duplicate(long long n, int copies, uint32_t *X, uint32_t *Y, float *VX, float *VY, float *VZ,
                            float *Z) {
    const long long tot = n * (long long)copies;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const long long k = t % n, d = n + t;
        const float vx = VX[k];
        X[d] = X[k]; Y[d] = Y[k];
        VX[d] = isnan(vx) ? __int_as_float(HOLE_NAN) : vx;
        VY[d] = VY[k]; VZ[d] = VZ[k];
        if (Z) Z[d] = Z[k];
    }
}

extern "C" int lepic_gpu_duplicate_particles(lepic_ctx *c, int32_t np_dup) {
    if (!c) return LEPIC_EINVAL;
    if (const int rm = materialize_all(c)) return rm;   // records of a pending sort moved first
    const int dup = np_dup < 0 ? -np_dup : np_dup;
    if (dup <= 1) return LEPIC_OK;
    int r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    const lepic_config &g = c->cfg;
    for (int s = 0; s < g.ntype; s++)   // restart.f90:117-121
        if ((long long)dup * c->hcnt->n_slots[s] > c->sp[s].cap) {
            c->last_err = "|np_dup| * np_tot exceeds the particle capacity (restart.f90:117-121)";
            return LEPIC_ECAPACITY;
        }
    for (int s = 0; s < g.ntype; s++) {
        SpeciesBuf &B = c->sp[s];
        const long long n = c->hcnt->n_slots[s];
        if (n > 0) {
            const long long tot = n * (dup - 1);
            k_duplicate<<<(unsigned)std::min<long long>(div_up(tot, 256), (long long)c->num_sms * 16), 256, 0,
                          c->stream>>>(n, dup - 1, B.X[B.cur], B.Y[B.cur], B.VX[B.cur], B.VY[B.cur], B.VZ[B.cur],
                                       B.Z[B.cur]);
            LCUDA(cudaGetLastError());
        }
        const long long slots = n * dup, alive = c->hcnt->n_alive[s] * dup;
        LCUDA(cudaMemcpyAsync(&c->dcnt->n_slots[s], &slots, sizeof(slots), cudaMemcpyHostToDevice, c->stream));
        LCUDA(cudaMemcpyAsync(&c->dcnt->n_alive[s], &alive, sizeof(alive), cudaMemcpyHostToDevice, c->stream));
        LCUDA(cudaStreamSynchronize(c->stream));   // the host values above are locals
    }
    r = lepic_gpu_sync(c);
    if (r != LEPIC_OK) return r;
    return lepic_gpu_charge_deposition(c);  // restart_OMP: np of every particle
}
