// B200 kernels of the shoebox integration path and their C ABI (include/xpgi.h).
//
// Work decomposition: one CTA per reflection. The CTA first maps its box pixels to the Kabsch frame (eps1/eps2,
// the pixel area J, u1/u2) in shared memory, then each thread owns whole pixel columns: the per-pixel terms stay in
// registers and the frame direction is walked with 65-bit masks (foreground frames, frames claimed by neighbours),
// so every voxel costs one coalesced 4-byte read per pass plus a handful of flops. Reductions accumulate in float64
// per thread and combine warp by warp in a fixed order: results do not depend on which other reflections share a
// launch.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <type_traits>

#include "xpgi_device.cuh"
#include "xpgi_internal.h"

using namespace xi;

namespace {

thread_local char g_err[512] = {0};

int fail(int code, const char* msg) {
    snprintf(g_err, sizeof g_err, "%s", msg);
    return code;
}

int cuda_check(const char* where) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof g_err, "%s: %s", where, cudaGetErrorString(e));
        return XI_E_CUDA;
    }
    return XI_OK;
}

constexpr float kSbOff = 3.0f;     // shoeboxes are stored as value + 3 (0 = unrecorded)

// neighbour data of a CTA: per active neighbour, squared normalised distances per column / row / frame
struct NbShared {
    int nact;
    int zmin[XI_MAX_K];             // frame of the smallest dz^2 of each active neighbour
    float x[XI_MAX_K], y[XI_MAX_K], z[XI_MAX_K], sx[XI_MAX_K], sz[XI_MAX_K];
};

// The per-axis terms of the active neighbours, in dynamic shared memory sized for the launch's neighbour columns
// and largest box: dx2 / dy2 (K x max_bx), dz2 (K x max_dz).
struct NbTab {
    float *dx2, *dy2, *dz2;
    int sxy, sz;
    __device__ __forceinline__ float& x2(int a, int i) const { return dx2[a * sxy + i]; }
    __device__ __forceinline__ float& y2(int a, int j) const { return dy2[a * sxy + j]; }
    __device__ __forceinline__ float* z2(int a) const { return dz2 + a * sz; }
};

__host__ __device__ inline size_t nb_bytes(int K, int max_bx, int max_dz) {
    return ((size_t)K * (2 * max_bx + max_dz) * sizeof(float) + 15) / 16 * 16;
}

__device__ __forceinline__ NbTab nb_tab(unsigned char* base, int K, int max_bx, int max_dz) {
    NbTab t;
    t.dx2 = reinterpret_cast<float*>(base);
    t.dy2 = t.dx2 + (size_t)K * max_bx;
    t.dz2 = t.dy2 + (size_t)K * max_bx;
    t.sxy = max_bx;
    t.sz = max_dz;
    return t;
}

// One neighbour column of a row, read ahead of its test by lane k of the warp that makes it.
struct NbColumn {
    float x, y, z, sx, sz;
    __device__ __forceinline__ void load(const XiRows& R, int row, int k) {
        const size_t o = (size_t)row * R.K + k;
        x = R.nbx[o];
        y = R.nby[o];
        z = R.nbz[o];
        sx = R.nbsx[o];
        sz = R.nbsz[o];
    }
};

__device__ __forceinline__ float frame_centre(int iz0, float fb, int z) { return (float)iz0 + fb * ((float)z + 0.5f); }

// Neighbour columns whose ellipsoid reaches the box (the separable pre-test of xpg/integrate_kernels.py:192-203;
// skipping the others is exact), by one warp: lane k tests column k, the passing columns are listed in column order.
__device__ __forceinline__ void neighbour_test(const NbColumn& c, int K, bool skip_first, int bx, const float* xs,
                                               const float* ys, float z_first, float z_last, NbShared& nb) {
    const int k = threadIdx.x & 31;
    bool on = false;
    if (k < K && !(k == 0 && skip_first)) {
        const float mx = (fminf(fmaxf(c.x, xs[0]), xs[bx - 1]) - c.x) / c.sx;
        const float my = (fminf(fmaxf(c.y, ys[0]), ys[bx - 1]) - c.y) / c.sx;
        const float mz = (fminf(fmaxf(c.z, z_first), z_last) - c.z) / c.sz;
        on = (mx * mx + my * my) + mz * mz < 1.0f;
    }
    const unsigned ball = __ballot_sync(0xffffffffu, on);
    if (on) {
        const int a = __popc(ball & ((1u << k) - 1u));
        nb.x[a] = c.x;
        nb.y[a] = c.y;
        nb.z[a] = c.z;
        nb.sx[a] = c.sx;
        nb.sz[a] = c.sz;
    }
    if (k == 0) nb.nact = __popc(ball);
}

// The active neighbours' per-axis terms, spread over the CTA (no barrier).
__device__ __forceinline__ void neighbour_axes(int Dz, int bx, const float* xs, const float* ys, int iz0, float fb,
                                               const NbShared& nb, const NbTab& tb) {
    const int each = 2 * bx + Dz;
    for (int q = threadIdx.x; q < nb.nact * each; q += blockDim.x) {
        const int a = q / each, e = q - a * each;
        if (e < 2 * bx) {
            const bool col = e < bx;
            const int i = col ? e : e - bx;
            const float d = ((col ? xs[i] : ys[i]) - (col ? nb.x[a] : nb.y[a])) / nb.sx[a];
            (col ? tb.x2(a, i) : tb.y2(a, i)) = d * d;
        } else {
            const int z = e - 2 * bx;
            const float dz = (frame_centre(iz0, fb, z) - nb.z[a]) / nb.sz[a];
            tb.z2(a)[z] = dz * dz;
        }
    }
}

// The frame of each neighbour's smallest dz^2 (the first such frame), a warp per neighbour (no barrier).
__device__ __forceinline__ void neighbour_zmin(int Dz, NbShared& nb, const NbTab& tb) {
    const int lane = threadIdx.x & 31;
    for (int a = threadIdx.x >> 5; a < nb.nact; a += blockDim.x >> 5) {
        const float* d2 = tb.z2(a);
        float best = d2[0];
        int bz = 0;
        for (int z = lane; z < Dz; z += 32)
            if (d2[z] < best || (z < bz && d2[z] == best)) {
                best = d2[z];
                bz = z;
            }
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_down_sync(0xffffffffu, best, o);
            const int oz = __shfl_down_sync(0xffffffffu, bz, o);
            if (ov < best || (ov == best && oz < bz)) {
                best = ov;
                bz = oz;
            }
        }
        if (lane == 0) nb.zmin[a] = bz;
    }
}

// Frames of pixel (i, j) inside any active neighbour's ellipsoid: ((dx^2 + dy^2) + dz^2 < 1). dz^2 over the frames
// is unimodal (the bin centres increase, float subtraction, division and squaring are monotone), so for a given
// dx^2 + dy^2 the frames that pass form one interval around the minimum: found by two binary searches on the same
// float comparisons as a full scan.
__device__ __forceinline__ Mask65 neighbour_frames(const NbShared& nb, const NbTab& tb, int i, int j, int Dz) {
    Mask65 m;
    m.clear();
    for (int a = 0; a < nb.nact; ++a) {
        const float dxy = tb.x2(a, i) + tb.y2(a, j);
        const float* d2 = tb.z2(a);
        const int zm = nb.zmin[a];
        if (!(dxy + d2[zm] < 1.0f)) continue;
        int lo = 0, hi = zm;                 // first z in [0, zm] that passes
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (dxy + d2[mid] < 1.0f) hi = mid; else lo = mid + 1;
        }
        const int z0 = lo;
        lo = zm;
        hi = Dz - 1;                         // last z in [zm, Dz - 1] that passes
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (dxy + d2[mid] < 1.0f) lo = mid; else hi = mid - 1;
        }
        const int z1 = lo;
        // bits z0..z1
        if (z0 < 64) {
            const int e = min(z1, 63);
            const unsigned long long upto = (e == 63) ? ~0ull : ((1ull << (e + 1)) - 1ull);
            m.lo |= upto & ~((1ull << z0) - 1ull);
        }
        if (z1 >= 64) m.hi |= 1u;            // Dz <= 65: bit 64 only
    }
    return m;
}

// the bits of frames z0 and on, up to 32 of them
__device__ __forceinline__ unsigned frames_from(const Mask65& m, int z0) {
    return z0 < 64 ? (unsigned)(m.lo >> z0) | (z0 > 32 ? m.hi << (64 - z0) : 0u) : m.hi;
}

// A thread's pixels of a box, tid, tid + blockDim.x, ..., with their column i and row j (stepped, not divided).
struct PixelWalk {
    int p, i, j, di, dj, bx;
    __device__ __forceinline__ explicit PixelWalk(int side) : p(threadIdx.x), bx(side) {
        j = p / bx;
        i = p - j * bx;
        dj = (int)blockDim.x / bx;
        di = (int)blockDim.x - dj * bx;
    }
    __device__ __forceinline__ void next() {
        p += blockDim.x;
        i += di;
        j += dj;
        if (i >= bx) {
            i -= bx;
            ++j;
        }
    }
};

// eps1, eps2 of a box's pixels into shared memory (no barrier).
__device__ __forceinline__ void box_eps(const XiDetector& det, const float S[3], const float e1[3], const float e2[3],
                                        int bx, const float* xs, const float* ys, float* e1s, float* e2s) {
    const int P = bx * bx;
    const float invS = 1.0f / norm3(S[0], S[1], S[2]);
    for (PixelWalk w(bx); w.p < P; w.next()) {
        float a, b;
        eps12(det, S, invS, e1, e2, xs[w.i], ys[w.j], &a, &b);
        e1s[w.p] = a;
        e2s[w.p] = b;
    }
}

// The pixel areas J from a box's eps1, eps2, and seff from the centre's (no barrier).
__device__ __forceinline__ void box_area(int bx, const float* e1s, const float* e2s, float sd, float* J_out,
                                         float* seff_out) {
    const int P = bx * bx;
    for (PixelWalk w(bx); w.p < P; w.next()) {
        const int p = w.p;
        float g[2][2];   // [field][axis x / y]
        const float* f[2] = {e1s, e2s};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float* F = f[q];
            // along x (columns)
            if (w.i == 0)
                g[q][0] = (-1.5f * F[p] + 2.0f * F[p + 1]) - 0.5f * F[p + 2];
            else if (w.i == bx - 1)
                g[q][0] = (0.5f * F[p - 2] - 2.0f * F[p - 1]) + 1.5f * F[p];
            else
                g[q][0] = (F[p + 1] - F[p - 1]) / 2.0f;
            // along y (rows)
            if (w.j == 0)
                g[q][1] = (-1.5f * F[p] + 2.0f * F[p + bx]) - 0.5f * F[p + 2 * bx];
            else if (w.j == bx - 1)
                g[q][1] = (0.5f * F[p - 2 * bx] - 2.0f * F[p - bx]) + 1.5f * F[p];
            else
                g[q][1] = (F[p + bx] - F[p - bx]) / 2.0f;
        }
        const float J = fabsf(g[0][0] * g[1][1] - g[1][0] * g[0][1]);
        J_out[p] = J;
        if (w.j == bx / 2 && w.i == bx / 2) {
            const float psz = sqrtf(J);
            const float q = psz / sd;
            *seff_out = sd * sqrtf(1.0f + (q * q) / 12.0f);
        }
    }
}

// ==================================================================================================================
// shared per-CTA helpers
// ==================================================================================================================

// Rocking-curve fractions of all Dz bins, in two steps: the Dz x 21 mixture terms spread over the CTA, then (after a
// barrier) each bin's terms summed in component order in float64 and rounded once (xpg/integrate_kernels.py:130-141,
// :255-262).
// Out of line, with one error function in it: see the note on the passes' code size at pass1_row.
__device__ __noinline__ void rocking_terms(int Dz, int iz0, float fb, float frames_phi0, float osc, float sm,
                                           const float* rcw, float phi, float zeta, float* terms) {
    const float s = sm / fmaxf(fabsf(zeta), 1e-3f);
    const float sw = (s * 0.25f) * kSqrt2;
    for (int q = threadIdx.x; q < Dz * XI_RC_K; q += blockDim.x) {
        const int z = q / XI_RC_K, k = q % XI_RC_K;
        float lo, hi;
        bin_limits(iz0, fb, z, frames_phi0, osc, &lo, &hi);
        const float c = (k == XI_RC_K - 1) ? 3.5f : (float)((double)k * 0.35 + (-3.5));
        const float cs = c * s;
        float e[2];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const float v = erf32((((h ? lo : hi) - phi) - cs) / sw);
            e[0] = h ? e[0] : v;
            e[1] = v;
        }
        terms[q] = (rcw[k] * 0.5f) * (e[0] - e[1]);
    }
}

__device__ __forceinline__ float rocking_sum(const float* terms, int z) {
    double acc = 0.0;
    for (int k = 0; k < XI_RC_K; ++k) acc += (double)terms[z * XI_RC_K + k];
    return (float)acc;
}

// The foreground frames (R >= 1e-3 * Rmax + 1e-6) as a mask, and Rmax, by a warp (every lane gets them).
__device__ __forceinline__ Mask65 foreground_frames(const float* fR, int Dz, float* Rmax_out) {
    const int lane = threadIdx.x & 31;
    float Rmax = fR[0];
    for (int z = lane; z < Dz; z += 32) Rmax = fmaxf(Rmax, fR[z]);
    for (int o = 16; o > 0; o >>= 1) Rmax = fmaxf(Rmax, __shfl_xor_sync(0xffffffffu, Rmax, o));
    const float thr = 1e-3f * Rmax + 1e-6f;
    const unsigned w0 = __ballot_sync(0xffffffffu, lane < Dz && fR[lane] >= thr);
    const unsigned w1 = __ballot_sync(0xffffffffu, lane + 32 < Dz && fR[lane + 32] >= thr);
    const unsigned w2 = __ballot_sync(0xffffffffu, lane + 64 < Dz && fR[lane + 64] >= thr);
    Mask65 m;
    m.lo = (unsigned long long)w0 | ((unsigned long long)w1 << 32);
    m.hi = w2 & 1u;
    *Rmax_out = Rmax;
    return m;
}

// Sums over 32 lanes of eight values a lane: lane l gets the sum of v[(l >> 2) & 7] (lanes 4 k .. 4 k + 3 the same one),
// in nine shuffles where eight sums take forty. The order of each sum is the same whatever the lane count of the CTA.
__device__ __forceinline__ float warp_sum8(const float (&v)[8]) {
    const int lane = threadIdx.x & 31;
    float a[4], b[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float keep = lane & 16 ? v[4 + j] : v[j], send = lane & 16 ? v[j] : v[4 + j];
        a[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float keep = lane & 8 ? a[2 + j] : a[j], send = lane & 8 ? a[j] : a[2 + j];
        b[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    const float keep = lane & 4 ? b[1] : b[0], send = lane & 4 ? b[0] : b[1];
    float c = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;
}

// Sums over 32 lanes of sixteen doubles a lane: lane l gets the sum of v[l >> 1] (sixteen exchanges, not eighty).
__device__ __forceinline__ double warp_sum16(const double (&v)[16]) {
    const int lane = threadIdx.x & 31;
    double a[8], b[4], c[2];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = (lane & 16 ? v[8 + j] : v[j]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? v[j] : v[8 + j], 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = (lane & 8 ? a[4 + j] : a[j]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? a[j] : a[4 + j], 8);
#pragma unroll
    for (int j = 0; j < 2; ++j) c[j] = (lane & 4 ? b[2 + j] : b[j]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? b[j] : b[2 + j], 4);
    double d = (lane & 2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, lane & 2 ? c[0] : c[1], 2);
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
}

// the sum over a warp in every lane
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per-CTA shared copies of the small tables every pixel reads: the panel maps (up to 16 panels) and the rocking-curve
// weights. Returns the detector description with its panel pointers redirected to the shared copies.
constexpr int kSmemPanels = 16;
struct CtaTables {
    float pan[6][3 * kSmemPanels];
    float rcw[XI_RC_K];
};

__device__ XiDetector cta_tables(const XiDetector& det, const XiBlock& B, CtaTables& T) {
    XiDetector d = det;
    const int np = det.n_panels;
    if (np <= kSmemPanels) {
        for (int r = threadIdx.x; r < 3 * np; r += blockDim.x) {
            T.pan[0][r] = det.P0[r];
            T.pan[1][r] = det.Bx[r];
            T.pan[2][r] = det.By[r];
            T.pan[3][r] = det.U1[r];
            T.pan[4][r] = det.U2[r];
            T.pan[5][r] = det.UN[r];
        }
        d.P0 = T.pan[0];
        d.Bx = T.pan[1];
        d.By = T.pan[2];
        d.U1 = T.pan[3];
        d.U2 = T.pan[4];
        d.UN = T.pan[5];
    }
    for (int k = threadIdx.x; k < XI_RC_K; k += blockDim.x) T.rcw[k] = B.rcw[k];
    return d;
}

// Asks for a shoebox of V floats in L2 (by one thread; whole 16-byte units), so that it comes from DRAM while the
// row's geometry is computed.
__device__ __forceinline__ void prefetch_box(const float* sb, int V) {
    const uintptr_t a = (reinterpret_cast<uintptr_t>(sb) + 15) & ~(uintptr_t)15;
    const uintptr_t e = reinterpret_cast<uintptr_t>(sb + V) & ~(uintptr_t)15;
    if (e > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
}

// Completes the staging of a shoebox in shared memory: waits for phase `parity` of the bulk copy's barrier (bounded;
// on a timeout the status word gets bit 2 and the values are copied with plain loads), or copies with plain loads
// when the row's arena offset is not 16-byte aligned. Ends with a barrier.
__device__ void stage_wait(bool tma, unsigned long long* bar, unsigned parity, float* stage, const float* sb, int V,
                           int* status) {
    bool ok = true;
    if (tma) ok = mbar_wait(bar, parity, 1ll << 24);
    if (!tma || !ok) {
        // (no barrier here: the wait may run out for some threads only; the others' share has arrived by the copy)
        if (!ok) atomicOr(status, 2);
        for (int v = threadIdx.x; v < V; v += blockDim.x) stage[v] = sb[v];
    } else {
        // the bulk copy moved whole 16-byte units; the last 0..3 values come with plain loads (no read past the row)
        for (int v = (V & ~3) + threadIdx.x; v < V; v += blockDim.x) stage[v] = sb[v];
    }
    __syncthreads();
}

// ==================================================================================================================
// pass 1
// ==================================================================================================================
constexpr int kClipCand = 1024;     // background voxels above the lowest clip threshold kept per CTA, at most
constexpr int kFgList = 2048;       // foreground pixels listed per CTA (pass C iterates them densely), at most
constexpr int kClipWarp = 256;      // candidates that one warp iterates alone
constexpr int kScan = 9;            // voxels of a pixel column that pass 1's scan takes together (depths: 3, 5, 9, 17, ...)
constexpr int kValid = 17;          // in pass 2, whose scan only compares
constexpr int kZBatch = 8;          // and pass C, whose frame sums go by eights
// The gather's threads per row and the frames of a box pixel that a thread reads together. Bound by memory latency
// (15 of 20 stall cycles) and by how many frames' pages are open at once: more frames in flight a thread make it slower
// (16 frames: 16.7 ms for the 16M-pixel sweep's 107,446 rows), more pixels of the same frames faster. 128 threads and
// 8 frames: 5.94 ms there and 5.10 ms for the 4M-pixel sweep's 90,287; 256 and 4: 5.06 and 4.44 ms; 512 and 4: 4.80 and
// 4.96 ms; 128 and 4: 5.75 and 4.96 ms. Two rules beside that:
// - where the launch's largest box is known to have no more than 128 pixels, 128 threads: the others only kept rows off
//   the SM (30,000 boxes of 9 x 9 x 5: 70 us with 128 and 8 frames, 79 with 256 and 4, 59 with 128 and 4; a fifth of the
//   rows, 11, 13.5 and 11). Not from 13 px on: 100 boxes of 13 x 13 x 17 6.6 us with 256, 9.4 with 128, 10,000 of
//   17 x 17 x 33 234 and 278.
// - float frames, which are not encoded after the load, are bound by the loads in flight: 128 threads up to 17 px (23,068
//   boxes of 17 x 17 x 9: 134 us with 128 and 8 frames, 146 with 256 and 4, 133 so), eight frames a thread from there on
//   (1,250 boxes of 73 x 73 x 9: 133, 149 and 132 us).
constexpr int kGatherThreads = 256;
constexpr int kGatherSmall = 11, kGatherSmallFloat = 17;  // largest side of a launch with half the threads
constexpr int kGatherBatch = 4, kGatherFloatBatch = 8;

// Dynamic shared memory of pass 1 for boxes up to max_bx pixels a side and max_dz bins with K neighbour columns: the
// neighbours' frame masks (8P) | geometry scratch eps1, then the background template (4P) | eps2, then the img2 counts
// (4P) | per pixel the number of clean foreground-frame voxels and the all-clean bit (P) | frame 64's neighbour bits,
// the foreground pixels and the background ring's (a bit each) | foreground list | rocking-curve terms, then the clip
// candidates | the neighbours' axis terms | staged shoebox.
struct Pass1Layout {
    int Pm, cap, fgcap;
    size_t e1, e2, imgn, hi, fg, ring, fgl, scr, nbt, stage, bytes;

    __host__ __device__ Pass1Layout(int max_bx, int max_dz, int K, bool staged) {
        Pm = max_bx * max_bx;
        cap = Pm * max_dz < kClipCand ? Pm * max_dz : kClipCand;
        fgcap = Pm < kFgList ? Pm : kFgList;
        e1 = (size_t)8 * Pm;
        e2 = e1 + (size_t)4 * Pm;
        imgn = e2 + (size_t)4 * Pm;
        hi = (imgn + Pm + 3) / 4 * 4;
        fg = hi + (max_dz > 64 ? (size_t)(Pm + 31) / 32 * 4 : 0);
        ring = fg + (size_t)(Pm + 31) / 32 * 4;
        fgl = ring + (size_t)(Pm + 31) / 32 * 4;
        scr = (fgl + (size_t)2 * fgcap + 15) / 16 * 16;
        const size_t c = (size_t)6 * cap, t = (size_t)max_dz * XI_RC_K * sizeof(float);
        nbt = (scr + (c > t ? c : t) + 15) / 16 * 16;
        stage = nbt + nb_bytes(K, max_bx, max_dz);
        bytes = stage + (staged ? ((size_t)Pm * max_dz * sizeof(float) + 15) / 16 * 16 : 0);
    }
};

// resident CTAs per SM the pass kernels are compiled for (registers per thread <= 65536 / (NT * blocks)): 64 registers
// in pass 1, 80 in pass 2
template <int NT> constexpr int min_ctas() { return 768 / NT; }
template <int NT> constexpr int min_ctas_pass1() { return 1024 / NT; }

// Pass 1 of one row, by the whole CTA. `bar`: the CTA's bulk-copy barrier (initialised once per CTA), `phase`: its
// next phase (advanced here when the row is staged by a bulk copy). The caller separates consecutive rows of a CTA
// with a barrier.
//
// Bound by instructions and by the latency of its serial steps, not by bytes: each voxel is read once from DRAM. So
// the scan of the box (pass A, 40% of a row's time when every voxel took its own tests) takes nine voxels at a time
// and tests them together (all valid, none above the lowest clip threshold): a batch that passes needs only its sums,
// one that fails makes its masks and splits its sums by them, from the same registers. Going voxel by voxel through such
// a batch, its values read again, was 1.25 times the time of one loop over all voxels where the background lies above
// the threshold (1,261 boxes of 31 x 31 x 33 with 20 counts a voxel: 0.527 ms, 0.662 so, 0.517 now), and most columns of
// a common box hold such a batch. The set-up steps share barriers, the clipping iterations run in one warp, and the
// per-frame sums of pass C reduce eight frames at a time (warp_sum8).
//
// Code size counts: the resident CTAs' warps are in different steps of a row, and with the loops over 32-frame words
// and the error functions unrolled or inlined several times, a third of the stalls were waits for instructions. What a
// row runs twice is one function. (Loads of the next batch ahead of the tests, in more registers, lost more by their
// code than they hid: 13.9 ms in place of 12.1 for the sweep below at that stage.)
//
// Before and after: 107,446 rows of the 16M-pixel geometry (90 frames, 2.6e9 voxels) 14.1 -> 9.3 ms, 4,096 boxes of
// 31 x 31 x 33 0.82 -> 0.48 ms, 40,001 of 9 x 9 x 5 0.90 -> 0.52 ms.
template <int NT, bool STAGED>
__device__ __forceinline__ void pass1_row(const XiDetector& det_g, const XiRows& R, const XiBlock& B,
                                          const float* __restrict__ arena, const XiPass1Out& O, int row, int max_bx,
                                          int max_dz, int* status, unsigned long long* bar, unsigned& phase) {
    extern __shared__ __align__(16) unsigned char dyn1[];
    constexpr int kW = NT / 32;
    __shared__ CtaTables T;
    __shared__ float xs[XI_MAX_BX], ys[XI_MAX_BX];
    __shared__ float fR[XI_MAX_DZ];
    __shared__ float4 fcol[XI_MAX_DZ];              // frame: (centre, e3, e3^2)
    __shared__ NbShared nb;
    __shared__ float s_e1[3], s_e2[3], s_S[3], s_zeta, s_seff, s_b;
    __shared__ Mask65 s_fgz;
    __shared__ unsigned s_rec[3];
    __shared__ int s_int[3];
    __shared__ double red[kW * 16];
    __shared__ double tot[16];
    __shared__ double fzw[kW][XI_MAX_DZ];
    // background voxels above the lowest possible clip threshold (the only ones the iterations can drop)
    __shared__ int s_ncand;
    __shared__ double s_nbg, s_fr;

    // the row's scalars, all asked for at once
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int Dz = R.Dz[row], bx = R.bx[row];
    NbColumn nbc;
    if (warp == kW - 1 && lane < R.K) nbc.load(R, row, lane);
    const int pxs = R.pxs ? R.pxs[row] : 1;
    const int ix0 = R.ix0[row], iy0 = R.iy0[row], iz0 = R.iz0[row];
    const float fb = R.fb[row];
    const float phi = R.phi[row];
    const float* sb = arena + R.sb_off[row];
    const int64_t po = R.pix_off[row], fo = R.frm_off[row];
    float S[3] = {0.0f, 0.0f, 0.0f};
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; ++c) S[c] = R.S[3 * row + c];
    if (Dz < 1 || Dz > max_dz || bx < 3 || bx > max_bx) {
        if (threadIdx.x == 0) atomicOr(status, 1);
        return;
    }
    const int P = bx * bx;
    const Pass1Layout L(max_bx, max_dz, R.K, STAGED);    // the tables are laid out for the launch's largest box
    unsigned long long* nblo = reinterpret_cast<unsigned long long*>(dyn1);
    float* e1s = reinterpret_cast<float*>(dyn1 + L.e1);
    float* e2s = reinterpret_cast<float*>(dyn1 + L.e2);
    float* brefs = e1s;                            // a pixel's own slot, once its u1 / u2 are out
    float* ics = e2s;
    unsigned char* imgn = dyn1 + L.imgn;            // per pixel: clean foreground-frame voxels | all-clean bit 7
    unsigned* nbhi = reinterpret_cast<unsigned*>(dyn1 + L.hi);
    unsigned* fgw = reinterpret_cast<unsigned*>(dyn1 + L.fg);
    unsigned* ringw = reinterpret_cast<unsigned*>(dyn1 + L.ring);
    unsigned short* fgl = reinterpret_cast<unsigned short*>(dyn1 + L.fgl);
    float* terms = reinterpret_cast<float*>(dyn1 + L.scr);
    float* cand_v = terms;
    unsigned short* cand_p = reinterpret_cast<unsigned short*>(dyn1 + L.scr + (size_t)4 * L.cap);
    float* stage = reinterpret_cast<float*>(dyn1 + L.stage);
    const NbTab tb = nb_tab(dyn1 + L.nbt, R.K, max_bx, max_dz);
    const float gain = B.gain, bias = R.sb_bias;
    const float* box = STAGED ? stage : sb;
    // the shoebox streams into shared memory (bulk copy) while the geometry below is computed
    const unsigned vbytes = (unsigned)(((size_t)Dz * P * sizeof(float)) & ~(size_t)15);   // whole 16-byte units
    const bool tma = STAGED && vbytes > 0 && ((reinterpret_cast<uintptr_t>(sb) & 15) == 0) &&
                     ((reinterpret_cast<uintptr_t>(stage) & 15) == 0);
    if (tma && threadIdx.x == 0) {
        mbar_expect_tx(bar, vbytes);
        bulk_copy_g2s(stage, sb, vbytes, bar);
    }
    if (!STAGED && threadIdx.x == 0) prefetch_box(sb, Dz * P);

    const XiDetector det = cta_tables(det_g, B, T);
    if (threadIdx.x == 0) {
        float e1[3], e2[3], zeta;
        kabsch_frame(S, B.s0, B.axis, e1, e2, &zeta);
        for (int c = 0; c < 3; ++c) { s_e1[c] = e1[c]; s_e2[c] = e2[c]; s_S[c] = S[c]; }
        s_zeta = zeta;
        s_ncand = 0;
    }
    if (threadIdx.x < 3) {
        s_rec[threadIdx.x] = 0u;
        s_int[threadIdx.x] = 0;
    }
    for (int i = threadIdx.x; i < bx; i += NT) {
        xs[i] = box_coord(ix0, i, pxs);
        ys[i] = box_coord(iy0, i, pxs);
    }
    if (max_dz > 64)
        for (int w = threadIdx.x; w < (P + 31) / 32; w += NT) nbhi[w] = 0u;
    __syncthreads();
    const float zeta = s_zeta;
    if (warp == kW - 1)
        neighbour_test(nbc, R.K, false, bx, xs, ys, frame_centre(iz0, fb, 0), frame_centre(iz0, fb, Dz - 1), nb);
    rocking_terms(Dz, iz0, fb, B.frames_phi0, B.osc, B.sm, T.rcw, phi, zeta, terms);
    for (int z = lane; z < Dz; z += 32) fzw[warp][z] = 0.0;
    __syncthreads();
    for (int z = NT - 1 - (int)threadIdx.x; z < Dz; z += NT) {     // (the last threads have the fewest pixels)
        fR[z] = rocking_sum(terms, z);
        float lo, hi;
        bin_limits(iz0, fb, z, B.frames_phi0, B.osc, &lo, &hi);
        const float e3 = zeta * (0.5f * (lo + hi) - phi);
        fcol[z] = make_float4(frame_centre(iz0, fb, z), e3, e3 * e3, 0.0f);
    }
    const int nact = nb.nact;
    if (nact) neighbour_axes(Dz, bx, xs, ys, iz0, fb, nb, tb);
    {
        float e1[3] = {s_e1[0], s_e1[1], s_e1[2]}, e2[3] = {s_e2[0], s_e2[1], s_e2[2]};
        const float Sr[3] = {s_S[0], s_S[1], s_S[2]};
        box_eps(det, Sr, e1, e2, bx, xs, ys, e1s, e2s);
    }
    __syncthreads();
    box_area(bx, e1s, e2s, B.sd, O.J + po, &s_seff);
    if (warp == kW - 1) {
        float Rmax;
        const Mask65 m = foreground_frames(fR, Dz, &Rmax);
        if (lane == 0) s_fgz = m;
    }
    if (nact) neighbour_zmin(Dz, nb, tb);
    const bool templ = det.bkg != nullptr;
    // The clip threshold (bp + 3 sqrt(gain max(bp, 0.5))) + 1 is non-decreasing in bp = b * bref >= 0 (every
    // float operation in it is monotone), so it never falls below its value at bp = 0: background voxels at or
    // below that bound pass every iteration. They are summed once; the others are listed for the iterations.
    int neg_bref = 0;
    if (templ)
        for (PixelWalk w(bx); w.p < P; w.next()) neg_bref |= (bkg_ref(det, xs[w.i], ys[w.j]) < 0.0f);
    const bool use_list = !__syncthreads_or(neg_bref);
    const Mask65 fgz = s_fgz;
    const float seff = s_seff;
    if (STAGED) {
        stage_wait(tma, bar, phase, stage, sb, Dz * P, status);
        if (tma) phase ^= 1u;
    }

    // ---- per pixel: u1 / u2 out, foreground / background ring, neighbour frames, and pass A: first background
    // estimate, counts, recorded frames, the b-independent part of img2. A pixel column's background counts are
    // summed in float32 (exact for detector counts: integers whose column sum stays below 2^24; a larger column is
    // summed again in float64) and its template weight as count * bref, so the float64 totals equal voxel-by-voxel
    // float64 sums.
    const float clip_floor = (0.0f + 3.0f * sqrtf(gain * fmaxf(0.0f, 0.5f))) + 1.0f;
    {
        Mask65 rec;
        rec.clear();
        int t_over = 0, t_fgm = 0, t_fgnb = 0;
        double a4[4] = {0.0, 0.0, 0.0, 0.0};         // counts, weights; of the voxels no iteration can drop
        PixelWalk px(bx);
        for (int p0 = 0; p0 < P; p0 += NT, px.next()) {
            const int p = px.p;
            bool fg2 = false, ring = false;
            if (p < P) {
                const float u1 = e1s[p] / seff, u2 = e2s[p] / seff;
                O.u1[po + p] = u1;
                O.u2[po + p] = u2;
                const float r2 = u1 * u1 + u2 * u2;
                fg2 = r2 <= kFgR2;
                ring = r2 >= kBgR2;
            }
            const unsigned ball = __ballot_sync(0xffffffffu, fg2), rball = __ballot_sync(0xffffffffu, ring);
            if (lane == 0 && p < P) {
                fgw[p >> 5] = ball;
                ringw[p >> 5] = rball;
            }
            if (p >= P) continue;
            float bref = 1.0f;
            if (templ) {
                bref = bkg_ref(det, xs[px.i], ys[px.j]);
                brefs[p] = bref;
            }
            Mask65 nbm;
            nbm.clear();
            if (nact) {
                nbm = neighbour_frames(nb, tb, px.i, px.j, Dz);
                nblo[p] = nbm.lo;
                if (nbm.hi) atomicOr(&nbhi[p >> 5], 1u << (p & 31));
            }
            float cs = 0.0f, cs0 = 0.0f, ic = 0.0f;
            int cn = 0, cn0 = 0, in_ = 0;
            bool okall = true;
            const float* col = box + p;
#pragma unroll 1
            for (int z0 = 0; z0 < Dz; z0 += kScan, col += (size_t)kScan * P) {
                const int nbat = min(kScan, Dz - z0);
                const unsigned all = (1u << nbat) - 1u;
                const unsigned ib = frames_from(fgz, z0) & all;   // its foreground frames (the same in every thread)
                const unsigned kb = frames_from(nbm, z0) & all;   // and its neighbours' frames
                float v[kScan];                            // independent loads in flight before any is used
#pragma unroll
                for (int u = 0; u < kScan; ++u) v[u] = u < nbat ? col[(size_t)u * P] : bias;
                bool ok = true, low = true;
#pragma unroll
                for (int u = 0; u < kScan; ++u) {
                    v[u] = v[u] - bias;
                    ok = ok && v[u] >= 0.0f;
                    low = low && v[u] <= clip_floor;       // (false of NaN)
                }
                unsigned vm = all, rm = all, om = 0u;      // valid, recorded, overloaded
                if (!ok) {
                    vm = rm = 0u;
#pragma unroll
                    for (int u = 0; u < kScan; ++u) {
                        vm |= (unsigned)(v[u] >= 0.0f) << u;
                        rm |= (unsigned)(v[u] > -2.5f) << u;
                        om |= (unsigned)(v[u] == -2.0f) << u;
                    }
                    vm &= all;
                    rm &= all;
                }
                const unsigned mine = vm & ~kb;            // valid and not a neighbour's
                if (ib) {
                    const unsigned m = ib & mine;
#pragma unroll
                    for (int u = 0; u < kScan; ++u)
                        if ((m >> u) & 1u) ic += v[u];
                }
                if (ring) {                                // background (the ring excludes the foreground ellipse)
                    unsigned hm = 0u;                      // its voxels above the lowest clip threshold
                    if (low) {
#pragma unroll
                        for (int u = 0; u < kScan; ++u)
                            if ((mine >> u) & 1u) cs0 += v[u];
                    } else {
#pragma unroll
                        for (int u = 0; u < kScan; ++u)
                            if ((mine >> u) & 1u) {
                                const bool up = !(v[u] <= clip_floor);
                                hm |= (unsigned)up << u;
                                cs0 += up ? 0.0f : v[u];
                                cs += up ? v[u] : 0.0f;
                            }
                    }
                    cn0 += __popc(mine & ~hm);
                    if (hm) {
                        cn += __popc(hm);
                        // listed while the list has room (a full list is not used, so it need not be counted on)
                        if (use_list && *(volatile int*)&s_ncand <= L.cap) {
                            int k = atomicAdd(&s_ncand, __popc(hm));
#pragma unroll 1
                            for (unsigned r = hm; r; r &= r - 1u, ++k)
                                if (k < L.cap) {           // (the value read again: the batch is near)
                                    cand_v[k] = col[(size_t)(__ffs(r) - 1) * P] - bias;
                                    cand_p[k] = (unsigned short)p;
                                }
                        }
                    }
                }
                if (z0 < 64) rec.lo |= (unsigned long long)rm << z0;
                if (z0 > 64 - kScan) rec.hi |= z0 < 64 ? rm >> (64 - z0) : rm;
                if (!ib) continue;
                const unsigned fgm = fg2 ? ib : 0u;       // foreground voxels of the batch
                t_over += __popc(fgm & om);
                t_fgm += __popc(fgm & ~vm & rm);
                t_fgnb += __popc(fgm & kb);
                const unsigned clean_fg = ib & vm & ~kb;   // foreground-frame voxels valid and not a neighbour's
                in_ += __popc(clean_fg);
                if (clean_fg != ib) okall = false;
            }
            double csd = (double)cs;
            if (cs >= 16777216.0f) {                     // float32 may have rounded: this column again in float64
                csd = 0.0;
                for (int z = 0; z < Dz; ++z) {
                    const float v = box[(size_t)z * P + p] - bias;
                    if (ring && v >= 0.0f && !nbm.get(z) && v > clip_floor) csd += (double)v;
                }
            }
            a4[0] += csd + (double)cs0;
            a4[1] += (double)(cn + cn0) * (double)bref;
            a4[2] += (double)cs0;
            a4[3] += (double)cn0 * (double)bref;
            ics[p] = ic;                                 // completed with the background after pass B
            imgn[p] = (unsigned char)(in_ | (okall ? 0x80 : 0));
        }
        const unsigned r3[3] = {(unsigned)rec.lo, (unsigned)(rec.lo >> 32), rec.hi};
#pragma unroll
        for (int w = 0; w < 3; ++w) {
            const unsigned r = __reduce_or_sync(0xffffffffu, r3[w]);
            if (lane == 0 && r) atomicOr(&s_rec[w], r);
        }
        const int t3[3] = {t_over, t_fgm, t_fgnb};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int t = __reduce_add_sync(0xffffffffu, t3[q]);
            if (lane == 0 && t) atomicAdd(&s_int[q], t);
        }
        block_sum<NT, 4>(a4, red, tot);
    }
    float b = (float)tot[0] / fmaxf((float)tot[1], 1e-6f);
    const double base_c = tot[2], base_b = tot[3];
    const int ncand = s_ncand;
    const bool listed = use_list && ncand <= L.cap;
    // the foreground pixels listed in pixel order: every warp scans the counts of the bit words, each fills its own
    // words' pixels (the list, and so every later sum over it, is the same on every run)
    int nfl = 0;
    {
        const int nw = (P + 31) / 32;
        for (int w0 = 0; w0 < nw; w0 += 32) {
            const unsigned word = w0 + lane < nw ? fgw[w0 + lane] : 0u;
            int incl = __popc(word);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int excl = nfl + incl - __popc(word);
            for (int w = warp; w < min(32, nw - w0); w += kW) {
                const unsigned bits = __shfl_sync(0xffffffffu, word, w);
                const int k = __shfl_sync(0xffffffffu, excl, w) + __popc(bits & ((1u << lane) - 1u));
                if (((bits >> lane) & 1u) && k < L.fgcap) fgl[k] = (unsigned short)(32 * (w0 + w) + lane);
            }
            nfl += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    // the rocking curve recorded
    if (warp == kW - 1) {
        double fr = 0.0;
        for (int z = lane; z < Dz; z += 32)
            if ((s_rec[z >> 5] >> (z & 31)) & 1u) fr += (double)fR[z];
        fr = warp_total(fr);
        if (lane == 0) s_fr = fr;
    }
    // ---- passes B: Poisson-aware clipped background, 4 iterations (background-ring pixels only)
    double nbg_d = 0.0;
    auto clip_threshold = [&](float bp) { return (bp + 3.0f * sqrtf(gain * fmaxf(bp, 0.5f))) + 1.0f; };
    auto clip_candidates = [&](int first, int step, double& sc, double& sw) {
        const float flat = clip_threshold(b * 1.0f);
        for (int k = first; k < ncand; k += step) {
            const float v = cand_v[k];
            const float bref = templ ? brefs[cand_p[k]] : 1.0f;
            if (v <= (templ ? clip_threshold(b * bref) : flat)) {
                sc += (double)v;
                sw += (double)bref;
            }
        }
    };
    if (listed && ncand <= kClipWarp) {                  // few candidates: one warp, no barriers
        if (warp == 0) {
            for (int it = 0; it < 4; ++it) {
                double sc = 0.0, sw = 0.0;
                clip_candidates(lane, 32, sc, sw);
                const double tc = base_c + warp_total(sc);
                nbg_d = base_b + warp_total(sw);
                const float was = b;
                b = (float)tc / fmaxf((float)nbg_d, 1e-6f);
                if (b == was && it) break;               // the same voxels again: so would every later iteration
            }
            if (lane == 0) {
                s_b = b;
                s_nbg = nbg_d;
            }
        }
        __syncthreads();
        b = s_b;
        nbg_d = s_nbg;
    } else {
        for (int it = 0; it < 4; ++it) {
            double a2[2] = {0.0, 0.0};
            if (listed) {
                clip_candidates(threadIdx.x, NT, a2[0], a2[1]);
            } else {
                for (int p = threadIdx.x; p < P; p += NT) {
                    if (!((ringw[p >> 5] >> (p & 31)) & 1u)) continue;
                    const float bref = templ ? brefs[p] : 1.0f;
                    const float thr = clip_threshold(b * bref);
                    Mask65 nbm;
                    nbm.clear();
                    if (nact) {
                        nbm.lo = nblo[p];
                        nbm.hi = max_dz > 64 ? (nbhi[p >> 5] >> (p & 31)) & 1u : 0u;
                    }
                    for (int z = 0; z < Dz; ++z) {
                        const float v = box[(size_t)z * P + p] - bias;
                        if (v >= 0.0f && !nbm.get(z) && v <= thr) {
                            a2[0] += (double)v;
                            a2[1] += (double)bref;
                        }
                    }
                }
            }
            block_sum<NT, 2>(a2, red, tot);
            const double tc = (listed ? base_c : 0.0) + tot[0];
            nbg_d = (listed ? base_b : 0.0) + tot[1];
            b = (float)tc / fmaxf((float)nbg_d, 1e-6f);
            __syncthreads();                             // tot is read before the next iteration's sums
        }
    }
    // ---- pass C: summation, centroid, moments, per-frame net over the listed foreground pixels; img2 ---------
    // img2 is linear in the background: each pixel's clean foreground-frame count sum (pass A) minus its count of
    // such voxels times b * bref. The foreground sums run over the pixel list (every lane a foreground pixel);
    // a column's sums are taken in float32 (<= 65 terms), then weighted by the pixel's constants and added in
    // float64; a frame's net sum is float32 over 32 pixels of the list, float64 beyond. (Also splitting the frames
    // over the warps, as a row may have few foreground pixels, cost more in longer code than it gave: 12.6 ms in place
    // of 12.1 for the 16M-pixel sweep's pass 1.)
    for (int p = threadIdx.x; p < P; p += NT) {
        const unsigned char m = imgn[p];
        O.img2[po + p] = ics[p] - (float)(m & 0x7f) * (b * (templ ? brefs[p] : 1.0f));
        O.all_valid2[po + p] = m >> 7;
    }
    double acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = 0.0;
    const bool fl_listed = nfl <= L.fgcap;
    const int n_items = fl_listed ? nfl : P;
    for (int k0 = 32 * warp; k0 < n_items; k0 += NT) {
        const int k = k0 + lane;
        int p = 0;
        bool have = k < n_items;
        if (have) {
            p = fl_listed ? (int)fgl[k] : k;
            have = fl_listed || ((fgw[p >> 5] >> (p & 31)) & 1u);
        }
        if (!__any_sync(0xffffffffu, have)) continue;      // warp-uniform: no foreground pixel in this warp
        float u1 = 0.f, u2 = 0.f, bref = 1.f;
        Mask65 nbm;
        nbm.clear();
        if (have) {
            u1 = O.u1[po + p];
            u2 = O.u2[po + p];
            if (templ) bref = brefs[p];
            if (nact) {
                nbm.lo = nblo[p];
                if (max_dz > 64) nbm.hi = (nbhi[p >> 5] >> (p & 31)) & 1u;
            }
        }
        const float bpix = b * bref;
        float c_net = 0.f, c_c = 0.f, c_w = 0.f, c_wz = 0.f, c_e3 = 0.f, c_e33 = 0.f;
        int c_n = 0, c_raw = 0;                              // exact: <= 65 counts below 2^23 each
        const float* col = box + p;
#pragma unroll 1
        for (int z0 = 0; z0 < Dz; z0 += kZBatch, col += (size_t)kZBatch * P) {
            const int nbat = min(kZBatch, Dz - z0);
            const unsigned ib = frames_from(fgz, z0), kb = frames_from(nbm, z0);
            float v[kZBatch];
#pragma unroll
            for (int u = 0; u < kZBatch; ++u) v[u] = have && u < nbat ? col[(size_t)u * P] : 0.0f;
#pragma unroll
            for (int u = 0; u < kZBatch; ++u) {
                const float c = v[u] - bias;
                const bool clean = have && u < nbat && c >= 0.0f && !((kb >> u) & 1u);
                const float cc = clean ? c : 0.0f;
                const float net = clean ? c - bpix : 0.0f;
                v[u] = net;
                if ((ib >> u) & 1u) {                  // a foreground frame (the same in every thread)
                    const float4 f = fcol[z0 + u];
                    c_n += clean ? 1 : 0;
                    c_net += net;
                    c_c += cc;
                    c_raw += (int)cc;
                    const float wpos = fmaxf(net, 0.0f);
                    c_w += wpos;
                    c_wz += wpos * f.x;
                    c_e3 += net * f.y;
                    c_e33 += net * f.z;
                }
            }
            const float s = warp_sum8(v);
            const int u = (lane >> 2) & 7;
            if ((lane & 3) == 0 && u < nbat) fzw[warp][z0 + u] += (double)s;
        }
        if (have && c_n > 0) {
            const int j = p / bx, i = p - j * bx;
            const float x = xs[i], y = ys[j];
            const float eps1 = u1 * seff, eps2 = u2 * seff;
            const float e12 = eps1 * eps1 + eps2 * eps2;
            acc[14] += (double)c_n;
            acc[0] += (double)c_n * (double)bref;             // sfb
            acc[1] += (double)c_net;                          // isum, and the moments' weight
            acc[2] += (double)c_c;                            // vsum counts
            acc[3] += (double)c_n * (double)bpix;             // vsum0
            acc[4] += (double)c_w;                            // sw
            acc[5] += (double)c_w * (double)x;
            acc[6] += (double)c_w * (double)y;
            acc[7] += (double)c_wz;
            acc[8] += (double)c_raw;                          // integer partial sums below 2^53: exact
            acc[9] += (double)c_net * (double)eps1;
            acc[10] += (double)c_net * (double)eps2;
            acc[11] += (double)c_net * (double)e12;
            acc[12] += (double)c_e3;
            acc[13] += (double)c_e33;
        }
    }
    {
        const double t = warp_sum16(acc);
        if (!(lane & 1)) red[warp * 16 + (lane >> 1)] = t;
        __syncthreads();
        if (threadIdx.x < 16) {
            double v = 0.0;
            for (int w = 0; w < kW; ++w) v += red[w * 16 + threadIdx.x];
            tot[threadIdx.x] = v;
        }
        __syncthreads();
    }
    for (int z = threadIdx.x; z < Dz; z += NT) {
        double s = 0.0;
        for (int w = 0; w < kW; ++w) s += fzw[w][z];
        O.fz[fo + z] = (float)s;
    }
    if (warp == 0) {
        // the row's quotients, one a lane: the centroid over sw (lanes 5..7), the moments over sws (lanes 9..13)
        const float sw = fmaxf((float)tot[4], 1e-6f);
        const float sws = fmaxf((float)tot[1], 1e-6f);
        const float num = lane < 15 ? (float)tot[lane] : 0.0f;
        const float q = num / (lane < 9 ? sw : sws);
        const float mu1 = __shfl_sync(0xffffffffu, q, 9), mu2 = __shfl_sync(0xffffffffu, q, 10);
        const float e12 = __shfl_sync(0xffffffffu, q, 11), mu3 = __shfl_sync(0xffffffffu, q, 12);
        const float e33 = __shfl_sync(0xffffffffu, q, 13);
        if (lane == 5) O.xo[row] = q;
        if (lane == 6) O.yo[row] = q;
        if (lane == 7) O.zo[row] = q;
        if (lane == 0) {
            const float nbg = (float)nbg_d;
            const float sfb = (float)tot[0];
            const float tail = ((sfb * sfb) * gain) * fmaxf(b, kVarFloor) / fmaxf(nbg, 1.0f);
            O.bg[row] = b;
            O.nbg[row] = nbg;
            O.isum[row] = (float)tot[1];
            O.vsum[row] = gain * (float)tot[2] + tail;
            O.vsum0[row] = gain * (float)tot[3] + tail;
            O.m_d[row] = ((e12 - mu1 * mu1) - mu2 * mu2) / 2.0f;
            O.m_m[row] = e33 - mu3 * mu3;
            O.frac_rec[row] = (float)s_fr;
            O.nfg[row] = (float)tot[14];
            O.zeta[row] = zeta;
            O.seff[row] = seff;
            O.n_over[row] = s_int[0];
            O.n_fg_masked[row] = s_int[1];
            O.n_fg_nb[row] = s_int[2];
            if (O.isum_raw) O.isum_raw[row] = (int64_t)tot[8];
        }
    }
}

// Pass 1, one CTA per row of `order` (one shoebox shape group per launch).
template <int NT, bool STAGED>
__global__ void __launch_bounds__(NT, min_ctas_pass1<NT>()) k_pass1(XiDetector det_g, XiRows R, XiBlock B,
                                                              const float* __restrict__ arena, XiPass1Out O,
                                                              const int32_t* __restrict__ order, int max_bx,
                                                              int max_dz, int* status) {
    __shared__ __align__(8) unsigned long long s_bar;
    if (STAGED) {
        if (threadIdx.x == 0) mbar_init(&s_bar, 1);
        __syncthreads();
    }
    unsigned phase = 0;
    pass1_row<NT, STAGED>(det_g, R, B, arena, O, order ? order[blockIdx.x] : blockIdx.x, max_bx, max_dz, status,
                          &s_bar, phase);
}

// A row set's description copied into the CTA's shared memory (all threads take the same branch: `cur` was read
// after a barrier); thread 0 records which set it holds once every thread has passed the test.
__device__ __forceinline__ void load_set(const XiRowSet* __restrict__ sets, int set, XiRowSet* buf, int* cur) {
    const int* src = reinterpret_cast<const int*>(sets + set);
    int* dst = reinterpret_cast<int*>(buf);
    for (int w = threadIdx.x; w < (int)(sizeof(XiRowSet) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    if (threadIdx.x == 0) *cur = set;
}

// Pass 1 over a queue of (set, row) items: resident CTAs take items in queue order until it is empty, so rows of
// any blocks and sweeps (of one size bin) share one launch with no tail between shape groups.
template <int NT, bool STAGED>
__global__ void __launch_bounds__(NT, min_ctas_pass1<NT>()) k_pass1_q(const XiRowSet* __restrict__ sets,
                                                                const int64_t* __restrict__ items, int n_items,
                                                                int max_bx, int max_dz, int max_k, int* queue,
                                                                int* status) {
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ XiRowSet s_set;
    __shared__ int s_item, s_cur;
    if (threadIdx.x == 0) {
        if (STAGED) mbar_init(&s_bar, 1);
        s_cur = -1;
    }
    unsigned phase = 0;
    for (;;) {
        __syncthreads();                 // the previous row's shared memory is free
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= n_items) return;
        const int64_t v = items[it];
        const int set = (int)(v >> 32);
        if (set != s_cur) load_set(sets, set, &s_set, &s_cur);
        if (s_set.rows.K > max_k) {          // neighbour tables are sized for max_k columns: skip, flag
            if (threadIdx.x == 0) atomicOr(status, 1);
            continue;
        }
        pass1_row<NT, STAGED>(s_set.det, s_set.rows, s_set.blk, s_set.arena, s_set.p1, (int)(v & 0xffffffffll),
                              max_bx, max_dz, status, &s_bar, phase);
    }
}

// ==================================================================================================================
// pass 2
// ==================================================================================================================
constexpr int kFitPix = 2048;       // pixels that may hold fitted voxels, listed per CTA when not all of the box's can
constexpr int kFitChunk = 9;        // frames of such a pixel that a thread takes
constexpr int kFitWarp = 128;       // listed voxels that a warp of the fit takes

__host__ __device__ inline int fit_chunks(int Dz) { return (Dz + kFitChunk - 1) / kFitChunk; }

// The fit's lists in shared memory: voxels, pixels listed, run bits. The bits cover the runs of every pixel where there
// is room, so that voxels are listed also in a row with more candidate pixels than their list holds (a wide spot in a
// 97 px box), and later rounds take only the runs that hold fitted voxels beside the list: 4,251 boxes of 97 x 97 x 1
// 10.1 -> 6.3 ms, 160 of 97 x 97 x 65 6.2 -> 3.5 ms.
struct Fit {
    int cap, pix, runs;
};

// Dynamic shared memory of pass 2 for boxes up to max_bx pixels a side and max_dz bins with K neighbour columns: the
// neighbours' frame masks (8P; first the partner's eps1 / eps2) | P2s (4P) | P2ps (4P) | background template (4P; first
// the partner's J) | frame 64's neighbour bits (one per pixel, only when boxes reach it) | the fit list (8 x cap; first
// the rocking-curve terms and the region's profile) | the pixels that may hold fitted voxels (2 x fitpix) | a bit for
// each run of frames (`runs`: of the listed pixels, or of every pixel) | the neighbours' axis terms | staged shoebox.
struct Pass2Layout {
    int Pm;
    size_t p2, pp2, bref, hi, list, prof, pix, rest, nbt, stage, bytes;

    __host__ __device__ Pass2Layout(int max_bx, int max_dz, int K, Fit fit, bool staged) {
        Pm = max_bx * max_bx;
        p2 = (size_t)8 * Pm;
        pp2 = p2 + (size_t)4 * Pm;
        bref = pp2 + (size_t)4 * Pm;
        hi = bref + (size_t)4 * Pm;
        list = (hi + (max_dz > 64 ? (size_t)(Pm + 31) / 32 * 4 : 0) + 15) / 16 * 16;
        prof = list + ((size_t)max_dz * XI_RC_K * sizeof(float) + 15) / 16 * 16;
        const size_t c = (size_t)8 * fit.cap, t = prof - list + XI_GRID * XI_GRID * sizeof(float);
        pix = list + ((c > t ? c : t) + 15) / 16 * 16;
        rest = (pix + (size_t)2 * fit.pix + 3) / 4 * 4;
        nbt = (rest + ((size_t)fit.runs + 31) / 32 * 4 + 15) / 16 * 16;
        stage = nbt + nb_bytes(K, max_bx, max_dz);
        bytes = stage + (staged ? ((size_t)Pm * max_dz * sizeof(float) + 15) / 16 * 16 : 0);
    }
};

// The warp's sums of v[A .. B - 1] in every lane, the exchanges of the values interleaved.
template <int A, int B, int NV>
__device__ __forceinline__ void warp_totals(double (&v)[NV]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int j = A; j < B; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
}

// Sums of v[0 .. A - 1], of v[A .. B - 1] if `mid` and of v[B ..] if `end` (the same in every thread; the others stay
// zero) over the first nw warps of the CTA, in every lane of them; `red`: 2 x (NT / 32) x 8 doubles, its halves taken in
// turn by `turn` (so one barrier a sum). Warps combine in warp order. Values are taken in groups whose exchanges
// interleave: one after the other they were a serial chain that a launch of few rows waits for (500 boxes of 9 x 9 x 5,
// one in ten with a partner: 31.5 us, 29.5 so; 40,001 of them 0.89 and 0.84 ms).
template <int A, int B, int NV>
__device__ __forceinline__ void group_sum(double (&v)[NV], bool mid, bool end, int nw, double* red, int stride, int turn) {
    double* r = red + (turn & 1) * stride;
    warp_totals<0, A>(v);
    if (mid) warp_totals<A, B>(v);
    if (end) warp_totals<B, NV>(v);
    if (nw == 1) return;
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int j = 0; j < NV; ++j) r[(threadIdx.x >> 5) * NV + j] = v[j];
    asm volatile("bar.sync 1, %0;" ::"r"(32 * nw) : "memory");
    auto combine = [&](auto lo, auto hi) {
        double t[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) t[j] = 0.0;
#pragma unroll 1
        for (int w = 0; w < nw; ++w)
#pragma unroll
            for (int j = lo.value; j < hi.value; ++j) t[j] += r[w * NV + j];
#pragma unroll
        for (int j = lo.value; j < hi.value; ++j) v[j] = t[j];
    };
    combine(std::integral_constant<int, 0>(), std::integral_constant<int, A>());
    if (mid) combine(std::integral_constant<int, A>(), std::integral_constant<int, B>());
    if (end) combine(std::integral_constant<int, B>(), std::integral_constant<int, NV>());
}

// Pass 2 of one row, by the whole CTA (barrier and phase as in pass1_row).
//
// Bound by instructions and by the latency of its serial steps, as pass 1. Only a few percent of a box's voxels enter
// the fit, those where the profile exceeds a hundredth of its largest value, while every voxel's validity counts (for
// the profile share on valid voxels). So the scan of the box tests validity alone (a compare a voxel, 17 loads in
// flight: 10.3 ms for the sweep below at that stage, 10.8 with nine), and the pixels whose column can hold fitted voxels
// are listed and taken again, a thread a run of up to nine frames. Six rounds of the fit then run on the compacted fitted
// voxels in few warps, with one barrier a round (none for one warp) and only the sums the row needs; the other warps are
// done.
// Where the list overflows, the runs that did not fit are taken from the box again in every round (the rows used to
// scan their whole box).
//
// Before and after: 107,446 rows of the 16M-pixel geometry (90 frames, 500 fitted voxels a row) 16.9 -> 8.8 ms, 4,096
// boxes of 31 x 31 x 33 (5,350 fitted) 2.88 -> 1.02 ms, 1,003 of 41 x 41 x 65 (21,000 fitted) 6.86 -> 1.35 ms, 40,001 of
// 9 x 9 x 5 1.28 -> 0.84 ms.
template <int NT, bool STAGED>
__device__ __forceinline__ void pass2_row(const XiDetector& det_g, const XiRows& R, const XiBlock& B,
                                          const float* __restrict__ arena, const float* __restrict__ prof,
                                          const XiPass2In& I2, const XiPass2Out& O, int row, int max_bx, int max_dz,
                                          const Fit& fit, int* status, unsigned long long* bar, unsigned& phase) {
    extern __shared__ __align__(16) unsigned char dyn2[];
    constexpr int kW = NT / 32;
    __shared__ CtaTables T;
    __shared__ int s_nlist, s_npix, s_end;
    __shared__ float xs[XI_MAX_BX], ys[XI_MAX_BX];
    __shared__ float fR[XI_MAX_DZ], fRp[XI_MAX_DZ];
    __shared__ NbShared nb;
    __shared__ float s_e1[3], s_e2[3], s_S[3], s_zetap, s_seffp;
    __shared__ double red[2 * kW * 8];
    __shared__ double tot[8];
    __shared__ float fmax_w[kW][2];

    // the row's scalars, all asked for at once
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int Dz = R.Dz[row], bx = R.bx[row];
    NbColumn nbc;
    if (warp == kW - 1 && lane < R.K) nbc.load(R, row, lane);
    const int pxs = R.pxs ? R.pxs[row] : 1;
    const int ix0 = R.ix0[row], iy0 = R.iy0[row], iz0 = R.iz0[row];
    const float fb = R.fb[row];
    const float phi = R.phi[row];
    const float hp = R.has_p[row];
    const bool has_p = hp > 0.5f;
    const float* sb = arena + R.sb_off[row];
    const int64_t po = R.pix_off[row];
    const float zeta = I2.zeta[row], seff = I2.seff[row];
    const float bg = I2.bg[row], nbgv = I2.nbg[row];
    const float* prof_g = prof + (size_t)R.region[row] * XI_GRID * XI_GRID;
    if (Dz < 1 || Dz > max_dz || bx < 3 || bx > max_bx) {
        if (threadIdx.x == 0) atomicOr(status, 1);
        return;
    }
    const int P = bx * bx;
    const Pass2Layout L(max_bx, max_dz, R.K, fit, STAGED);
    const int cap = fit.cap;
    unsigned long long* nblo = reinterpret_cast<unsigned long long*>(dyn2);
    float* e1s = reinterpret_cast<float*>(dyn2);          // partner geometry, before nblo is written
    float* e2s = e1s + L.Pm;
    float* P2s = reinterpret_cast<float*>(dyn2 + L.p2);
    float* P2ps = reinterpret_cast<float*>(dyn2 + L.pp2);
    float* brefs = reinterpret_cast<float*>(dyn2 + L.bref);
    float* Jps = brefs;                                   // partner J, before brefs is written
    unsigned* nbhi = max_dz > 64 ? reinterpret_cast<unsigned*>(dyn2 + L.hi) : nullptr;   // frame 64's bits
    float* ul_v = reinterpret_cast<float*>(dyn2 + L.list);                               // fit list: net counts
    float* terms = ul_v;                                  // rocking-curve terms, before the fit list is written
    unsigned* ul_i = reinterpret_cast<unsigned*>(ul_v + cap);                            // fit list: z << 16 | pixel
    unsigned short* pixl = reinterpret_cast<unsigned short*>(dyn2 + L.pix);
    unsigned* rest = reinterpret_cast<unsigned*>(dyn2 + L.rest);                         // runs beside the list
    float* stage = reinterpret_cast<float*>(dyn2 + L.stage);                             // 16-byte aligned
    const NbTab tb = nb_tab(dyn2 + L.nbt, R.K, max_bx, max_dz);
    const float gain = B.gain, bias = R.sb_bias;
    const float* box = STAGED ? stage : sb;
    float* prof_r = reinterpret_cast<float*>(dyn2 + L.prof);
    for (int q = threadIdx.x; q < XI_GRID * XI_GRID; q += NT) prof_r[q] = prof_g[q];
    const XiDetector det = cta_tables(det_g, B, T);
    const bool templ = det.bkg != nullptr;
    const unsigned vbytes = (unsigned)(((size_t)Dz * P * sizeof(float)) & ~(size_t)15);   // whole 16-byte units
    const bool tma = STAGED && vbytes > 0 && ((reinterpret_cast<uintptr_t>(sb) & 15) == 0) &&
                     ((reinterpret_cast<uintptr_t>(stage) & 15) == 0);
    if (tma && threadIdx.x == 0) {
        mbar_expect_tx(bar, vbytes);
        bulk_copy_g2s(stage, sb, vbytes, bar);
    }
    if (!STAGED && threadIdx.x == 0) prefetch_box(sb, Dz * P);

    for (int i = threadIdx.x; i < bx; i += NT) {
        xs[i] = box_coord(ix0, i, pxs);
        ys[i] = box_coord(iy0, i, pxs);
    }
    if (threadIdx.x == 0) {
        s_nlist = 0;
        s_npix = 0;
        s_end = cap;
        if (has_p) {
            float S[3] = {R.pS[3 * row], R.pS[3 * row + 1], R.pS[3 * row + 2]};
            float e1[3], e2[3], zp;
            kabsch_frame(S, B.s0, B.axis, e1, e2, &zp);
            for (int c = 0; c < 3; ++c) { s_e1[c] = e1[c]; s_e2[c] = e2[c]; s_S[c] = S[c]; }
            s_zetap = zp;
        }
    }
    __syncthreads();
    if (warp == kW - 1)
        neighbour_test(nbc, R.K, has_p, bx, xs, ys, frame_centre(iz0, fb, 0), frame_centre(iz0, fb, Dz - 1), nb);
    rocking_terms(Dz, iz0, fb, B.frames_phi0, B.osc, B.sm, T.rcw, phi, zeta, terms);
    __syncthreads();
    for (int z = threadIdx.x; z < Dz; z += NT) {
        fR[z] = rocking_sum(terms, z);
        if (!has_p) fRp[z] = 0.0f;
    }
    const int nact = nb.nact;
    if (nact) neighbour_axes(Dz, bx, xs, ys, iz0, fb, nb, tb);
    if (has_p) {
        float e1[3] = {s_e1[0], s_e1[1], s_e1[2]}, e2[3] = {s_e2[0], s_e2[1], s_e2[2]};
        float S[3] = {s_S[0], s_S[1], s_S[2]};
        box_eps(det, S, e1, e2, bx, xs, ys, e1s, e2s);
        __syncthreads();                                  // the row's own terms are summed
        rocking_terms(Dz, iz0, fb, B.frames_phi0, B.osc, B.sm, T.rcw, R.pphi[row], s_zetap, terms);
        box_area(bx, e1s, e2s, B.sd, Jps, &s_seffp);
        __syncthreads();
        for (int z = threadIdx.x; z < Dz; z += NT) fRp[z] = rocking_sum(terms, z);
    }
    __syncthreads();
    // per-pixel profile planes; the profile maxima follow from them (f32 products are monotone in R)
    float Rmax, Rpmax = 0.0f;
    const Mask65 fgz = foreground_frames(fR, Dz, &Rmax);
    if (has_p) {
        Rpmax = fRp[0];
        for (int z = lane; z < Dz; z += 32) Rpmax = fmaxf(Rpmax, fRp[z]);
        for (int o = 16; o > 0; o >>= 1) Rpmax = fmaxf(Rpmax, __shfl_xor_sync(0xffffffffu, Rpmax, o));
    }
    if (nact) neighbour_zmin(Dz, nb, tb);
    float pm_t = 0.0f, ppm_t = 0.0f;
    for (int p = threadIdx.x; p < P; p += NT) {
        const float J = I2.J[po + p];
        const float v = profile_value(prof_r, I2.u1[po + p], I2.u2[po + p], J, seff);
        P2s[p] = v;
        pm_t = fmaxf(pm_t, v * Rmax);
        if (has_p) {
            // the partner's u1 / u2 are eps / seff
            const float vp = profile_value(prof_r, e1s[p] / s_seffp, e2s[p] / s_seffp, Jps[p], s_seffp);
            P2ps[p] = vp;
            ppm_t = fmaxf(ppm_t, (vp * Rpmax) * hp);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        pm_t = fmaxf(pm_t, __shfl_down_sync(0xffffffffu, pm_t, o));
        ppm_t = fmaxf(ppm_t, __shfl_down_sync(0xffffffffu, ppm_t, o));
    }
    if (lane == 0) {
        fmax_w[warp][0] = pm_t;
        fmax_w[warp][1] = ppm_t;
    }
    if (nbhi)
        for (int w = threadIdx.x; w < (P + 31) / 32; w += NT) nbhi[w] = 0u;
    for (int w = threadIdx.x; w < (min(P * fit_chunks(Dz), fit.runs) + 31) / 32; w += NT) rest[w] = 0u;
    __syncthreads();                                      // (partner scratch free)
    float pmax = 0.0f, ppmax = 0.0f;
#pragma unroll
    for (int w = 0; w < kW; ++w) {
        pmax = fmaxf(pmax, fmax_w[w][0]);
        ppmax = fmaxf(ppmax, fmax_w[w][1]);
    }
    const float pthr = 0.01f * pmax;
    const float ppthr = 0.01f * fmaxf(ppmax, 1e-12f);
    if (STAGED) {
        stage_wait(tma, bar, phase, stage, sb, Dz * P, status);
        if (tma) phase ^= 1u;
    }
    // frame sums of the rocking curve: a pixel's profile total is P2 * sum_z R (all frames) and its foreground
    // share P2 * sum_{z in fgz} R, both taken per pixel in float64; p_valid subtracts the frames a pixel loses
    // (masked voxels, neighbours), summed per column
    double r_all = 0.0, r_fg = 0.0;
    for (int z = lane; z < Dz; z += 32) {
        r_all += (double)fR[z];
        if (fgz.get(z)) r_fg += (double)fR[z];
    }
    r_all = warp_total(r_all);
    r_fg = warp_total(r_fg);

    // ---- every voxel's validity, the profile sums, and the pixels that may hold fitted voxels
    double a8[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // s_net, s_w, p_total, p_valid, p_fgn, a110, C0, nuse
    {
        PixelWalk px(bx);
        for (int p0 = 0; p0 < P; p0 += NT, px.next()) {
            const int p = px.p;
            bool may = false;
            if (p < P) {
                const float P2 = P2s[p];
                const float u1 = I2.u1[po + p], u2 = I2.u2[po + p];
                const bool fg2 = (u1 * u1 + u2 * u2) <= kFgR2;
                // (products of non-negative factors are monotone; a negative one is looked at voxel by voxel)
                may = P2 * Rmax > pthr || P2 < 0.0f;
                if (has_p) {
                    const float P2p = P2ps[p];
                    may = may || (P2p * Rpmax) * hp > ppthr || P2p < 0.0f;
                }
                if (templ) brefs[p] = bkg_ref(det, xs[px.i], ys[px.j]);
                Mask65 nbm;
                nbm.clear();
                if (nact) {
                    nbm = neighbour_frames(nb, tb, px.i, px.j, Dz);
                    nblo[p] = nbm.lo;
                    if (nbm.hi) atomicOr(&nbhi[p >> 5], 1u << (p & 31));
                }
                float lost = 0.0f;                   // rocking-curve weight of the frames this pixel loses
                const float* col = box + p;
                for (int z0 = 0; z0 < Dz; z0 += kValid, col += (size_t)kValid * P) {
                    const int nbat = min(kValid, Dz - z0);
                    const unsigned kb = frames_from(nbm, z0) & ((1u << nbat) - 1u);
                    float v[kValid];
#pragma unroll
                    for (int u = 0; u < kValid; ++u) v[u] = u < nbat ? col[(size_t)u * P] : bias;
                    bool ok = kb == 0u;
#pragma unroll
                    for (int u = 0; u < kValid; ++u) ok = ok && v[u] >= bias;      // value >= 0
                    if (ok) continue;
#pragma unroll
                    for (int u = 0; u < kValid; ++u)
                        if (u < nbat && !(v[u] >= bias && !((kb >> u) & 1u))) lost += fR[z0 + u];
                }
                const double tp = (double)P2 * r_all;
                a8[2] += tp;
                a8[3] += tp - (double)P2 * (double)lost;
                if (fg2) a8[4] += (double)P2 * r_fg;
            }
            const unsigned ball = __ballot_sync(0xffffffffu, may);
            if (ball) {
                int base = 0;
                if (lane == 0) base = atomicAdd(&s_npix, __popc(ball));
                base = __shfl_sync(0xffffffffu, base, 0) + __popc(ball & ((1u << lane) - 1u));
                if (may && base < fit.pix) pixl[base] = (unsigned short)p;
            }
        }
    }
    __syncthreads();
    // a plain row (no partner, no background template) keeps the fitted voxels' profile values, others their places
    const bool plain = !has_p && !templ;
    // ---- the fitted voxels: runs of frames of the listed pixels (of every pixel when the list overflows)
    const bool pix_listed = s_npix <= fit.pix;
    const int npix = pix_listed ? s_npix : P;
    const int nchunk = fit_chunks(Dz), clen = (Dz + nchunk - 1) / nchunk;
    const int n_run = npix * nchunk;
    const bool kept = n_run <= fit.runs;                  // the runs have their bits (else no voxel is listed)
    // run k: its pixel and first frame; f(frame of the run, raw value, pv, ppv) for every fitted voxel of it
    auto run_of = [&](int k, int& p, int& z0) {
        const int c = k / npix, q = k - c * npix;
        p = pix_listed ? (int)pixl[q] : q;
        z0 = c * clen;
    };
    auto fitted_of = [&](int p, int z0, auto&& f) {
        const int zn = min(clen, Dz - z0);
        const float P2 = P2s[p], P2p = has_p ? P2ps[p] : 0.0f;
        const float* col = box + (size_t)z0 * P + p;
        float v[kFitChunk], pv[kFitChunk], ppv[kFitChunk];
#pragma unroll
        for (int u = 0; u < kFitChunk; ++u) {
            const bool in = u < zn;
            pv[u] = in ? P2 * fR[z0 + u] : 0.0f;
            ppv[u] = in && has_p ? (P2p * fRp[z0 + u]) * hp : 0.0f;
            v[u] = in && (pv[u] > pthr || ppv[u] > ppthr) ? col[(size_t)u * P] : bias - 1.0f;
        }
        unsigned nbm = 0u;                                // the run's frames claimed by a neighbour
        if (nact) {
            if (z0 < 64) nbm = (unsigned)(nblo[p] >> z0);
            if (nbhi && z0 + kFitChunk > 64) nbm |= ((nbhi[p >> 5] >> (p & 31)) & 1u) << (64 - z0);
        }
#pragma unroll
        for (int u = 0; u < kFitChunk; ++u)
            if (v[u] >= bias && !((nbm >> u) & 1u)) f(u, v[u], pv[u], ppv[u]);
    };
    for (int k0 = 0; k0 < n_run; k0 += NT) {
        const int k = k0 + threadIdx.x;
        int p = 0, z0 = 0;
        unsigned m = 0u;
        if (k < n_run) {
            run_of(k, p, z0);
            fitted_of(p, z0, [&](int u, float, float, float) { m |= 1u << u; });
        }
        // warp-aggregated append: a lane's entries follow the entries of the lanes before it
        const int c = __popc(m);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int wtot = __shfl_sync(0xffffffffu, incl, 31);
        if (!wtot) continue;
        int at = 0;
        if (lane == 31) at = atomicAdd(&s_nlist, wtot);
        at = __shfl_sync(0xffffffffu, at, 31) + incl - c;
        const float bref = templ ? brefs[p] : 1.0f;
        const float bpix = bg * bref;
        const float iv0 = __frcp_rn(gain * fmaxf(bpix, kVarFloor));
        const float P2 = P2s[p], P2p = has_p ? P2ps[p] : 0.0f;
        a8[7] += (double)c;
        // a run that does not fit whole is left to the later passes (at most one straddles the list's end)
        const bool fits = at + c <= cap;
        if (c && !fits) {
            if (at < cap) s_end = at;
            if (kept) atomicOr(&rest[k >> 5], 1u << (k & 31));
        }
#pragma unroll 1
        for (unsigned r = m; r; r &= r - 1u, ++at) {
            const int z = z0 + __ffs(r) - 1;
            const float net = (box[(size_t)z * P + p] - bias) - bpix;
            const float pv = P2 * fR[z];
            const float ppv = has_p ? (P2p * fRp[z]) * hp : 0.0f;
            a8[0] += (double)net;
            a8[1] += (double)(pv + ppv);
            a8[5] += (double)((pv * pv) * iv0);
            a8[6] += (double)((pv * bref) * iv0);
            if (fits && kept) {
                ul_v[at] = net;
                ul_i[at] = plain ? __float_as_uint(pv) : ((unsigned)z << 16) | (unsigned)p;
            }
        }
    }
    block_sum<NT, 8>(a8, red, tot);
    const double s_net_use = tot[0];
    const float p_total = (float)tot[2], p_valid = (float)tot[3], p_fgn = (float)tot[4];
    const double a110 = fmax(tot[5], 1e-12), C0 = tot[6];
    const float nuse = (float)tot[7];
    float I = (float)tot[0] / fmaxf((float)tot[1], 1e-6f), Ip = I * hp;
    // listed voxels, and whether runs are left beside them (all of them when there was no room for the runs' bits)
    const bool whole = kept && s_nlist <= cap;
    const int nlist = whole ? s_nlist : kept ? s_end : 0;

    // ---- the fit, in the first nw warps: kFitWarp listed voxels a warp, all warps when runs are left
    const int nw = whole ? min(kW, max(1, (nlist + kFitWarp - 1) / kFitWarp)) : kW;
    if (warp >= nw) return;
    const int nt = 32 * nw;
    // every fitted voxel of this thread: f(net, pv, ppv, bpix, bref)
    auto each_fitted = [&](auto&& f) {
#pragma unroll 1
        for (int k = threadIdx.x; k < nlist; k += nt) {
            const float net = ul_v[k];
            const unsigned id = ul_i[k];
            float pv = __uint_as_float(id), ppv = 0.0f, bref = 1.0f;
            if (!plain) {
                const int z = (int)(id >> 16), p = (int)(id & 0xffffu);
                pv = P2s[p] * fR[z];
                if (has_p) ppv = (P2ps[p] * fRp[z]) * hp;
                if (templ) bref = brefs[p];
            }
            f(net, pv, ppv, bg * bref, bref);
        }
        if (whole) return;
#pragma unroll 1
        for (int k = threadIdx.x; k < n_run; k += NT) {
            if (kept && !((rest[k >> 5] >> (k & 31)) & 1u)) continue;
            int p, z0;
            run_of(k, p, z0);
            const float bref = templ ? brefs[p] : 1.0f;
            const float bpix = bg * bref;
            fitted_of(p, z0, [&](int, float v, float pv, float ppv) { f((v - bias) - bpix, pv, ppv, bpix, bref); });
        }
    };
    constexpr int kStride = kW * 8;
    int turn = 0;
    // ---- IRLS: Poisson-weighted 2x2 normal equations, float64 sums, N_IRLS iterations; the last iteration's
    // weights also give C of the variance tail and the sum of the fitted profile values
    double a11 = 0.0, a12 = 0.0, a22 = 1.0, b1 = 0.0, b2 = 0.0, det2 = 1.0, Cc = 0.0, swp = 0.0;
#pragma unroll 1
    for (int it = 0; it < kIrls; ++it) {
        const bool last = it == kIrls - 1;
        const float Ipos = fmaxf(I, 0.0f), Ippos = fmaxf(Ip, 0.0f);
        double a7[7] = {0, 0, 0, 0, 0, 0, 0};   // a11, b1, a12, a22, b2, C, sum p
        each_fitted([&](float net, float pv, float ppv, float bpix, float bref) {
            float mu = bpix + Ipos * pv;
            if (has_p) mu = mu + Ippos * ppv;
            const float iv = __frcp_rn(gain * fmaxf(mu, kVarFloor));
            a7[0] += (double)((pv * pv) * iv);
            a7[1] += (double)((pv * net) * iv);
            if (has_p) {
                a7[2] += (double)((pv * ppv) * iv);
                a7[3] += (double)((ppv * ppv) * iv);
                a7[4] += (double)((ppv * net) * iv);
            }
            if (last) {
                a7[5] += (double)((pv * bref) * iv);
                a7[6] += (double)pv;
            }
        });
        group_sum<2, 5>(a7, has_p, last, nw, red, kStride, turn++);
        a11 = a7[0];
        b1 = a7[1];
        if (has_p) {
            a12 = a7[2];
            a22 = a7[3];
            b2 = a7[4];
        }
        Cc = a7[5];
        swp = a7[6];
        det2 = fmax(a11 * a22 - a12 * a12, 1e-30);
        I = (float)((a22 * b1 - a12 * b2) / det2);
        if (has_p || last) Ip = (float)((a11 * b2 - a12 * b1) / det2 * (double)hp);
    }
    const float Ippos = fmaxf(Ip, 0.0f);
    const float pm = (float)swp / fmaxf(nuse, 1.0f);
    // mean residual over the fitted voxels (with a partner the residual removes the partner's fitted share)
    double s_resid = s_net_use;
    if (has_p) {
        double a1[1] = {0.0};
        each_fitted([&](float net, float pv, float ppv, float bpix, float bref) {
            a1[0] += (double)(net - Ippos * ppv);
        });
        group_sum<1, 1>(a1, false, false, nw, red, kStride, turn++);
        s_resid = a1[0];
    }
    const float nm = (float)s_resid / fmaxf(nuse, 1.0f);
    // ---- profile / residual correlation
    double a3[3] = {0.0, 0.0, 0.0};
    each_fitted([&](float net, float pv, float ppv, float bpix, float bref) {
        const float resid = has_p ? net - Ippos * ppv : net;
        const float dp = pv - pm, dn = resid - nm;
        a3[0] += (double)(dp * dn);
        a3[1] += (double)(dp * dp);
        a3[2] += (double)(dn * dn);
    });
    group_sum<3, 3>(a3, false, false, nw, red, kStride, turn++);
    if (threadIdx.x == 0) {
        const double var_b = (double)gain * fmax((double)bg, (double)kVarFloor) / fmax((double)nbgv, 1.0);
        const double a11i = a22 / det2;
        const double varI = a11i + (Cc * a11i) * (Cc * a11i) * var_b;
        const double infl = a11i * a11;
        const double var0 = (1.0 / a110 + (C0 / a110) * (C0 / a110) * var_b) * fmax(infl, 1.0);
        const float sdd = (float)a3[0], spp = (float)a3[1], snn = (float)a3[2];
        O.iprf[row] = I;
        O.vprf[row] = (float)varI;
        O.vprf0[row] = (float)var0;
        O.corr[row] = sdd / sqrtf(fmaxf(spp * snn, 1e-20f));
        O.p_valid[row] = p_valid;
        O.p_total[row] = p_total;
        O.ipartner[row] = Ip;
        O.rho[row] = has_p ? (float)(a12 / sqrt(fmax(a11 * a22, 1e-30))) : 0.0f;
        O.p_fg[row] = p_fgn / fmaxf(p_total, 1e-9f);
    }
}

// Pass 2, one CTA per row of `order` (one shoebox shape group per launch).
template <int NT, bool STAGED>
__global__ void __launch_bounds__(NT, min_ctas<NT>()) k_pass2(XiDetector det_g, XiRows R, XiBlock B,
                                                              const float* __restrict__ arena,
                                                              const float* __restrict__ prof, XiPass2In I2,
                                                              XiPass2Out O, const int32_t* __restrict__ order,
                                                              int max_bx, int max_dz, Fit fit, int* status) {
    __shared__ __align__(8) unsigned long long s_bar;
    if (STAGED) {
        if (threadIdx.x == 0) mbar_init(&s_bar, 1);
        __syncthreads();
    }
    unsigned phase = 0;
    pass2_row<NT, STAGED>(det_g, R, B, arena, prof, I2, O, order ? order[blockIdx.x] : blockIdx.x, max_bx, max_dz,
                          fit, status, &s_bar, phase);
}

// Pass 2 over a queue of (set, row) items (as k_pass1_q); a set's pass-1 outputs are its pass-2 inputs.
template <int NT, bool STAGED>
__global__ void __launch_bounds__(NT, min_ctas<NT>()) k_pass2_q(const XiRowSet* __restrict__ sets,
                                                                const int64_t* __restrict__ items, int n_items,
                                                                int max_bx, int max_dz, int max_k, Fit fit,
                                                                int* queue, int* status) {
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ XiRowSet s_set;
    __shared__ int s_item, s_cur;
    if (threadIdx.x == 0) {
        if (STAGED) mbar_init(&s_bar, 1);
        s_cur = -1;
    }
    unsigned phase = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= n_items) return;
        const int64_t v = items[it];
        const int set = (int)(v >> 32);
        if (set != s_cur) load_set(sets, set, &s_set, &s_cur);
        if (s_set.rows.K > max_k) {
            if (threadIdx.x == 0) atomicOr(status, 1);
            continue;
        }
        XiPass2In in;
        in.zeta = s_set.p1.zeta;
        in.seff = s_set.p1.seff;
        in.J = s_set.p1.J;
        in.u1 = s_set.p1.u1;
        in.u2 = s_set.p1.u2;
        in.bg = s_set.p1.bg;
        in.nbg = s_set.p1.nbg;
        pass2_row<NT, STAGED>(s_set.det, s_set.rows, s_set.blk, s_set.arena, s_set.prof, in, s_set.p2,
                              (int)(v & 0xffffffffll), max_bx, max_dz, fit, status, &s_bar, phase);
    }
}

// ==================================================================================================================
// gather and bin decode
// ==================================================================================================================
__device__ __forceinline__ float prepared_pixel(const XiFrames& F, const void* frame, int y, int x) {
    // one detector pixel of a frame as XPG's readers deliver it, with the mask ceiling applied
    if (y < 0 || y >= F.ny || x < 0 || x >= F.nx) return -1.0f;
    const size_t idx = (size_t)y * F.nx + x;
    float v;
    if (F.is_float) {
        v = ((const float*)frame)[idx];
    } else {
        const uint32_t r = ((const uint32_t*)frame)[idx];
        if (r == 0xFFFFFFFFu || r < F.min_valid) v = -1.0f;
        else if (r >= F.overload) v = -2.0f;
        else v = (float)r;
    }
    if (F.mask && F.mask[idx] == 0) v = fminf(v, -1.0f);
    return v;
}

// the raw value of a pixel known to be inside the frame, encoded as XPG's readers deliver it (mask applied later)
__device__ __forceinline__ float encode_raw(const XiFrames& F, uint32_t r) {
    if (r == 0xFFFFFFFFu || r < F.min_valid) return -1.0f;
    if (r >= F.overload) return -2.0f;
    return (float)r;
}

__device__ __forceinline__ float box_value(const XiFrames& F, const void* frame, int sy, int sx, int s) {
    if (s == 1) return prepared_pixel(F, frame, sy, sx);
    // s x s super-pixel (xpg/integrate.py:682-699): incomplete super-pixels at the far edges are masked
    if (sy < 0 || sx < 0 || sy >= F.ny / s || sx >= F.nx / s) return -1.0f;
    float sum = 0.0f, mn = 0.0f;
    for (int a = 0; a < s; ++a)
        for (int c = 0; c < s; ++c) {
            const float v = prepared_pixel(F, frame, sy * s + a, sx * s + c);
            if (a == 0 && c == 0) { sum = v; mn = v; }
            else { sum = sum + v; mn = fminf(mn, v); }
        }
    if (mn < 0.0f) return mn <= -1.5f ? -2.0f : -1.0f;
    return sum;
}

// The gather of one row's box from the frames of a wedge, by the whole CTA; plain rows NB frames at a time.
template <int NB>
__device__ __forceinline__ void gather_row(const XiFrames& F, const XiGatherRows& G, float* __restrict__ arena,
                                           int32_t* __restrict__ cnt, int row) {
    const int iz0 = G.iz0[row], fb = G.fb[row], Dz = G.Dz[row], bx = G.bx[row];
    const int s = G.pxs ? G.pxs[row] : 1;
    const int ix0 = G.ix0[row], iy0 = G.iy0[row];
    const int P = bx * bx;
    const int span = Dz * fb;
    const int w0 = max(0, iz0 - F.first_fi), w1 = min(F.n_frames, iz0 + span - F.first_fi);
    float* dst = arena + G.sb_off[row];
    const size_t fstride = (size_t)F.ny * F.nx * (F.is_float ? sizeof(float) : sizeof(uint32_t));
    if (fb == 1 && s == 1) {
        // plain rows: a thread owns box pixels and reads a pixel's frames NB at a time (independent loads in flight);
        // the pixel's bounds and mask are looked up once
        const size_t fpix = (size_t)F.ny * F.nx;
        for (int p = threadIdx.x; p < P; p += blockDim.x) {
            const int y = iy0 + p / bx, x = ix0 + p % bx;
            const bool inside = y >= 0 && y < F.ny && x >= 0 && x < F.nx;
            const size_t idx = inside ? (size_t)y * F.nx + x : 0;
            const bool masked = inside && F.mask && F.mask[idx] == 0;
            const int k0 = F.first_fi - iz0;                  // box frame of wedge frame 0
            for (int w = w0; w < w1; w += NB) {
                float vv[NB];
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    vv[u] = -1.0f;
                    const int ww = w + u;
                    if (inside && ww < w1) {
                        const size_t o = (size_t)ww * fpix + idx;
                        vv[u] = F.is_float ? ((const float*)F.data)[o] : encode_raw(F, ((const uint32_t*)F.data)[o]);
                    }
                }
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    const int ww = w + u;
                    if (ww >= w1 || (F.frame_ok && !F.frame_ok[ww])) continue;
                    const float v = masked ? fminf(vv[u], -1.0f) : vv[u];
                    dst[(size_t)(k0 + ww) * P + p] = v + kSbOff;
                }
            }
        }
        return;
    }
    for (int w = w0; w < w1; ++w) {
        if (F.frame_ok && !F.frame_ok[w]) continue;
        const int fi = F.first_fi + w;
        const int k = fi - iz0;
        const void* frame = (const char*)F.data + (size_t)w * fstride;
        if (fb == 1) {
            float* slot = dst + (size_t)k * P;
            for (int p = threadIdx.x; p < P; p += blockDim.x) {
                const int i = p % bx, j = p / bx;
                slot[p] = box_value(F, frame, iy0 + j, ix0 + i, s) + kSbOff;
            }
        } else {
            const int kb = k / fb;
            float* slot = dst + (size_t)kb * P;
            for (int p = threadIdx.x; p < P; p += blockDim.x) {
                const int i = p % bx, j = p / bx;
                float v = box_value(F, frame, iy0 + j, ix0 + i, s);
                if (v < 0.0f) v = (v == -2.0f) ? __int_as_float(0x7fc00000) : __int_as_float(0x7f800000);
                slot[p] = slot[p] + v;
            }
            if (threadIdx.x == 0) cnt[G.cnt_off[row] + kb] += 1;
        }
    }
}

template <int NB>
__global__ void k_gather(XiFrames F, XiGatherRows G, float* __restrict__ arena, int32_t* __restrict__ cnt,
                         const int32_t* __restrict__ order) {
    gather_row<NB>(F, G, arena, cnt, order ? order[blockIdx.x] : blockIdx.x);
}

// The gather of one wedge with the frames and rows read from a device descriptor when the kernel runs, so that one
// launch captured in a CUDA graph serves every wedge of a block: CTAs stride over the step's rows.
__global__ void k_gather_step(const XiGatherStep* __restrict__ step, XiGatherRows G, float* __restrict__ arena,
                              int32_t* __restrict__ cnt) {
    const XiFrames F = step->frames;
    const int n = step->n_order;
    if (F.n_frames <= 0) return;
    for (int k = blockIdx.x; k < n; k += gridDim.x) gather_row<kGatherBatch>(F, G, arena, cnt, step->order[k]);
}


__global__ void k_decode_bins(XiGatherRows G, float* __restrict__ arena, const int32_t* __restrict__ cnt) {
    const int row = G.order ? G.order[blockIdx.x] : blockIdx.x;
    if (G.cnt_off[row] < 0) return;
    const int Dz = G.Dz[row], bx = G.bx[row], fb = G.fb[row];
    const int P = bx * bx;
    float* a = arena + G.sb_off[row];
    const int32_t* c = cnt + G.cnt_off[row];
    for (int v = threadIdx.x; v < Dz * P; v += blockDim.x) {
        const int z = v / P;
        float x = a[v];
        if (isnan(x)) x = -2.0f;
        else if (isinf(x)) x = -1.0f;
        x = x + kSbOff;
        if (c[z] < fb) x = 0.0f;
        a[v] = x;
    }
}

// zero the arena slots of the listed rows (rows the gather does not write in full: binned rows accumulate, rows whose
// frames reach beyond the run's). A row's slot is Dz * bx^2 floats rounded up to 4 and starts on 16 bytes.
__global__ void k_zero_rows(XiGatherRows G, float* __restrict__ arena) {
    const int row = G.order ? G.order[blockIdx.x] : blockIdx.x;
    const int64_t v = (int64_t)G.Dz[row] * G.bx[row] * G.bx[row];
    const int64_t n4 = (v + 3) / 4;
    float4* a = reinterpret_cast<float4*>(arena + G.sb_off[row]);
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int64_t i = threadIdx.x; i < n4; i += blockDim.x) a[i] = z;
}

// ==================================================================================================================
// profile accumulation and finalisation
// ==================================================================================================================
__global__ void k_accumulate(XiRows R, XiPass1Out O, const uint8_t* __restrict__ sel, int strong_test,
                             int n_regions, double* __restrict__ num, double* __restrict__ den) {
    const int row = R.order ? R.order[blockIdx.x] : blockIdx.x;
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        bool ok = true;
        if (strong_test) {
            // strong, fully recorded, unobstructed (xpg/integrate.py:531-533), float64 on the float32 outputs
            const double isum = (double)O.isum[row], vs = (double)O.vsum[row];
            ok = (isum > 0.0) && (isum / sqrt(fmax(vs, 1e-6)) > 10.0) && O.n_over[row] == 0 &&
                 (double)O.frac_rec[row] > 0.95 && O.n_fg_nb[row] == 0 && O.n_fg_masked[row] == 0;
        }
        if (sel && !sel[row]) ok = false;
        const int reg = R.region[row];
        if (reg < 0 || reg >= n_regions) ok = false;
        s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) return;
    const int bx = R.bx[row];
    const int P = bx * bx;
    const int64_t po = R.pix_off[row];
    const float isum = fmaxf(O.isum[row], 1e-6f);
    const float seff = O.seff[row];
    const float s2 = seff * seff;
    double* nr = num + (size_t)R.region[row] * XI_GRID * XI_GRID;
    double* dr = den + (size_t)R.region[row] * XI_GRID * XI_GRID;
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        const float dens = (O.img2[po + p] / isum) / fmaxf(O.J[po + p] / s2, 1e-12f);
        GridCell g = grid_cell(O.u1[po + p], O.u2[po + p]);
        if (!(O.all_valid2[po + p] && g.inside)) continue;
        const float w00 = (1.0f - g.t1) * (1.0f - g.t2), w10 = g.t1 * (1.0f - g.t2);
        const float w01 = (1.0f - g.t1) * g.t2, w11 = g.t1 * g.t2;
        const int b = g.i2 * XI_GRID + g.i1;
        atomicAdd(nr + b, (double)(w00 * dens));
        atomicAdd(dr + b, (double)w00);
        atomicAdd(nr + b + 1, (double)(w10 * dens));
        atomicAdd(dr + b + 1, (double)w10);
        atomicAdd(nr + b + XI_GRID, (double)(w01 * dens));
        atomicAdd(dr + b + XI_GRID, (double)w01);
        atomicAdd(nr + b + XI_GRID + 1, (double)(w11 * dens));
        atomicAdd(dr + b + XI_GRID + 1, (double)w11);
    }
}

__global__ void k_finalize(const double* __restrict__ num, const double* __restrict__ den, float* __restrict__ prof) {
    // one CTA per region (xpg/integrate.py:546-555); the Gaussian prior is float32-rounded as XPG's table
    const int r = blockIdx.x;
    constexpr int G2 = XI_GRID * XI_GRID;
    __shared__ double pr[G2];
    __shared__ double part[32];
    const double du = (9.0 / (XI_GRID - 1)) * (9.0 / (XI_GRID - 1));
    for (int q = threadIdx.x; q < G2; q += blockDim.x) {
        const int iy = q / XI_GRID, ix = q % XI_GRID;
        // numpy.linspace(-4.5, 4.5, 41): i * step + start, the last point exactly 4.5
        const double step = 9.0 / (XI_GRID - 1);
        const double u1 = ix == XI_GRID - 1 ? 4.5 : (double)ix * step + (-4.5);
        const double u2 = iy == XI_GRID - 1 ? 4.5 : (double)iy * step + (-4.5);
        const float gauss = (float)(exp(-0.5 * (u1 * u1 + u2 * u2)) / (2.0 * 3.141592653589793));
        const float g3 = 3.0f * gauss;                 // XPG: 3.0 * (float32 table) stays float32
        const double n = num[(size_t)r * G2 + q], d = den[(size_t)r * G2 + q];
        const double dens = d > 0.0 ? n / fmax(d, 1e-12) : 0.0;
        const double emp = fmax(dens, 0.0);
        const double v = (d * emp + (double)g3) / (d + 3.0);
        pr[q] = v;
    }
    __syncthreads();
    // sum in index order by one warp (fixed order), then normalise
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int q = threadIdx.x; q < G2; q += 32) s += pr[q];
        part[threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < 32; ++q) s += part[q];
        part[0] = fmax(s * du, 1e-12);
    }
    __syncthreads();
    const double norm = part[0];
    for (int q = threadIdx.x; q < G2; q += blockDim.x) prof[(size_t)r * G2 + q] = (float)(pr[q] / norm);
}

// status word of the kernels (rows skipped for an unsupported shape)
__device__ int g_status = 0;

int* status_ptr() {
    static int* p = nullptr;
    int dev = -1;
    cudaGetDevice(&dev);
    static int pdev = -2;
    if (p == nullptr || pdev != dev) {
        if (cudaGetSymbolAddress((void**)&p, g_status) != cudaSuccess) return nullptr;
        pdev = dev;
    }
    return p;
}

int rows_check(const XiRows* R) {
    if (!R) return fail(XI_E_ARG, "rows: null");
    if (R->n < 0 || (R->order && R->n_order < 0)) return fail(XI_E_ARG, "rows: negative count");
    if (R->K < 0 || R->K > XI_MAX_K) return fail(XI_E_LIMIT, "rows: neighbour columns beyond XI_MAX_K");
    if (R->max_bx < 3 || R->max_bx > XI_MAX_BX || R->max_dz < 1 || R->max_dz > XI_MAX_DZ)
        return fail(XI_E_LIMIT, "rows: max_bx / max_dz outside 3..97 / 1..65");
    return XI_OK;
}

template <int NT, bool STAGED>
int launch_pass1(const XiDetector* det, const XiRows* R, const XiBlock* B, const float* arena, XiPass1Out* O,
                 cudaStream_t s, int nblk) {
    const size_t sm = Pass1Layout(R->max_bx, R->max_dz, R->K, STAGED).bytes;
    cudaFuncSetAttribute(k_pass1<NT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_pass1<NT, STAGED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    k_pass1<NT, STAGED><<<nblk, NT, sm, s>>>(*det, *R, *B, arena, *O, R->order, R->max_bx, R->max_dz,
                                              status_ptr());
    return cuda_check("xi_pass1");
}

template <int NT, bool STAGED>
int launch_pass2(const XiDetector* det, const XiRows* R, const XiBlock* B, const float* arena, const float* prof,
                 const XiPass2In* in, XiPass2Out* O, cudaStream_t s, int nblk, Fit fit) {
    const size_t sm = Pass2Layout(R->max_bx, R->max_dz, R->K, fit, STAGED).bytes;
    cudaFuncSetAttribute(k_pass2<NT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_pass2<NT, STAGED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    k_pass2<NT, STAGED><<<nblk, NT, sm, s>>>(*det, *R, *B, arena, prof, *in, *O, R->order, R->max_bx, R->max_dz,
                                              fit, status_ptr());
    return cuda_check("xi_pass2");
}

__global__ void k_zero_int(int* p) { *p = 0; }

// Resident CTAs of a persistent launch: as many as the SMs hold at once (at least one).
template <typename K>
int resident_grid(K kernel, int nt, size_t smem, int n_items) {
    int dev = 0, n_sm = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, nt, smem) != cudaSuccess)
        return -1;
    const long long g = (long long)(per_sm > 0 ? per_sm : 1) * n_sm;
    return (int)(g < n_items ? g : n_items);
}

template <int NT, bool STAGED>
int launch_pass1_q(const XiRowSet* sets, const int64_t* items, int n_items, int max_bx, int max_dz, int K, int* queue,
                   cudaStream_t s) {
    const size_t sm = Pass1Layout(max_bx, max_dz, K, STAGED).bytes;
    cudaFuncSetAttribute(k_pass1_q<NT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_pass1_q<NT, STAGED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    const int grid = resident_grid(k_pass1_q<NT, STAGED>, NT, sm, n_items);
    if (grid <= 0) return cuda_check("xi_pass1_batched: occupancy");
    k_zero_int<<<1, 1, 0, s>>>(queue);
    k_pass1_q<NT, STAGED><<<grid, NT, sm, s>>>(sets, items, n_items, max_bx, max_dz, K, queue, status_ptr());
    return cuda_check("xi_pass1_batched");
}

template <int NT, bool STAGED>
int launch_pass2_q(const XiRowSet* sets, const int64_t* items, int n_items, int max_bx, int max_dz, int K, Fit fit,
                   int* queue, cudaStream_t s) {
    const size_t sm = Pass2Layout(max_bx, max_dz, K, fit, STAGED).bytes;
    cudaFuncSetAttribute(k_pass2_q<NT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k_pass2_q<NT, STAGED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    const int grid = resident_grid(k_pass2_q<NT, STAGED>, NT, sm, n_items);
    if (grid <= 0) return cuda_check("xi_pass2_batched: occupancy");
    k_zero_int<<<1, 1, 0, s>>>(queue);
    k_pass2_q<NT, STAGED><<<grid, NT, sm, s>>>(sets, items, n_items, max_bx, max_dz, K, fit, queue, status_ptr());
    return cuda_check("xi_pass2_batched");
}

// Dynamic shared memory available beside the kernels' static arrays (bytes).
constexpr size_t kStageBudget = 190 * 1024;

// Dynamic shared memory of a pass-2 CTA of nt threads when n share an SM: 228 KB an SM, of which each CTA loses 1 KB and
// its static arrays (at most 4,032 bytes of 64 threads, 4,304 of 128, 4,848 of 256).
constexpr size_t pass2_share(int n, int nt) {
    return (size_t)228 * 1024 / n - 1024 - (nt == 64 ? 4096 : nt == 128 ? 4352 : 4864);
}

// Launch tuning (xi_tune): the largest shoebox each pass stages in shared memory, and the fit-list capacity of
// pass 2. Larger staging overlaps the box read with the set-up but costs resident CTAs per SM.
size_t g_stage_max[2] = {48 * 1024, 48 * 1024};
int g_list_cap[2] = {2048, 2048};   // boxes up to XI_PASS2_LARGE_VOXELS voxels, larger boxes: the least list (pass2_plan)
int g_wide_nt = 256;          // threads per CTA of the pass kernels for boxes over 200 pixels (128 or 256)

// Pass 1 stages boxes of up to g_stage_max[0] bytes when they fit beside the per-pixel tables.
bool pass1_staged(int max_bx, int max_dz, int K) {
    return (size_t)max_bx * max_bx * max_dz * sizeof(float) <= g_stage_max[0] &&
           Pass1Layout(max_bx, max_dz, K, true).bytes <= kStageBudget;
}

// threads of a pass CTA for boxes up to max_bx pixels a side
int pass_threads(int max_bx) {
    const int P = max_bx * max_bx;
    return P <= 96 ? 64 : P <= 200 || g_wide_nt == 128 ? 128 : 256;
}

// Pass 2's shared-memory plan for boxes up to max_bx pixels a side and max_dz bins with K neighbour columns: whether
// the box is staged, and the fit's lists. First the CTAs that an SM holds: as many as the registers allow, fewer where
// the tables with the least list (g_list_cap voxels, or the whole box) need more room than their share. Then what that
// share leaves goes to the box, staged where it is small and costs no CTA, to the runs' bits and the list of pixels (of all of
// the box's pixels where the least list still fits, else of kFitPix) and to the list of voxels. Runs that
// do not fit the list are taken from the box in every round; the second least list is for launches whose largest box
// exceeds XI_PASS2_LARGE_VOXELS voxels or XI_PASS2_LARGE_DEPTH bins; 0 voxels: no list.
// A CTA counts for more than a staged box or a longer list. With the list sized first, to a third of an SM, and the box
// beside it, 31 x 31 x 9, 17 x 17 x 33, 23 x 23 x 17, 25 x 25 x 17, 41 x 41 x 5 and 13 x 13 x 65 boxes ran one or two CTAs
// fewer (4,624, 4,194, 4,447, 3,764, 4,759 and 3,641 boxes: 731, 646, 678, 1,159, 868 and 738 us; 483, 504, 528, 418, 598
// and 441 us so), and boxes whose tables alone exceed a third kept 2,048 voxels whatever was free (55 x 55 x 33, 400 boxes,
// 946 -> 717 us; 73 x 73 x 9, 834 boxes, 1,565 -> 898 us; 73 x 73 x 1, 7,506 boxes, 8.86 -> 3.83 ms). A longer least list
// costs CTAs in turn: 8,192 voxels for the larger boxes, 1,003 boxes of 41 x 41 x 65: 2.15 ms, 1.34 so.
int pass2_plan(int max_bx, int max_dz, int K, bool* staged, Fit* fit) {
    const size_t P = (size_t)max_bx * max_bx;
    const size_t V = P * max_dz;
    const size_t chunks = (size_t)fit_chunks(max_dz);
    auto lists = [&](size_t cap, size_t pix, size_t run_pix) {
        return Fit{(int)cap, (int)pix, (int)(run_pix * chunks)};
    };
    auto bytes = [&](size_t cap, size_t pix, size_t run_pix, bool box) {
        return Pass2Layout(max_bx, max_dz, K, lists(cap, pix, run_pix), box).bytes;
    };
    const int nt = pass_threads(max_bx);
    if (bytes(0, 0, 0, false) > pass2_share(1, nt))
        return fail(XI_E_LIMIT, "pass 2: box too large (per-pixel tables exceed shared memory)");
    const bool large = V > (size_t)XI_PASS2_LARGE_VOXELS || max_dz > XI_PASS2_LARGE_DEPTH;
    const size_t want = (size_t)g_list_cap[large ? 1 : 0], least = V < want ? V : want;
    size_t pix = P < (size_t)kFitPix ? P : (size_t)kFitPix;
    auto ctas = [&](bool box) {                           // an SM holds with the least list (0: not even one)
        int n = 768 / nt;
        while (n > 0 && bytes(least, pix, pix, box) > pass2_share(n, nt)) --n;
        return n;
    };
    const int n = ctas(false);
    *staged = V * sizeof(float) <= g_stage_max[1] && n > 0 && ctas(true) == n;
    const size_t room = pass2_share(n > 0 ? n : 1, nt);
    while (pix > 0 && bytes(0, pix, pix, *staged) > room) pix /= 2;
    size_t run_pix = pix;
    if (bytes(least, pix, P, *staged) <= room) run_pix = P;
    if (bytes(least, P, P, *staged) <= room) pix = P;
    // voxels of a list in `room` (beyond the room that it shares with the rocking-curve terms and the profile)
    const Pass2Layout base(max_bx, max_dz, K, lists(0, pix, run_pix), *staged);
    const size_t most = ((base.pix - base.list) + (room - base.bytes)) / 16 * 16 / 8;
    *fit = lists(want ? (V < most ? V : most) : 0, pix, run_pix);
    return XI_OK;
}

}  // namespace

// ==================================================================================================================
// C ABI
// ==================================================================================================================
extern "C" {

const char* xi_last_error(void) { return g_err; }

int xi_version(void) { return 3; }

int xi_tune(int key, long long value) {
    if (key == XI_TUNE_PASS1_STAGE_BYTES || key == XI_TUNE_PASS2_STAGE_BYTES) {
        if (value < 0 || value > (long long)kStageBudget) return fail(XI_E_LIMIT, "xi_tune: staging bytes");
        g_stage_max[key == XI_TUNE_PASS1_STAGE_BYTES ? 0 : 1] = (size_t)value;
        return XI_OK;
    }
    if (key == XI_TUNE_WIDE_THREADS) {
        if (value != 128 && value != 256) return fail(XI_E_LIMIT, "xi_tune: threads per CTA (128 or 256)");
        g_wide_nt = (int)value;
        return XI_OK;
    }
    if (key == XI_TUNE_PASS2_LIST_CAP || key == XI_TUNE_PASS2_LIST_CAP_LARGE) {
        if (value < 0 || value > 16384) return fail(XI_E_LIMIT, "xi_tune: list capacity");
        g_list_cap[key == XI_TUNE_PASS2_LIST_CAP ? 0 : 1] = (int)value;
        return XI_OK;
    }
    return fail(XI_E_ARG, "xi_tune: unknown key");
}

int xi_status(void* stream) {
    int* p = status_ptr();
    if (!p) return fail(XI_E_CUDA, "status word unavailable");
    int h = 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemcpyAsync(&h, p, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return cuda_check("xi_status");
    if (h) {
        int zero = 0;
        cudaMemcpyAsync(p, &zero, sizeof(int), cudaMemcpyHostToDevice, s);
        cudaStreamSynchronize(s);
        return fail(XI_E_SHAPE, "a row's shoebox shape exceeded the call's shape hint; the row was skipped");
    }
    return XI_OK;
}


int xi_status_copy(int* host_dst, void* stream) {
    int* p = status_ptr();
    if (!p) return fail(XI_E_CUDA, "status word unavailable");
    if (!host_dst) return fail(XI_E_ARG, "xi_status_copy: null destination");
    if (cudaMemcpyAsync(host_dst, p, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream) != cudaSuccess)
        return cuda_check("xi_status_copy");
    return XI_OK;
}


int xi_pass1(const XiDetector* det, const XiRows* R, const XiBlock* B, const float* arena, XiPass1Out* O,
             void* stream) {
    if (!det || !B || !arena || !O) return fail(XI_E_ARG, "xi_pass1: null argument");
    int rc = rows_check(R);
    if (rc) return rc;
    const int nblk = R->order ? R->n_order : R->n;
    if (nblk == 0) return XI_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t P = (size_t)R->max_bx * R->max_bx;
    const bool staged = pass1_staged(R->max_bx, R->max_dz, R->K);
    if (staged) {
        if (P <= 96) return launch_pass1<64, true>(det, R, B, arena, O, s, nblk);
        if (P <= 200 || g_wide_nt == 128) return launch_pass1<128, true>(det, R, B, arena, O, s, nblk);
        return launch_pass1<256, true>(det, R, B, arena, O, s, nblk);
    }
    if (P <= 96) return launch_pass1<64, false>(det, R, B, arena, O, s, nblk);
    if (P <= 200 || g_wide_nt == 128) return launch_pass1<128, false>(det, R, B, arena, O, s, nblk);
    return launch_pass1<256, false>(det, R, B, arena, O, s, nblk);
}


int xi_pass2(const XiDetector* det, const XiRows* R, const XiBlock* B, const float* arena, const float* prof,
             const XiPass2In* in, XiPass2Out* O, void* stream) {
    if (!det || !B || !arena || !prof || !in || !O) return fail(XI_E_ARG, "xi_pass2: null argument");
    int rc = rows_check(R);
    if (rc) return rc;
    const int nblk = R->order ? R->n_order : R->n;
    if (nblk == 0) return XI_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t P = (size_t)R->max_bx * R->max_bx;
    bool staged = false;
    Fit fit{0, 0, 0};
    rc = pass2_plan(R->max_bx, R->max_dz, R->K, &staged, &fit);
    if (rc) return rc;
    if (staged) {
        if (P <= 96) return launch_pass2<64, true>(det, R, B, arena, prof, in, O, s, nblk, fit);
        if (P <= 200 || g_wide_nt == 128) return launch_pass2<128, true>(det, R, B, arena, prof, in, O, s, nblk, fit);
        return launch_pass2<256, true>(det, R, B, arena, prof, in, O, s, nblk, fit);
    }
    if (P <= 96) return launch_pass2<64, false>(det, R, B, arena, prof, in, O, s, nblk, fit);
    if (P <= 200 || g_wide_nt == 128) return launch_pass2<128, false>(det, R, B, arena, prof, in, O, s, nblk, fit);
    return launch_pass2<256, false>(det, R, B, arena, prof, in, O, s, nblk, fit);
}

static int batched_check(const XiRowSet* sets, const int64_t* items, int n_items, int max_bx, int max_dz, int max_k,
                         int* queue, const char* who) {
    if (n_items < 0) return fail(XI_E_ARG, who);
    if (n_items && (!sets || !items || !queue)) return fail(XI_E_ARG, who);
    if (max_bx < 3 || max_bx > XI_MAX_BX || max_dz < 1 || max_dz > XI_MAX_DZ || max_k < 0 || max_k > XI_MAX_K)
        return fail(XI_E_LIMIT, "batched pass: max_bx / max_dz / max_k outside 3..97 / 1..65 / 0..16");
    return XI_OK;
}

int xi_pass1_batched(const XiRowSet* sets, const int64_t* items, int n_items, int max_bx, int max_dz, int max_k,
                     int* queue, void* stream) {
    int rc = batched_check(sets, items, n_items, max_bx, max_dz, max_k, queue, "xi_pass1_batched: bad argument");
    if (rc || n_items == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t P = (size_t)max_bx * max_bx;
    if (pass1_staged(max_bx, max_dz, max_k)) {
        if (P <= 96) return launch_pass1_q<64, true>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
        if (P <= 200 || g_wide_nt == 128) return launch_pass1_q<128, true>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
        return launch_pass1_q<256, true>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
    }
    if (P <= 96) return launch_pass1_q<64, false>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
    if (P <= 200 || g_wide_nt == 128) return launch_pass1_q<128, false>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
    return launch_pass1_q<256, false>(sets, items, n_items, max_bx, max_dz, max_k, queue, s);
}

int xi_pass2_batched(const XiRowSet* sets, const int64_t* items, int n_items, int max_bx, int max_dz, int max_k,
                     int* queue, void* stream) {
    int rc = batched_check(sets, items, n_items, max_bx, max_dz, max_k, queue, "xi_pass2_batched: bad argument");
    if (rc || n_items == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t P = (size_t)max_bx * max_bx;
    bool staged = false;
    Fit fit{0, 0, 0};
    rc = pass2_plan(max_bx, max_dz, max_k, &staged, &fit);
    if (rc) return rc;
    if (staged) {
        if (P <= 96) return launch_pass2_q<64, true>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
        if (P <= 200 || g_wide_nt == 128) return launch_pass2_q<128, true>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
        return launch_pass2_q<256, true>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
    }
    if (P <= 96) return launch_pass2_q<64, false>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
    if (P <= 200 || g_wide_nt == 128) return launch_pass2_q<128, false>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
    return launch_pass2_q<256, false>(sets, items, n_items, max_bx, max_dz, max_k, fit, queue, s);
}

int xi_gather(const XiFrames* F, const XiGatherRows* G, float* arena, int32_t* cnt, void* stream) {
    if (!F || !G || !arena || !F->data) return fail(XI_E_ARG, "xi_gather: null argument");
    if (F->n_frames < 0 || F->ny <= 0 || F->nx <= 0 || G->n < 0) return fail(XI_E_ARG, "xi_gather: bad sizes");
    const int nblk = G->order ? G->n_order : G->n;
    if (nblk == 0 || F->n_frames == 0) return XI_OK;
    const bool small = G->max_bx > 0 && G->max_bx <= (F->is_float ? kGatherSmallFloat : kGatherSmall);
    const int nt = small ? kGatherThreads / 2 : kGatherThreads;
    cudaStream_t s = (cudaStream_t)stream;
    if (F->is_float && !small)
        k_gather<kGatherFloatBatch><<<nblk, nt, 0, s>>>(*F, *G, arena, cnt, G->order);
    else
        k_gather<kGatherBatch><<<nblk, nt, 0, s>>>(*F, *G, arena, cnt, G->order);
    return cuda_check("xi_gather");
}

int xi_gather_step(const XiGatherStep* step, const XiGatherRows* G, float* arena, int32_t* cnt, int grid,
                   void* stream) {
    if (!step || !G || !arena) return fail(XI_E_ARG, "xi_gather_step: null argument");
    if (grid <= 0 || G->n < 0) return fail(XI_E_ARG, "xi_gather_step: bad sizes");
    k_gather_step<<<grid, kGatherThreads, 0, (cudaStream_t)stream>>>(step, *G, arena, cnt);
    return cuda_check("xi_gather_step");
}

int xi_decode_bins(const XiGatherRows* G, float* arena, const int32_t* cnt, void* stream) {
    if (!G || !arena || !cnt) return fail(XI_E_ARG, "xi_decode_bins: null argument");
    if (G->n == 0) return XI_OK;
    const int nblk = G->order ? G->n_order : G->n;
    if (nblk <= 0) return XI_OK;
    k_decode_bins<<<nblk, 256, 0, (cudaStream_t)stream>>>(*G, arena, cnt);
    return cuda_check("xi_decode_bins");
}

int xi_zero_rows(const XiGatherRows* G, float* arena, void* stream) {
    if (!G || !arena) return fail(XI_E_ARG, "xi_zero_rows: null argument");
    const int nblk = G->order ? G->n_order : G->n;
    if (nblk <= 0) return XI_OK;
    if (((uintptr_t)arena & 15) != 0) return fail(XI_E_ARG, "xi_zero_rows: arena not on 16 bytes");
    k_zero_rows<<<nblk, 256, 0, (cudaStream_t)stream>>>(*G, arena);
    return cuda_check("xi_zero_rows");
}

int xi_accumulate(const XiRows* R, const XiPass1Out* p1, const uint8_t* sel, int strong_test, int n_regions,
                  double* num, double* den, void* stream) {
    if (!R || !p1 || !num || !den) return fail(XI_E_ARG, "xi_accumulate: null argument");
    if (n_regions <= 0) return fail(XI_E_ARG, "xi_accumulate: n_regions");
    const int nblk = R->order ? R->n_order : R->n;
    if (nblk == 0) return XI_OK;
    k_accumulate<<<nblk, 128, 0, (cudaStream_t)stream>>>(*R, *p1, sel, strong_test, n_regions, num, den);
    return cuda_check("xi_accumulate");
}

int xi_finalize_profiles(const double* num, const double* den, int n_regions, float* prof, void* stream) {
    if (!num || !den || !prof || n_regions <= 0) return fail(XI_E_ARG, "xi_finalize_profiles: bad argument");
    k_finalize<<<n_regions, 256, 0, (cudaStream_t)stream>>>(num, den, prof);
    return cuda_check("xi_finalize_profiles");
}

}  // extern "C"

int xi_fail(int code, const char* msg) { return fail(code, msg); }
int xi_cuda_check(const char* where) { return cuda_check(where); }
