// Forward-model likelihood passes (XPG's pixel-level forward integrator, xpg/forward/): the fused scatter / gather
// of the separable profile factors of reflections' boxes into / from a dense window of voxels, the work of
// xpg/forward/kernels.py:34-103 (Triton) and of the eager passes WindowModel.mu / grad_ratio / grad_newton
// (xpg/forward/model.py:476-577).
//
// A warp (or, of few reflections, a CTA of four) takes a reflection: a lane holds a pixel of its box (the terms'
// factors P and the voxel's place in the window, looked up once) and walks the box's frames inside the window, four
// voxels in flight: f = sum_t R[t, row, z] * P[t, row, y, x], and either adds I f + beta to the window voxel (scatter:
// float atomics, several reflections share voxels) or accumulates the weighted sums of the row in float64 (gather),
// reduced over the warp or CTA and added once to the row's output.
// Frames outermost, a CTA of 128 a reflection, each voxel's place in the window by 64-bit products and a division, was
// bound by instructions: 544, 889 and 860 us for the scatter and the two gathers of 60,000 boxes of 9 x 13 x 13 voxels
// with two terms in a 40 x 1024 x 1024 window. So arranged: 268, 472 and 371 us. The scatter is bound by the L2's
// atomics, the ratio gather by DRAM (68% of its peak: the boxes' 52-byte rows lie anywhere in 420 MB, and come in
// 64-byte pieces), the Newton gather by its two IEEE quotients a voxel.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "xpgi.h"

namespace {

thread_local char g_err[256] = {0};

int fm_fail(int code, const char* msg) {
    snprintf(g_err, sizeof g_err, "%s", msg);
    return code;
}

constexpr int kFmThreads = 128;
constexpr int kFmBatch = 4;                  // voxels of a pixel in flight

// A reflection's box in the window: its frames z0 .. z1 - 1 that lie in it, and the index of voxel (0, 0, 0).
struct Box {
    int64_t ky0, kx0, first, plane;
    int z0, z1;
};

__device__ __forceinline__ Box box_of(const XiFmBoxes& B, const XiFmWindow& W, int row) {
    Box o;
    const int64_t kz0 = B.iz0[row] - W.f0;
    o.ky0 = B.iy0[row] - W.y0;
    o.kx0 = B.ix0[row] - W.x0;
    o.plane = (int64_t)W.ny * W.nx;
    o.first = (kz0 * W.ny + o.ky0) * W.nx + o.kx0;
    const int64_t lo = kz0 < 0 ? -kz0 : 0, hi = W.nf - kz0;
    o.z0 = (int)(lo < B.Dz ? lo : B.Dz);
    o.z1 = (int)(hi < B.Dz ? (hi > 0 ? hi : 0) : B.Dz);
    return o;
}

// The terms' factors of one pixel of a box (T: their number, or 0: B.n_terms, up to 4).
template <int T>
struct Factors {
    static constexpr int N = T ? T : 4;
    float p[N];
    const float* r[N];

    __device__ __forceinline__ int terms(const XiFmBoxes& B) const { return T ? T : B.n_terms; }
    __device__ __forceinline__ void row(const XiFmBoxes& B, int row) {
#pragma unroll
        for (int t = 0; t < N; ++t)
            if (t < terms(B)) r[t] = B.R + ((size_t)t * B.n + row) * B.Dz;
    }
    __device__ __forceinline__ void pixel(const XiFmBoxes& B, int row, int px) {
        const size_t bb = (size_t)B.b * B.b;
#pragma unroll
        for (int t = 0; t < N; ++t)
            if (t < terms(B)) p[t] = __ldg(B.P + ((size_t)t * B.n + row) * bb + px);
    }
    // f on frame z: the terms' products rounded, then summed in term order
    __device__ __forceinline__ float at(const XiFmBoxes& B, int z) const {
        float f = __ldg(r[0] + z) * p[0];
#pragma unroll
        for (int t = 1; t < N; ++t)
            if (t < terms(B)) f = f + __ldg(r[t] + z) * p[t];
        return f;
    }
};

// The row and first pixel of a thread: WPR warps (1 or 4) a row.
template <int WPR>
__device__ __forceinline__ int row_of() {
    return WPR == 1 ? (int)(blockIdx.x * (kFmThreads / 32) + threadIdx.x / 32) : (int)blockIdx.x;
}

template <int T, int WPR>
__global__ void __launch_bounds__(kFmThreads) k_fm_scatter(XiFmBoxes B, XiFmWindow W, const float* __restrict__ I,
                                                           const float* __restrict__ beta, float* __restrict__ mu) {
    const int row = row_of<WPR>();
    if (row >= B.n) return;
    const Box o = box_of(B, W, row);
    const float Ir = I[row];
    const float br = beta ? beta[row] : 0.0f;
    const int bb = B.b * B.b;
    Factors<T> F;
    F.row(B, row);
    for (int px = WPR == 1 ? threadIdx.x & 31 : threadIdx.x; px < bb; px += 32 * WPR) {
        const int y = px / B.b, x = px - y * B.b;
        const int64_t ky = o.ky0 + y, kx = o.kx0 + x;
        if (ky < 0 || ky >= W.ny || kx < 0 || kx >= W.nx) continue;
        F.pixel(B, row, px);
        float* v = mu + o.first + (int64_t)y * W.nx + x + o.z0 * o.plane;
#pragma unroll 4
        for (int z = o.z0; z < o.z1; ++z, v += o.plane) {
            float val = F.at(B, z) * Ir;
            if (beta) val = val + br;
            atomicAdd(v, val);
        }
    }
}

// a / m with the zero counts, which most voxels have, kept off the division's slow path (a zero numerator takes it)
__device__ __forceinline__ float quotient(float a, float m) {
    const float q = (a == 0.0f ? 1.0f : a) / m;
    return a == 0.0f ? (m != 0.0f && m == m ? 0.0f : __int_as_float(0x7fc00000)) : q;
}

// one voxel's terms of a row's sums; a voxel without a count (ns < 0) has none
template <int MODE>
__device__ __forceinline__ void add(float f, float ns, float m, float a, double& acc, double& accd) {
    const bool on = ns >= 0.0f;
    if (MODE == 0) {
        const float t = f * quotient(a, m);
        acc += (double)(on ? t : 0.0f);
    } else {
        const float t = f * (1.0f - quotient(fmaxf(ns, 0.0f), m)), d = (f * f) / fmaxf(m, 1e-6f);
        acc += (double)(on ? t : 0.0f);
        accd += (double)(on ? d : 0.0f);
    }
}

template <typename NST, int MODE, int T, int WPR>
__global__ void __launch_bounds__(kFmThreads) k_fm_gather(XiFmBoxes B, XiFmWindow W, const int64_t* __restrict__ rows,
                                                          const float* __restrict__ A, const float* __restrict__ M,
                                                          const NST* __restrict__ NS, float* __restrict__ g,
                                                          float* __restrict__ fd) {
    const int row = row_of<WPR>();
    double acc = 0.0, accd = 0.0;
    if (row < B.n) {
        const Box o = box_of(B, W, row);
        const int bb = B.b * B.b;
        Factors<T> F;
        F.row(B, row);
        for (int px = WPR == 1 ? threadIdx.x & 31 : threadIdx.x; px < bb; px += 32 * WPR) {
            const int y = px / B.b, x = px - y * B.b;
            const int64_t ky = o.ky0 + y, kx = o.kx0 + x;
            if (ky < 0 || ky >= W.ny || kx < 0 || kx >= W.nx) continue;
            F.pixel(B, row, px);
            int64_t v = o.first + (int64_t)y * W.nx + x + o.z0 * o.plane;
            int z = o.z0;
            // full batches without a branch a voxel (a masked voxel adds zero), then the frames left over
            for (; z + kFmBatch <= o.z1; z += kFmBatch) {
                float ns[kFmBatch], m[kFmBatch], a[kFmBatch];
#pragma unroll
                for (int u = 0; u < kFmBatch; ++u, v += o.plane) {
                    ns[u] = (float)__ldg(NS + v);
                    m[u] = __ldg(M + v);
                    if (MODE == 0) a[u] = __ldg(A + v);
                }
#pragma unroll
                for (int u = 0; u < kFmBatch; ++u) add<MODE>(F.at(B, z + u), ns[u], m[u], a[u], acc, accd);
            }
            for (; z < o.z1; ++z, v += o.plane)
                add<MODE>(F.at(B, z), (float)__ldg(NS + v), __ldg(M + v), MODE == 0 ? __ldg(A + v) : 0.0f, acc, accd);
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (MODE == 1) accd += __shfl_down_sync(0xffffffffu, accd, off);
    }
    if (WPR > 1) {
        __shared__ double s_acc[2][WPR];
        if ((threadIdx.x & 31) == 0) {
            s_acc[0][threadIdx.x / 32] = acc;
            s_acc[1][threadIdx.x / 32] = accd;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            acc = accd = 0.0;
            for (int w = 0; w < WPR; ++w) {
                acc += s_acc[0][w];
                accd += s_acc[1][w];
            }
        }
    }
    if (row < B.n && (WPR == 1 ? (threadIdx.x & 31) == 0 : threadIdx.x == 0)) {
        const int64_t r = rows ? rows[row] : row;
        atomicAdd(g + r, (float)acc);
        if (MODE == 1) atomicAdd(fd + r, (float)accd);
    }
}

int check_boxes(const XiFmBoxes* B, const XiFmWindow* W) {
    if (!B || !W) return fm_fail(XI_E_ARG, "forward pass: null argument");
    if (B->n < 0 || B->n_terms < 1 || B->n_terms > 4 || B->Dz < 1 || B->b < 1)
        return fm_fail(XI_E_ARG, "forward pass: bad box shape (n >= 0, 1..4 terms, Dz >= 1, b >= 1)");
    if (B->n > 0 && (!B->R || !B->P || !B->iz0 || !B->iy0 || !B->ix0))
        return fm_fail(XI_E_ARG, "forward pass: null factor or origin array");
    if (W->nf < 0 || W->ny < 0 || W->nx < 0) return fm_fail(XI_E_ARG, "forward pass: negative window size");
    return XI_OK;
}

int launch_check(const char* who) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof g_err, "%s: %s", who, cudaGetErrorString(e));
        return XI_E_CUDA;
    }
    return XI_OK;
}

// A warp a reflection where that fills the device, else a CTA (the two gathers of 60,000 boxes of 9 x 13 x 13 voxels:
// 472 and 371 us by warps, 515 and 427 by CTAs; of 5,000 boxes 57 and 52 us by warps, 52 and 45 by CTAs). A box of at
// most 32 pixels has no work for a second warp, one of up to 64 little: warps too, from 148 x 8 rows on of the latter
// (ratio gather of 9,471 boxes of 3 x 1 x 1 with three terms 27.1 us by CTAs, 11.2 by warps, of 1 x 7 x 7 14.4 and 8.1;
// 2,000 of 9 x 7 x 7 8.6 and 7.3, but 500 of them 5.1 and 6.1).
bool warp_rows(const XiFmBoxes& B) {
    const int64_t px = (int64_t)B.b * B.b;
    return B.n >= 148 * 64 || px <= 32 || (px <= 64 && B.n >= 148 * 8);
}

template <int T>
void launch_scatter(const XiFmBoxes& B, const XiFmWindow& W, const float* I, const float* beta, float* mu,
                    cudaStream_t s) {
    if (warp_rows(B)) k_fm_scatter<T, 1><<<(B.n - 1) / 4 + 1, kFmThreads, 0, s>>>(B, W, I, beta, mu);
    else k_fm_scatter<T, 4><<<B.n, kFmThreads, 0, s>>>(B, W, I, beta, mu);
}

template <typename NST, int MODE, int T>
void launch_gather(const XiFmBoxes& B, const XiFmWindow& W, const int64_t* rows, const float* A, const float* M,
                   const void* NS, float* g, float* fd, cudaStream_t s) {
    const NST* ns = static_cast<const NST*>(NS);
    if (warp_rows(B)) k_fm_gather<NST, MODE, T, 1><<<(B.n - 1) / 4 + 1, kFmThreads, 0, s>>>(B, W, rows, A, M, ns, g, fd);
    else k_fm_gather<NST, MODE, T, 4><<<B.n, kFmThreads, 0, s>>>(B, W, rows, A, M, ns, g, fd);
}

template <typename NST, int MODE, typename... Args>
void launch_terms(const XiFmBoxes& B, Args... a) {
    if (B.n_terms == 1) launch_gather<NST, MODE, 1>(B, a...);
    else if (B.n_terms == 2) launch_gather<NST, MODE, 2>(B, a...);
    else launch_gather<NST, MODE, 0>(B, a...);
}

template <typename NST>
void launch_mode(const XiFmBoxes& B, const XiFmWindow& W, const int64_t* rows, const float* A, const float* M,
                 const void* NS, int mode, float* g, float* fd, cudaStream_t s) {
    if (mode == 0) launch_terms<NST, 0>(B, W, rows, A, M, NS, g, fd, s);
    else launch_terms<NST, 1>(B, W, rows, A, M, NS, g, fd, s);
}

}  // namespace

extern "C" {

const char* xi_fm_last_error(void) { return g_err; }

int xi_fm_scatter(const XiFmBoxes* boxes, const XiFmWindow* win, const float* I, const float* beta, float* mu,
                  void* stream) {
    int rc = check_boxes(boxes, win);
    if (rc) return rc;
    if (boxes->n == 0) return XI_OK;
    if (!I || !mu) return fm_fail(XI_E_ARG, "xi_fm_scatter: null I or mu");
    if (boxes->n_terms == 1) launch_scatter<1>(*boxes, *win, I, beta, mu, (cudaStream_t)stream);
    else if (boxes->n_terms == 2) launch_scatter<2>(*boxes, *win, I, beta, mu, (cudaStream_t)stream);
    else launch_scatter<0>(*boxes, *win, I, beta, mu, (cudaStream_t)stream);
    return launch_check("xi_fm_scatter");
}

int xi_fm_gather(const XiFmBoxes* boxes, const XiFmWindow* win, const int64_t* rows, const float* A, const float* M,
                 const void* NS, int ns_type, int mode, float* g, float* fd, void* stream) {
    int rc = check_boxes(boxes, win);
    if (rc) return rc;
    if (boxes->n == 0) return XI_OK;
    if (!M || !NS || !g) return fm_fail(XI_E_ARG, "xi_fm_gather: null M, NS or g");
    if (mode == 0 && !A) return fm_fail(XI_E_ARG, "xi_fm_gather: mode 0 needs A");
    if (mode == 1 && !fd) return fm_fail(XI_E_ARG, "xi_fm_gather: mode 1 needs fd");
    if (mode != 0 && mode != 1) return fm_fail(XI_E_ARG, "xi_fm_gather: mode 0 or 1");
    cudaStream_t s = (cudaStream_t)stream;
    switch (ns_type) {
        case XI_FM_NS_I16: launch_mode<int16_t>(*boxes, *win, rows, A, M, NS, mode, g, fd, s); break;
        case XI_FM_NS_I32: launch_mode<int32_t>(*boxes, *win, rows, A, M, NS, mode, g, fd, s); break;
        case XI_FM_NS_F32: launch_mode<float>(*boxes, *win, rows, A, M, NS, mode, g, fd, s); break;
        default: return fm_fail(XI_E_ARG, "xi_fm_gather: ns_type");
    }
    return launch_check("xi_fm_gather");
}

}  // extern "C"
