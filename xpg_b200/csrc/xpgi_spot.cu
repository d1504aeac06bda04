// Strong-pixel classifier of spot finding (include/xpgi.h, "Spot finding"): XPG's dispersion test and its extended
// second pass (xpg/spotfind.py:27-97) on float32 frames, bit for bit. Both passes need, per pixel, window sums of the
// valid-pixel count, the values and their squares, each sum over its window in increasing coordinate from zero (along
// x for every row, then the row sums along y: the order the reference's pooling sums in; zero outside the frame).
//
// The work is instructions (float adds, shared-memory reads), not bytes (16 B a pixel over the two launches): a warp
// marches a strip of 64 columns down the frame, four rows a step. A lane owns two adjacent columns, so a staged value
// feeds two horizontal sums, and a row's sums, kept in a ring of rows in shared memory, feed four vertical ones; the
// sums of value and square are one packed float pair (add.rn.f32x2: two IEEE adds an instruction); the counts are
// integers (bit windows along x, running sums along y); the tests' roots and quotients are computed only where bounds
// leave the test open. One warp a CTA: with four, and a strip of 256 columns, warps waited for one another (1.6 ms in
// place of 1.4 at that stage). Against a thread a pixel with both window loops in shared memory (32 x 8 tiles, 46 x
// 22 staged for the second pass): four 4148 x 4362 frames 4.19 -> 1.13 ms, one 1030 x 1065 frame 76 -> 44 us
// (first pass alone: 1.35 -> 0.38 ms, 26 -> 18 us), windows of half widths 0 to 8, square and not, of four such frames
// 0.27 to 0.56 of the time.
// The first launch of an extended call finds the strong pixels and writes the background pixels (those not within
// 1 px of one) and the pixels within 2 px of one; the second re-estimates the background and classifies.
// Small frames have too few strips for that (a warp's march is one long chain of steps); they take the tiles (below).
#include <cuda_runtime.h>
#include <stdint.h>

#include "xpgi.h"
#include "xpgi_internal.h"

namespace {

constexpr int kNT = 32;                      // threads of a CTA: one warp, so that no warp waits for another
constexpr int kPx = 2;                       // adjacent columns of a thread
constexpr int kCols = kNT * kPx;             // columns of a strip
constexpr int kStep = 4;                     // rows of a step
constexpr int kRing = 16;                    // bit rows kept by a first pass (a power of two)
constexpr int kMaxHalf = 2 * XI_SPOT_MAX_HALF + 1;
constexpr float kDispersionSigmaB = 6.0f;

typedef unsigned long long pair_t;           // (sum, sum of squares): two floats

__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
    pair_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ pair_t pack2(float a, float b) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void unpack2(pair_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

// Shared memory of a CTA for half widths hx, hy: the ring of horizontal sums (2 hy + 4 rows) and counts, four staged
// rows of values and of weight bits, the bit rows of the first pass (25.6 KB at most).
struct Layout {
    int ring, width, words;                  // rows of the ring; staged values and weight words of a row
    size_t cnt, raw, bits, flag, bytes;

    __host__ __device__ Layout(int hx, int hy) {
        ring = 2 * hy + kStep;
        width = (kCols + 2 * hx + 3) / 4 * 4;
        words = (kCols + 2 * hx + kNT - 1) / kNT + 2;
        cnt = (size_t)ring * kCols * sizeof(pair_t);
        raw = cnt + (size_t)ring * kNT * sizeof(uint16_t);
        bits = raw + (size_t)kStep * width * sizeof(pair_t);
        flag = bits + (size_t)kStep * words * sizeof(uint32_t);
        bytes = flag + (size_t)2 * kRing * 2 * sizeof(uint32_t);
    }
};

// The window sums of the CTA's strip: columns x0 .. x0 + 63, four rows a step, a thread's two columns in its
// registers. H >= 0: both half widths, known at compile time (loops unrolled); H < 0: hx, hy. A pixel enters with
// weight 1 where it is valid (SEL false) or where its flag in sel is set.
template <int H, bool SEL>
struct Strip {
    static constexpr int kLoads = (kCols + 2 * (H >= 0 ? H : kMaxHalf) + kNT - 1) / kNT;
    const float* img;
    const uint8_t* sel;
    int ny, nx, x0, hx_, hy_;
    Layout L;
    unsigned char* sm;
    float v[kStep][kLoads];                  // the next rows, on their way from memory
    uint8_t w[SEL ? kStep : 1][SEL ? kLoads : 1];
    unsigned cols;                           // which of the thread's staged columns lie in the frame
    uint32_t n2;                             // weights of the 2 hy rows before the next one, 16 bits a column
    int slot;                                // ring row of the next staged row

    __device__ Strip(const float* i, const uint8_t* s, int ny_, int nx_, int x, int hx__, int hy__, unsigned char* m)
        : img(i), sel(s), ny(ny_), nx(nx_), x0(x), hx_(hx__), hy_(hy__), L(H >= 0 ? H : hx__, H >= 0 ? H : hy__),
          sm(m), cols(0), n2(0), slot(0) {
        for (int k = 0; k < kLoads; ++k) {
            const int c = threadIdx.x + k * kNT, xx = x0 - hx() + c;
            if (c < kCols + 2 * hx() && xx >= 0 && xx < nx) cols |= 1u << k;
        }
    }
    __device__ __forceinline__ int hx() const { return H >= 0 ? H : hx_; }
    __device__ __forceinline__ int hy() const { return H >= 0 ? H : hy_; }
    __device__ __forceinline__ ulonglong2* ring(int row) const {
        return reinterpret_cast<ulonglong2*>(sm) + (size_t)row * kNT + threadIdx.x;
    }
    __device__ __forceinline__ uint16_t* ring_n() const { return reinterpret_cast<uint16_t*>(sm + L.cnt) + threadIdx.x; }
    __device__ __forceinline__ int wrap(int row) const { return row >= L.ring ? row - L.ring : row; }
    __device__ __forceinline__ static uint32_t wide(uint16_t c) { return (c & 0xffu) | ((uint32_t)(c >> 8) << 16); }

    // rows y .. y + rows - 1 into registers (invalid outside the frame)
    __device__ __forceinline__ void fetch(int y, int rows) {
        const int64_t at = (int64_t)y * nx + (x0 - hx() + (int)threadIdx.x);
#pragma unroll
        for (int r = 0; r < kStep; ++r) {
            const bool in = r < rows && y + r >= 0 && y + r < ny;
            const int64_t o = at + (int64_t)r * nx;
#pragma unroll
            for (int k = 0; k < kLoads; ++k) {
                const bool on = in && ((cols >> k) & 1u);
                v[r][k] = on ? __ldg(img + o + k * kNT) : -1.0f;
                if (SEL) w[r][k] = on ? __ldg(sel + o + k * kNT) : 0;
            }
        }
    }

    // the fetched rows into shared memory: value and square of every pixel that counts, the weights as bits
    __device__ __forceinline__ void stage(int rows) {
        pair_t* raw = reinterpret_cast<pair_t*>(sm + L.raw) + threadIdx.x;
        uint32_t* bits = reinterpret_cast<uint32_t*>(sm + L.bits);
        __syncwarp();                                   // the last step's readers are done
#pragma unroll
        for (int r = 0; r < kStep; ++r) {
            if (r >= rows) break;
#pragma unroll
            for (int k = 0; k < kLoads; ++k) {
                if (H < 0 && k * kNT >= kCols + 2 * hx()) break;
                const bool on = SEL ? w[SEL ? r : 0][SEL ? k : 0] != 0 : v[r][k] >= 0.0f;
                const unsigned ball = __ballot_sync(0xffffffffu, on);
                const float x = on ? v[r][k] : 0.0f;
                if ((k + 1) * kNT <= kCols || (int)threadIdx.x + k * kNT < L.width) raw[r * L.width + k * kNT] = pack2(x, x * x);
                if (threadIdx.x == 0) bits[r * L.words + k] = ball;
            }
        }
        __syncwarp();
    }

    // the staged rows' horizontal sums and counts of the thread's columns into the ring
    __device__ __forceinline__ void horizontal(int rows) {
        const ulonglong2* raw = reinterpret_cast<const ulonglong2*>(sm + L.raw) + threadIdx.x;
        const int b = kPx * threadIdx.x, sh = b & 31;
        const uint32_t* bits = reinterpret_cast<const uint32_t*>(sm + L.bits) + b / 32;
        const int wd = 2 * hx();                           // last offset of a window
#pragma unroll 2
        for (int r = 0; r < rows; ++r, raw += L.width / 2, bits += L.words) {
            pair_t a[kPx] = {0ull, 0ull};
#pragma unroll
            for (int k0 = 0; k0 < (H >= 0 ? 2 * H + kPx : 2 * kMaxHalf + kPx); k0 += 2) {
                if (H < 0 && k0 >= wd + kPx) break;
                const ulonglong2 f = raw[k0 / 2];
                if (k0 <= wd) a[0] = add2(a[0], f.x);
                if (k0 >= 1) a[1] = add2(a[1], f.x);
                if (k0 + 1 <= wd) a[0] = add2(a[0], f.y);
                a[1] = add2(a[1], f.y);
            }
            const int row = wrap(slot + r);
            *ring(row) = make_ulonglong2(a[0], a[1]);
            unsigned c0, c1;
            if (H >= 0 && 2 * H + kPx <= 32) {
                const uint32_t win = __funnelshift_r(bits[0], bits[1], sh);
                c0 = __popc(win & ((2u << wd) - 1u));
                c1 = c0 + ((win >> (wd + 1)) & 1u) - (win & 1u);
            } else {
                unsigned long long win = (((unsigned long long)bits[1] << 32) | bits[0]) >> sh;
                if (sh) win |= (unsigned long long)bits[2] << (64 - sh);
                c0 = __popcll(win & ((2ull << wd) - 1ull));
                c1 = c0 + (unsigned)((win >> (wd + 1)) & 1ull) - (unsigned)(win & 1ull);
            }
            ring_n()[row * kNT] = (uint16_t)(c0 | (c1 << 8));
        }
    }

    // the first 2 hy rows of the windows of row y (the rows from y - hy on)
    __device__ __forceinline__ void start(int y) {
        fetch(y - hy(), min(kStep, 2 * hy()));
        for (int done = 0; done < 2 * hy(); done += kStep) {
            const int rows = min(kStep, 2 * hy() - done);
            stage(rows);
            // the next group: more rows of the start, or the four rows of the first step
            fetch(y - hy() + done + rows, done + rows < 2 * hy() ? min(kStep, 2 * hy() - done - rows) : kStep);
            horizontal(rows);
            for (int r = 0; r < rows; ++r) n2 += wide(ring_n()[wrap(slot + r) * kNT]);
            slot = wrap(slot + rows);
        }
        if (hy() == 0) fetch(y, kStep);
    }

    // the window sums of rows y .. y + 3 of the thread's columns (s: value and square; n: counts, 16 bits a column);
    // rows y + 4 + hy .. on their way
    __device__ __forceinline__ void step(int y, pair_t (&s)[kStep][kPx], uint32_t (&n)[kStep]) {
        fetch(y + hy() + kStep, kStep);
        horizontal(kStep);
        const int first = wrap(slot + kStep);              // ring row of row y - hy
        slot = first;
#pragma unroll
        for (int j = 0; j < kStep; ++j)
#pragma unroll
            for (int q = 0; q < kPx; ++q) s[j][q] = 0ull;
        int row = first;
#pragma unroll
        for (int i = 0; i < (H >= 0 ? 2 * H + kStep : 2 * kMaxHalf + kStep); ++i) {
            if (H < 0 && i >= 2 * hy() + kStep) break;
            const ulonglong2 u = *ring(row);
#pragma unroll
            for (int j = 0; j < kStep; ++j)
                if (i >= j && i - j <= 2 * hy()) {
                    s[j][0] = add2(s[j][0], u.x);
                    s[j][1] = add2(s[j][1], u.y);
                }
            row = wrap(row + 1);
        }
        int lead = wrap(first + 2 * hy()), tail = first;
#pragma unroll
        for (int j = 0; j < kStep; ++j) {
            n[j] = n2 + wide(ring_n()[lead * kNT]);
            n2 = n[j] - wide(ring_n()[tail * kNT]);
            lead = wrap(lead + 1);
            tail = wrap(tail + 1);
        }
    }
};

// The two tests of a pixel against multiples of a sigma that involve a root are first made with bounds that hold for
// any rounding of the exact expressions; only a pixel the bounds leave open takes the exact ones (a bright or a
// borderline pixel, well under one in a thousand), so the roots and quotients of the others are not computed.

// false: (d > k * sqrt(s2)) does not hold for any s2 >= v, however it is rounded
__device__ __forceinline__ bool may_exceed(float d, float k, float v) {
    return k < 0.0f || (d > 0.0f && !(1.001f * (d * d) < (k * k) * v));
}

// The exact tests, kept out of line: inlined for each of a lane's eight pixels they made the loop overrun the
// instruction cache (2.0 ms for four 4148 x 4362 frames, 1.6 out of line).
__device__ __noinline__ bool dispersed(float p, float n, float s1, float s2, float gain, float n_s) {
    const float nn = fmaxf(n, 2.0f);
    const float mean = s1 / nn;
    const float var = fmaxf((s2 - s1 * mean) / (nn - 1.0f), 0.0f);
    const float thr = gain * (1.0f + kDispersionSigmaB * sqrtf(2.0f / (nn - 1.0f)));
    return var > thr * fmaxf(mean, 1e-6f) && (p - mean) > n_s * sqrtf(gain * fmaxf(mean, 1.0f));
}

__device__ __noinline__ bool at_most(float p, float n, float s1, float gain, float bgp) {
    const float mean = s1 / fmaxf(n, 2.0f);
    return p <= mean + bgp * sqrtf(gain * fmaxf(mean, 0.5f));
}

__device__ __noinline__ bool exceeds(float p, float n, float s1, float s2, float gain, float sp) {
    const float nn = fmaxf(n, 2.0f);
    const float mean = s1 / nn;
    const float var = fmaxf((s2 - s1 * mean) / (nn - 1.0f), 0.0f);
    const float sig = sqrtf(fmaxf(gain * fmaxf(mean, 0.5f), var));
    return (p - mean) > sp * sig;
}

// The pixels of rows y .. y + 3 in the thread's columns (-1 outside the frame), read ahead of their sums.
struct Pixels {
    float p[kStep][kPx];
    __device__ __forceinline__ Pixels(const float* img, int ny, int nx, int y, int x) {
#pragma unroll
        for (int r = 0; r < kStep; ++r)
#pragma unroll
            for (int q = 0; q < kPx; ++q) {
                const bool in = y + r >= 0 && y + r < ny && x + q >= 0 && x + q < nx;
                p[r][q] = in ? __ldg(img + (int64_t)(y + r) * nx + x + q) : -1.0f;
            }
    }
};

// The dispersion test (xpg/spotfind.py:41-54): strong pixel and local mean. BG: instead of the mean, the background
// pixels of the extended pass (xpg/spotfind.py:78-79): valid, not within 1 px of a strong one, at most mean +
// background_pixel x sigma; and in place of the strong pixels those within 2 px of one, all the second pass asks of
// them (looked up there, 25 flags a candidate, they were most of a small frame's time). A CTA then computes two rows
// and columns more on each side than it writes, and writes a step's rows later, when the rows below them are known.
template <int H, bool BG>
__global__ void __launch_bounds__(kNT) k_spot_first(const float* __restrict__ img, int ny, int nx, int hx, int hy,
                                                    int rows, float gain, float n_s, float min_local, float bgp,
                                                    uint8_t* __restrict__ strong, uint8_t* __restrict__ bg,
                                                    float* __restrict__ mean) {
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int kEdge = BG ? 2 : 0;
    const size_t f0 = (size_t)blockIdx.z * ny * nx;
    const int x0 = blockIdx.x * (kCols - 2 * kEdge) - kEdge, y0 = blockIdx.y * rows, y1 = min(y0 + rows, ny);
    Strip<H, false> S(img + f0, nullptr, ny, nx, x0, hx, hy, sm);
    // bit rows of the strong pixels and of the background candidates, row y at y & 15: the even columns, the odd ones.
    // A step reads rows y - 8 .. y - 1 and writes y .. y + 3: no barrier between the two.
    uint32_t* sw = reinterpret_cast<uint32_t*>(sm + S.L.flag);
    uint32_t* cw = sw + kRing * 2;
    const int lane = threadIdx.x;
    const int x = x0 + kPx * (int)threadIdx.x;
    S.start(y0 - kEdge);
    // (BG: a step more, in which the last rows are written)
    for (int y = y0 - kEdge; y < y1 + kEdge + (BG ? kStep : 0); y += kStep) {
        S.stage(kStep);                                    // (its barriers also close the last step's bit rows)
        if (BG && y > y0 + 1) {
            // rows y - 6 .. y - 3: lanes 0..7 make the words of four rows, even and odd columns
            uint32_t nr = 0u, b = 0u;
            if (lane < 2 * kStep) {
                const int yy = y - 6 + lane / 2, odd = lane & 1;
                uint32_t near1 = 0u;
#pragma unroll
                for (int d = -2; d <= 2; ++d) {
                    const uint32_t* w = sw + ((yy + d) & (kRing - 1)) * 2;
                    const uint32_t e = w[0], o = w[1];
                    const uint32_t m1 = e | o | (odd ? e >> 1 : o << 1);             // columns within 1
                    nr |= m1 | (odd ? (o << 1) | (o >> 1) : (e << 1) | (e >> 1));    // and within 2
                    if (d >= -1 && d <= 1) near1 |= m1;
                }
                b = cw[(yy & (kRing - 1)) * 2 + odd] & ~near1;
            }
#pragma unroll
            for (int r = 0; r < kStep; ++r) {
                const int yy = y - 6 + r;
                const int64_t o = (int64_t)f0 + (int64_t)yy * nx + x;
#pragma unroll
                for (int q = 0; q < kPx; ++q) {
                    const uint32_t s_ = __shfl_sync(0xffffffffu, nr, 2 * r + q);
                    const uint32_t b_ = __shfl_sync(0xffffffffu, b, 2 * r + q);
                    const int c = kPx * threadIdx.x + q;
                    if (yy >= y0 && yy < y1 && c >= kEdge && c < kCols - kEdge && x + q < nx) {
                        strong[o + q] = (s_ >> lane) & 1u;
                        bg[o + q] = (b_ >> lane) & 1u;
                    }
                }
            }
        }
        if (BG && y >= y1 + kEdge) break;
        const Pixels px(img + f0, ny, nx, y, x);
        pair_t s[kStep][kPx];
        uint32_t n[kStep];
        S.step(y, s, n);
#pragma unroll
        for (int r = 0; r < kStep; ++r) {
            const int yy = y + r;
#pragma unroll
            for (int q = 0; q < kPx; ++q) {
                const float p = px.p[r][q];
                float s1, s2;
                unpack2(s[r][q], s1, s2);
                const float nf = (float)((n[r] >> (16 * q)) & 0xffffu);
                const bool valid = p >= 0.0f;
                const float nn = fmaxf(nf, 2.0f);
                // the mean, or (not written out) within 1e-6 of it, for the bounds
                const float m = BG ? __fdividef(s1, nn) : s1 / nn;
                bool on = false;
                if (valid && nf >= min_local && may_exceed(p - m * (BG ? 0.99999f : 1.0f), n_s, gain * fmaxf(m, 1.0f)))
                    on = dispersed(p, nf, s1, s2, gain, n_s);
                if (!BG) {
                    if (yy < y1 && x + q < nx) {
                        const int64_t o = (int64_t)f0 + (int64_t)yy * nx + x + q;
                        strong[o] = on ? 1 : 0;
                        mean[o] = m;
                    }
                    continue;
                }
                const float v = gain * fmaxf(m, 0.5f), reach = fabsf(bgp) * (v * rsqrtf(v));
                const float over = p - (m + copysignf(reach, bgp));
                bool cand = valid && over < 0.0f;
                if (valid && !(fabsf(over) > 1e-4f * (m + reach))) cand = at_most(p, nf, s1, gain, bgp);
                const unsigned ws = __ballot_sync(0xffffffffu, on), wc = __ballot_sync(0xffffffffu, cand);
                if (lane == 0) {
                    sw[(yy & (kRing - 1)) * 2 + q] = ws;
                    cw[(yy & (kRing - 1)) * 2 + q] = wc;
                }
            }
        }
    }
}

// The extended pass (xpg/spotfind.py:80-91): the background re-estimated over the wider window of background pixels;
// a pixel within 2 px of first-pass signal is strong when it exceeds it by signal_pixel sigma.
template <int H>
__global__ void __launch_bounds__(kNT) k_spot_extended(const float* __restrict__ img, int ny, int nx, int hx, int hy,
                                                       int rows, float gain, float sp, float min_local4,
                                                       const uint8_t* __restrict__ bg, const uint8_t* __restrict__ near,
                                                       uint8_t* __restrict__ strong, float* __restrict__ mean) {
    extern __shared__ __align__(16) unsigned char sm[];
    const size_t f0 = (size_t)blockIdx.z * ny * nx;
    const int x0 = blockIdx.x * kCols, y0 = blockIdx.y * rows, y1 = min(y0 + rows, ny);
    Strip<H, true> S(img + f0, bg + f0, ny, nx, x0, hx, hy, sm);
    const int x = x0 + kPx * (int)threadIdx.x;
    S.start(y0);
    for (int y = y0; y < y1; y += kStep) {
        S.stage(kStep);
        const Pixels px(img + f0, ny, nx, y, x);
        pair_t s[kStep][kPx];
        uint32_t n[kStep];
        S.step(y, s, n);
#pragma unroll
        for (int r = 0; r < kStep; ++r) {
            const int yy = y + r;
            const int64_t o = (int64_t)f0 + (int64_t)yy * nx + x;
#pragma unroll
            for (int q = 0; q < kPx; ++q) {
                if (yy >= y1 || x + q >= nx) continue;
                const float p = px.p[r][q];
                float sum, sq;
                unpack2(s[r][q], sum, sq);
                const float nf = (float)((n[r] >> (16 * q)) & 0xffffu);
                const float nn = fmaxf(nf, 2.0f);
                const float m = sum / nn;
                bool st = false;
                if (p >= 0.0f && nf >= min_local4 && may_exceed(p - m, sp, gain * fmaxf(m, 0.5f)))
                    st = exceeds(p, nf, sum, sq, gain, sp) && near[o + q];
                strong[o + q] = st ? 1 : 0;
                mean[o + q] = m;
            }
        }
    }
}

// ---- tiles: a thread a pixel, a CTA a 32 x 8 tile of one frame. The tile and its halo are staged in shared memory, summed
// along x for every staged row, then along y for every pixel, in the same order as the strips' sums.

constexpr int kTW = 32, kTH = 8, kTile = kTW * kTH;

// window sums of the valid-pixel count, the values and their squares
struct Sums {
    float n, s1, s2;
};

// The sums of this thread's pixel over the pixels that enter: the valid ones, or those whose flag in sel is set.
__device__ Sums tile_sums(const float* __restrict__ img, const uint8_t* __restrict__ sel, int ny, int nx, int hx, int hy,
                          float* sm) {
    const int W = kTW + 2 * hx, H = kTH + 2 * hy;
    float* tw = sm;                   // staged weights, H x W
    float* tx = tw + H * W;           // staged values
    float* hw = tx + H * W;           // sums along x, H x kTW
    float* hs = hw + H * kTW;
    float* hq = hs + H * kTW;
    const int x0 = blockIdx.x * kTW - hx, y0 = blockIdx.y * kTH - hy;
    for (int i = threadIdx.x; i < H * W; i += kTile) {
        const int r = i / W, c = i % W;
        const int y = y0 + r, x = x0 + c;
        float w = 0.0f, v = 0.0f;
        if (y >= 0 && y < ny && x >= 0 && x < nx) {
            const size_t k = (size_t)y * nx + x;
            const float p = img[k];
            const bool on = sel ? sel[k] != 0 : p >= 0.0f;
            w = on ? 1.0f : 0.0f;
            v = on ? p : 0.0f;
        }
        tw[i] = w;
        tx[i] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < H * kTW; i += kTile) {
        const int r = i / kTW, c = i % kTW;
        float a = 0.0f, s = 0.0f, q = 0.0f;
        for (int d = 0; d <= 2 * hx; ++d) {
            const float v = tx[r * W + c + d];
            a = a + tw[r * W + c + d];
            s = s + v;
            q = q + v * v;
        }
        hw[i] = a;
        hs[i] = s;
        hq[i] = q;
    }
    __syncthreads();
    const int r = threadIdx.x / kTW, c = threadIdx.x % kTW;
    Sums o{0.0f, 0.0f, 0.0f};
    for (int d = 0; d <= 2 * hy; ++d) {
        const int k = (r + d) * kTW + c;
        o.n = o.n + hw[k];
        o.s1 = o.s1 + hs[k];
        o.s2 = o.s2 + hq[k];
    }
    return o;
}

size_t tile_smem(int hx, int hy) {                         // (38.3 KB at most)
    const size_t W = kTW + 2 * hx, H = kTH + 2 * hy;
    return (2 * H * W + 3 * H * kTW) * sizeof(float);
}

__device__ bool any_flag(const uint8_t* f, int ny, int nx, int y, int x, int r) {
    for (int yy = max(y - r, 0); yy <= min(y + r, ny - 1); ++yy)
        for (int xx = max(x - r, 0); xx <= min(x + r, nx - 1); ++xx)
            if (f[(size_t)yy * nx + xx]) return true;
    return false;
}

// the dispersion test: first-pass strong mask and local mean
__global__ void __launch_bounds__(kTile) k_spot_tile_first(const float* __restrict__ img, int ny, int nx, int hx, int hy,
                                                           float gain, float n_s, float min_local,
                                                           uint8_t* __restrict__ strong, float* __restrict__ mean) {
    extern __shared__ __align__(16) unsigned char sm[];
    const size_t f0 = (size_t)blockIdx.z * ny * nx;
    const Sums t = tile_sums(img + f0, nullptr, ny, nx, hx, hy, reinterpret_cast<float*>(sm));
    const int y = blockIdx.y * kTH + threadIdx.x / kTW, x = blockIdx.x * kTW + threadIdx.x % kTW;
    if (y >= ny || x >= nx) return;
    const size_t k = f0 + (size_t)y * nx + x;
    const float p = img[k];
    strong[k] = p >= 0.0f && t.n >= min_local && dispersed(p, t.n, t.s1, t.s2, gain, n_s) ? 1 : 0;
    mean[k] = t.s1 / fmaxf(t.n, 2.0f);
}

// the background pixels of the extended pass
__global__ void __launch_bounds__(kTile) k_spot_tile_background(const float* __restrict__ img, int ny, int nx,
                                                                const uint8_t* __restrict__ strong,
                                                                const float* __restrict__ mean, float gain, float bgp,
                                                                uint8_t* __restrict__ bg) {
    const int y = blockIdx.y * kTH + threadIdx.x / kTW, x = blockIdx.x * kTW + threadIdx.x % kTW;
    if (y >= ny || x >= nx) return;
    const size_t f0 = (size_t)blockIdx.z * ny * nx, k = f0 + (size_t)y * nx + x;
    const float p = img[k], m = mean[k];
    const float sigma = sqrtf(gain * fmaxf(m, 0.5f));
    bg[k] = p >= 0.0f && !any_flag(strong + f0, ny, nx, y, x, 1) && p <= m + bgp * sigma ? 1 : 0;
}

// the extended pass
__global__ void __launch_bounds__(kTile) k_spot_tile_extended(const float* __restrict__ img, int ny, int nx, int hx,
                                                              int hy, float gain, float sp, float min_local4,
                                                              const uint8_t* __restrict__ bg,
                                                              const uint8_t* __restrict__ first,
                                                              uint8_t* __restrict__ strong, float* __restrict__ mean) {
    extern __shared__ __align__(16) unsigned char sm[];
    const size_t f0 = (size_t)blockIdx.z * ny * nx;
    const Sums t = tile_sums(img + f0, bg + f0, ny, nx, hx, hy, reinterpret_cast<float*>(sm));
    const int y = blockIdx.y * kTH + threadIdx.x / kTW, x = blockIdx.x * kTW + threadIdx.x % kTW;
    if (y >= ny || x >= nx) return;
    const size_t k = f0 + (size_t)y * nx + x;
    const float p = img[k];
    const bool st = p >= 0.0f && t.n >= min_local4 && exceeds(p, t.n, t.s1, t.s2, gain, sp);
    strong[k] = st && any_flag(first + f0, ny, nx, y, x, 2) ? 1 : 0;
    mean[k] = t.s1 / fmaxf(t.n, 2.0f);
}

// ---- the choice

constexpr int kSms = 148;                    // of a B200

// CTAs of strips of `rows` rows
int64_t strip_ctas(bool extended, int n_frames, int ny, int nx, int rows) {
    const int cols = extended ? kCols - 4 : kCols;
    return (int64_t)((nx + cols - 1) / cols) * ((ny + rows - 1) / rows) * n_frames;
}

// Strips where they are enough to hide a march's latency, else tiles. Strips of few rows recompute the rows of their
// windows above them: square windows with unrolled loops (half widths 2 to 4) still gain in four rows, the others
// want strips of twelve, the widest extended ones more of them. One frame, strips against tiles:
//   half width 3: 260 x 256 7.7 / 8.0 us plain, 23 / 19 extended; 512 x 512 9 / 11, 26 / 29; 768 x 768 11 / 16, 35 / 50
//   half width 5: 512 x 512 12.8 / 12.2 plain, 43 / 35 extended; 768 x 768 16 / 20, 81 / 64; 1000 x 1000 26 / 31, 73 / 97
//   half width 8: 260 x 256 17 / 9, 60 / 24; 896 x 900 34 / 33, 163 / 117; 1030 x 1065 32 / 42, 139 / 146
constexpr int kWideCtas = kSms * 12;
bool use_strips(const XiSpotParams& p, int n_frames, int ny, int nx) {
    const bool ext = p.extended != 0;
    const int wide = p.nbx > p.nby ? p.nbx : p.nby;
    if (p.nbx == p.nby && wide >= 2 && wide <= 4) return strip_ctas(ext, n_frames, ny, nx, 4) >= kSms * (ext ? 6 : 3);
    if (!ext && wide < 7) return strip_ctas(ext, n_frames, ny, nx, 4) >= kSms * 10;
    return strip_ctas(ext, n_frames, ny, nx, 12) >= (ext && wide >= 7 ? kWideCtas : kSms * 8);
}

// Rows a CTA marches down: long strips recompute little (the 2 hy rows above the first one), short ones fill the
// device: the longest of 60, 28 and 12 that gives every SM eight CTAs, else 4. (All of them 4 k: an extended first pass
// computes two rows more above and below, which are whole steps too.)
int strip_rows(int n_frames, int ny, int strips) {
    for (int rows : {60, 28, 12})
        if ((int64_t)strips * ((ny + rows - 1) / rows) * n_frames >= kSms * 8) return rows;
    return 4;
}

template <typename K, typename... A>
void launch(K kernel, int cols, int hx, int hy, int n_frames, int ny, int nx, cudaStream_t s, const float* img, A... a) {
    const size_t sm = Layout(hx, hy).bytes;
    const int strips = (nx + cols - 1) / cols, rows = strip_rows(n_frames, ny, strips);
    kernel<<<dim3((unsigned)strips, (unsigned)((ny + rows - 1) / rows), (unsigned)n_frames), kNT, sm, s>>>(
        img, ny, nx, hx, hy, rows, a...);
}

// Window loops unrolled for square windows of half width 2 to 4 (the finder's own default is 3) and the second
// pass's 5, 7 and 9 that follow from them; any other window takes the same kernel with loops of run-time length.
template <bool BG, typename... A>
void launch_first(int hx, int hy, int cols, int n_frames, int ny, int nx, cudaStream_t s, const float* img, A... a) {
    const int h = hx == hy ? hx : -1;
    if (h == 2) launch(k_spot_first<2, BG>, cols, hx, hy, n_frames, ny, nx, s, img, a...);
    else if (h == 3) launch(k_spot_first<3, BG>, cols, hx, hy, n_frames, ny, nx, s, img, a...);
    else if (h == 4) launch(k_spot_first<4, BG>, cols, hx, hy, n_frames, ny, nx, s, img, a...);
    else launch(k_spot_first<-1, BG>, cols, hx, hy, n_frames, ny, nx, s, img, a...);
}

template <typename... A>
void launch_extended(int hx, int hy, int n_frames, int ny, int nx, cudaStream_t s, const float* img, A... a) {
    const int h = hx == hy ? hx : -1;
    if (h == 5) launch(k_spot_extended<5>, kCols, hx, hy, n_frames, ny, nx, s, img, a...);
    else if (h == 7) launch(k_spot_extended<7>, kCols, hx, hy, n_frames, ny, nx, s, img, a...);
    else if (h == 9) launch(k_spot_extended<9>, kCols, hx, hy, n_frames, ny, nx, s, img, a...);
    else launch(k_spot_extended<-1>, kCols, hx, hy, n_frames, ny, nx, s, img, a...);
}

}  // namespace

extern "C" size_t xi_spot_workspace(int n_frames, int ny, int nx) {
    if (n_frames < 0 || ny < 0 || nx < 0) return 0;
    const size_t n = (size_t)n_frames * ny * nx;
    const size_t flags = (n + 255) / 256 * 256;
    // the first pass's flags (strong, or near a strong pixel; background), and its mean for as many pixels as tiles are
    // taken for (so that the scratch of a batch serves a shorter one)
    const size_t most = (size_t)kWideCtas * (kCols - 4) * 12;
    return 2 * flags + (n < most ? n : most) * sizeof(float);
}

extern "C" int xi_spot_strong(const float* img, int n_frames, int ny, int nx, float gain, const XiSpotParams* p,
                              uint8_t* strong, float* mean, void* ws, size_t ws_bytes, void* stream) {
    if (!p || n_frames < 0 || ny < 0 || nx < 0) return xi_fail(XI_E_ARG, "xi_spot_strong: null argument or size");
    const size_t n = (size_t)n_frames * ny * nx;
    if (n == 0) return XI_OK;
    if (!img || !strong || !mean) return xi_fail(XI_E_ARG, "xi_spot_strong: null pointer");
    if (p->nbx < 0 || p->nby < 0 || p->nbx > XI_SPOT_MAX_HALF || p->nby > XI_SPOT_MAX_HALF)
        return xi_fail(XI_E_LIMIT, "xi_spot_strong: window half-size beyond XI_SPOT_MAX_HALF");
    if (n_frames > 65535) return xi_fail(XI_E_LIMIT, "xi_spot_strong: more than 65535 frames in one call");
    cudaStream_t s = (cudaStream_t)stream;
    const float ml = (float)p->min_local;
    const bool strips = use_strips(*p, n_frames, ny, nx);
    const dim3 grid((unsigned)((nx + kTW - 1) / kTW), (unsigned)((ny + kTH - 1) / kTH), (unsigned)n_frames);
    if (!p->extended && !strips) {
        k_spot_tile_first<<<grid, kTile, tile_smem(p->nbx, p->nby), s>>>(img, ny, nx, p->nbx, p->nby, gain,
                                                                         p->signal_pixel, ml, strong, mean);
        return xi_cuda_check("xi_spot_strong");
    }
    if (!p->extended) {
        launch_first<false>(p->nbx, p->nby, kCols, n_frames, ny, nx, s, img, gain, p->signal_pixel, ml, 0.0f, strong,
                            (uint8_t*)nullptr, mean);
        return xi_cuda_check("xi_spot_strong");
    }
    if (!ws || ws_bytes < xi_spot_workspace(n_frames, ny, nx)) return xi_fail(XI_E_ARG, "xi_spot_strong: workspace");
    uint8_t* near = static_cast<uint8_t*>(ws);
    uint8_t* bg = near + (n + 255) / 256 * 256;
    if (!strips) {
        uint8_t* first = near;
        float* mean1 = reinterpret_cast<float*>(bg + (n + 255) / 256 * 256);
        const int hx2 = 2 * p->nbx + 1, hy2 = 2 * p->nby + 1;
        k_spot_tile_first<<<grid, kTile, tile_smem(p->nbx, p->nby), s>>>(img, ny, nx, p->nbx, p->nby, gain,
                                                                         p->signal_pixel, ml, first, mean1);
        k_spot_tile_background<<<grid, kTile, 0, s>>>(img, ny, nx, first, mean1, gain, p->background_pixel, bg);
        k_spot_tile_extended<<<grid, kTile, tile_smem(hx2, hy2), s>>>(img, ny, nx, hx2, hy2, gain, p->signal_pixel,
                                                                      4.0f * ml, bg, first, strong, mean);
        return xi_cuda_check("xi_spot_strong");
    }
    launch_first<true>(p->nbx, p->nby, kCols - 4, n_frames, ny, nx, s, img, gain, p->signal_pixel, ml,
                       p->background_pixel, near, bg, (float*)nullptr);
    launch_extended(2 * p->nbx + 1, 2 * p->nby + 1, n_frames, ny, nx, s, img, gain, p->signal_pixel, 4.0f * ml, bg, near,
                    strong, mean);
    return xi_cuda_check("xi_spot_strong");
}
