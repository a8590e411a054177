// UpsampleBicubic2d forward and backward (cubic convolution with A = -0.75, no antialiasing), NCHW and NHWC.
//
// Forward: a thread owns one or two adjacent elements of an output row and walks down a band of rows, keeping the
// four horizontal sums of the current source rows in registers; the sixteen clamped taps are combined in the
// reference's order (four row sums left to right, then the column sum), every operation rounded on its own, so
// fp32 results carry the bits of a serial CPU statement of
// image/resize_bicubic_v2/op_kernel/arch35/resize_bicubic_v2_simt_base.h:23-120. The four special schedules of
// resize_bicubic_v2_simt_nchw.h:50-90 (copy, one input pixel, one output pixel, integer positions) are selected on
// the host with the reference's rule and are plain copies here too.
//
// Backward: one thread per grad_input element gathers the grads that reach it, walking them in ascending
// (row, column) order. The walk, its start, its end and the coefficient expressions are those of the reference's
// gather kernel (image/resize_bicubic_v2_grad/op_kernel/arch35/resize_bicubic_v2_grad_simt_determine.h:95-350):
// an axis on which the element is interior is walked by distance to the source position, a first or last index
// tap by tap with clamped destinations. The sum has a fixed order, so results are reproducible from run to run
// and fp32 results carry the bits of that kernel run serially. The column side of the walk is the same for every
// row, so each thread evaluates it once into a shared-memory list.
//
// Calls at exactly 2x on NCHW tensors (scales 0.5 with half-pixel coordinates: every source coordinate is exact and
// the coefficients are a handful of constants, evaluated on the host) have kernels of their own in both directions:
// Bicubic2dFwdX2Kernel and Bicubic2dBwdX2Kernel stage a band of rows in shared memory as fp32 once and work from
// register windows; their terms, order and rounding are those of the general kernels.
#include <algorithm>
#include <vector>

#include "launch_util.cuh"

namespace opscv {
namespace {

constexpr int kThreads = 256;
constexpr float kA = -0.75f;

// ((a + 2) x - (a + 3)) x x + 1
__device__ __forceinline__ float Conv1(float x)
{
    return Add(Mul(Mul(Sub(Mul(kA + 2.0f, x), kA + 3.0f), x), x), 1.0f);
}
// ((a x - 5 a) x + 8 a) x - 4 a
__device__ __forceinline__ float Conv2(float x)
{
    return Sub(Mul(Add(Mul(Sub(Mul(kA, x), 5.0f * kA), x), 8.0f * kA), x), 4.0f * kA);
}
__device__ __forceinline__ void TapCoeff(float t, float (&c)[4])
{
    c[0] = Conv2(Add(t, 1.0f));
    c[1] = Conv1(t);
    const float u = Sub(1.0f, t);
    c[2] = Conv1(u);
    c[3] = Conv2(Add(u, 1.0f)); // the forward kernel writes 2 - t; see FwdCoeff
}
// resize_bicubic_v2_simt_base.h:33-41: the last argument is 2 - t (the backward kernels use (1 - t) + 1)
__device__ __forceinline__ void FwdCoeff(float t, float (&c)[4])
{
    c[0] = Conv2(Add(t, 1.0f));
    c[1] = Conv1(t);
    c[2] = Conv1(Sub(1.0f, t));
    c[3] = Conv2(Sub(2.0f, t));
}
// resize_bicubic_v2_grad_base.h:44-56
__device__ __forceinline__ float PointCoeff(float d)
{
    if (d <= 1.0f) {
        return Conv1(d);
    }
    if (d < 2.0f) {
        return Conv2(d);
    }
    return 0.0f;
}
__device__ __forceinline__ int32_t ClampIdx(long long v, int32_t last)
{
    return static_cast<int32_t>(v < 0 ? 0 : (v > last ? last : v));
}
__device__ __forceinline__ int32_t ClampIdx32(int32_t v, int32_t last) { return min(max(v, 0), last); }

struct BicubicGeom {
    int64_t rows;  // forward: planes * hout; backward: planes * hin
    int32_t hin, win, hout, wout;
    int32_t chan;  // NHWC: channels; NCHW: 1
    float scaleH, scaleW, invH, invW;
    int32_t align; // backward: align_corners; forward: !halfPixel
    int32_t schedule;
};

// Copy schedules (one input pixel, one output pixel, integer source positions): no arithmetic.
template <typename T, bool NHWC>
__global__ void __launch_bounds__(kThreads) Bicubic2dFwdCopyKernel(const T* __restrict__ x, T* __restrict__ y, BicubicGeom g)
{
    const int32_t inner = g.wout * g.chan;
    const int64_t planeIn = static_cast<int64_t>(g.hin) * g.win * g.chan;
    const int64_t rowIn = static_cast<int64_t>(g.win) * g.chan;
    for (int64_t row = blockIdx.y; row < g.rows; row += gridDim.y) {
        const int64_t plane = row / g.hout;
        const int32_t H = static_cast<int32_t>(row - plane * g.hout);
        const float oh = g.align ? Mul(static_cast<float>(H), g.scaleH)
                                 : Sub(Mul(Add(static_cast<float>(H), 0.5f), g.scaleH), 0.5f);
        const T* px = x + plane * planeIn;
        const T* r1 = px + ClampIdx(static_cast<long long>(floorf(oh)), g.hin - 1) * rowIn;
        T* py = y + row * inner;
        for (int32_t t = blockIdx.x * kThreads + threadIdx.x; t < inner; t += gridDim.x * kThreads) {
            const int32_t W = NHWC ? t / g.chan : t;
            const int32_t c = NHWC ? t - W * g.chan : 0;
            if (g.schedule == 2 || g.schedule == 3) { // one input pixel / one output pixel: x[plane][0][0]
                py[t] = px[c];
                continue;
            }
            const float ow = g.align ? Mul(static_cast<float>(W), g.scaleW)
                                     : Sub(Mul(Add(static_cast<float>(W), 0.5f), g.scaleW), 0.5f);
            const long long left = static_cast<long long>(floorf(ow));
            py[t] = r1[static_cast<int64_t>(ClampIdx(left, g.win - 1)) * g.chan + c]; // integer positions
        }
    }
}

// General schedule. A thread owns V adjacent elements of an output row (one column for NHWC: its channel of one
// pixel) and walks down a band of output rows. The four horizontal sums that an output row needs are kept in
// registers and shifted as the source row advances: an input row's horizontal sum is computed once per band and
// column instead of once per output row that uses it, and the vertical combination stays the reference's
// left-to-right sum of four products, so the bits do not change.
template <typename T, bool NHWC, int V>
__global__ void __launch_bounds__(kThreads) Bicubic2dFwdKernel(const T* __restrict__ x, T* __restrict__ y, BicubicGeom g,
                                                                int32_t bandRows, int32_t bands)
{
    // per output row of the band: the source row above the four taps and the four vertical coefficients, evaluated
    // once per band by the block instead of once per row by every thread
    extern __shared__ float sRow[];
    float* sCh = sRow;                                                   // [bandRows][4]
    int32_t* sTop = reinterpret_cast<int32_t*>(sRow + 4 * bandRows);     // [bandRows]
    const int32_t inner = g.wout * g.chan;
    const int32_t t0 = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    const bool active = t0 < inner;
    const int64_t planeIn = static_cast<int64_t>(g.hin) * g.win * g.chan;
    const int64_t rowIn = static_cast<int64_t>(g.win) * g.chan;
    // per-column taps and weights (V columns)
    int32_t off[V][4];
    float cw[V][4];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int32_t t = active ? t0 + v : 0;
        const int32_t W = NHWC ? t / g.chan : t;
        const int32_t c = NHWC ? t - W * g.chan : 0;
        const float ow = g.align ? Mul(static_cast<float>(W), g.scaleW)
                                 : Sub(Mul(Add(static_cast<float>(W), 0.5f), g.scaleW), 0.5f);
        const float fw = floorf(ow);
        const long long left = static_cast<long long>(fw);
        FwdCoeff(Sub(ow, fw), cw[v]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            off[v][j] = ClampIdx(left - 1 + j, g.win - 1) * g.chan + c;
        }
    }
    int32_t tableBand = -1;
    for (int64_t item = blockIdx.y; item < g.rows; item += gridDim.y) { // g.rows = planes * bands here
        const int64_t plane = item / bands;
        const int32_t band = static_cast<int32_t>(item - plane * bands);
        const int32_t h0 = band * bandRows;
        const int32_t h1 = min(h0 + bandRows, g.hout);
        if (band != tableBand) { // uniform over the block
            __syncthreads();
            for (int32_t r = threadIdx.x; r < h1 - h0; r += blockDim.x) {
                const int32_t H = h0 + r;
                const float oh = g.align ? Mul(static_cast<float>(H), g.scaleH)
                                         : Sub(Mul(Add(static_cast<float>(H), 0.5f), g.scaleH), 0.5f);
                const float fh = floorf(oh);
                float ch[4];
                FwdCoeff(Sub(oh, fh), ch);
                // tops outside [-2, hin + 1] clamp every tap to the same row as the bound does
                const float lim = fminf(fmaxf(fh, -2.0f), static_cast<float>(g.hin) + 1.0f);
                sTop[r] = static_cast<int32_t>(lim);
                sCh[4 * r + 0] = ch[0];
                sCh[4 * r + 1] = ch[1];
                sCh[4 * r + 2] = ch[2];
                sCh[4 * r + 3] = ch[3];
            }
            __syncthreads();
            tableBand = band;
        }
        if (!active) {
            continue;
        }
        const T* px = x + plane * planeIn;
        T* py = y + (plane * g.hout + h0) * static_cast<int64_t>(inner) + t0;
        float rs[V][4];
        int32_t curTop = 0;
        bool have = false;
        auto rowSums = [&](int32_t srcRow, int slot) {
            const T* r = px + ClampIdx32(srcRow, g.hin - 1) * rowIn;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float v0 = DType<T>::Load(r + off[v][0]), v1 = DType<T>::Load(r + off[v][1]),
                            v2 = DType<T>::Load(r + off[v][2]), v3 = DType<T>::Load(r + off[v][3]);
                rs[v][slot] = Add(Add(Add(Mul(v0, cw[v][0]), Mul(v1, cw[v][1])), Mul(v2, cw[v][2])), Mul(v3, cw[v][3]));
            }
        };
        for (int32_t r = 0; r < h1 - h0; ++r, py += inner) {
            const int32_t top = sTop[r];
            const float4 ch = *reinterpret_cast<const float4*>(sCh + 4 * r);
            const int32_t shift = top - curTop;
            if (!have || shift < 0 || shift >= 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    rowSums(top - 1 + k, k);
                }
                have = true;
            } else {
                for (int32_t sft = 0; sft < shift; ++sft) {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        rs[v][0] = rs[v][1];
                        rs[v][1] = rs[v][2];
                        rs[v][2] = rs[v][3];
                    }
                    rowSums(curTop + sft + 3, 3);
                }
            }
            curTop = top;
            float out[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                out[v] = Add(Add(Add(Mul(rs[v][0], ch.x), Mul(rs[v][1], ch.y)), Mul(rs[v][2], ch.z)), Mul(rs[v][3], ch.w));
            }
            StorePack<T, V>(py, out);
        }
    }
}

// General schedule, NCHW, tiled through shared memory. A block takes a (plane, band of output rows) item: it loads
// the source rows the band touches once (converted to fp32), forms every horizontal sum of those rows once,
// a[source row][output column], and then combines four rows of `a` per output row with 16-byte shared-memory loads.
// The sums are the expressions of the kernel above in the same order, so the bits are the same; what changes is
// that a tap is loaded and converted once per block instead of once per output column that uses it, and that the
// column coefficients live in registers for all the rows of the tile.
constexpr int kFwdWalk = 16; // output rows that a thread walks in the narrow vertical pass
struct BicubicTile {
    int32_t bandRows; // output rows per item
    int32_t bands;
    int32_t maxSrc;   // most source rows any band touches
    int32_t tw;       // threads along a row in the horizontal pass (power of two)
    int32_t pw;       // threads along a row in the vertical pass (power of two)
};

__host__ __device__ __forceinline__ int32_t FwdTop(int32_t H, float scaleH, int32_t align, int32_t hin, float (*ch)[4])
{
#ifdef __CUDA_ARCH__
    const float oh = align ? Mul(static_cast<float>(H), scaleH) : Sub(Mul(Add(static_cast<float>(H), 0.5f), scaleH), 0.5f);
    const float fh = floorf(oh);
    if (ch != nullptr) {
        FwdCoeff(Sub(oh, fh), *ch);
    }
#else
    (void)ch;
    float oh;
    if (align) {
        oh = static_cast<float>(H) * scaleH;
    } else {
        const float t = (static_cast<float>(H) + 0.5f) * scaleH;
        oh = t - 0.5f;
    }
    const float fh = floorf(oh);
#endif
    // tops outside [-2, hin + 1] clamp every tap to the same row as the bound does
    return static_cast<int32_t>(fminf(fmaxf(fh, -2.0f), static_cast<float>(hin) + 1.0f));
}

template <typename T, int V>
__global__ void __launch_bounds__(kThreads) Bicubic2dFwdTileKernel(const T* __restrict__ x, T* __restrict__ y, BicubicGeom g,
                                                                   BicubicTile tile, int64_t items)
{
    extern __shared__ __align__(16) float sTile[];
    float* sCh = sTile;                                           // [bandRows][4], read as float4
    float* sA = sCh + 4 * tile.bandRows;                          // [maxSrc][wout], 16-byte aligned rows when V >= 4
    float* sX = sA + static_cast<size_t>(tile.maxSrc) * g.wout;   // [maxSrc][win]
    int32_t* sTop = reinterpret_cast<int32_t*>(sX + static_cast<size_t>(tile.maxSrc) * g.win); // [bandRows]
    const int32_t tid = threadIdx.x;
    const int32_t tx = tid & (tile.tw - 1), ty = tid / tile.tw, tyN = kThreads / tile.tw;
    const int32_t px_ = tid & (tile.pw - 1), py_ = tid / tile.pw, pyN = kThreads / tile.pw;
    const int32_t packs = g.wout / V;
    const bool pairAligned = (g.wout & 1) == 0; // rows of sums start on 8-byte boundaries
    const int64_t planeIn = static_cast<int64_t>(g.hin) * g.win;
    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const int64_t plane = item / tile.bands;
        const int32_t band = static_cast<int32_t>(item - plane * tile.bands);
        const int32_t h0 = band * tile.bandRows;
        const int32_t nOut = min(tile.bandRows, g.hout - h0);
        __syncthreads(); // the previous item's tiles are no longer read
        for (int32_t r = tid; r < nOut; r += kThreads) {
            float ch[4];
            sTop[r] = FwdTop(h0 + r, g.scaleH, g.align, g.hin, &ch);
            *reinterpret_cast<float4*>(sCh + 4 * r) = make_float4(ch[0], ch[1], ch[2], ch[3]);
        }
        __syncthreads();
        const int32_t srcLo = ClampIdx32(sTop[0] - 1, g.hin - 1);
        const int32_t srcHi = ClampIdx32(sTop[nOut - 1] + 2, g.hin - 1);
        const int32_t nSrc = min(srcHi - srcLo + 1, tile.maxSrc);
        const T* px = x + plane * planeIn + static_cast<int64_t>(srcLo) * g.win;
        for (int32_t i = tid; i < nSrc * g.win; i += kThreads) {
            sX[i] = DType<T>::Load(px + i);
        }
        __syncthreads();
        // horizontal sums: a thread keeps the taps and coefficients of two adjacent columns for all the rows of the
        // tile. When the second column's window is the first one's moved on by zero or one source pixel (any
        // up-scale) the two sums share their tap reads: five shared-memory loads instead of eight.
        for (int32_t w = 2 * tx; w < g.wout; w += 2 * tile.tw) {
            float cw0[4], cw1[4];
            long long left0, left1;
            {
                const float ow = g.align ? Mul(static_cast<float>(w), g.scaleW)
                                         : Sub(Mul(Add(static_cast<float>(w), 0.5f), g.scaleW), 0.5f);
                const float fw = floorf(ow);
                left0 = static_cast<long long>(fw);
                FwdCoeff(Sub(ow, fw), cw0);
            }
            const bool two = w + 1 < g.wout;
            {
                const float ow = g.align ? Mul(static_cast<float>(w + 1), g.scaleW)
                                         : Sub(Mul(Add(static_cast<float>(w + 1), 0.5f), g.scaleW), 0.5f);
                const float fw = floorf(ow);
                left1 = static_cast<long long>(fw);
                FwdCoeff(Sub(ow, fw), cw1);
            }
            const int32_t o0 = ClampIdx(left0 - 1, g.win - 1), o1 = ClampIdx(left0, g.win - 1),
                          o2 = ClampIdx(left0 + 1, g.win - 1), o3 = ClampIdx(left0 + 2, g.win - 1),
                          o4 = ClampIdx(left0 + 3, g.win - 1);
            const long long step = left1 - left0;
            if (two && (step == 0 || step == 1)) {
                for (int32_t r = ty; r < nSrc; r += tyN) {
                    const float* row = sX + r * g.win;
                    const float v0 = row[o0], v1 = row[o1], v2 = row[o2], v3 = row[o3];
                    const float v4 = step == 1 ? row[o4] : 0.0f;
                    const float u0 = step == 1 ? v1 : v0, u1 = step == 1 ? v2 : v1, u2 = step == 1 ? v3 : v2,
                                u3 = step == 1 ? v4 : v3;
                    float2 a;
                    a.x = Add(Add(Add(Mul(v0, cw0[0]), Mul(v1, cw0[1])), Mul(v2, cw0[2])), Mul(v3, cw0[3]));
                    a.y = Add(Add(Add(Mul(u0, cw1[0]), Mul(u1, cw1[1])), Mul(u2, cw1[2])), Mul(u3, cw1[3]));
                    if (pairAligned) {
                        *reinterpret_cast<float2*>(sA + r * g.wout + w) = a;
                    } else {
                        sA[r * g.wout + w] = a.x;
                        sA[r * g.wout + w + 1] = a.y;
                    }
                }
            } else {
                const int32_t q0 = ClampIdx(left1 - 1, g.win - 1), q1 = ClampIdx(left1, g.win - 1),
                              q2 = ClampIdx(left1 + 1, g.win - 1), q3 = ClampIdx(left1 + 2, g.win - 1);
                for (int32_t r = ty; r < nSrc; r += tyN) {
                    const float* row = sX + r * g.win;
                    sA[r * g.wout + w] = Add(Add(Add(Mul(row[o0], cw0[0]), Mul(row[o1], cw0[1])), Mul(row[o2], cw0[2])), Mul(row[o3], cw0[3]));
                    if (two) {
                        sA[r * g.wout + w + 1] = Add(Add(Add(Mul(row[q0], cw1[0]), Mul(row[q1], cw1[1])), Mul(row[q2], cw1[2])), Mul(row[q3], cw1[3]));
                    }
                }
            }
        }
        __syncthreads();
        T* py = y + (plane * g.hout + h0) * static_cast<int64_t>(g.wout);
        const int32_t segs = (nOut + kFwdWalk - 1) / kFwdWalk;
        if (V <= 2 && g.scaleH < 1.0f && packs * segs >= kThreads) {
            // Rows that allow no wider store than two elements: a thread walks kFwdWalk output rows down its columns with
            // the four sums in registers. An up-scale moves the window on by at most one source row per output row, so
            // most rows load one sum or none; with four loads and four row offsets per output the pass was bound by
            // instruction issue (fp32 8x64 planes 60x80 -> 150x199: 80 instructions per output, 81 % of the issue slots; 46 -> 37 us).
            // Columns and segments of rows share one index, so that no thread is idle at any width. A down-scale loads four
            // sums per row all the same, and a tile with fewer walks than threads leaves some idle: both take a thread per
            // output (bf16 4x50 planes 45x44 -> 26x27: 8.3 us by walks, 6.4).
            for (int32_t i = tid; i < packs * segs; i += kThreads) {
                const int32_t seg = i / packs, p = i - seg * packs;
                const int32_t r1 = min(nOut, (seg + 1) * kFwdWalk);
                const float* col = sA + p * V;
                T* dst = py + static_cast<int64_t>(seg * kFwdWalk) * g.wout + p * V;
                int32_t cur = INT32_MIN / 2;
                float a[4][V];
                auto load = [&](int32_t row, float (&v)[V]) {
                    const float* src = col + (ClampIdx32(row, g.hin - 1) - srcLo) * g.wout;
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        v[e] = src[e];
                    }
                };
                for (int32_t r = seg * kFwdWalk; r < r1; ++r, dst += g.wout) {
                    const int32_t top = sTop[r];
                    const float4 ch = *reinterpret_cast<const float4*>(sCh + 4 * r);
                    if (top == cur + 1) {
#pragma unroll
                        for (int e = 0; e < V; ++e) {
                            a[0][e] = a[1][e];
                            a[1][e] = a[2][e];
                            a[2][e] = a[3][e];
                        }
                        load(top + 2, a[3]);
                    } else if (top != cur) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            load(top - 1 + k, a[k]);
                        }
                    }
                    cur = top;
                    float out[V];
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        out[e] = Add(Add(Add(Mul(a[0][e], ch.x), Mul(a[1][e], ch.y)), Mul(a[2][e], ch.z)), Mul(a[3][e], ch.w));
                    }
                    StorePack<T, V>(dst, out);
                }
            }
            continue;
        }
        // vertical combination, V adjacent outputs per thread
        constexpr int C = V / 4 > 0 ? V / 4 : 1;
        constexpr int L = V < 4 ? V : 4;
        for (int32_t p = px_; p < packs; p += tile.pw) {
            for (int32_t r = py_; r < nOut; r += pyN) {
                const int32_t top = sTop[r];
                const float4 ch = *reinterpret_cast<const float4*>(sCh + 4 * r);
                const float* a0 = sA + (ClampIdx32(top - 1, g.hin - 1) - srcLo) * g.wout + p * V;
                const float* a1 = sA + (ClampIdx32(top, g.hin - 1) - srcLo) * g.wout + p * V;
                const float* a2 = sA + (ClampIdx32(top + 1, g.hin - 1) - srcLo) * g.wout + p * V;
                const float* a3 = sA + (ClampIdx32(top + 2, g.hin - 1) - srcLo) * g.wout + p * V;
                float out[V];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    float r0[L], r1[L], r2[L], r3[L];
                    LoadPack<float, L>(a0 + c * L, r0);
                    LoadPack<float, L>(a1 + c * L, r1);
                    LoadPack<float, L>(a2 + c * L, r2);
                    LoadPack<float, L>(a3 + c * L, r3);
#pragma unroll
                    for (int v = 0; v < L; ++v) {
                        out[c * L + v] = Add(Add(Add(Mul(r0[v], ch.x), Mul(r1[v], ch.y)), Mul(r2[v], ch.z)), Mul(r3[v], ch.w));
                    }
                }
                StorePack<T, V>(py + static_cast<int64_t>(r) * g.wout + p * V, out);
            }
        }
    }
}

__device__ __forceinline__ float BwdSrc(float scale, int32_t idx, int32_t align)
{
    return align ? Mul(scale, static_cast<float>(idx)) : Sub(Mul(scale, Add(static_cast<float>(idx), 0.5f)), 0.5f);
}

// First grads index of the walk for grad_input index yIdx (resize_bicubic_v2_grad_simt_determine.h:95-113)
__device__ __forceinline__ int32_t WalkStart(int32_t yIdx, float inverse, float offset)
{
    const float v = ceilf(Sub(Mul(Add(Sub(static_cast<float>(yIdx), 2.0f), offset), inverse), offset));
    const long long s = static_cast<long long>(v);
    return static_cast<int32_t>(s < 0 ? 0 : (s > INT32_MAX ? INT32_MAX : s));
}

// One grad_input element by the reference's walk, with nothing cached: the coefficients of a column are evaluated
// again for every row. Used for elements whose column list does not fit the shared-memory lists of the kernel
// below (an extent of 1 makes every grads index a tap of the single element).
template <typename T>
__device__ float BwdElementDirect(const T* __restrict__ pg, const BicubicGeom& g, int32_t yh, int32_t yw, int32_t c,
                                  int64_t rowGo, float offset)
{
    const int32_t hStart = WalkStart(yh, g.invH, offset);
    const float rhStart = Sub(Mul(Add(static_cast<float>(hStart), offset), g.scaleH), offset);
    const bool borderH = yh == 0 || yh == g.hin - 1;
    const int32_t wStart = WalkStart(yw, g.invW, offset);
    const float rwStart = Sub(Mul(Add(static_cast<float>(wStart), offset), g.scaleW), offset);
    const bool borderW = yw == 0 || yw == g.win - 1;
    float add = 0.0f;
    float rh = rhStart;
    for (int32_t h = hStart; h < g.hout; ++h, rh = BwdSrc(g.scaleH, h, g.align)) {
        float chTap[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float chPoint = 0.0f;
        long long fh = 0;
        if (borderH) {
            fh = static_cast<long long>(floorf(rh));
            if (yh == 0 && fh > 1 && g.hin > 1) {
                break;
            }
            TapCoeff(Sub(rh, static_cast<float>(fh)), chTap);
        } else {
            if (!(rh < Add(static_cast<float>(yh), 2.0f))) {
                break;
            }
            chPoint = PointCoeff(fabsf(Sub(rh, static_cast<float>(yh))));
        }
        const T* prow = pg + h * rowGo + c;
        float rw = rwStart;
        for (int32_t w = wStart; w < g.wout; ++w, rw = BwdSrc(g.scaleW, w, g.align)) {
            float cwTap[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            float cwPoint = 0.0f;
            long long fw = 0;
            if (borderW) {
                fw = static_cast<long long>(floorf(rw));
                if (yw == 0 && fw > 1 && g.win > 1) {
                    break;
                }
                TapCoeff(Sub(rw, static_cast<float>(fw)), cwTap);
            } else {
                if (!(rw < Add(static_cast<float>(yw), 2.0f))) {
                    break;
                }
                cwPoint = PointCoeff(fabsf(Sub(rw, static_cast<float>(yw))));
            }
            const float gv = DType<T>::Load(prow + static_cast<int64_t>(w) * g.chan);
            if (!borderH && !borderW) {
                add = Add(add, Mul(Mul(gv, chPoint), cwPoint));
            } else if (!borderH) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (ClampIdx(fw - 1 + j, g.win - 1) == yw) {
                        add = Add(add, Mul(Mul(gv, chPoint), cwTap[j]));
                    }
                }
            } else if (!borderW) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (ClampIdx(fh - 1 + i, g.hin - 1) == yh) {
                        add = Add(add, Mul(Mul(gv, chTap[i]), cwPoint));
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (ClampIdx(fh - 1 + i, g.hin - 1) == yh && ClampIdx(fw - 1 + j, g.win - 1) == yw) {
                            add = Add(add, Mul(Mul(gv, chTap[i]), cwTap[j]));
                        }
                    }
                }
            }
        }
    }
    return add;
}

// The gather with the column side of the walk cached. A thread owns one element position of a grad_input row
// (column yw; for NHWC also its channel) and keeps it while the block moves over rows and planes. It first walks
// the grads columns once, exactly as the reference does, and stores every grads column that reaches it with its
// coefficients (one for an interior yw, up to three matching taps in tap order for a first or last yw) in its own
// column of a shared-memory table. For each grads row h of the row walk it then has one coefficient (interior yh) or
// the matching tap coefficients in tap order (first or last yh), and adds (g * cH) * cW over the columns, for each of
// them with the row taps outside the column taps. That is the order and the rounding of the reference's four walks,
// so the sum has the same bits. The additions of a thread are one chain; what it must not wait for one by one are the
// loads, so the grads values of kListBatch columns are fetched before the first of them is used (border columns of
// fp32 8x64 planes 60x80 <- 150x199: 58 us with one load at a time, 38 us in batches).
// The blocks of a launch divide its element positions (of all columns, or of the first and the last) by x and its rows by y;
// colsPB positions per block, further threads take further rows.
constexpr int kListBatch = 8;
constexpr int kListTaps = 3; // a fourth needs an extent of 1
constexpr int kListThreads = 128;
constexpr int kListBytes = 4 + 4 * kListTaps; // per column and thread
constexpr int kInteriorBytes = 4;             // and of a list of interior columns
struct ListShape {
    int32_t colsPB, entries, x, y;
};

template <typename T, bool NHWC>
__device__ __forceinline__ void BwdListBlock(const T* __restrict__ go, T* __restrict__ gi, const BicubicGeom& g,
                                             int32_t maxW, int32_t colsPB, bool borderOnly, float* sList, int32_t blockX,
                                             int64_t blockY, int64_t blocksY)
{
    const int32_t nt = blockDim.x, tid = threadIdx.x;
    float* sCoef = sList; // [maxW][kListTaps][nt]
    int32_t* sCol = reinterpret_cast<int32_t*>(sList + static_cast<size_t>(maxW) * kListTaps * nt); // column << 2 | taps
    const int32_t inner = g.win * g.chan;
    const int32_t rowsPB = nt / colsPB;
    const int32_t rowLane = tid / colsPB;
    const int32_t pos = blockX * colsPB + (tid - rowLane * colsPB);
    if (rowLane >= rowsPB || pos >= (borderOnly ? 2 * g.chan : inner)) {
        return;
    }
    int32_t t = pos;
    if (borderOnly) {
        const int32_t side = NHWC ? pos / g.chan : pos;
        t = side == 0 ? pos : inner - 2 * g.chan + pos; // column 0 or column win - 1, same channel
    }
    const int32_t yw = NHWC ? t / g.chan : t;
    const int32_t c = NHWC ? t - yw * g.chan : 0;
    const int64_t planeGo = static_cast<int64_t>(g.hout) * g.wout * g.chan;
    const int64_t rowGo = static_cast<int64_t>(g.wout) * g.chan;
    const float offset = g.align ? 0.0f : 0.5f;
    const bool borderW = yw == 0 || yw == g.win - 1;

    // the column walk, once
    int32_t cnt = 0;
    bool overflow = false;
    const int32_t wStart = WalkStart(yw, g.invW, offset);
    {
        float rw = Sub(Mul(Add(static_cast<float>(wStart), offset), g.scaleW), offset);
        for (int32_t w = wStart; w < g.wout && !overflow; ++w, rw = BwdSrc(g.scaleW, w, g.align)) {
            if (borderW) {
                const long long fw = static_cast<long long>(floorf(rw));
                if (yw == 0 && fw > 1 && g.win > 1) {
                    break;
                }
                float cwTap[4];
                TapCoeff(Sub(rw, static_cast<float>(fw)), cwTap);
                int n = 0;
                overflow = cnt >= maxW || w >= (1 << 29);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (!overflow && ClampIdx(fw - 1 + j, g.win - 1) == yw) {
                        if (n < kListTaps) {
                            sCoef[(cnt * kListTaps + n) * nt + tid] = cwTap[j];
                            ++n;
                        } else {
                            overflow = true;
                        }
                    }
                }
                if (n > 0 && !overflow) {
                    sCol[cnt * nt + tid] = w << 2 | n;
                    ++cnt;
                }
            } else {
                if (!(rw < Add(static_cast<float>(yw), 2.0f))) {
                    break;
                }
                overflow = cnt >= maxW || w >= (1 << 29);
                if (!overflow) {
                    sCoef[cnt * kListTaps * nt + tid] = PointCoeff(fabsf(Sub(rw, static_cast<float>(yw))));
                    sCol[cnt * nt + tid] = w << 2 | 1;
                    ++cnt;
                }
            }
        }
    }

    for (int64_t row = blockY * rowsPB + rowLane; row < g.rows; row += blocksY * rowsPB) {
        const int64_t plane = row / g.hin;
        const int32_t yh = static_cast<int32_t>(row - plane * g.hin);
        const T* pg = go + plane * planeGo;
        T* po = gi + row * inner;
        if (overflow) {
            po[t] = DType<T>::FromF(BwdElementDirect<T>(pg, g, yh, yw, c, rowGo, offset));
            continue;
        }
        const bool borderH = yh == 0 || yh == g.hin - 1;
        const int32_t hStart = WalkStart(yh, g.invH, offset);
        float rh = Sub(Mul(Add(static_cast<float>(hStart), offset), g.scaleH), offset);
        float add = 0.0f;
        for (int32_t h = hStart; h < g.hout; ++h, rh = BwdSrc(g.scaleH, h, g.align)) {
            const T* prow = pg + h * rowGo + c;
            float chv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            int nH = 1;
            if (!borderH) {
                if (!(rh < Add(static_cast<float>(yh), 2.0f))) {
                    break;
                }
                chv[0] = PointCoeff(fabsf(Sub(rh, static_cast<float>(yh))));
            } else {
                const long long fh = static_cast<long long>(floorf(rh));
                if (yh == 0 && fh > 1 && g.hin > 1) {
                    break;
                }
                float chTap[4];
                TapCoeff(Sub(rh, static_cast<float>(fh)), chTap);
                nH = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (ClampIdx(fh - 1 + i, g.hin - 1) == yh) {
                        // compacted in tap order without dynamic register indexing
                        chv[3] = chTap[i];
                        if (nH == 0) chv[0] = chTap[i];
                        if (nH == 1) chv[1] = chTap[i];
                        if (nH == 2) chv[2] = chTap[i];
                        ++nH;
                    }
                }
            }
            for (int32_t k0 = 0; k0 < cnt; k0 += kListBatch) {
                float gv[kListBatch];
                int32_t taps[kListBatch];
#pragma unroll
                for (int u = 0; u < kListBatch; ++u) {
                    gv[u] = 0.0f;
                    taps[u] = 0;
                    if (k0 + u < cnt) {
                        const int32_t col = sCol[(k0 + u) * nt + tid];
                        gv[u] = DType<T>::Load(prow + static_cast<int64_t>(col >> 2) * g.chan);
                        taps[u] = col & 3;
                    }
                }
#pragma unroll
                for (int u = 0; u < kListBatch; ++u) {
                    if (taps[u] == 0) {
                        break;
                    }
                    const float* cu = sCoef + (k0 + u) * kListTaps * nt + tid;
                    for (int i = 0; i < nH; ++i) {
                        const float gc = Mul(gv[u], i == 0 ? chv[0] : (i == 1 ? chv[1] : (i == 2 ? chv[2] : chv[3])));
#pragma unroll
                        for (int j = 0; j < kListTaps; ++j) {
                            if (j < taps[u]) {
                                add = Add(add, Mul(gc, cu[j * nt]));
                            }
                        }
                    }
                }
            }
        }
        po[t] = DType<T>::FromF(add);
    }
}

// The same for the interior columns, whose grads columns follow one another from the start of the walk with one coefficient
// each: a list is its coefficients, 4 bytes per column and thread, and a term is one load, two products and one addition.
// All terms of a batch are formed before the first is added. What bounds it is instruction issue on the terms, which the general
// block spends on columns, taps and bounds as well (fp32 8x38 planes 97x104 <- 35x712: 377 us by general lists).
template <typename T, bool NHWC>
__device__ __forceinline__ void BwdInteriorListBlock(const T* __restrict__ go, T* __restrict__ gi, const BicubicGeom& g,
                                                     int32_t maxW, int32_t colsPB, float* sCoef, int32_t blockX, int64_t blockY,
                                                     int64_t blocksY)
{
    const int32_t nt = blockDim.x, tid = threadIdx.x; // sCoef: [maxW][nt]
    const int32_t inner = g.win * g.chan;
    const int32_t rowsPB = nt / colsPB, rowLane = tid / colsPB;
    const int32_t pos = blockX * colsPB + (tid - rowLane * colsPB);
    if (rowLane >= rowsPB || pos >= inner - 2 * g.chan) {
        return;
    }
    const int32_t t = pos + g.chan;
    const int32_t yw = NHWC ? t / g.chan : t;
    const int32_t c = NHWC ? t - yw * g.chan : 0;
    const int64_t rowGo = static_cast<int64_t>(g.wout) * g.chan, planeGo = g.hout * rowGo;
    const float offset = g.align ? 0.0f : 0.5f;
    const int32_t wStart = WalkStart(yw, g.invW, offset);
    const float* coef = sCoef + tid;
    int32_t cnt = 0;
    bool overflow = false;
    for (int32_t w = wStart; w < g.wout; ++w) {
        const float rw = BwdSrc(g.scaleW, w, g.align);
        if (!(rw < Add(static_cast<float>(yw), 2.0f))) {
            break;
        }
        overflow = cnt >= maxW;
        if (overflow) {
            break;
        }
        sCoef[cnt * nt + tid] = PointCoeff(fabsf(Sub(rw, static_cast<float>(yw))));
        ++cnt;
    }
    const int32_t step = NHWC ? g.chan : 1;
    for (int64_t row = blockY * rowsPB + rowLane; row < g.rows; row += blocksY * rowsPB) {
        const int64_t plane = row / g.hin;
        const int32_t yh = static_cast<int32_t>(row - plane * g.hin);
        const T* pg = go + plane * planeGo;
        T* dst = gi + row * inner + t;
        if (overflow) {
            *dst = DType<T>::FromF(BwdElementDirect<T>(pg, g, yh, yw, c, rowGo, offset));
            continue;
        }
        const bool borderH = yh == 0 || yh == g.hin - 1;
        float add = 0.0f;
        for (int32_t h = WalkStart(yh, g.invH, offset); h < g.hout; ++h) {
            const float rh = BwdSrc(g.scaleH, h, g.align);
            float chv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            int nH = 1;
            if (!borderH) {
                if (!(rh < Add(static_cast<float>(yh), 2.0f))) {
                    break;
                }
                chv[0] = PointCoeff(fabsf(Sub(rh, static_cast<float>(yh))));
            } else {
                const long long fh = static_cast<long long>(floorf(rh));
                if (yh == 0 && fh > 1 && g.hin > 1) {
                    break;
                }
                float chTap[4];
                TapCoeff(Sub(rh, static_cast<float>(fh)), chTap);
                nH = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (ClampIdx(fh - 1 + i, g.hin - 1) == yh) { // compacted in tap order
                        chv[3] = chTap[i];
                        if (nH == 0) chv[0] = chTap[i];
                        if (nH == 1) chv[1] = chTap[i];
                        if (nH == 2) chv[2] = chTap[i];
                        ++nH;
                    }
                }
            }
            const T* p = pg + h * rowGo + static_cast<int64_t>(wStart) * step + c;
            const float* cp = coef;
            int32_t k = 0;
            if (nH == 1) {
                const float ch = chv[0];
#pragma unroll 1
                for (; k + kListBatch <= cnt; k += kListBatch, p += kListBatch * static_cast<int64_t>(step), cp += kListBatch * nt) {
                    float term[kListBatch];
#pragma unroll
                    for (int u = 0; u < kListBatch; ++u) {
                        term[u] = DType<T>::Load(p + u * step);
                    }
#pragma unroll
                    for (int u = 0; u < kListBatch; ++u) {
                        term[u] = Mul(Mul(term[u], ch), cp[u * nt]);
                    }
#pragma unroll
                    for (int u = 0; u < kListBatch; ++u) {
                        add = Add(add, term[u]);
                    }
                }
                float term[kListBatch]; // what is left, all loads in flight as well
#pragma unroll
                for (int u = 0; u < kListBatch - 1; ++u) {
                    term[u] = k + u < cnt ? DType<T>::Load(p + u * step) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < kListBatch - 1; ++u) {
                    if (k + u < cnt) {
                        add = Add(add, Mul(Mul(term[u], ch), cp[u * nt]));
                    }
                }
            } else {
#pragma unroll 4
                for (; k < cnt; ++k, p += step, cp += nt) {
                    const float gv = DType<T>::Load(p), cw = *cp;
                    for (int i = 0; i < nH; ++i) {
                        add = Add(add, Mul(Mul(gv, i == 0 ? chv[0] : (i == 1 ? chv[1] : (i == 2 ? chv[2] : chv[3]))), cw));
                    }
                }
            }
        }
        *dst = DType<T>::FromF(add);
    }
}

// All columns by lists (scales beyond four, user scales that contradict the extents, extents of two): the border columns in
// the first blocks, whose chains are the longest, the interior ones behind them.
template <typename T, bool NHWC>
__global__ void __launch_bounds__(kListThreads) Bicubic2dBwdListKernel(const T* __restrict__ go, T* __restrict__ gi, BicubicGeom g,
                                                                        ListShape border, ListShape interior)
{
    extern __shared__ __align__(16) float sList[];
    const int32_t block = blockIdx.x, borders = border.x * border.y;
    if (g.win <= 2) {
        BwdListBlock<T, NHWC>(go, gi, g, border.entries, border.colsPB, false, sList, block % border.x,
                                         block / border.x, border.y);
    } else if (block < borders) {
        BwdListBlock<T, NHWC>(go, gi, g, border.entries, border.colsPB, true, sList, block % border.x,
                                         block / border.x, border.y);
    } else {
        BwdInteriorListBlock<T, NHWC>(go, gi, g, interior.entries, interior.colsPB, sList, (block - borders) % interior.x,
                                      (block - borders) / interior.x, interior.y);
    }
}

// ---- the same gather for the interior columns (1 .. win - 2): a walk down the grads rows --------------------------
// A thread owns one element position of a grad_input row and a block a band of grad_input rows. The thread walks down
// the grads rows that feed the band and keeps one sum open for every grad_input row whose walk includes the current
// grads row (at most kOpen: the walk spans four source pixels, one more through rounding), so a grads value is loaded
// and converted once per column that it feeds instead of once per term. A grad_input row takes its terms in ascending
// grads row and, within one, ascending grads column, each (g * cH) * cW with its own roundings: the order and the bits
// of the reference's walk. What bounds the kernel is instruction issue on those terms: two packed products per pair of
// terms and one add per term, which cannot be packed because the terms of a sum follow one another.
// The column side of the walk (at most K columns, one coefficient each) stays in registers; the row side is evaluated
// once per block into shared-memory records. First and last rows take up to four taps per grads row: they ride along
// in the blocks whose band holds them. The first and the last column are list blocks, the first blocks of the same grid,
// so that their long chains run under the walk. fp32 8x64 planes 60x80 <- 150x199: 230 us as two launches that loaded
// every term -> 80 us.
constexpr int kOpen = 5;
constexpr int kWalkThreads = 128;
constexpr int kWalkMaxRows = 448; // grads rows that a band may read (their records stay below 48 KB)

struct WalkRecord {
    float c[kOpen];   // coefficients of the open rows, from `first` on
    int32_t first, count;
    int32_t edge;     // bits 0..3: taps of this grads row that land on row 0, bits 4..7: on row hin - 1
    float tap[4];     // their coefficients
    float pad[4];
};
static_assert(sizeof(WalkRecord) == 64, "records are read as 16-byte words");
static_assert(kListThreads == kWalkThreads, "list blocks and walk blocks share a grid");

// walkX: blocks of one band; the first list.x * list.y blocks of the grid are list blocks.
struct WalkShape {
    int64_t positions; // planes * interior element positions of a row
    int32_t bandRows, maxRows, walkX;
    ListShape list;
};

template <typename T, bool NHWC, int K>
__global__ void __launch_bounds__(kWalkThreads, (NHWC && K > 14) ? 3 : ((NHWC || K > 14) ? 4 : 5))
    Bicubic2dBwdWalkKernel(const T* __restrict__ go, T* __restrict__ gi, BicubicGeom g, WalkShape ws)
{
    extern __shared__ __align__(16) float sWalk[];
    const int32_t lists = ws.list.x * ws.list.y;
    if (static_cast<int32_t>(blockIdx.x) < lists) {
        BwdListBlock<T, NHWC>(go, gi, g, ws.list.entries, ws.list.colsPB, true, sWalk,
                                         static_cast<int32_t>(blockIdx.x) % ws.list.x,
                                         static_cast<int32_t>(blockIdx.x) / ws.list.x, ws.list.y);
        return;
    }
    const int32_t walkBlock = static_cast<int32_t>(blockIdx.x) - lists;
    const int32_t band = walkBlock / ws.walkX;
    WalkRecord* rec = reinterpret_cast<WalkRecord*>(sWalk);
    int32_t* rowStart = reinterpret_cast<int32_t*>(rec + ws.maxRows);
    int32_t* rowEnd = rowStart + ws.bandRows;
    const float offset = g.align ? 0.0f : 0.5f;
    const int32_t y0 = band * ws.bandRows, y1 = min(y0 + ws.bandRows, g.hin);
    const int32_t yi0 = max(y0, 1), yi1 = min(y1, g.hin - 1); // interior rows of the band
    for (int32_t r = threadIdx.x; r < y1 - y0; r += blockDim.x) {
        const int32_t y = y0 + r;
        const int32_t h0 = min(WalkStart(y, g.invH, offset), g.hout);
        int32_t h = h0;
        if (y == g.hin - 1) {
            h = g.hout;
        } else {
            while (h < g.hout) {
                const float rh = BwdSrc(g.scaleH, h, g.align);
                if (y == 0 ? static_cast<long long>(floorf(rh)) > 1 : !(rh < Add(static_cast<float>(y), 2.0f))) {
                    break;
                }
                ++h;
            }
        }
        rowStart[r] = h0;
        rowEnd[r] = h;
    }
    __syncthreads();
    // starts and ends grow with the row
    const int32_t hLo = rowStart[0], hHi = min(rowEnd[y1 - 1 - y0], hLo + ws.maxRows);
    for (int32_t h = hLo + threadIdx.x; h < hHi; h += blockDim.x) {
        const float rh = BwdSrc(g.scaleH, h, g.align);
        WalkRecord w{};
        int32_t y = yi0, yEnd = yi1; // the first interior row whose walk has not ended
        while (y < yEnd) {
            const int32_t mid = (y + yEnd) >> 1;
            if (rowEnd[mid - y0] <= h) {
                y = mid + 1;
            } else {
                yEnd = mid;
            }
        }
        w.first = y;
#pragma unroll
        for (int a = 0; a < kOpen; ++a) {
            if (y + a < yi1 && rowStart[y + a - y0] <= h) {
                w.c[a] = PointCoeff(fabsf(Sub(rh, static_cast<float>(y + a))));
                w.count = a + 1;
            }
        }
        const bool top = y0 == 0 && h >= rowStart[0] && h < rowEnd[0];
        const bool bottom = y1 == g.hin && h >= rowStart[y1 - 1 - y0] && h < rowEnd[y1 - 1 - y0];
        if (top || bottom) {
            const long long fh = static_cast<long long>(floorf(rh));
            TapCoeff(Sub(rh, static_cast<float>(fh)), w.tap);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int32_t dst = ClampIdx(fh - 1 + i, g.hin - 1);
                w.edge |= (top && dst == 0) ? 1 << i : 0;
                w.edge |= (bottom && dst == g.hin - 1) ? 16 << i : 0;
            }
        }
        rec[h - hLo] = w;
    }
    __syncthreads();

    const int64_t pos = static_cast<int64_t>(walkBlock - band * ws.walkX) * blockDim.x + threadIdx.x;
    if (pos >= ws.positions) {
        return;
    }
    const int32_t inner = g.win * g.chan;
    const int32_t perPlane = inner - 2 * g.chan;
    const int64_t plane = ws.positions <= INT32_MAX
                              ? static_cast<int64_t>(static_cast<uint32_t>(pos) / static_cast<uint32_t>(perPlane))
                              : pos / perPlane;
    const int32_t t = static_cast<int32_t>(pos - plane * perPlane) + g.chan; // skip column 0
    const int32_t yw = NHWC ? t / g.chan : t;
    const int32_t c = NHWC ? t - yw * g.chan : 0;
    const int64_t rowGo = static_cast<int64_t>(g.wout) * g.chan;
    const T* pg = go + plane * g.hout * rowGo;
    T* po = gi + plane * g.hin * static_cast<int64_t>(inner) + t;

    // the column walk, once; slots past it keep the coefficient 0
    F2 cw[K / 2];
    int32_t cnt = 0;
    const int32_t wStart = WalkStart(yw, g.invW, offset);
    {
        float cws[K];
        bool done = false;
#pragma unroll
        for (int k = 0; k < K + 1; ++k) {
            const int32_t w = wStart + k;
            if (k < K) {
                cws[k < K ? k : 0] = 0.0f;
            }
            if (!done && w < g.wout) {
                const float rw = BwdSrc(g.scaleW, w, g.align);
                if (!(rw < Add(static_cast<float>(yw), 2.0f))) {
                    done = true;
                } else if (k == K) {
                    cnt = -1; // does not fit the registers
                } else {
                    cws[k < K ? k : 0] = PointCoeff(fabsf(Sub(rw, static_cast<float>(yw))));
                    cnt = k + 1;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < K / 2; ++k) {
            cw[k] = MakeF2(cws[2 * k], cws[2 * k + 1]);
        }
    }
    if (cnt < 0) {
        for (int32_t y = y0; y < y1; ++y) {
            po[static_cast<int64_t>(y) * inner] = DType<T>::FromF(BwdElementDirect<T>(pg, g, y, yw, c, rowGo, offset));
        }
        return;
    }
    const int32_t colStep = NHWC ? g.chan : 1; // a compile-time 1 for NCHW
    const T* pw = pg + hLo * rowGo + static_cast<int64_t>(wStart) * colStep + c;

    float acc[kOpen];
#pragma unroll
    for (int a = 0; a < kOpen; ++a) {
        acc[a] = 0.0f;
    }
    float top = 0.0f, bottom = 0.0f;
    int32_t cur = yi0;
    auto finish = [&]() { // the oldest open row is complete
        po[static_cast<int64_t>(cur) * inner] = DType<T>::FromF(acc[0]);
#pragma unroll
        for (int a = 0; a + 1 < kOpen; ++a) {
            acc[a] = acc[a + 1];
        }
        acc[kOpen - 1] = 0.0f;
        ++cur;
    };
    T raw[K]; // the next grads row, in flight; slots past the walk stay 0
#pragma unroll
    for (int k = 0; k < K; ++k) {
        raw[k] = DType<T>::FromF(0.0f);
        if (k < cnt && hLo < hHi) {
            raw[k] = __ldg(pw + k * colStep);
        }
    }
    for (int32_t h = hLo; h < hHi; ++h) {
        F2 gv[K / 2];
#pragma unroll
        for (int k = 0; k < K / 2; ++k) {
            gv[k] = MakeF2(DType<T>::ToF(raw[2 * k]), DType<T>::ToF(raw[2 * k + 1]));
        }
        pw += rowGo;
        if (h + 1 < hHi) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (k < cnt) {
                    raw[k] = __ldg(pw + k * colStep);
                }
            }
        }
        const WalkRecord& r = rec[h - hLo];
        const float4 r0 = *reinterpret_cast<const float4*>(&r);
        const float4 r1 = *(reinterpret_cast<const float4*>(&r) + 1);
        const float ch[kOpen] = {r0.x, r0.y, r0.z, r0.w, r1.x};
        const int32_t first = __float_as_int(r1.y), count = __float_as_int(r1.z), edge = __float_as_int(r1.w);
        while (cur < first) {
            finish();
        }
#pragma unroll
        for (int a = 0; a < kOpen; ++a) {
            if (a < count) { // the same for the whole block
                const F2 c2 = MakeF2(ch[a], ch[a]);
#pragma unroll
                for (int k = 0; k < K / 2; ++k) {
                    float p0, p1;
                    SplitF2(Mul2(Mul2(gv[k], c2), cw[k]), p0, p1);
                    // a slot past the walk gives a zero, which cannot change a sum that started from +0
                    acc[a] = Add(acc[a], p0);
                    acc[a] = Add(acc[a], p1);
                }
            }
        }
        if (edge != 0) { // first or last row: the taps of one grads value before those of the next
#pragma unroll
            for (int k = 0; k < K / 2; ++k) {
                float gs[2], cs[2];
                SplitF2(gv[k], gs[0], gs[1]);
                SplitF2(cw[k], cs[0], cs[1]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (2 * k + u < cnt) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float term = Mul(Mul(gs[u], r.tap[i]), cs[u]);
                            if ((edge >> i) & 1) {
                                top = Add(top, term);
                            }
                            if ((edge >> (i + 4)) & 1) {
                                bottom = Add(bottom, term);
                            }
                        }
                    }
                }
            }
        }
    }
    while (cur < yi1) {
        finish();
    }
    if (y0 == 0) {
        po[0] = DType<T>::FromF(top);
    }
    if (y1 == g.hin) {
        po[static_cast<int64_t>(g.hin - 1) * inner] = DType<T>::FromF(bottom);
    }
}

// ---- backward at exactly 2x (scales 0.5, align_corners = false), NCHW --------------------------------------------
// At this scale every source coordinate w / 2 - 0.25 is exact, so the walk of an interior grad_input index y visits
// the grads indices 2y - 3 .. 2y + 4 (those inside the image) and the coefficient of the k-th of them is the same
// number PointCoeff(|k / 2 - 1.75|) for every y. A block stages the grads rows of a band of grad_input rows in shared
// memory as fp32 (each grads value is loaded and converted once instead of sixteen times), with zero columns either
// side: a term whose grads column lies outside the image then adds a zero, which leaves a round-to-nearest sum that
// started from +0 unchanged, so the window of a column needs no bounds. A thread owns two adjacent grad_input
// columns of one row and reads their ten grads columns of a grads row as three 16-byte shared-memory loads. The
// first and last row and column, whose walk has up to three clamped taps per grads index, take their (index,
// coefficient) entries from four lists that the block builds with the reference's walk; the border columns are items
// of their own behind the pairs, so that their longer loop does not run in the warps of the interior. Terms, their
// (row, column, row tap, column tap) order and their rounding are those of the other two backward kernels.
// n / d for n * d < 2^32 as the high half of one 32-bit multiply: m = floor(2^32 / d) + 1 (the usual round-up
// reciprocal; exact because n * (m * d - 2^32) < 2^32 there). d = 1 has no 32-bit reciprocal and is tested for. The
// item loops below split an item index into (row, position) with it.
struct FastDiv {
    uint32_t m, d;
};
inline FastDiv MakeFastDiv(uint32_t d) { return FastDiv{d > 1 ? static_cast<uint32_t>((1ULL << 32) / d + 1) : 0u, d}; }
__device__ __forceinline__ uint32_t DivBy(uint32_t n, FastDiv f) { return f.d > 1 ? __umulhi(n, f.m) : n; }

constexpr int kX2Pad = 4;     // zero columns left of a staged grads row (the window of column 0 starts at -4)
constexpr int kX2Groups = 5;  // grads indices in the walk of a first or last index at 2x
constexpr int kX2Slots = 3;   // clamped taps of one grads index that fall on it (four only for an extent of 1)
constexpr int kX2Threads = 256;

// The walk of a first or last grad_input index in slot form: grads indices start .. start + 4, up to three tap
// coefficients each in tap order; bit 3m + t of mask says that slot t of group m holds a term.
constexpr int kX2Flat = 9;    // terms of such a walk when the extent is at least 2
struct X2BorderList {
    int32_t start;
    uint32_t mask;
    float coef[kX2Groups * kX2Slots];
    // the same terms one after the other in walk order, filled up with (column -1, 0): a term of the zero column
    // adds nothing, so a loop over all kX2Flat entries needs no test
    int32_t flatIdx[kX2Flat];
    float flatCoef[kX2Flat];
    int32_t terms;
};

struct X2BorderLists {
    X2BorderList l[4]; // 0 first column, 1 last column, 2 first row, 3 last row
    float interior[8]; // coefficient of the k-th grads index of an interior walk: PointCoeff(|k / 2 - 1.75|)
};

// The reference's walk for a first or last index at scale 0.5, on the host: this file's host code is compiled with
// floating-point contraction off, so every operation below rounds as the device's non-fused multiply and add do
// (and at this scale the coordinates and the fractions 0.25 / 0.75 are exact anyway).
namespace x2host {
inline float Conv1(float x) { return ((((kA + 2.0f) * x) - (kA + 3.0f)) * x) * x + 1.0f; }
inline float Conv2(float x) { return ((((kA * x) - 5.0f * kA) * x) + 8.0f * kA) * x - 4.0f * kA; }
inline float PointCoeff(float d) { return d <= 1.0f ? Conv1(d) : (d < 2.0f ? Conv2(d) : 0.0f); }
inline void FwdCoeff(float t, float (&c)[4])
{
    c[0] = Conv2(t + 1.0f);
    c[1] = Conv1(t);
    c[2] = Conv1(1.0f - t);
    c[3] = Conv2(2.0f - t);
}
inline X2BorderList BorderList(int32_t yIdx, int32_t in, int32_t out)
{
    X2BorderList list;
    const int32_t start = std::max(2 * yIdx - 3, 0); // ceil((y - 2 + 0.5) * 2 - 0.5), clamped at 0
    uint32_t mask = 0;
    for (int k = 0; k < kX2Groups * kX2Slots; ++k) {
        list.coef[k] = 0.0f;
    }
    for (int32_t o = start; o < out && o - start < kX2Groups; ++o) {
        const float r = (static_cast<float>(o) + 0.5f) * 0.5f - 0.5f;
        const long long f = static_cast<long long>(std::floor(r));
        if (yIdx == 0 && f > 1 && in > 1) {
            break;
        }
        const float t = r - static_cast<float>(f);
        const float u = 1.0f - t;
        const float tap[4] = {Conv2(t + 1.0f), Conv1(t), Conv1(u), Conv2(u + 1.0f)};
        int slot = 0;
        for (int j = 0; j < 4; ++j) {
            const long long idx = std::min<long long>(std::max<long long>(f - 1 + j, 0), in - 1);
            if (idx == yIdx && slot < kX2Slots) {
                list.coef[(o - start) * kX2Slots + slot] = tap[j];
                mask |= 1u << ((o - start) * kX2Slots + slot);
                ++slot;
            }
        }
    }
    list.start = start;
    list.mask = mask;
    list.terms = 0;
    for (int k = 0; k < kX2Flat; ++k) {
        list.flatIdx[k] = -1;
        list.flatCoef[k] = 0.0f;
    }
    for (int k = 0; k < kX2Groups * kX2Slots; ++k) {
        if (mask & (1u << k)) {
            if (list.terms < kX2Flat) {
                list.flatIdx[list.terms] = start + k / kX2Slots;
                list.flatCoef[list.terms] = list.coef[k];
            }
            ++list.terms;
        }
    }
    return list;
}
} // namespace x2host

// The four corners of a plane at 2x: both walks have clamped taps, so a grads value meets up to three row
// coefficients times up to three column coefficients, row taps outside column taps. One thread per plane and corner,
// the corner uniform over a block, so every slot test is uniform; grads straight from global memory.
template <typename T>
__device__ __forceinline__ void X2Corner(const T* __restrict__ go, T* __restrict__ gi, const BicubicGeom& g, int64_t plane,
                                         int corner, const X2BorderLists& lists)
{
    // corner: 0 (0, 0), 1 (0, win - 1), 2 (hin - 1, 0), 3 (hin - 1, win - 1)
    const X2BorderList& rows = lists.l[2 + (corner >> 1)];
    const X2BorderList& cols = lists.l[corner & 1];
    const uint32_t rmask = rows.mask, cmask = cols.mask;
    const T* pg = go + plane * (static_cast<int64_t>(g.hout) * g.wout);
    float add = 0.0f;
#pragma unroll
    for (int mr = 0; mr < kX2Groups; ++mr) {
        const uint32_t rbits = (rmask >> (mr * kX2Slots)) & 7u;
        if (rbits == 0) {
            continue;
        }
        const T* prow = pg + static_cast<int64_t>(rows.start + mr) * g.wout;
#pragma unroll
        for (int m = 0; m < kX2Groups; ++m) {
            const uint32_t cbits = (cmask >> (m * kX2Slots)) & 7u;
            if (cbits == 0) {
                continue;
            }
            const float gv = DType<T>::Load(prow + cols.start + m);
#pragma unroll
            for (int i = 0; i < kX2Slots; ++i) {
                if (rbits & (1u << i)) {
                    const float gch = Mul(gv, rows.coef[mr * kX2Slots + i]);
#pragma unroll
                    for (int t = 0; t < kX2Slots; ++t) {
                        if (cbits & (1u << t)) {
                            add = Add(add, Mul(gch, cols.coef[m * kX2Slots + t]));
                        }
                    }
                }
            }
        }
    }
    const int32_t yh = (corner >> 1) ? g.hin - 1 : 0, yw = (corner & 1) ? g.win - 1 : 0;
    gi[(plane * g.hin + yh) * g.win + yw] = DType<T>::FromF(add);
}

template <typename T>
__global__ void __launch_bounds__(kX2Threads) Bicubic2dBwdX2Kernel(const T* __restrict__ go, T* __restrict__ gi, BicubicGeom g,
                                                                   int32_t bandRows, int32_t bands, int32_t pitch,
                                                                   int32_t vecLoad, const X2BorderLists lists,
                                                                   int64_t planes, int32_t cornerBlocks)
{
    extern __shared__ __align__(16) float sG[]; // (2 * bandRows + 6) grads rows of `pitch` floats
    const X2BorderList* sL = lists.l;
    const int32_t tid = threadIdx.x, nt = blockDim.x;
    if (static_cast<int32_t>(blockIdx.x) < cornerBlocks) {
        // the first blocks of the grid take the corners of all planes (four blocks per nt planes); they are resident
        // next to band blocks from the start, so their chains of dependent additions cost no time of their own
        const int64_t cp = static_cast<int64_t>(blockIdx.x >> 2) * nt + tid;
        if (cp < planes) {
            X2Corner<T>(go, gi, g, cp, static_cast<int>(blockIdx.x & 3), lists);
        }
        return;
    }
    const uint32_t bandBlock = blockIdx.x - cornerBlocks;
    const int64_t plane = bandBlock / bands;
    const int32_t band = static_cast<int32_t>(bandBlock - plane * bands);
    const int32_t yhA = band * bandRows, yhB = min(yhA + bandRows, g.hin);
    const int32_t hBase = 2 * yhA - 3; // grads row of shared-memory row 0
    const int32_t hLo = max(hBase, 0), hHi = min(2 * (yhB - 1) + 4, g.hout - 1);
    const int32_t nRows = hHi - hLo + 1;

    const float* c = lists.interior;
    {
        // zero rows where the band's window leaves the image, zero columns either side of a row, as 8-byte stores (wout is even)
        const int32_t rowsTop = hLo - hBase, rowsAll = 2 * (yhB - yhA) + 6;
        const int32_t rowsZero = rowsAll - nRows; // above the first image row and below the last
        for (int32_t i = tid; i < rowsZero * (pitch / 4); i += nt) {
            const int32_t r = i / (pitch / 4), k = i - r * (pitch / 4);
            const int32_t row = r < rowsTop ? r : nRows + r;
            *reinterpret_cast<float4*>(sG + row * pitch + 4 * k) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        float* sRow0 = sG + (hLo - hBase) * pitch;
        const int32_t padPairs = (pitch - g.wout) / 2;
        for (int32_t i = tid; i < nRows * padPairs; i += nt) {
            const int32_t r = i / padPairs, k = i - r * padPairs;
            *reinterpret_cast<float2*>(sRow0 + r * pitch + (k < kX2Pad / 2 ? 2 * k : g.wout + 2 * k)) = make_float2(0.0f, 0.0f);
        }
        const T* pg = go + plane * (static_cast<int64_t>(g.hout) * g.wout) + static_cast<int64_t>(hLo) * g.wout;
        float* sBase = sRow0 + kX2Pad;
        // a thread keeps its position in a row and steps over rows: one division per thread instead of one per load
        if (vecLoad) {
            constexpr int VL = 16 / sizeof(T);
            const int32_t packs = g.wout / VL;
            const int32_t lanesPerRow = min(packs, nt), rowsPerPass = nt / lanesPerRow;
            const int32_t r0 = tid / lanesPerRow, p0 = tid - r0 * lanesPerRow;
            if (r0 < rowsPerPass) {
                for (int32_t r = r0; r < nRows; r += rowsPerPass) {
                    for (int32_t p = p0; p < packs; p += lanesPerRow) {
                        float v[VL];
                        LoadPackLdg<T, VL>(pg + r * g.wout + p * VL, v);
                        float4* dst = reinterpret_cast<float4*>(sBase + r * pitch + p * VL);
#pragma unroll
                        for (int m = 0; m < VL / 4; ++m) {
                            dst[m] = make_float4(v[4 * m], v[4 * m + 1], v[4 * m + 2], v[4 * m + 3]);
                        }
                    }
                }
            }
        } else {
            const int32_t lanesPerRow = min(g.wout, nt), rowsPerPass = nt / lanesPerRow;
            const int32_t r0 = tid / lanesPerRow, w0 = tid - r0 * lanesPerRow;
            if (r0 < rowsPerPass) {
                for (int32_t r = r0; r < nRows; r += rowsPerPass) {
                    for (int32_t w = w0; w < g.wout; w += lanesPerRow) {
                        sBase[r * pitch + w] = DType<T>::Load(pg + r * g.wout + w);
                    }
                }
            }
        }
    }
    __syncthreads();

    const int32_t pairs = (g.win + 1) / 2;
    const int32_t bandN = yhB - yhA;
    const int32_t nPair = bandN * pairs;
    const int32_t borderBase = (nPair + 31) & ~31;      // first columns from here, one per row of the band
    const int32_t borderBase1 = borderBase + ((bandN + 31) & ~31); // last columns: other warps, so that the slot
    const int32_t total = borderBase1 + bandN;                 // tests below are uniform over a warp
    T* pgi = gi + (plane * g.hin + yhA) * g.win;
    for (int32_t item = tid; item < total; item += nt) {
        if (item < nPair) {
            const int32_t r = item / pairs, q = item - r * pairs;
            const int32_t yh = yhA + r;
            const float* sw = sG + 4 * q; // grads column 4q - 4
            float a0 = 0.0f, a1 = 0.0f;
            if (yh != 0 && yh != g.hin - 1) {
                const float4* row = reinterpret_cast<const float4*>(sw + (2 * yh - 3 - hBase) * pitch);
#pragma unroll
                for (int j = 0; j < 8; ++j, row += pitch / 4) {
                    { // rows above or below the image are zero rows: their terms add nothing
                        const float4 A = row[0], B = row[1], C = row[2];
                        const float v[12] = {A.x, A.y, A.z, A.w, B.x, B.y, B.z, B.w, C.x, C.y, C.z, C.w};
                        float gc[10];
#pragma unroll
                        for (int k = 0; k < 10; ++k) {
                            gc[k] = Mul(v[1 + k], c[j]);
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            a0 = Add(a0, Mul(gc[k], c[k]));
                            a1 = Add(a1, Mul(gc[2 + k], c[k]));
                        }
                    }
                }
            } else {
                const X2BorderList& rows = sL[yh == 0 ? 2 : 3];
                const uint32_t mask = rows.mask;
#pragma unroll 1
                for (int m = 0; m < kX2Groups; ++m) {
                    const uint32_t bits = (mask >> (m * kX2Slots)) & 7u;
                    if (bits == 0) {
                        continue;
                    }
                    const float ch0 = rows.coef[m * kX2Slots], ch1 = rows.coef[m * kX2Slots + 1],
                                ch2 = rows.coef[m * kX2Slots + 2];
                    const float4* row = reinterpret_cast<const float4*>(sw + (rows.start + m - hBase) * pitch);
                    const float4 A = row[0], B = row[1], C = row[2];
                    const float v[12] = {A.x, A.y, A.z, A.w, B.x, B.y, B.z, B.w, C.x, C.y, C.z, C.w};
#pragma unroll
                    for (int k = 0; k < 8; ++k) { // slots fill in tap order, so bit 0 is set whenever the group is
                        a0 = Add(a0, Mul(Mul(v[1 + k], ch0), c[k]));
                        a1 = Add(a1, Mul(Mul(v[3 + k], ch0), c[k]));
                        if (bits & 2u) {
                            a0 = Add(a0, Mul(Mul(v[1 + k], ch1), c[k]));
                            a1 = Add(a1, Mul(Mul(v[3 + k], ch1), c[k]));
                        }
                        if (bits & 4u) {
                            a0 = Add(a0, Mul(Mul(v[1 + k], ch2), c[k]));
                            a1 = Add(a1, Mul(Mul(v[3 + k], ch2), c[k]));
                        }
                    }
                }
            }
            T* po = pgi + static_cast<int64_t>(r) * g.win;
            const int32_t yw0 = 2 * q;
            if (yw0 >= 1 && yw0 <= g.win - 2) {
                po[yw0] = DType<T>::FromF(a0);
            }
            if (yw0 + 1 <= g.win - 2) {
                po[yw0 + 1] = DType<T>::FromF(a1);
            }
        } else if (item >= borderBase) {
            // a first or last column of an interior row: the terms of its walk as one list
            const int32_t side = item >= borderBase1 ? 1 : 0;
            const int32_t r = item - (side ? borderBase1 : borderBase);
            if (r >= bandN) {
                continue;
            }
            const int32_t yh = yhA + r;
            if (yh == 0 || yh == g.hin - 1) {
                continue; // the four corners of a plane: the corner blocks
            }
            const X2BorderList& cols = sL[side];
            float add = 0.0f;
            int32_t wI[kX2Flat];
            float cw[kX2Flat];
#pragma unroll
            for (int e = 0; e < kX2Flat; ++e) {
                wI[e] = cols.flatIdx[e];
                cw[e] = cols.flatCoef[e];
            }
            const float* prow = sG + (2 * yh - 3 - hBase) * pitch + kX2Pad;
#pragma unroll
            for (int j = 0; j < 8; ++j, prow += pitch) {
#pragma unroll
                for (int e = 0; e < kX2Flat; ++e) {
                    add = Add(add, Mul(Mul(prow[wI[e]], c[j]), cw[e]));
                }
            }
            pgi[static_cast<int64_t>(r) * g.win + (side ? g.win - 1 : 0)] = DType<T>::FromF(add);
        }
    }
}

// ---- forward at exactly 2x (half-pixel coordinates, scales 0.5), NCHW ---------------------------------------------
// Output index 2i has the source coordinate i - 0.25 (window i - 2 .. i + 1, fraction 0.75), output index 2i + 1 has
// i + 0.25 (window i - 1 .. i + 2, fraction 0.25), all exact: two sets of four coefficients serve the whole image
// and come from the host. A block stages the source rows of a band (with the two rows above and below it, clamped)
// as fp32 with replicated columns either side, so that neither pass clamps an index; pass A forms the
// horizontal sums of every staged row, eight adjacent output columns per thread from eight source values (four
// 8-byte shared-memory loads, two 16-byte stores); pass B gives a thread four adjacent columns of the four output rows
// of two source rows: six 16-byte loads of sums, four stores. Sums and products in the order of the general kernels.
struct X2FwdCoef {
    float even[4]; // FwdCoeff(0.75): output indices 2i
    float odd[4];  // FwdCoeff(0.25): output indices 2i + 1
};

// FULL: every group of four output columns is whole and every row 8- or 16-byte aligned (one store per group).
template <typename T, bool FULL>
__global__ void __launch_bounds__(kX2Threads) Bicubic2dFwdX2Kernel(const T* __restrict__ x, T* __restrict__ y, BicubicGeom g,
                                                                   int32_t bandRows, int32_t bands, int32_t vecIn,
                                                                   int32_t vecOut, const X2FwdCoef cf, const FastDiv halfPacks,
                                                                   const FastDiv packsDiv)
{
    extern __shared__ __align__(16) float sm[];
    const int32_t tid = threadIdx.x, nt = blockDim.x;
    const int32_t pitchX = g.win + 4 + (g.win & 1); // two replicated columns left, two or three right (even pitch)
    const int32_t packs = (g.wout + 3) / 4, pitchH = 4 * packs; // an odd input width leaves the last pack half used
    const int64_t plane = blockIdx.x / bands;
    const int32_t band = static_cast<int32_t>(blockIdx.x - plane * bands);
    const int32_t rA = band * bandRows, rB = min(rA + bandRows, g.hin);
    const int32_t nSlots = rB - rA + 4; // slot s holds source row clamp(rA - 2 + s)
    float* sX = sm;
    float* sH = sm + (((bandRows + 4) * pitchX + 3) & ~3);
    const T* px = x + plane * (static_cast<int64_t>(g.hin) * g.win);
    {
        for (int32_t i = tid; i < 2 * nSlots; i += nt) { // the replicated columns
            const int32_t sl = i >> 1, right = i & 1;
            const int32_t row = ClampIdx32(rA - 2 + sl, g.hin - 1);
            const float v = DType<T>::Load(px + static_cast<int64_t>(row) * g.win + (right ? g.win - 1 : 0));
            if (right) {
                for (int32_t k = g.win + 2; k < pitchX; ++k) {
                    sX[sl * pitchX + k] = v;
                }
            } else {
                *reinterpret_cast<float2*>(sX + sl * pitchX) = make_float2(v, v);
            }
        }
        if (vecIn) {
            constexpr int VL = 16 / sizeof(T);
            const int32_t packs = g.win / VL;
            const int32_t lanesPerRow = min(packs, nt), rowsPerPass = nt / lanesPerRow;
            const int32_t s0 = tid / lanesPerRow, p0 = tid - s0 * lanesPerRow;
            if (s0 < rowsPerPass) {
                for (int32_t sl = s0; sl < nSlots; sl += rowsPerPass) {
                    const T* prow = px + static_cast<int64_t>(ClampIdx32(rA - 2 + sl, g.hin - 1)) * g.win;
                    for (int32_t pk = p0; pk < packs; pk += lanesPerRow) {
                        float v[VL];
                        LoadPackLdg<T, VL>(prow + pk * VL, v);
                        float2* dst = reinterpret_cast<float2*>(sX + sl * pitchX + 2 + pk * VL);
#pragma unroll
                        for (int m = 0; m < VL / 2; ++m) {
                            dst[m] = make_float2(v[2 * m], v[2 * m + 1]);
                        }
                    }
                }
            }
        } else {
            const int32_t lanesPerRow = min(g.win, nt), rowsPerPass = nt / lanesPerRow;
            const int32_t s0 = tid / lanesPerRow, w0 = tid - s0 * lanesPerRow;
            if (s0 < rowsPerPass) {
                for (int32_t sl = s0; sl < nSlots; sl += rowsPerPass) {
                    const T* prow = px + static_cast<int64_t>(ClampIdx32(rA - 2 + sl, g.hin - 1)) * g.win;
                    for (int32_t w = w0; w < g.win; w += lanesPerRow) {
                        sX[sl * pitchX + 2 + w] = DType<T>::Load(prow + w);
                    }
                }
            }
        }
    }
    __syncthreads();
    // Both passes use the packed fp32 operations: two sums that share their coefficients go through one instruction
    // per product and per addition (AddProduct2 keeps the product's own rounding), so the bits are the scalar ones.
    const F2 E0 = MakeF2(cf.even[0], cf.even[0]), E1 = MakeF2(cf.even[1], cf.even[1]), E2 = MakeF2(cf.even[2], cf.even[2]),
             E3 = MakeF2(cf.even[3], cf.even[3]);
    const F2 O0 = MakeF2(cf.odd[0], cf.odd[0]), O1 = MakeF2(cf.odd[1], cf.odd[1]), O2 = MakeF2(cf.odd[2], cf.odd[2]),
             O3 = MakeF2(cf.odd[3], cf.odd[3]);
    // ((t0 c0 + t1 c1) + t2 c2) + t3 c3 on both halves
    auto blend = [](F2 t0, F2 t1, F2 t2, F2 t3, F2 c0, F2 c1, F2 c2, F2 c3) {
        F2 acc = AddProduct2(Mul2(t1, c1), Mul2(t0, c0));
        acc = AddProduct2(Mul2(t2, c2), acc);
        return AddProduct2(Mul2(t3, c3), acc);
    };
    // pass A: eight adjacent sums of a staged row from eight source values (the second four only where they exist).
    // Output columns 4q and 4q + 2 share the even coefficients and have windows one source pixel apart, 4q + 1 and
    // 4q + 3 likewise with the odd ones: each pair is one packed chain, and a group of four sums is stored in the
    // order (0, 2, 1, 3), which pass B undoes when it stores.
    for (int32_t item = tid; item < nSlots * static_cast<int32_t>(halfPacks.d); item += nt) {
        const int32_t sl = DivBy(item, halfPacks), q = 2 * (item - sl * static_cast<int32_t>(halfPacks.d));
        if (sl >= nSlots || q >= packs) {
            continue; // cannot happen for item below the bound; keeps a wrong quotient from leaving the tiles
        }
        const float2* src = reinterpret_cast<const float2*>(sX + sl * pitchX + 2 * q); // source columns 2q - 2 ..
        const float2 a = src[0], b = src[1], c = src[2];
        const F2 A = MakeF2(a.x, a.y), B = MakeF2(b.x, b.y), C = MakeF2(c.x, c.y);
        const F2 AB = MakeF2(a.y, b.x), BC = MakeF2(b.y, c.x);
        F2* dst = reinterpret_cast<F2*>(sH + sl * pitchH + 4 * q);
        struct alignas(16) Quad {
            F2 lo, hi;
        };
        Quad h;
        h.lo = blend(A, AB, B, BC, E0, E1, E2, E3);  // columns 4q, 4q + 2
        h.hi = blend(AB, B, BC, C, O0, O1, O2, O3);  // columns 4q + 1, 4q + 3
        *reinterpret_cast<Quad*>(dst) = h;
        if (q + 1 < packs) {
            const float2 d = src[3];
            const F2 D = MakeF2(d.x, d.y), CD = MakeF2(c.y, d.x);
            h.lo = blend(B, BC, C, CD, E0, E1, E2, E3);
            h.hi = blend(BC, C, CD, D, O0, O1, O2, O3);
            *reinterpret_cast<Quad*>(dst + 2) = h;
        }
    }
    __syncthreads();
    // pass B: four adjacent columns of the four output rows of two source rows (two where the band ends)
    T* py = y + (plane * g.hout + 2 * rA) * static_cast<int64_t>(g.wout);
    const int32_t rows = rB - rA;
    const int32_t step = packs;
    // lo = columns (0, 2), hi = columns (1, 3) of the group; valid = columns of the group inside the row (4, or 2 in
    // the last group of a row whose width is not a multiple of 4); vecOut = elements per store the rows allow
    auto store = [&](T* dst, F2 lo, F2 hi, int32_t valid) {
        float vals[4];
        SplitF2(lo, vals[0], vals[2]);
        SplitF2(hi, vals[1], vals[3]);
        if (FULL) {
            StorePack<T, 4>(dst, vals);
        } else if (vecOut == 2) {
            const float a[2] = {vals[0], vals[1]}, b[2] = {vals[2], vals[3]};
            StorePack<T, 2>(dst, a);
            if (valid > 2) {
                StorePack<T, 2>(dst + 2, b);
            }
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                if (v < valid) {
                    dst[v] = DType<T>::FromF(vals[v]);
                }
            }
        }
    };
    for (int32_t item = tid; item < ((rows + 1) / 2) * packs; item += nt) {
        const int32_t r2 = DivBy(item, packsDiv), q = item - r2 * packs;
        const int32_t r = 2 * r2;
        if (r >= rows || q < 0 || q >= packs) {
            continue; // as in pass A
        }
        const float4* col = reinterpret_cast<const float4*>(sH + r * pitchH + 4 * q); // slots r .. r + 5
        const float4 R0 = col[0], R1 = col[step], R2 = col[2 * step], R3 = col[3 * step], R4 = col[4 * step];
        const F2 l0 = MakeF2(R0.x, R0.y), h0 = MakeF2(R0.z, R0.w), l1 = MakeF2(R1.x, R1.y), h1 = MakeF2(R1.z, R1.w),
                 l2 = MakeF2(R2.x, R2.y), h2 = MakeF2(R2.z, R2.w), l3 = MakeF2(R3.x, R3.y), h3 = MakeF2(R3.z, R3.w),
                 l4 = MakeF2(R4.x, R4.y), h4 = MakeF2(R4.z, R4.w);
        T* dst = py + static_cast<int64_t>(2 * r) * g.wout + 4 * q;
        const int32_t valid = FULL ? 4 : min(4, g.wout - 4 * q);
        store(dst, blend(l0, l1, l2, l3, E0, E1, E2, E3), blend(h0, h1, h2, h3, E0, E1, E2, E3), valid);
        store(dst + g.wout, blend(l1, l2, l3, l4, O0, O1, O2, O3), blend(h1, h2, h3, h4, O0, O1, O2, O3), valid);
        if (r + 1 < rows) {
            const float4 R5 = col[5 * step];
            const F2 l5 = MakeF2(R5.x, R5.y), h5 = MakeF2(R5.z, R5.w);
            store(dst + 2 * g.wout, blend(l1, l2, l3, l4, E0, E1, E2, E3), blend(h1, h2, h3, h4, E0, E1, E2, E3), valid);
            store(dst + 3 * g.wout, blend(l2, l3, l4, l5, O0, O1, O2, O3), blend(h2, h3, h4, h5, O0, O1, O2, O3), valid);
        }
    }
}

// Band height and block size of the 2x kernel. false: the kernel does not apply.
struct X2Launch {
    int32_t bandRows, bands, threads, pitch;
    size_t smem;
};
bool PlanBwdX2(const BicubicGeom& g, bool nhwc, X2Launch* out)
{
    if (nhwc || g.align || g.scaleH != 0.5f || g.scaleW != 0.5f || g.invH != 2.0f || g.invW != 2.0f ||
        g.hin < 2 || g.win < 2 || g.hout != 2 * g.hin || g.wout != 2 * g.win || g.wout > (1 << 20)) {
        return false;
    }
    const int32_t pitch = (g.wout + 12 + 3) & ~3;
    const int32_t pairs = (g.win + 1) / 2;
    // Bands as tall as 32 KB of staged rows allow (measured at 56 x 56 planes: taller bands stage fewer halo rows and
    // pay the per-block set-up less often, 301 us at 28 rows against 337 us at 14; a whole plane per block, 58 KB,
    // leaves too few blocks per SM: 341 us), equal over the plane; then the block size that wastes the fewest warp
    // slots over the passes of the item loop.
    const size_t rowBytes = static_cast<size_t>(pitch) * sizeof(float);
    int32_t bh = static_cast<int32_t>(std::min<int64_t>((32 * 1024 / rowBytes - 6) / 2, g.hin));
    if (bh < 1) {
        bh = 1;
    }
    if ((2 * bh + 6) * rowBytes > 48 * 1024) {
        return false;
    }
    const int32_t nb = (g.hin + bh - 1) / bh;
    bh = (g.hin + nb - 1) / nb;
    const int64_t warpItems = CeilDiv(static_cast<int64_t>(bh) * pairs, 32) + 2 * CeilDiv(bh, 32);
    double best = 0.0;
    for (int32_t threads = 128; threads <= kX2Threads; threads += 32) {
        const int64_t warps = threads / 32;
        const double fill = static_cast<double>(warpItems) / static_cast<double>(CeilDiv(warpItems, warps) * warps);
        if (fill > best) { // ties go to the smaller block: more blocks per SM to overlap staging with arithmetic
            best = fill;
            *out = X2Launch{bh, nb, threads, pitch, (2 * bh + 6) * rowBytes};
        }
    }
    const int64_t planes = g.rows / g.hin;
    return planes * out->bands + 4 * CeilDiv(planes, out->threads) <= INT32_MAX;
}

dim3 RowGrid(int64_t rows, int64_t inner)
{
    const int64_t gx = std::min<int64_t>(std::max<int64_t>(CeilDiv(inner, kThreads), 1), 64);
    const int64_t cap = std::max<int64_t>(static_cast<int64_t>(NumSMs()) * 16 / gx, 1);
    const int64_t gy = std::min<int64_t>(std::max<int64_t>(rows, 1), std::min<int64_t>(cap, 65535));
    return dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy), 1);
}

// ---- launch shapes of the general backward ------------------------------------------------------------------------
// A launch of `positions` element positions per row, lists of `bytes` per column, `threads` threads per block. Columns of one
// list: four source pixels for an interior column, two and a half for a first or last one (three, for user scales). Lists that
// would not fit make their thread fall back to the uncached walk, so the bound only has to be good, not safe; a
// single-column image (every grads column is a tap) always falls back.
ListShape PlanBwdList(const BicubicGeom& g, int64_t positions, int bytes, int threads, double span)
{
    const double perScale = g.invW > 0.0f ? static_cast<double>(g.invW) : 1.0;
    const int64_t maxW = static_cast<int64_t>(std::ceil(span * perScale)) + 4;
    const int64_t cap = (bytes == kInteriorBytes ? 96 : 192) * 1024 / (bytes * threads);
    ListShape l;
    l.colsPB = static_cast<int32_t>(std::min<int64_t>(threads, positions));
    const int rowsPB = threads / l.colsPB;
    l.entries = static_cast<int32_t>(std::max<int64_t>(4, std::min<int64_t>(maxW, cap)));
    l.x = static_cast<int32_t>(CeilDiv(positions, l.colsPB));
    const int64_t gyCap = std::max<int64_t>(static_cast<int64_t>(NumSMs()) * 32 / l.x, 1);
    l.y = static_cast<int32_t>(std::min<int64_t>(std::min<int64_t>(CeilDiv(g.rows, rowsPB), gyCap), 65535));
    return l;
}
size_t ListSmem(const ListShape& l, int bytes, int threads)
{
    return static_cast<size_t>(l.entries) * threads * bytes;
}

// The list kernel alone.
struct BwdListPlan {
    ListShape border, interior;
    int32_t threads;
    int64_t blocks;
    size_t smem;
};
BwdListPlan PlanBwdLists(const BicubicGeom& g)
{
    const int64_t inner = static_cast<int64_t>(g.win) * g.chan;
    BwdListPlan p{};
    if (g.win <= 2) {
        p.threads = kListThreads;
        p.border = PlanBwdList(g, inner, kListBytes, p.threads, 4.0);
    } else {
        // equal shares of a row for its blocks, so that none of them is nearly empty, and no more threads than that needs:
        // fewer threads leave room for longer lists
        const int64_t positions = inner - 2LL * g.chan, share = CeilDiv(positions, CeilDiv(positions, kListThreads));
        p.threads = static_cast<int32_t>(std::max<int64_t>(64, (share + 31) / 32 * 32));
        p.border = PlanBwdList(g, 2LL * g.chan, kListBytes, p.threads, 3.0);
        p.interior = PlanBwdList(g, positions, kInteriorBytes, p.threads, 4.0);
        p.blocks = static_cast<int64_t>(p.interior.x) * p.interior.y;
        p.smem = ListSmem(p.interior, kInteriorBytes, p.threads);
    }
    p.blocks += static_cast<int64_t>(p.border.x) * p.border.y;
    p.smem = std::max(p.smem, ListSmem(p.border, kListBytes, p.threads));
    return p;
}

// Interior columns by the row walk, the two border columns apart; false where the list kernel serves the call.
struct BwdWalkPlan {
    WalkShape ws;
    int64_t bands, blocks;
    size_t smem;
};
bool PlanBwdWalk(const BicubicGeom& g, BwdWalkPlan* plan)
{
    constexpr size_t kMostSmem = 48 * 1024; // four blocks per SM
    const int64_t inner = static_cast<int64_t>(g.win) * g.chan;
    const double perScale = g.invW > 0.0f ? static_cast<double>(g.invW) : 1.0;
    // columns of the longest interior walk: 4 / scale within two source pixels either side, one more for rounding
    const int64_t walk = static_cast<int64_t>(std::ceil(4.0 * perScale)) + 1;
    // The bound on open rows holds while the start of a walk (from the inverse scale) and its end (from the scale) speak of
    // the same positions: a quarter of a source pixel for the two scales, another quarter for the rounding of positions up to
    // 2^20 rows and 2^22 grads rows. The last row's walk runs to the end of the grads, which a user scale can put anywhere.
    const double rowsPerRow = g.invH;
    const double drift = g.invH > 0.0f && g.scaleH > 0.0f ? std::fabs(static_cast<double>(g.scaleH) * g.invH - 1.0) *
                                                                (static_cast<double>(g.hin) + 2.0 * rowsPerRow + 4.0)
                                                          : 1.0;
    if (walk > 17 || g.win <= 2 || g.hin <= 2 || g.hin > (1 << 20) || g.hout > (1 << 22) || !(drift < 0.25) ||
        !(8.0 * rowsPerRow + 8.0 < kWalkMaxRows) ||
        !(static_cast<double>(g.hout) <= (static_cast<double>(g.hin) + 2.0) * rowsPerRow + 2.0)) {
        return false;
    }
    const int64_t planes = g.rows / g.hin;
    const ListShape l = PlanBwdList(g, 2LL * g.chan, kListBytes, kListThreads, 4.0);
    WalkShape& ws = plan->ws;
    ws = WalkShape{};
    ws.positions = planes * (inner - 2LL * g.chan);
    const int64_t gx = CeilDiv(ws.positions, kWalkThreads);
    // grads rows of a band: four source pixels beyond it, and the rounding of its ends
    auto bandReads = [&](int64_t band) { return static_cast<int64_t>((static_cast<double>(band) + 5.0) * rowsPerRow) + 4; };
    // shared memory: a record per grads row, start and end of every row of the band (which are what fills it where a band
    // reads few rows, in a strong vertical down-scale)
    auto bandSmem = [&](int64_t band) { return static_cast<size_t>(bandReads(band)) * sizeof(WalkRecord) + static_cast<size_t>(band) * 8; };
    // Bands: every band re-reads four source pixels' worth of grads rows; fewer than five blocks per SM leave each of them
    // waiting on its own loads (about 0.25 us a row), more share the issue slots (about 0.06 us a row). A tall plane needs
    // more than 256 of them for its records to fit (fp32 1x40000x64 <- 160000x256: 247 us, by lists 1352).
    double bestTime = 0.0;
    for (int64_t b = 1; b <= g.hin && (b <= 256 || g.hin / b >= 16); b += b < 256 ? 1 : b / 16) {
        const int64_t band = CeilDiv(g.hin, b);
        const int64_t reads = bandReads(band);
        if (reads > kWalkMaxRows || bandSmem(band) > kMostSmem) {
            continue;
        }
        const double k = static_cast<double>(CeilDiv(gx * CeilDiv(g.hin, band), NumSMs()));
        const double time = (static_cast<double>(reads) + 8.0) * std::max(0.25 * std::ceil(k / 5.0), 0.06 * k);
        if (ws.bandRows == 0 || time < bestTime * 0.98) {
            ws.bandRows = static_cast<int32_t>(band);
            bestTime = time;
        }
    }
    if (ws.bandRows == 0) {
        return false;
    }
    plan->bands = CeilDiv(g.hin, ws.bandRows);
    plan->blocks = gx * plan->bands + static_cast<int64_t>(l.x) * l.y;
    if (plan->blocks > INT32_MAX) {
        return false;
    }
    ws.maxRows = static_cast<int32_t>(bandReads(ws.bandRows));
    ws.walkX = static_cast<int32_t>(gx);
    ws.list = l;
    plan->smem = std::max(ListSmem(l, kListBytes, kListThreads), bandSmem(ws.bandRows));
    return true;
}

BicubicGeom BwdGeom(Layout lay, const Shape4& sh, float scaleH, float scaleW, float invH, float invW, bool align)
{
    const bool nhwc = lay == kNHWC;
    BicubicGeom g;
    g.rows = (nhwc ? sh.n : sh.n * sh.c) * sh.hin;
    g.hin = sh.hin;
    g.win = sh.win;
    g.hout = sh.hout;
    g.wout = sh.wout;
    g.chan = nhwc ? static_cast<int32_t>(sh.c) : 1;
    g.scaleH = scaleH;
    g.scaleW = scaleW;
    g.invH = invH;
    g.invW = invW;
    g.align = align ? 1 : 0;
    g.schedule = 0;
    return g;
}

} // namespace

cudaError_t Bicubic2dFwd(Dt dt, Layout lay, const void* x, void* y, Shape4 sh, float scaleH, float scaleW,
                         bool halfPixel, int32_t schedule, cudaStream_t s)
{
    const bool nhwc = lay == kNHWC;
    const int64_t planes = nhwc ? sh.n : sh.n * sh.c;
    BicubicGeom g;
    g.rows = planes * sh.hout;
    g.hin = sh.hin;
    g.win = sh.win;
    g.hout = sh.hout;
    g.wout = sh.wout;
    g.chan = nhwc ? static_cast<int32_t>(sh.c) : 1;
    g.scaleH = scaleH;
    g.scaleW = scaleW;
    g.invH = g.invW = 0.0f;
    g.align = halfPixel ? 0 : 1;
    g.schedule = schedule;
    const int64_t inner = static_cast<int64_t>(g.wout) * g.chan;
    if (schedule != 0) {
        const dim3 grid = RowGrid(g.rows, inner);
        OPSCV_DISPATCH_DT(dt, T, {
            if (nhwc) {
                Bicubic2dFwdCopyKernel<T, true><<<grid, kThreads, 0, s>>>(static_cast<const T*>(x), static_cast<T*>(y), g);
            } else {
                Bicubic2dFwdCopyKernel<T, false><<<grid, kThreads, 0, s>>>(static_cast<const T*>(x), static_cast<T*>(y), g);
            }
        });
        CountLaunch();
        return cudaGetLastError();
    }
    if (!nhwc && halfPixel && scaleH == 0.5f && scaleW == 0.5f && g.hout == 2 * g.hin && g.wout == 2 * g.win &&
        g.win <= (1 << 20)) {
        // exactly 2x: bands of source rows whose staged rows and horizontal sums take about 32 KB
        const size_t pitchX = static_cast<size_t>(g.win) + 4 + (g.win & 1), pitchH = (static_cast<size_t>(g.wout) + 3) / 4 * 4;
        const size_t slotBytes = (pitchX + pitchH) * sizeof(float);
        int32_t bh = static_cast<int32_t>(std::min<int64_t>(static_cast<int64_t>(32 * 1024 / slotBytes) - 4, g.hin));
        bh = std::max(bh, 1);
        const int32_t nb = (g.hin + bh - 1) / bh;
        bh = (g.hin + nb - 1) / nb;
        const size_t smem = ((static_cast<size_t>(bh + 4) * pitchX + 3) / 4 * 4 + static_cast<size_t>(bh + 4) * pitchH) * sizeof(float);
        if (smem <= 48 * 1024 && planes * nb <= INT32_MAX) {
            X2FwdCoef cf;
            x2host::FwdCoeff(0.75f, cf.even);
            x2host::FwdCoeff(0.25f, cf.odd);
            const int threads = 128; // measured at 56 x 56 planes: 101 us against 109 us with 256 (more blocks per SM overlap the three phases)
            OPSCV_DISPATCH_DT(dt, T, {
                const int vecIn = (g.win % (16 / sizeof(T)) == 0 && Aligned(x, 16)) ? 1 : 0;
                const int vecOut = (g.wout % 4 == 0 && Aligned(y, 4 * sizeof(T))) ? 4 : (Aligned(y, 2 * sizeof(T)) ? 2 : 1);
                auto k = vecOut == 4 ? Bicubic2dFwdX2Kernel<T, true> : Bicubic2dFwdX2Kernel<T, false>;
                k<<<static_cast<unsigned>(planes * nb), threads, smem, s>>>(
                    static_cast<const T*>(x), static_cast<T*>(y), g, bh, nb, vecIn, vecOut, cf,
                    MakeFastDiv(static_cast<uint32_t>(((g.wout + 3) / 4 + 1) / 2)), MakeFastDiv(static_cast<uint32_t>((g.wout + 3) / 4)));
            });
            CountLaunch();
            return cudaGetLastError();
        }
    }
    if (!nhwc) {
        // the shared-memory tile form: the largest band of output rows whose tiles fit 64 KB
        const int es = DtSize(dt);
        int v = 16 / es;
        while (v > 1 && (g.wout % v != 0 || !Aligned(y, static_cast<size_t>(v) * es))) {
            v >>= 1;
        }
        std::vector<int32_t> top(static_cast<size_t>(g.hout));
        for (int32_t H = 0; H < g.hout; ++H) {
            top[H] = FwdTop(H, g.scaleH, g.align, g.hin, nullptr);
        }
        auto clampRow = [&](int32_t r) { return std::min(std::max(r, 0), g.hin - 1); };
        BicubicTile tile{};
        size_t smem = 0;
        for (int32_t band = g.hout; band >= 4; band = (band + 1) / 2) {
            int32_t worst = 0;
            for (int32_t h0 = 0; h0 < g.hout; h0 += band) {
                const int32_t h1 = std::min(h0 + band, g.hout);
                worst = std::max(worst, clampRow(top[h1 - 1] + 2) - clampRow(top[h0] - 1) + 1);
            }
            const size_t need = (static_cast<size_t>(worst) * (static_cast<size_t>(g.wout) + g.win) + 5u * band) * sizeof(float);
            if (need <= 64u * 1024u) {
                tile.bandRows = band;
                tile.bands = static_cast<int32_t>(CeilDiv(g.hout, band));
                tile.maxSrc = worst;
                smem = need;
                break;
            }
            if (band == 4) {
                break;
            }
        }
        // a band must still be long enough to amortise the three extra source rows it loads
        if (smem != 0 && (tile.bandRows >= 16 || tile.bands == 1)) {
            int tw = 1; // one thread per pair of columns in the horizontal pass
            while (tw < (g.wout + 1) / 2 && tw < kThreads) {
                tw <<= 1;
            }
            int pw = 1;
            while (pw < g.wout / v && pw < kThreads) {
                pw <<= 1;
            }
            tile.tw = tw;
            tile.pw = pw;
            const int64_t items = planes * tile.bands;
            const int64_t perSm = std::max<int64_t>(1, std::min<int64_t>(8, (200u * 1024u) / smem));
            const unsigned grid = static_cast<unsigned>(std::min<int64_t>(items, static_cast<int64_t>(NumSMs()) * perSm * 4));
            cudaError_t attr = cudaSuccess;
            OPSCV_DISPATCH_DT(dt, T, {
                const T* px = static_cast<const T*>(x);
                T* py = static_cast<T*>(y);
                OPSCV_DISPATCH_VEC(v, V, {
                    if constexpr (V * sizeof(T) <= 16) {
                        if (smem > 48u * 1024u) {
                            attr = cudaFuncSetAttribute(Bicubic2dFwdTileKernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        static_cast<int>(smem));
                        }
                        if (attr == cudaSuccess) {
                            Bicubic2dFwdTileKernel<T, V><<<grid, kThreads, smem, s>>>(px, py, g, tile, items);
                        }
                    }
                });
            });
            if (attr != cudaSuccess) {
                return attr;
            }
            CountLaunch();
            return cudaGetLastError();
        }
    }
    // Two elements per thread for 16-bit tensors (4-byte stores) when rows allow it. Bands: enough (plane, band)
    // items to fill the device a few times over, but at least 16 output rows each, since every band starts by
    // computing four horizontal sums afresh.
    const int v = (DtSize(dt) == 2 && inner % 2 == 0 && Aligned(y, 4)) ? 2 : 1;
    // a block as wide as the row when the row is short, so that no warp of it is idle
    const int threads = static_cast<int>(std::min<int64_t>(kThreads, (CeilDiv(inner, v) + 31) / 32 * 32));
    const int64_t colBlocks = CeilDiv(CeilDiv(inner, v), threads);
    const int64_t want = static_cast<int64_t>(NumSMs()) * 8 * 4;
    int64_t bands = std::max<int64_t>(1, std::min<int64_t>(CeilDiv(want, std::max<int64_t>(planes * colBlocks, 1)),
                                                           std::max<int32_t>(sh.hout / 16, 1)));
    int32_t bandRows = static_cast<int32_t>(CeilDiv(sh.hout, bands));
    bandRows = std::min<int32_t>(bandRows, 2048); // 40 KB of row coefficients at most
    bands = CeilDiv(sh.hout, bandRows);
    const size_t smem = static_cast<size_t>(bandRows) * 5 * sizeof(float);
    g.rows = planes * bands;
    const dim3 grid(static_cast<unsigned>(colBlocks), static_cast<unsigned>(std::min<int64_t>(g.rows, 65535)), 1);
    OPSCV_DISPATCH_DT(dt, T, {
        const T* px = static_cast<const T*>(x);
        T* py = static_cast<T*>(y);
        if (nhwc) {
            if (v == 2) {
                Bicubic2dFwdKernel<T, true, 2><<<grid, threads, smem, s>>>(px, py, g, bandRows, static_cast<int32_t>(bands));
            } else {
                Bicubic2dFwdKernel<T, true, 1><<<grid, threads, smem, s>>>(px, py, g, bandRows, static_cast<int32_t>(bands));
            }
        } else {
            if (v == 2) {
                Bicubic2dFwdKernel<T, false, 2><<<grid, threads, smem, s>>>(px, py, g, bandRows, static_cast<int32_t>(bands));
            } else {
                Bicubic2dFwdKernel<T, false, 1><<<grid, threads, smem, s>>>(px, py, g, bandRows, static_cast<int32_t>(bands));
            }
        }
    });
    CountLaunch();
    return cudaGetLastError();
}

cudaError_t Bicubic2dBwd(Dt dt, Layout lay, const void* go, void* gi, Shape4 sh, float scaleH, float scaleW,
                         float invH, float invW, bool align, cudaStream_t s)
{
    const bool nhwc = lay == kNHWC;
    const BicubicGeom g = BwdGeom(lay, sh, scaleH, scaleW, invH, invW, align);
    const double perScale = invW > 0.0f ? static_cast<double>(invW) : 1.0;
    cudaError_t err = cudaSuccess;
    auto launchList = [&]() {
        const BwdListPlan l = PlanBwdLists(g);
        OPSCV_DISPATCH_DT(dt, T, {
            auto kernel = nhwc ? Bicubic2dBwdListKernel<T, true> : Bicubic2dBwdListKernel<T, false>;
            if (l.smem > 48 * 1024) {
                err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(l.smem));
            }
            if (err == cudaSuccess) {
                kernel<<<static_cast<unsigned>(l.blocks), l.threads, l.smem, s>>>(
                    static_cast<const T*>(go), static_cast<T*>(gi), g, l.border, l.interior);
            }
        });
        CountLaunch();
    };
    X2Launch x2;
    X2BorderLists lists;
    bool useX2 = PlanBwdX2(g, nhwc, &x2);
    if (useX2) {
        lists.l[0] = x2host::BorderList(0, g.win, g.wout);
        lists.l[1] = x2host::BorderList(g.win - 1, g.win, g.wout);
        lists.l[2] = x2host::BorderList(0, g.hin, g.hout);
        lists.l[3] = x2host::BorderList(g.hin - 1, g.hin, g.hout);
        for (const X2BorderList& l : lists.l) {
            useX2 = useX2 && l.terms <= kX2Flat;
        }
        for (int k = 0; k < 8; ++k) {
            lists.interior[k] = x2host::PointCoeff(std::fabs(0.5f * static_cast<float>(k) - 1.75f));
        }
    }
    if (useX2) {
        const int64_t planes = g.rows / g.hin;
        OPSCV_DISPATCH_DT(dt, T, {
            const int vec = (g.wout % (16 / sizeof(T)) == 0 && Aligned(go, 16)) ? 1 : 0;
            const int32_t cornerBlocks = 4 * static_cast<int32_t>(CeilDiv(planes, x2.threads));
            Bicubic2dBwdX2Kernel<T><<<static_cast<unsigned>(planes * x2.bands + cornerBlocks), x2.threads, x2.smem, s>>>(
                static_cast<const T*>(go), static_cast<T*>(gi), g, x2.bandRows, x2.bands, x2.pitch, vec, lists, planes,
                cornerBlocks);
        });
        CountLaunch();
        return cudaGetLastError();
    }
    BwdWalkPlan plan;
    if (!PlanBwdWalk(g, &plan)) {
        launchList();
        return err != cudaSuccess ? err : cudaGetLastError();
    }
    OPSCV_DISPATCH_DT(dt, T, {
        auto launch = [&](auto columns) {
            constexpr int K = decltype(columns)::value;
            auto kernel = nhwc ? Bicubic2dBwdWalkKernel<T, true, K> : Bicubic2dBwdWalkKernel<T, false, K>;
            if (plan.smem > 48 * 1024) {
                err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(plan.smem));
            }
            if (err == cudaSuccess) {
                kernel<<<static_cast<unsigned>(plan.blocks), kWalkThreads, plan.smem, s>>>(
                    static_cast<const T*>(go), static_cast<T*>(gi), g, plan.ws);
            }
        };
        // A walk spans four source pixels: at most ceil(4 / scale) columns, with a margin for rounding (a column whose walk is
        // longer all the same takes the uncached walk).
        const int64_t columns = static_cast<int64_t>(std::ceil(4.0 * perScale + 0.02));
        if (columns <= 6) {
            launch(std::integral_constant<int, 6>{});
        } else if (columns <= 8) {
            launch(std::integral_constant<int, 8>{});
        } else if (columns <= 10) {
            launch(std::integral_constant<int, 10>{});
        } else if (columns <= 12) {
            launch(std::integral_constant<int, 12>{});
        } else if (columns <= 14) {
            launch(std::integral_constant<int, 14>{});
        } else {
            launch(std::integral_constant<int, 18>{});
        }
    });
    CountLaunch();
    return err != cudaSuccess ? err : cudaGetLastError();
}

bool DebugBicubic2dBwd(Layout lay, Shape4 sh, float scaleH, float scaleW, float invH, float invW, bool align, int64_t values[8])
{
    const BicubicGeom g = BwdGeom(lay, sh, scaleH, scaleW, invH, invW, align);
    X2Launch x2;
    BwdWalkPlan p;
    if (PlanBwdX2(g, lay == kNHWC, &x2) || !PlanBwdWalk(g, &p)) {
        return false;
    }
    const int64_t v[8] = {p.ws.bandRows, p.ws.maxRows, kOpen, 0, 0, 0, p.bands, static_cast<int64_t>(p.smem)};
    std::copy(v, v + 8, values);
    return true;
}

} // namespace opscv
