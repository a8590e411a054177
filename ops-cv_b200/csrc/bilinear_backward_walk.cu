// UpsampleBilinear2dBackward, the row walks that serve up-scales by whole factors or not, up to where the grads of one group
// (below) no longer fit the shared memory of a block: NCHW rows of 4096 grads columns at small factors, of fp32 2048 at a
// factor of eight and 1280 at sixteen; NHWC a factor of about ten.
//
// Both kernels use the same view of an axis: lo(d), the lower of the two grad_input indices that grads index d feeds,
// grows with d, so the grads indices with lo = y form one run ("group" y). grad_input index y is fed by group y - 1
// (through the upper tap, weight delta) and by group y (through the lower tap, weight 1 - delta); the last index gets
// both taps of its own group. A thread that walks down the grads rows therefore keeps two sums open, the row of the
// current group and the next one, and a row is finished when its group ends. Indices and weights are evaluated where
// they are needed with the expressions of LerpEntry (variant 1): no table launch precedes these kernels.
//
//   * NCHW (BilinearBwdColumnsKernel): vertical sums first. A thread owns V adjacent grads columns and reads every
//     grads row of its band exactly once, in whole coalesced lines; a finished row of vertical sums goes to shared
//     memory and the block reduces it horizontally. Work per grads element does not grow with the scale.
//   * NHWC (BilinearBwdNHWCWalkKernel): a thread owns 16 bytes of channels of one grad_input column, reads the grads
//     pixels that feed the column and adds the reference scatter kernel's products in its serial order, so the bits are
//     those of the scatter; each grads pixel is read by the two columns that it feeds, next to each other in one block.
//
// Reference arithmetic: image/resize_bilinear_v2_grad/op_kernel/arch35/resize_bilinear_v2_grad_simt.h:107-152.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cp_async.cuh"
#include "launch_util.cuh"

namespace opscv {
namespace {

// One axis of the scatter: grads index d reads source position (d + offset) * scale - offset.
struct BwdAxis {
    float scale, offset;
    int32_t last; // grad_input extent - 1
    int32_t out;  // grads extent
};

BwdAxis MakeAxis(const AxisGeom& g, bool halfPixel)
{
    return BwdAxis{g.scale, halfPixel ? 0.5f : 0.0f, g.in - 1, g.out};
}

// Host and device evaluate the same single-precision operations (host code is compiled without contraction).
__host__ __device__ __forceinline__ float BwdPosition(const BwdAxis& a, int32_t d)
{
#ifdef __CUDA_ARCH__
    const float src = Sub(Mul(Add(static_cast<float>(d), a.offset), a.scale), a.offset);
#else
    const float scaled = (static_cast<float>(d) + a.offset) * a.scale;
    const float src = scaled - a.offset;
#endif
    return src < 0.0f ? 0.0f : src;
}
__host__ __device__ __forceinline__ int32_t BwdLower(const BwdAxis& a, int32_t d)
{
#ifdef __CUDA_ARCH__
    return min(__float2int_rd(BwdPosition(a, d)), a.last);
#else
    const float lo = std::floor(BwdPosition(a, d));
    return lo < static_cast<float>(a.last) ? static_cast<int32_t>(lo) : a.last;
#endif
}
__device__ __forceinline__ float BwdDelta(const BwdAxis& a, int32_t d)
{
    const float src = BwdPosition(a, d);
    const int32_t lo = min(__float2int_rd(src), a.last);
    return fminf(fmaxf(Sub(src, static_cast<float>(lo)), 0.0f), 1.0f);
}
// First grads index whose lower tap is y or more (0 for y <= 0, the extent if there is none): a guess from the inverse
// of the position formula, set right by stepping.
__host__ __device__ __forceinline__ int32_t GroupStart(const BwdAxis& a, int32_t y)
{
    if (y <= 0) {
        return 0;
    }
    if (y > a.last) {
        return a.out;
    }
#ifdef __CUDA_ARCH__
    const float guess = __fdividef(static_cast<float>(y) + a.offset, a.scale) - a.offset;
#else
    const float guess = (static_cast<float>(y) + a.offset) / a.scale - a.offset;
#endif
    int32_t d = guess > 0.0f ? (guess < static_cast<float>(a.out) ? static_cast<int32_t>(guess) : a.out) : 0;
    while (d > 0 && BwdLower(a, d - 1) >= y) {
        --d;
    }
    while (d < a.out && BwdLower(a, d) < y) {
        ++d;
    }
    return d;
}

// V sums of a thread. Pairs are kept packed for the whole walk: as scalars that are packed around every operation they
// cost a register move per operand (counted on the NHWC kernel: 80 of its 320 instructions per row and warp).
template <int V>
struct Sums {
    static constexpr int kPairs = V / 2;
    F2 p[kPairs > 0 ? kPairs : 1];
    float s; // V == 1
    __device__ __forceinline__ void Clear()
    {
#pragma unroll
        for (int k = 0; k < kPairs; ++k) {
            p[k] = MakeF2(0.0f, 0.0f);
        }
        s = 0.0f;
    }
    __device__ __forceinline__ void Get(float (&v)[V]) const
    {
        if constexpr (V == 1) {
            v[0] = s;
        } else {
#pragma unroll
            for (int k = 0; k < kPairs; ++k) {
                SplitF2(p[k], v[2 * k], v[2 * k + 1]);
            }
        }
    }
    // += w * v, fused
    __device__ __forceinline__ void Fma(F2 w, float w1, const float (&v)[V])
    {
        if constexpr (V == 1) {
            s = fmaf(w1, v[0], s);
        } else {
#pragma unroll
            for (int k = 0; k < kPairs; ++k) {
                p[k] = Fma2(w, MakeF2(v[2 * k], v[2 * k + 1]), p[k]);
            }
        }
    }
};

struct ColumnsShape {
    int32_t hin, win, hout, wout;
    int32_t planesPerBlock;
    int32_t team;        // threads of a plane: thread k owns grads columns k, k + team, ...
    int32_t bandRows;    // grad_input rows per block
    int32_t dRowCap;     // most grads rows any band reads
    int32_t stageGroups; // groups per stage of the ring
    int32_t stages;      // of the ring: 2 or 3
    int32_t slotBytes;   // bytes of a stage of one plane
    int32_t lanesLog;    // log2 of the lanes that share one horizontal sum
};
constexpr int kColumnsBatch = 4; // parked rows that are reduced together

size_t ColumnsSmem(const ColumnsShape& q)
{
    return static_cast<size_t>(q.stages) * q.planesPerBlock * q.slotBytes +
           4 * (static_cast<size_t>(2 * q.stageGroups * q.planesPerBlock + 1) * q.wout + (q.win + 2) +
                (q.bandRows + q.stageGroups + 3) + q.dRowCap);
}

// grid = (plane groups, bands); block = the teams of its planes, K grads columns per thread, and one warp more that
// copies. The grads rows stream through a ring of stages in shared memory, each the rows of stageGroups groups:
// one run of memory per plane, copied in 16-byte pieces whatever its alignment (a slot keeps the run's offset within its
// first 16 bytes). The finished rows of vertical sums of a stage are parked in one of two buffers and reduced behind the
// barrier that the next stage needs anyway: one barrier per stage.
template <typename TIn, typename TOut, int K>
__global__ void __launch_bounds__(544, 2)
    BilinearBwdColumnsKernel(const TIn* __restrict__ go, TOut* __restrict__ gi, int64_t planes, ColumnsShape q,
                             BwdAxis ah, BwdAxis aw)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int32_t stageBytes = q.planesPerBlock * q.slotBytes;
    float* buf = reinterpret_cast<float*>(smemRaw + q.stages * stageBytes); // [2][groups][planes][wout]
    const int32_t rowFloats = q.planesPerBlock * q.wout, bufFloats = q.stageGroups * rowFloats;
    float* dCol = buf + 2 * bufFloats;                                             // upper-tap weights of the columns
    int32_t* xStart = reinterpret_cast<int32_t*>(dCol + q.wout);                   // group starts of columns -1 .. win
    int32_t* yStart = xStart + q.win + 2;                                          // group starts of rows ya - 1 .. yb
    float* dRow = reinterpret_cast<float*>(yStart + q.bandRows + q.stageGroups + 3); // upper-tap weights of the rows

    const int32_t tid = threadIdx.x, nthreads = blockDim.x;
    const int64_t pBase = static_cast<int64_t>(blockIdx.x) * q.planesPerBlock;
    const int32_t np = static_cast<int32_t>(min(static_cast<int64_t>(q.planesPerBlock), planes - pBase));
    const int32_t ya = blockIdx.y * q.bandRows, yb = min(q.hin, ya + q.bandRows);
    // groups of rows ya - 1 .. yb - 1, then empty ones up to a whole stage
    const int32_t groups = yb - ya + 1, stages = (groups + q.stageGroups - 1) / q.stageGroups;
    for (int32_t k = tid; k <= stages * q.stageGroups; k += nthreads) {
        yStart[k] = GroupStart(ah, min(ya - 1 + k, yb));
    }
    for (int32_t k = tid; k < q.win + 2; k += nthreads) {
        xStart[k] = GroupStart(aw, k - 1);
    }
    for (int32_t j = tid; j < q.wout; j += nthreads) {
        dCol[j] = BwdDelta(aw, j);
    }
    __syncthreads();
    const int32_t is = yStart[0], ie = yStart[groups];
    for (int32_t i = tid; i < ie - is; i += nthreads) {
        dRow[i] = BwdDelta(ah, is + i);
    }
    const int32_t rowBytes = q.wout * static_cast<int32_t>(sizeof(TIn));
    const char* first = reinterpret_cast<const char*>(go);

    if (tid >= nthreads - 32) { // the copying warp
        const int32_t lane = tid & 31;
        const char* end = reinterpret_cast<const char*>(go + planes * q.hout * q.wout);
        const int64_t planeBytes = static_cast<int64_t>(q.hout) * rowBytes;
        const char* run0 = first + pBase * planeBytes + static_cast<int64_t>(is) * rowBytes;
        int32_t slot = 0;
        auto issue = [&](int32_t st) {
            if (st < stages) {
                const int32_t rows = yStart[(st + 1) * q.stageGroups] - yStart[st * q.stageGroups];
                const char* run = run0;
                uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smemRaw)) + slot * stageBytes + 16 * lane;
                for (int32_t p = 0; p < np && rows > 0; ++p, run += planeBytes, d += q.slotBytes) {
                    const int32_t mis = static_cast<int32_t>(reinterpret_cast<uintptr_t>(run) & 15);
                    const int32_t granules = (mis + rows * rowBytes + 15) >> 4;
                    const char* a = run - mis + 16 * lane;
                    if (run - mis >= first && run - mis + 16 * static_cast<int64_t>(granules) <= end) {
                        for (int32_t g = lane; g < granules; g += 32) {
                            CpAsync16(d + 16 * (g - lane), a);
                            a += 512;
                        }
                    } else { // the first or the last run of the tensor: no 16-byte piece reaches past its ends
                        for (int32_t g = lane; g < granules; g += 32, a += 512) {
                            if (a >= first && a + 16 <= end) {
                                CpAsync16(d + 16 * (g - lane), a);
                                continue;
                            }
                            TIn* e = reinterpret_cast<TIn*>(smemRaw + slot * stageBytes + p * q.slotBytes + 16 * g);
                            for (int32_t b = 0; b < 16 / static_cast<int32_t>(sizeof(TIn)); ++b) {
                                const char* v = a + b * sizeof(TIn);
                                if (v >= first && v < end) {
                                    e[b] = *reinterpret_cast<const TIn*>(v);
                                }
                            }
                        }
                    }
                }
                run0 += static_cast<int64_t>(rows) * rowBytes;
            }
            slot = slot + 1 == q.stages ? 0 : slot + 1;
            CpAsyncCommit();
        };
        for (int32_t st = 0; st < q.stages - 1; ++st) {
            issue(st);
        }
        for (int32_t st = 0; st < stages; ++st) {
            if (q.stages == 2) {
                CpAsyncWait<0>();
            } else {
                CpAsyncWait<1>();
            }
            __syncthreads(); // stage st has arrived, and everyone is done with stage st - 1
            issue(st + q.stages - 1);
        }
        __syncthreads();
        return;
    }

    const int32_t pl = tid / q.team, k0 = tid - pl * q.team;
    const bool active = pl < np;
    const uint32_t planeLow =
        static_cast<uint32_t>(reinterpret_cast<uintptr_t>(go + (pBase + (active ? pl : 0)) * q.hout * q.wout));
    const unsigned char* ring = smemRaw + (active ? pl : 0) * q.slotBytes;
    int32_t colByte[K]; // offsets of this thread's columns in a row; columns past the row repeat its last one
#pragma unroll
    for (int m = 0; m < K; ++m) {
        colByte[m] = min(k0 + m * q.team, q.wout - 1) * static_cast<int32_t>(sizeof(TIn));
    }
    float* mine = buf + (active ? pl : 0) * q.wout + k0;

    // Horizontal sums: item (plane, column) goes to `lanes` adjacent threads. A thread nearly always has one item at
    // most (the host picks K no larger than the scale): its window and, where they are few, its weights stay in registers.
    const int32_t workers = nthreads - 32;
    const int32_t lanes = 1 << q.lanesLog, sub = tid & (lanes - 1);
    const int32_t items = np * q.win;
    struct Window {
        int32_t at;           // first column, in the parked row
        int32_t col;          // first column
        int32_t count, upper; // columns of this lane: all, and those of group x - 1
        TOut* out;
        bool last;
    };
    auto window = [&](int32_t item) {
        Window w;
        const int32_t p = item / q.win, x = item - p * q.win;
        w.col = xStart[x] + sub;
        w.count = max(0, (xStart[x + 2] - w.col + lanes - 1) >> q.lanesLog);
        w.upper = max(0, (xStart[x + 1] - w.col + lanes - 1) >> q.lanesLog);
        w.at = p * q.wout + w.col;
        w.out = gi + ((pBase + p) * q.hin + ya) * static_cast<int64_t>(q.win) + x;
        w.last = x == aw.last;
        return w;
    };
    auto reduce = [&](const Window& w, const float* parked) {
        float a = 0.0f;
        const float* v = parked + w.at;
        const float* d = dCol + w.col;
        int32_t t = 0;
        for (; t < w.upper; ++t, v += lanes, d += lanes) { // group x - 1: upper taps
            a = fmaf(*d, *v, a);
        }
        if (!w.last) {
            for (; t < w.count; ++t, v += lanes, d += lanes) { // group x: lower taps
                a = fmaf(Sub(1.0f, *d), *v, a);
            }
        } else { // the last column takes both taps of its group
            for (; t < w.count; ++t, v += lanes, d += lanes) {
                a = fmaf(Sub(1.0f, *d), *v, a);
                a = fmaf(*d, *v, a);
            }
        }
        return a;
    };
    // Two columns per thread go with scales of two to four, where a sum has six or seven taps up to a scale of three (bf16 400
    // planes 100x130 <- 187x383: 80 us by tiles, 88 with five held, 60 with seven); with one it has five at most.
    constexpr int kHeld = K == 2 ? 7 : 5, kBatch = kColumnsBatch;
    const bool hasItem = (tid >> q.lanesLog) < items;
    const bool warpHasItems = ((tid & ~31) >> q.lanesLog) < items;
    const bool moreRounds = (items << q.lanesLog) > workers;
    Window own{};
    if (hasItem) {
        own = window(tid >> q.lanesLog);
    }
    const bool few = own.count <= kHeld && lanes == 1;
    float held[kHeld];
    uint32_t twins = 0; // taps of the last column with a second weight of exactly zero: 0 * Inf must still give NaN
#pragma unroll
    for (int t = 0; t < kHeld; ++t) {
        held[t] = 0.0f;
        if (t < own.count && few) {
            const float d = dCol[own.col + t];
            held[t] = t < own.upper ? d : Sub(1.0f, d);
            if (own.last && t >= own.upper) { // both taps
                held[t] = Add(held[t], d);
                twins |= d == 0.0f || d == 1.0f ? 1u << t : 0u;
            }
        }
    }
    const bool allFew = __all_sync(0xffffffffu, few);
    // the rows parked by one stage, y0 = row of the first within the band
    auto horizontal = [&](const float* parked, int32_t y0, int32_t count) {
        if (!warpHasItems) {
            return;
        }
        if (allFew && count == kBatch) { // a whole stage of rows: each tap's test and weight serve all of them
            float a[kBatch];
#pragma unroll
            for (int y = 0; y < kBatch; ++y) {
                a[y] = 0.0f;
            }
            const float* v = parked + own.at;
#pragma unroll
            for (int t = 0; t < kHeld; ++t) {
                if (t < own.count) {
#pragma unroll
                    for (int y = 0; y < kBatch; ++y) {
                        a[y] = fmaf(held[t], v[y * rowFloats + t], a[y]);
                    }
                }
            }
            if (twins != 0) {
                for (int32_t t = 0; t < own.count; ++t) {
                    for (int y = 0; y < kBatch && ((twins >> t) & 1u) != 0; ++y) {
                        a[y] = fmaf(0.0f, v[y * rowFloats + t], a[y]);
                    }
                }
            }
#pragma unroll
            for (int y = 0; y < kBatch; ++y) {
                if (hasItem) {
                    own.out[y * static_cast<int64_t>(q.win)] = DType<TOut>::FromF(a[y]);
                }
            }
            own.out += kBatch * static_cast<int64_t>(q.win);
            if (!moreRounds) {
                return;
            }
        }
        const bool ownDone = allFew && count == kBatch;
        for (int32_t y = y0; y < y0 + count; ++y, parked += rowFloats) {
            if (!ownDone) {
                float a = reduce(own, parked);
                for (int32_t m = lanes >> 1; m > 0; m >>= 1) {
                    a += __shfl_xor_sync(0xffffffffu, a, m);
                }
                if (hasItem && sub == 0) {
                    *own.out = DType<TOut>::FromF(a);
                }
                own.out += q.win;
            }
            if (moreRounds) {
                for (int32_t idx = tid + workers; idx - (tid & 31) < (items << q.lanesLog); idx += workers) {
                    const bool valid = (idx >> q.lanesLog) < items;
                    Window w{};
                    if (valid) {
                        w = window(idx >> q.lanesLog);
                    }
                    float b = reduce(w, parked);
                    for (int32_t m = lanes >> 1; m > 0; m >>= 1) {
                        b += __shfl_xor_sync(0xffffffffu, b, m);
                    }
                    if (valid && sub == 0) {
                        w.out[static_cast<int64_t>(y) * q.win] = DType<TOut>::FromF(b);
                    }
                }
            }
        }
    };

    Sums<K> lo, hi;
    lo.Clear();
    hi.Clear();
    int32_t slot = 0, half = 0;
    int32_t parkedFirst = 0, parkedRows = 0; // rows (within the band) parked by the stage before
    int32_t row = is, rowEnd = is;
    const float* d = dRow;
    for (int32_t st = 0; st < stages; ++st) {
        __syncthreads(); // the stage has arrived, and the parked rows of the stage before are whole
        horizontal(buf + (bufFloats - half), parkedFirst, parkedRows);
        const unsigned char* src =
            ring + slot * stageBytes + ((planeLow + static_cast<uint32_t>(row) * static_cast<uint32_t>(rowBytes)) & 15u);
        parkedRows = 0;
        float* park = mine + half;
        const int32_t g1 = min((st + 1) * q.stageGroups, groups);
        for (int32_t grp = st * q.stageGroups; grp < g1; ++grp) { // the group of grad_input row ya - 1 + grp
            rowEnd = yStart[grp + 1];
            const bool last = ya - 1 + grp == ah.last;
            auto addRow = [&](const unsigned char* at, float wHi) {
                const float wLo = Sub(1.0f, wHi);
                float v[K];
#pragma unroll
                for (int m = 0; m < K; ++m) {
                    v[m] = DType<TIn>::ToF(*reinterpret_cast<const TIn*>(at + colByte[m]));
                }
                lo.Fma(MakeF2(wLo, wLo), wLo, v);
                if (!last) {
                    hi.Fma(MakeF2(wHi, wHi), wHi, v);
                } else { // the last row takes both taps of its group
                    lo.Fma(MakeF2(wHi, wHi), wHi, v);
                }
            };
#pragma unroll 1
            for (; row + 2 <= rowEnd; row += 2, src += 2 * rowBytes, d += 2) {
                addRow(src, d[0]);
                addRow(src + rowBytes, d[1]);
            }
            if (row < rowEnd) {
                addRow(src, d[0]);
                ++row;
                src += rowBytes;
                ++d;
            }
            if (grp > 0) { // grad_input row ya - 1 + grp is finished
                float sums[K];
                lo.Get(sums);
#pragma unroll
                for (int m = 0; m < K; ++m) {
                    if (active && k0 + m * q.team < q.wout) {
                        park[m * q.team] = sums[m];
                    }
                }
                park += rowFloats;
                ++parkedRows;
            }
            lo = hi;
            hi.Clear();
        }
        parkedFirst = max(st * q.stageGroups - 1, 0);
        half = bufFloats - half;
        slot = slot + 1 == q.stages ? 0 : slot + 1;
    }
    __syncthreads();
    horizontal(buf + (bufFloats - half), parkedFirst, parkedRows);
}

// One weight applied to one grads pixel: acc += (wx * wy) * v with the reference's three roundings, wx and wy in both
// halves. FUSE: the host has checked that the product with any value of the grads type is exact, so one fused
// multiply-add gives the bits.
template <int V, bool FUSE>
__device__ __forceinline__ void AddTap(Sums<V>& acc, F2 wx, F2 wy, const float (&v)[V])
{
    const F2 w = Mul2(wx, wy);
#pragma unroll
    for (int k = 0; k < V / 2; ++k) {
        const F2 x = MakeF2(v[2 * k], v[2 * k + 1]);
        acc.p[k] = FUSE ? Fma2(w, x, acc.p[k]) : AddProduct2(Mul2(w, x), acc.p[k]);
    }
}

struct WalkShape {
    int32_t groups; // channel vectors of a pixel
    int32_t hin, win, hout, wout;
    int32_t slice;     // channel vectors per block
    int32_t tileX;     // grad_input columns per block
    int32_t images;    // images per block
    int32_t bandRows;  // grad_input rows per block
    int32_t segPixels; // most grads pixels of a row that any tile reads
    int32_t stageRows; // most grads rows per stage of the ring
    int32_t dRowCap;   // most grads rows any band reads
};
constexpr int kWalkStages = 3;
constexpr int kWalkThreads = 224; // and a copying warp: four blocks of 64 registers a thread per SM

size_t WalkSmem(const WalkShape& q)
{
    return static_cast<size_t>(kWalkStages) * q.stageRows * q.images * q.segPixels * q.slice * 16 +
           4 * (static_cast<size_t>(q.bandRows) + 3 + q.dRowCap + q.segPixels);
}

// grid = (channel slices x column tiles, image groups, bands). A thread owns one 16-byte channel vector of one
// grad_input column; one warp more copies the grads pixels that the block's columns read, stageRows rows of a group at a
// time, into a ring in shared memory (every pixel crosses from L2 once per block).
template <typename T, typename TOut, bool FUSE>
__global__ void __launch_bounds__(kWalkThreads + 32, 4)
    BilinearBwdNHWCWalkKernel(const T* __restrict__ go, TOut* __restrict__ gi, int64_t n, WalkShape q, BwdAxis ah,
                              BwdAxis aw)
{
    constexpr int V = 16 / sizeof(T);
    constexpr int kHeld = 4; // column weights kept in registers: all of them up to a scale of about 2
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int32_t segment = q.segPixels * q.slice; // 16-byte vectors of one row of one image
    const int32_t imageVecs = q.stageRows * segment, stageVecs = q.images * imageVecs;
    uint4* ring = reinterpret_cast<uint4*>(smemRaw);
    int32_t* yStart = reinterpret_cast<int32_t*>(ring + kWalkStages * stageVecs); // group starts of rows ya - 1 .. yb
    float* dRow = reinterpret_cast<float*>(yStart + q.bandRows + 3);              // upper-tap weights of the grads rows
    float* dPix = dRow + q.dRowCap;                                               // and of the tile's grads columns

    const int32_t tiles = static_cast<int32_t>(CeilDiv(q.win, q.tileX));
    const int32_t tile = blockIdx.x % tiles, firstGroup = blockIdx.x / tiles * q.slice;
    const int32_t xa = tile * q.tileX, xb = min(q.win, xa + q.tileX);
    const int32_t ya = blockIdx.z * q.bandRows, yb = min(q.hin, ya + q.bandRows), rowGroups = yb - ya + 1;
    const int32_t ja = GroupStart(aw, xa - 1), pixels = GroupStart(aw, xb) - ja;
    for (int32_t k = threadIdx.x; k <= rowGroups; k += blockDim.x) {
        yStart[k] = GroupStart(ah, ya - 1 + k);
    }
    for (int32_t p = threadIdx.x; p < pixels; p += blockDim.x) {
        dPix[p] = BwdDelta(aw, ja + p);
    }
    __syncthreads();
    const int32_t is = yStart[0], count = yStart[rowGroups] - is;
    for (int32_t i = threadIdx.x; i < count; i += blockDim.x) {
        dRow[i] = BwdDelta(ah, is + i);
    }
    const int64_t pixelElems = static_cast<int64_t>(q.groups) * V, rowElems = q.wout * pixelElems;
    const int64_t image0 = static_cast<int64_t>(blockIdx.y) * q.images;

    if (threadIdx.x >= blockDim.x - 32) { // the copying warp
        const int32_t lane = threadIdx.x & 31;
        const int32_t images = static_cast<int32_t>(min(static_cast<int64_t>(q.images), n - image0));
        const int32_t vecs = min(q.slice, q.groups - firstGroup);
        const uint32_t ringAt = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
        const int64_t imageBytes = q.hout * rowElems * static_cast<int64_t>(sizeof(T));
        const int64_t rowBytes = rowElems * static_cast<int64_t>(sizeof(T)), pixelBytes = q.groups * 16;
        const char* next = reinterpret_cast<const char*>(go) + image0 * imageBytes + is * rowBytes + ja * pixelBytes +
                           firstGroup * 16;
        int32_t group = 0, row = is, slot = 0;
        auto issue = [&]() {
            while (group + 1 < rowGroups && row >= yStart[group + 1]) {
                ++group;
            }
            const int32_t rows = max(0, min(q.stageRows, yStart[group + 1] - row));
            for (int32_t im = 0; im < images; ++im) {
                const char* a = next + im * imageBytes;
                uint32_t d = ringAt + static_cast<uint32_t>(slot * stageVecs + im * imageVecs) * 16u;
                for (int32_t r = 0; r < rows; ++r, a += rowBytes, d += static_cast<uint32_t>(segment) * 16u) {
                    if (vecs == q.groups) { // whole pixels: one run of memory
                        const char* v = a + 16 * lane;
                        uint32_t e = d + 16u * lane;
#pragma unroll 4
                        for (int32_t g = lane; g < pixels * vecs; g += 32, v += 512, e += 512) {
                            CpAsync16(e, v);
                        }
                    } else {
                        const char* v = a + 16 * lane;
                        uint32_t e = d + 16u * lane;
                        for (int32_t p = 0; p < pixels && lane < vecs; ++p, v += pixelBytes, e += 16u * q.slice) {
                            CpAsync16(e, v);
                        }
                    }
                }
            }
            CpAsyncCommit();
            row += rows;
            next += rows * rowBytes;
            slot = slot + 1 == kWalkStages ? 0 : slot + 1;
        };
        for (int st = 0; st < kWalkStages - 1; ++st) {
            issue();
        }
        for (int32_t k = 0; k < rowGroups; ++k) {
            for (int32_t i = yStart[k]; i < yStart[k + 1]; i += q.stageRows) {
                CpAsyncWait<kWalkStages - 2>();
                __syncthreads(); // the stage has arrived, and everyone is done with the one before
                issue();
            }
        }
        return;
    }

    const int32_t perImage = q.tileX * q.slice;
    const int32_t img = threadIdx.x / perImage, in = threadIdx.x - img * perImage;
    const int32_t xl = in / q.slice, g = in - xl * q.slice, x = xa + xl;
    const bool active = img < q.images && image0 + img < n && firstGroup + g < q.groups && x < xb;
    const int32_t js = GroupStart(aw, x - 1), jm = GroupStart(aw, x), taps = active ? GroupStart(aw, x + 1) - js : 0;
    const int32_t upperTaps = jm - js;
    const bool lastCol = x == aw.last;
    F2 wx[kHeld];
#pragma unroll
    for (int t = 0; t < kHeld; ++t) {
        const float d = BwdDelta(aw, js + t), w = js + t < jm ? d : Sub(1.0f, d);
        wx[t] = MakeF2(w, w);
    }
    const uint4* firstTap = ring + (active ? img * imageVecs + (js - ja) * q.slice + g : 0);
    const float* tapWeight = dPix + (active ? js - ja : 0);
    TOut* dst = gi + (((image0 + img) * q.hin + ya) * q.win + x) * pixelElems + static_cast<int64_t>(firstGroup + g) * V;
    const int64_t dstStep = q.win * pixelElems;
    const bool four = taps == kHeld && !lastCol;
    const float* d = dRow;
    const uint4* stageAt = firstTap;
    int32_t slot = 0;
    Sums<V> even, odd; // the open rows: they trade places from group to group
    even.Clear();
    odd.Clear();
    // the rows of group k: into `lo` (grad_input row ya - 1 + k, which it finishes) and `hi` (the next row)
    auto walkGroup = [&](int32_t k, Sums<V>& lo, Sums<V>& hi) {
        int32_t rows = yStart[k + 1] - yStart[k];
        const bool lastRow = ya - 1 + k == ah.last;
        while (rows > 0) {
            const int32_t part = min(rows, q.stageRows);
            __syncthreads();
            const uint4* row = stageAt;
            for (int32_t r = 0; r < part; ++r, row += segment) {
                const float upper = *d++, lower = Sub(1.0f, upper);
                const F2 wLo = MakeF2(lower, lower), wHi = MakeF2(upper, upper);
                if (four && !lastRow) {
                    uint4 raw[kHeld];
#pragma unroll
                    for (int t = 0; t < kHeld; ++t) {
                        raw[t] = row[t * q.slice];
                    }
#pragma unroll
                    for (int t = 0; t < kHeld; ++t) {
                        float v[V];
                        UnpackToF<T, V>(reinterpret_cast<const Pack<T, V>&>(raw[t]), v);
                        AddTap<V, FUSE>(lo, wx[t], wLo, v);
                        AddTap<V, FUSE>(hi, wx[t], wHi, v);
                    }
                } else {
                    // any number of taps; the last column and the last row take both taps of their group: up to four
                    // products of a pixel, in the order TL, TR, BL, BR of the scatter
                    const uint4* at = row;
#pragma unroll 1
                    for (int32_t t = 0; t < taps; ++t, at += q.slice) {
                        const bool twin = lastCol && t >= upperTaps;
                        const float dx1 = tapWeight[t], w1 = t < upperTaps ? dx1 : Sub(1.0f, dx1);
                        const F2 dx = MakeF2(dx1, dx1), w = MakeF2(w1, w1);
                        const uint4 raw = *at;
                        float v[V];
                        UnpackToF<T, V>(reinterpret_cast<const Pack<T, V>&>(raw), v);
                        AddTap<V, FUSE>(lo, w, wLo, v);
                        if (twin) {
                            AddTap<V, FUSE>(lo, dx, wLo, v);
                        }
                        if (lastRow) {
                            AddTap<V, FUSE>(lo, w, wHi, v);
                            if (twin) {
                                AddTap<V, FUSE>(lo, dx, wHi, v);
                            }
                        } else {
                            AddTap<V, FUSE>(hi, w, wHi, v);
                            if (twin) {
                                AddTap<V, FUSE>(hi, dx, wHi, v);
                            }
                        }
                    }
                }
            }
            rows -= part;
            ++slot;
            stageAt += stageVecs;
            if (slot == kWalkStages) {
                slot = 0;
                stageAt = firstTap;
            }
        }
        if (k > 0 && active) {
            float out[V];
            lo.Get(out);
            StorePack<TOut, V>(dst, out);
            dst += dstStep;
        }
        lo.Clear();
    };
#pragma unroll 1
    for (int32_t k = 0; k < rowGroups; k += 2) {
        walkGroup(k, even, odd);
        if (k + 1 < rowGroups) {
            walkGroup(k + 1, odd, even);
        }
    }
}

// A user scale that runs past the input makes one long group of the last index; the direct kernels serve it.
bool Overshoots(const BwdAxis& a)
{
    const int64_t lastGroup = a.out - static_cast<int64_t>(GroupStart(a, a.last));
    return static_cast<float>(lastGroup) > 1.0f / a.scale + 2.0f && a.last > 0;
}

// Most grads indices that `groups` adjacent groups hold: the ends of the axis, where indices are clamped, exactly;
// elsewhere the integers in an interval of groups / scale, widened at both ends by the rounding of the positions.
// In units of an index, index + offset is off by nothing below 2^23 and by 1/2 below 2^24, the product and the difference by
// index * 2^-24 each: together at most 1/2 below 2^22, 5/2 below 2^24. From there on indices share a position and no such
// bound holds.
constexpr int32_t kMostExtent = 1 << 24;
int32_t MostRows(const BwdAxis& a, int32_t groups)
{
    const double inner = groups / static_cast<double>(a.scale) + (a.out <= kMostExtent / 4 ? 2.0 : 6.0);
    const int32_t most = inner < a.out ? static_cast<int32_t>(inner) : a.out;
    return std::max({most, GroupStart(a, groups), a.out - GroupStart(a, a.last - groups + 1)});
}

// Rows of a band: the blocks of all bands run in waves of `slots` resident blocks, and a band costs its own rows, one
// more group of grads rows and its start (about two rows). Tall planes are cut into more than 64 bands while a band keeps
// eight rows: a few images of one would leave most SMs idle and each block a long walk (fp32 NHWC 1x100000x4x8 <- 250000x9:
// 2663 us in 64 bands).
int32_t PickBandRows(int32_t rows, int64_t blocksPerBand, int64_t slots)
{
    int32_t best = rows;
    double bestCost = 1e30;
    for (int32_t bands = 1; bands <= rows && (bands <= 64 || rows / bands >= 8); bands += bands < 64 ? 1 : bands / 16) {
        const int32_t r = static_cast<int32_t>(CeilDiv(rows, bands));
        const double cost = static_cast<double>(CeilDiv(blocksPerBand * CeilDiv(rows, r), slots)) * (r + 3);
        if (cost < bestCost) {
            bestCost = cost;
            best = r;
        }
    }
    return static_cast<int32_t>(std::max<int64_t>(best, CeilDiv(rows, 65535)));
}

// Launch shape of the column kernel.
struct ColumnsPlan {
    ColumnsShape q;
    int32_t k, threads, bands; // columns per thread
    int64_t planeGroups;
    size_t smem;
};
constexpr int32_t kColumnsThreads = 256; // per block, to aim for

// With so many planes per block; false where that needs more than mostSmem bytes of shared memory.
bool PlanColumnsOf(int32_t planesPerBlock, size_t mostSmem, int es, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw,
                   ColumnsPlan* plan)
{
    const int64_t planes = sh.n * sh.c;
    ColumnsShape& q = plan->q;
    q = ColumnsShape{};
    q.hin = sh.hin;
    q.win = sh.win;
    q.hout = sh.hout;
    q.wout = sh.wout;
    q.team = static_cast<int32_t>(CeilDiv(sh.wout, plan->k));
    q.planesPerBlock = planesPerBlock;
    const int32_t threads = static_cast<int32_t>(CeilDiv(q.planesPerBlock * q.team, 32)) * 32 + 32; // and the copying warp
    const int64_t planeGroups = CeilDiv(planes, q.planesPerBlock);
    // about eight grads rows per stage, no more than some twelve kilobytes of them; three stages unless they are large
    const int32_t rowBytes = sh.wout * es;
    const float perGroup = std::max(1.0f / ah.scale, 1.0f);
    q.stageGroups = static_cast<int32_t>(std::min(8.0f, 12288.0f / (static_cast<float>(rowBytes) * q.planesPerBlock)) / perGroup);
    q.stageGroups = std::max(1, std::min(q.stageGroups, kColumnsBatch));
    const int64_t slotBytes = (static_cast<int64_t>(MostRows(ah, q.stageGroups)) * rowBytes + 30) / 16 * 16;
    if (slotBytes * q.planesPerBlock > static_cast<int64_t>(mostSmem)) {
        return false;
    }
    q.slotBytes = static_cast<int32_t>(slotBytes);
    q.stages = q.slotBytes * q.planesPerBlock <= 14 * 1024 ? 3 : 2;
    const int64_t resident = std::max<int64_t>(1, std::min<int64_t>(1024 / threads + 1, (200 << 10) / (ColumnsSmem(q) + 2048)));
    q.bandRows = PickBandRows(sh.hin, planeGroups, static_cast<int64_t>(NumSMs()) * resident);
    const int32_t bands = static_cast<int32_t>(CeilDiv(sh.hin, q.bandRows));
    q.dRowCap = MostRows(ah, q.bandRows + 1);
    // a horizontal sum is shared by as many lanes as there are threads for each output of a row
    const int32_t perOutput = (threads - 32) / std::max(1, q.planesPerBlock * q.win);
    while (q.lanesLog < 3 && (2 << q.lanesLog) <= perOutput) {
        ++q.lanesLog;
    }
    plan->threads = threads;
    plan->bands = bands;
    plan->planeGroups = planeGroups;
    plan->smem = ColumnsSmem(q);
    return plan->smem <= mostSmem && planeGroups <= 0x7fffffff && bands <= 65535;
}

// False where the kernel does not take the call.
bool PlanColumns(int es, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw, ColumnsPlan* plan)
{
    // columns per thread: at least as many as the width of a row needs, and no more than leave a thread for every horizontal
    // sum of a finished row (a second round of sums costs as much as the walk: fp32 400 planes 72x225 <- 108x337, 89 us)
    int32_t& k = plan->k;
    k = 1;
    while (k < 8 && CeilDiv(sh.wout, k) > 512) {
        k *= 2;
    }
    while (k < 8 && CeilDiv(sh.wout, 2 * k) >= sh.win && (k < 4 || k * (kColumnsThreads + 64) < sh.wout)) {
        k *= 2;
    }
    const int32_t team = static_cast<int32_t>(CeilDiv(sh.wout, k));
    if (team > 512) {
        return false;
    }
    // A stage holds a whole group of grads rows, which grows with the scale. Two blocks per SM, with fewer planes each if need
    // be; a single block of one plane beats the kernel without a walk by far (fp32 4
    // planes 160x160 <- 1280x1280: 569 us without, 15 with).
    int32_t planes = static_cast<int32_t>(std::max<int64_t>(1, std::min<int64_t>(sh.n * sh.c, kColumnsThreads / team)));
    for (; planes > 1; planes = (planes + 1) / 2) {
        if (PlanColumnsOf(planes, 96 * 1024, es, sh, ah, aw, plan)) {
            return true;
        }
    }
    return PlanColumnsOf(1, 224 * 1024, es, sh, ah, aw, plan);
}

// Many grads at small scales: the tile kernel, whose work per grad_input element grows with the scale in both axes and whose
// start does not count then, is the faster one. us by tiles and by walks, 400 planes 100x130, bf16 / fp32: 1.1x 29 / 31 and
// 38 / 37, 1.3x1.2 31 / 35 and 39 / 39, 1.5x 35 / 43 and 51 / 51, 2x 78 / 101 and 55 / 57; 84 planes 240x320, 1.6x1.2 34 / 43 and
// 44 / 43. With 25 planes the walks lead throughout.
bool TilesPay(int es, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw)
{
    const double grads = static_cast<double>(sh.n) * sh.c * sh.hout * sh.wout;
    return grads >= 3.5e6 && static_cast<double>(ah.scale) * aw.scale > 1.0 / (es == 2 ? 2.4 : 1.75);
}

template <typename TIn, typename TOut>
bool LaunchColumns(const void* go, void* gi, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw, bool tiles, cudaStream_t s)
{
    ColumnsPlan plan;
    if ((tiles && TilesPay(static_cast<int>(sizeof(TIn)), sh, ah, aw)) ||
        !PlanColumns(static_cast<int>(sizeof(TIn)), sh, ah, aw, &plan)) {
        return false;
    }
    const dim3 grid(static_cast<unsigned>(plan.planeGroups), static_cast<unsigned>(plan.bands));
    auto launch = [&](auto kernel) {
        if (plan.smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          static_cast<int>(plan.smem)) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        kernel<<<grid, plan.threads, plan.smem, s>>>(static_cast<const TIn*>(go), static_cast<TOut*>(gi), sh.n * sh.c, plan.q,
                                                     ah, aw);
        return true;
    };
    switch (plan.k) {
        case 1: return launch(BilinearBwdColumnsKernel<TIn, TOut, 1>);
        case 2: return launch(BilinearBwdColumnsKernel<TIn, TOut, 2>);
        case 4: return launch(BilinearBwdColumnsKernel<TIn, TOut, 4>);
        default: return launch(BilinearBwdColumnsKernel<TIn, TOut, 8>);
    }
}

// Most significant bits that a weight of this axis can have. With scale = odd * 2^e a position is a multiple of 2^e, or of
// 2^(e - 1) with the half-pixel offset (rounding moves it to a coarser multiple), and so are a weight and its complement.
// From the scale alone: a look at every index took 193 us per axis and call at 4096 indices and a scale of two.
int AxisBits(const BwdAxis& a)
{
    int exponent = 0;
    const float m = std::frexp(a.scale, &exponent); // scale = m * 2^exponent, m in [0.5, 1)
    uint32_t digits = static_cast<uint32_t>(std::ldexp(m, 24));
    int e = exponent - 24;
    for (; (digits & 1u) == 0; digits >>= 1) { // scale is not zero
        ++e;
    }
    return std::max(1, std::min(24, (a.offset > 0.0f ? 1 : 0) - e));
}

// Launch shape of the NHWC kernel; false where it does not take the call.
struct WalkPlan {
    WalkShape q;
    int32_t tiles, slices, threads, bands;
    int64_t imageGroups;
    size_t smem;
};
bool PlanNHWC(int es, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw, WalkPlan* plan)
{
    const int v = 16 / es;
    if (sh.c % v != 0) {
        return false;
    }
    WalkShape& q = plan->q;
    q = WalkShape{};
    q.groups = static_cast<int32_t>(sh.c / v);
    q.hin = sh.hin;
    q.win = sh.win;
    q.hout = sh.hout;
    q.wout = sh.wout;
    const int32_t slices = static_cast<int32_t>(CeilDiv(q.groups, 32));
    q.slice = static_cast<int32_t>(CeilDiv(q.groups, slices));
    q.tileX = std::min(sh.win, kWalkThreads / q.slice);
    q.tileX = static_cast<int32_t>(CeilDiv(sh.win, CeilDiv(sh.win, q.tileX))); // equal tiles
    q.images = static_cast<int32_t>(std::max<int64_t>(1, std::min<int64_t>(sh.n, kWalkThreads / (q.tileX * q.slice))));
    // A single narrow image leaves a block a warp: on a tall one the gather kernel, with a thread per element, is faster
    // (fp32 1x100000x4x8 <- 250000x9: 104 us against 239, 10000 rows: 25 against 34 us, 500 rows: 21 us both).
    if (q.images * q.tileX * q.slice <= 32 && sh.hin > 1024) {
        return false;
    }
    const int32_t tiles = static_cast<int32_t>(CeilDiv(sh.win, q.tileX));
    q.segPixels = MostRows(aw, q.tileX + 1);
    // a whole group per stage where that is some eighteen kilobytes at most
    const int64_t rowBytes = std::max<int64_t>(1, static_cast<int64_t>(q.images) * q.segPixels * q.slice * 16);
    const int32_t groupRows = static_cast<int32_t>(std::min(std::ceil(1.0f / ah.scale), static_cast<float>(sh.hout)));
    q.stageRows = std::max(1, static_cast<int32_t>(std::min<int64_t>(groupRows, 18 * 1024 / rowBytes)));
    const int64_t imageGroups = CeilDiv(sh.n, q.images);
    const int32_t threads = static_cast<int32_t>(CeilDiv(q.images * q.tileX * q.slice, 32)) * 32 + 32; // and the copying warp
    const int64_t resident = std::max<int64_t>(1, std::min<int64_t>(1024 / threads, (220 << 10) / (WalkSmem(q) + 2048)));
    q.bandRows = PickBandRows(sh.hin, imageGroups * tiles * slices, static_cast<int64_t>(NumSMs()) * resident);
    const int32_t bands = static_cast<int32_t>(CeilDiv(sh.hin, q.bandRows));
    q.dRowCap = MostRows(ah, q.bandRows + 1);
    plan->tiles = tiles;
    plan->slices = slices;
    plan->threads = threads;
    plan->bands = bands;
    plan->imageGroups = imageGroups;
    plan->smem = WalkSmem(q);
    return plan->smem <= 112 * 1024 && imageGroups <= 65535 && bands <= 65535;
}

template <typename T, typename TOut>
bool LaunchNHWC(const void* go, void* gi, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw, cudaStream_t s)
{
    constexpr int V = 16 / sizeof(T);
    WalkPlan plan;
    if (!Aligned(go, 16) || !Aligned(gi, V * sizeof(TOut)) || !PlanNHWC(static_cast<int>(sizeof(T)), sh, ah, aw, &plan)) {
        return false;
    }
    const WalkShape& q = plan.q;
    const size_t smem = plan.smem;
    const int mant = std::is_same<T, __half>::value ? 11 : 8; // significand bits of T
    const bool fuse = sizeof(T) == 2 && AxisBits(ah) + AxisBits(aw) + mant <= 24;
    const dim3 grid(static_cast<unsigned>(plan.tiles * plan.slices), static_cast<unsigned>(plan.imageGroups),
                    static_cast<unsigned>(plan.bands));
    const int32_t threads = plan.threads;
    auto launch = [&](auto kernel) {
        if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     static_cast<int>(smem)) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        kernel<<<grid, threads, smem, s>>>(static_cast<const T*>(go), static_cast<TOut*>(gi), sh.n, q, ah, aw);
        return true;
    };
    if constexpr (sizeof(T) == 2) {
        if (fuse) {
            return launch(BilinearBwdNHWCWalkKernel<T, TOut, true>);
        }
    }
    return launch(BilinearBwdNHWCWalkKernel<T, TOut, false>);
}

template <typename TIn, typename TOut>
bool Launch(Layout lay, const void* go, void* gi, const Shape4& sh, const BwdAxis& ah, const BwdAxis& aw, bool tiles,
            cudaStream_t s)
{
    return lay == kNCHW ? LaunchColumns<TIn, TOut>(go, gi, sh, ah, aw, tiles, s) : LaunchNHWC<TIn, TOut>(go, gi, sh, ah, aw, s);
}

// An up-scale whose groups follow from the scale, at extents for which MostRows holds.
bool Walkable(const BwdAxis& a)
{
    return a.scale > 0.0f && a.scale <= 1.0f && a.out <= kMostExtent && a.last < kMostExtent && !Overshoots(a);
}

} // namespace

bool DebugBilinearBwdWalk(int es, Layout lay, Shape4 sh, AxisGeom gh, AxisGeom gw, bool halfPixel, bool tiles, int64_t values[8])
{
    const BwdAxis ah = MakeAxis(gh, halfPixel), aw = MakeAxis(gw, halfPixel);
    if (!Walkable(ah) || !Walkable(aw)) {
        return false;
    }
    if (lay == kNCHW) {
        ColumnsPlan p;
        if ((tiles && TilesPay(es, sh, ah, aw)) || !PlanColumns(es, sh, ah, aw, &p)) {
            return false;
        }
        const int64_t stage = (p.q.slotBytes - 15) / (sh.wout * static_cast<int64_t>(es));
        const int64_t v[8] = {p.q.bandRows, p.q.dRowCap, p.q.stageGroups, stage, p.k, p.q.planesPerBlock, p.bands,
                              static_cast<int64_t>(p.smem)};
        std::copy(v, v + 8, values);
        return true;
    }
    WalkPlan p;
    if (!PlanNHWC(es, sh, ah, aw, &p)) {
        return false;
    }
    const int64_t v[8] = {p.q.bandRows, p.q.dRowCap, p.q.tileX, p.q.segPixels, p.slices, p.q.images, AxisBits(ah) + AxisBits(aw),
                          static_cast<int64_t>(p.smem)};
    std::copy(v, v + 8, values);
    return true;
}

bool BilinearBwdWalk(Dt dtIn, Dt dtOut, Layout lay, const void* go, void* gi, Shape4 sh, AxisGeom gh, AxisGeom gw,
                     bool halfPixel, bool tiles, cudaStream_t s)
{
    const BwdAxis ah = MakeAxis(gh, halfPixel), aw = MakeAxis(gw, halfPixel);
    if (!Walkable(ah) || !Walkable(aw)) {
        return false;
    }
    if (dtIn == dtOut) {
        OPSCV_DISPATCH_DT(dtIn, T, { return (Launch<T, T>(lay, go, gi, sh, ah, aw, tiles, s)); });
    }
    if (dtIn == Dt::F32 && dtOut == Dt::F16) {
        return Launch<float, __half>(lay, go, gi, sh, ah, aw, tiles, s);
    }
    return dtIn == Dt::F32 && dtOut == Dt::BF16 && Launch<float, __nv_bfloat16>(lay, go, gi, sh, ah, aw, tiles, s);
}

} // namespace opscv
