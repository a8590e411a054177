// UpsampleBicubic2dAA forward and backward (NCHW).
//
// The anti-aliased bicubic filter is separable: out[i][j] = sum_m wH[i][m] * sum_n wW[j][n] * x[hmin_i+m][wmin_j+n]
// with per-axis windows and normalised weights that depend only on the output index. tables.cu builds those
// windows / weights once per call; the kernels here never evaluate the cubic.
//
// Forward
//   * streaming kernel (down-scaling, the common case): a block owns a band of output rows of one plane and
//     streams the input rows that band needs exactly once, 16 bytes per thread, fully coalesced. Each thread
//     owns four input columns and carries a small ring of partial sums, one per output row whose vertical window
//     is currently open (an input row touches only ~support/scale output rows). When an output row's window
//     closes, its vertically filtered row (still at input width) goes to shared memory and the block applies the
//     horizontal filter, each thread producing output columns with its weights held in registers.
//     Input is read once from HBM, nothing but the output is written.
//   * direct kernel (any shape): one thread per output element, double loop over the window in the reference's
//     accumulation order (rows outer, columns inner).
// Backward
//   * gather kernel: one thread per grad_input element sums the outputs whose windows cover it, rows outer,
//     columns inner; deterministic. A block-tiled variant serves the down-scaling case, where each output row
//     fans out to many input rows.
//   * atomic kernel: the reference's scatter with fp32 atomics (selectable).
//
// Reference arithmetic: image/upsample_bicubic2d_aa/op_kernel/arch35/upsample_bicubic2d_aa_simt_base.h:52-127,
// image/upsample_bicubic2d_aa_grad/op_kernel/arch35/upsample_bicubic2d_aa_grad_simt_base.h:32-102 and
// upsample_bicubic2d_aa_grad_simt_base_deter.h:30-122.
#include <algorithm>

#include "launch_util.cuh"

namespace opscv {
namespace {

constexpr int kThreads = 256;

// ---- forward, direct ----------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads)
    AAFwdDirectKernel(const T* __restrict__ x, T* __restrict__ y, int32_t hin, int32_t win, int32_t hout,
                      int32_t wout, AAAxis th, AAAxis tw, int64_t total)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int64_t row = idx / wout;
        const int32_t w = static_cast<int32_t>(idx - row * wout);
        const int64_t p = row / hout;
        const int32_t h = static_cast<int32_t>(row - p * hout);
        const int32_t hmin = __ldg(th.xmin + h), hsz = __ldg(th.xsize + h);
        const int32_t wmin = __ldg(tw.xmin + w), wsz = __ldg(tw.xsize + w);
        const float* wh = th.w + static_cast<int64_t>(h) * th.taps;
        const float* ww = tw.w + static_cast<int64_t>(w) * tw.taps;
        const T* xp = x + p * hin * static_cast<int64_t>(win);
        float value = 0.0f;
        for (int32_t m = 0; m < hsz; ++m) {
            const float weightH = __ldg(wh + m);
            const T* xr = xp + static_cast<int64_t>(hmin + m) * win + wmin;
            for (int32_t n = 0; n < wsz; ++n) {
                // value += x * weightsH * weightsW  (simt_base.h:121)
                value = Add(value, Mul(Mul(DType<T>::Load(xr + n), weightH), __ldg(ww + n)));
            }
        }
        y[idx] = DType<T>::FromF(value);
    }
}

// ---- forward, streaming (down-scaling) -----------------------------------------------------------------------
// Per input row r, the outputs whose vertical window covers r form a short run: an output covers r iff its centre lies in
// [r + 0.5 - support, r + 0.5 + support). Centres are `scale` apart and support is 2 * scale (cubic) or scale (triangle),
// so for scale >= 1 that is 4 or 2 outputs, one more through rounding (up to kAAMostRows rows: centres and window ends are off
// by 3/8 at most there, past 2^23 rows by more than one): NS = 5 or 3 open sums. The table launch writes, once
// per call, one 32-byte record per input row (AATablesAndRangesKernel): the weights of the run, its start and its length.
constexpr int32_t kAAMostRows = 1 << 22;
constexpr int kSlots = kAASlots;
constexpr int kSlotStride = kAASlotStride;
constexpr int kFlushBatch = 4;        // output rows per horizontal pass of the streaming forward kernel
constexpr int kStreamThreads = 512;   // most threads of a block of the register-prefetch variant (64 registers each)
constexpr int kRingThreads = 256;     // the bulk-copy variant: up to 255 registers per thread

// ---- bulk asynchronous copies (global -> shared) with mbarrier completion ----------------------------------------
// Used by the streaming forward kernel to keep whole input rows in flight without holding them in registers.
// Every wait is bounded: a wait that runs out bumps g_asyncCopyTimeouts (read by AsyncCopyTimeouts()), the block
// waits (bounded again) for the copies it still has in flight and returns, so the context stays usable.
__device__ unsigned int g_asyncCopyTimeouts = 0;
constexpr uint32_t kWaitLimit = 1u << 22;

__device__ __forceinline__ uint32_t SmemAddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void BarrierInit(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void BarrierInitFence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Arms the barrier for `bytes` of copy traffic and starts one row copy that completes on it. dst, src and bytes are
// multiples of 16.
__device__ __forceinline__ void BulkLoadRow(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     SmemAddr(dst)),
                 "l"(src), "r"(bytes), "r"(SmemAddr(bar))
                 : "memory");
}
__device__ __forceinline__ bool BarrierWait(uint64_t* bar, uint32_t parity, uint32_t limit)
{
    const uint32_t addr = SmemAddr(bar);
    for (uint32_t it = 0; it < limit; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(addr), "r"(parity)
                     : "memory");
        if (ok) {
            return true;
        }
    }
    return false;
}

// The parked rows are skewed by one float per 32 columns: the horizontal pass reads them at a stride of `scale`
// columns per lane, and without the skew lanes 32 / scale apart would always meet in one bank.
__host__ __device__ __forceinline__ int32_t Skew(int32_t col) { return col + (col >> 5); }
__host__ __device__ __forceinline__ int32_t ParkedRowFloats(int32_t win) { return (Skew(win) + 4) & ~3; }

// grid = (planes, bands); a band is `bandRows` output rows. A thread owns VC input columns of every row, in groups of
// LV adjacent ones, and keeps one partial sum per open output row (NS of them) for each. LV is the widest load that every
// row of the plane is aligned for (rows of an odd width start at every element offset: LV = 1); the groups of a thread
// are a block width apart, so a load instruction of a warp reads one contiguous run at any LV.
// What bounds it is instruction issue and the latency of the row loads (photographs, fp32: 96 instructions per warp and
// row before sums were kept in packed pairs, with 56 % of the issue slots busy). 16x3x720x1280 fp16 -> 333x592, whole
// call: 112 -> 87 us with four columns per thread (three blocks per SM) instead of eight and a band per model.
// Shared memory: the vertically filtered row being flushed, the records of the band's input rows with every weight twice
// (the operand of a packed multiply-add needs no register moves), and (wTaps > 0) the horizontal weights of all output
// columns, transposed.
// Two ways of bringing the input rows in:
//   BULK = false: every thread loads its own columns, PF rows ahead, into registers;
//   BULK = true : thread 0 starts one bulk asynchronous copy per row into a ring of ringGroups * PF row slots in
//                 shared memory (completion on one mbarrier per slot); the rows of a group of PF are consumed by all
//                 threads from shared memory, and after a block barrier the group's slots are refilled with the rows
//                 ringGroups groups ahead. Whole rows are in flight at no register cost.
template <typename T, int NS, int VC, int LV, int MAXT, bool BULK>
__global__ void __launch_bounds__(MAXT, BULK ? 1 : 2)
    AAFwdStreamKernel(const T* __restrict__ x, T* __restrict__ y, int32_t hin, int32_t win, int32_t hout,
                      int32_t wout, AAAxis th, AAAxis tw, const float* __restrict__ wrow, int32_t bandRows,
                      int32_t metaRows, int32_t wTaps, int32_t ringGroups)
{
    // input rows in flight per thread / rows per ring group: what 64 registers hold without spills beside the sums
    constexpr int PF = (BULK || (NS == 3 && LV * sizeof(T) >= 4 && LV > 1) || (sizeof(T) == 2 && LV == 4)) ? 4 : 2;
    constexpr int NL = VC / LV;            // loads per row
    constexpr int RW = (NS + 1) / 2;       // 16-byte words per shared record: NS weights twice, start, run length
    extern __shared__ __align__(16) float smemAll[];
    // BULK: the ring comes first (16-byte aligned slots of one row each), then the slot barriers
    const uint32_t rowBytes = static_cast<uint32_t>(win) * sizeof(T);
    const int32_t ringSlots = BULK ? ringGroups * PF : 0;
    unsigned char* ring = reinterpret_cast<unsigned char*>(smemAll);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + static_cast<size_t>(ringSlots) * rowBytes);
    float* smemF = reinterpret_cast<float*>(bars + ((ringSlots + 1) & ~1));
    const int32_t winPad = ParkedRowFloats(win);
    float* rowbufs = smemF;                                           // [kFlushBatch][winPad]
    ulonglong2* msm = reinterpret_cast<ulonglong2*>(smemF + kFlushBatch * winPad); // [metaRows][RW]
    float* wsm = reinterpret_cast<float*>(msm + RW * metaRows);       // [wTaps][wout]
    const int64_t p = blockIdx.x;
    const int32_t i0 = blockIdx.y * bandRows, i1 = min(hout, i0 + bandRows);
    // a window of a user scale may start past the input: it is empty, and a band of such windows reads no rows
    const int32_t rlo = min(__ldg(th.xmin + i0), hin);
    const int32_t rhi = min(min(__ldg(th.xmin + i1 - 1) + __ldg(th.xsize + i1 - 1), rlo + metaRows), hin);
    // Column ownership: load l of a thread covers columns l * (blockDim.x * LV) + threadIdx.x * LV ..
    const int32_t groupSpan = blockDim.x * LV;
    const int32_t c = threadIdx.x * LV;
    T* yp = y + p * hout * static_cast<int64_t>(wout);

    for (int32_t e = threadIdx.x; e < rhi - rlo; e += blockDim.x) {
        const float* src = wrow + static_cast<int64_t>(rlo + e) * kSlotStride;
        float* dst = reinterpret_cast<float*>(msm + e * RW);
#pragma unroll
        for (int a = 0; a < NS; ++a) {
            const float w = __ldg(src + a);
            dst[2 * a] = w;
            dst[2 * a + 1] = w;
        }
        dst[2 * NS] = __ldg(src + kSlots);
        dst[2 * NS + 1] = __ldg(src + kSlots + 1);
    }
    for (int32_t j = threadIdx.x; j < wout && wTaps > 0; j += blockDim.x) {
        const int32_t n = min(__ldg(tw.xsize + j), wTaps);
        for (int32_t t = 0; t < n; ++t) {
            wsm[t * wout + j] = __ldg(tw.w + static_cast<int64_t>(j) * tw.taps + t);
        }
    }
    __syncthreads();

    F2 acc[NS][VC / 2];
#pragma unroll
    for (int a = 0; a < NS; ++a) {
#pragma unroll
        for (int k = 0; k < VC / 2; ++k) {
            acc[a][k] = MakeF2(0.0f, 0.0f);
        }
    }
    // Completed output rows (vertical results, taken from the oldest accumulator slot) are parked in shared memory,
    // kFlushBatch rows at a time, and the horizontal filter then runs over the whole batch: a thread takes one
    // output column of all the batch's rows, so every weight is loaded once per batch and the rows give
    // independent accumulation chains. Output rows complete in increasing order, so a batch is rows
    // batchRow0 .. batchRow0 + pending - 1.
    int32_t pending = 0, batchRow0 = 0;
    auto runBatch = [&]() {
        __syncthreads(); // the batch's rows are written
        for (int32_t j = threadIdx.x; j < wout; j += blockDim.x) {
            const int32_t m = __ldg(tw.xmin + j), n = __ldg(tw.xsize + j);
            const float* wj = tw.w + static_cast<int64_t>(j) * tw.taps;
            float v[kFlushBatch];
#pragma unroll
            for (int bb = 0; bb < kFlushBatch; ++bb) {
                v[bb] = 0.0f;
            }
            // rows past `pending` hold stale values; their sums are not stored
            if (wTaps > 0) {
                const float* wp = wsm + j;
#pragma unroll 4
                for (int32_t t = 0; t < n; ++t) {
                    const float w = wp[t * wout];
                    const float* xr = rowbufs + Skew(m + t);
#pragma unroll
                    for (int bb = 0; bb < kFlushBatch; ++bb) {
                        v[bb] = fmaf(w, xr[bb * winPad], v[bb]);
                    }
                }
            } else {
                for (int32_t t = 0; t < n; ++t) {
                    const float w = __ldg(wj + t);
                    const float* xr = rowbufs + Skew(m + t);
#pragma unroll
                    for (int bb = 0; bb < kFlushBatch; ++bb) {
                        v[bb] = fmaf(w, xr[bb * winPad], v[bb]);
                    }
                }
            }
#pragma unroll
            for (int bb = 0; bb < kFlushBatch; ++bb) {
                if (bb < pending) {
                    yp[static_cast<int64_t>(batchRow0 + bb) * wout + j] = DType<T>::FromF(v[bb]);
                }
            }
        }
        __syncthreads(); // the rows have been read: the buffer can take the next batch
        pending = 0;
    };
    auto flush = [&](int32_t i) {
        if (pending == 0) {
            batchRow0 = i;
        }
        float* rowbuf = rowbufs + pending * winPad;
        float done[VC];
#pragma unroll
        for (int k = 0; k < VC / 2; ++k) {
            SplitF2(acc[0][k], done[2 * k], done[2 * k + 1]);
        }
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            const int32_t col = l * groupSpan + c;
            if (col < win) { // scalar stores: under the skew they are conflict-free across the warp
                const int32_t sc = Skew(col); // col is a multiple of LV: its LV <= 8 columns share one skew
#pragma unroll
                for (int k = 0; k < LV; ++k) {
                    rowbuf[sc + k] = done[l * LV + k];
                }
            }
        }
        if (++pending == kFlushBatch) {
            runBatch();
        }
    };
    auto shift = [&]() {
#pragma unroll
        for (int a = 0; a + 1 < NS; ++a) {
#pragma unroll
            for (int k = 0; k < VC / 2; ++k) {
                acc[a][k] = acc[a + 1][k];
            }
        }
#pragma unroll
        for (int k = 0; k < VC / 2; ++k) {
            acc[NS - 1][k] = MakeF2(0.0f, 0.0f);
        }
    };
    // Input rows are fetched PF rows ahead into fixed registers (the row loop is unrolled by PF; rotating a queue
    // through moves would make every iteration wait for the newest load), or ringGroups groups ahead into the ring.
    using Vec = Pack<T, LV>;
    Vec q[PF][NL];
    const T* xrows = x + (p * hin + rlo) * static_cast<int64_t>(win); // row rlo of this plane
    const T* xnext = xrows + c;                                       // next row to fetch (register path)
    int32_t rnext = rlo;
    auto fetch = [&](Vec (&dst)[NL]) {
        if (rnext < rhi) {
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                if (l * groupSpan + c < win) {
                    dst[l] = *reinterpret_cast<const Vec*>(xnext + l * groupSpan);
                }
            }
        }
        xnext += win;
        ++rnext;
    };
    // BULK: thread 0 starts the copies of group `grp` (rows rlo + grp * PF ..) into the group's slots
    auto issueGroup = [&](int32_t grp) {
        const int32_t slot0 = (grp % ringGroups) * PF;
#pragma unroll
        for (int f = 0; f < PF; ++f) {
            const int32_t rr = grp * PF + f; // row index relative to rlo
            if (rlo + rr < rhi) {
                BulkLoadRow(ring + static_cast<size_t>(slot0 + f) * rowBytes, xrows + static_cast<int64_t>(rr) * win,
                            rowBytes, bars + slot0 + f);
            }
        }
    };
    if (BULK) {
        if (threadIdx.x == 0) {
            for (int32_t sl = 0; sl < ringSlots; ++sl) {
                BarrierInit(bars + sl, 1);
            }
            BarrierInitFence();
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int32_t grp = 0; grp < ringGroups; ++grp) {
                issueGroup(grp);
            }
        }
    } else {
#pragma unroll
        for (int f = 0; f < PF; ++f) {
            fetch(q[f]);
        }
    }
    int32_t curStart = rlo < rhi ? static_cast<int32_t>(msm[RW - 1].y & 0xffffffffu) : i0;
    for (int32_t r0 = rlo; r0 < rhi; r0 += PF) {
        const int32_t grp = (r0 - rlo) / PF;
        const int32_t slot0 = BULK ? (grp % ringGroups) * PF : 0;
        if (BULK) {
            // wait for the rows of this group; the outcome is made uniform so that the block leaves together
            const uint32_t parity = static_cast<uint32_t>(grp / ringGroups) & 1u;
            bool ok = true;
#pragma unroll
            for (int f = 0; f < PF; ++f) {
                if (r0 + f < rhi) {
                    ok = BarrierWait(bars + slot0 + f, parity, kWaitLimit) && ok;
                }
            }
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) {
                    atomicAdd(&g_asyncCopyTimeouts, 1u);
                    // copies still in flight target this block's shared memory: give them a bounded chance to land
                    for (int32_t g2 = grp; g2 < grp + ringGroups; ++g2) {
                        for (int f = 0; f < PF; ++f) {
                            if (rlo + g2 * PF + f < rhi) {
                                BarrierWait(bars + (g2 % ringGroups) * PF + f,
                                            static_cast<uint32_t>(g2 / ringGroups) & 1u, 1u << 16);
                            }
                        }
                    }
                }
                return;
            }
        }
#pragma unroll
        for (int f = 0; f < PF; ++f) {
            const int32_t r = r0 + f;
            if (r < rhi) {
                const ulonglong2* m = msm + (r - rlo) * RW;
                const ulonglong2 mLast = m[RW - 1];
                const int32_t s = static_cast<int32_t>(mLast.y & 0xffffffffu), cnt = static_cast<int32_t>(mLast.y >> 32);
                while (curStart < s) { // outputs before start(r) no longer receive rows: complete
                    if (curStart >= i0 && curStart < i1) {
                        flush(curStart);
                    }
                    shift();
                    ++curStart;
                }
                float xv[VC];
                if (BULK) {
                    const T* srow = reinterpret_cast<const T*>(ring + static_cast<size_t>(slot0 + f) * rowBytes);
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        Vec v{};
                        if (l * groupSpan + c < win) {
                            v = *reinterpret_cast<const Vec*>(srow + l * groupSpan + c);
                        }
                        float part[LV];
                        UnpackToF<T, LV>(v, part);
#pragma unroll
                        for (int k = 0; k < LV; ++k) {
                            xv[l * LV + k] = part[k];
                        }
                    }
                } else {
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        float part[LV];
                        UnpackToF<T, LV>(q[f][l], part);
#pragma unroll
                        for (int k = 0; k < LV; ++k) {
                            xv[l * LV + k] = part[k];
                        }
                    }
                }
                // Slots past the run are not touched (an Inf / NaN input must not leak in). Away from the first and last
                // rows the run fills all slots but the last, which one test then covers: photographs 487 -> 463 us against a test
                // per slot. With three slots the tests are few and the other form's registers cost more (87 -> 92 us).
                F2 xp[VC / 2];
#pragma unroll
                for (int k = 0; k < VC / 2; ++k) {
                    xp[k] = MakeF2(xv[2 * k], xv[2 * k + 1]);
                }
                auto slot = [&](int a, F2 w) {
#pragma unroll
                    for (int k = 0; k < VC / 2; ++k) {
                        acc[a][k] = Fma2(w, xp[k], acc[a][k]);
                    }
                };
                if (NS > 3 && cnt >= NS - 1) {
#pragma unroll
                    for (int a = 0; a + 1 < NS; a += 2) {
                        const ulonglong2 w = m[a / 2];
                        slot(a, F2{w.x});
                        slot(a + 1, F2{w.y});
                    }
                    if (cnt == NS) {
                        slot(NS - 1, F2{mLast.x});
                    }
                } else {
#pragma unroll
                    for (int a = 0; a < NS; ++a) {
                        if (a < cnt) {
                            slot(a, a == NS - 1 ? F2{mLast.x} : F2{a % 2 == 0 ? m[a / 2].x : m[a / 2].y});
                        }
                    }
                }
                if (!BULK) {
                    fetch(q[f]);
                }
            }
        }
        if (BULK) {
            __syncthreads(); // every thread has read the group's slots: they can be refilled
            if (threadIdx.x == 0 && rlo + (grp + ringGroups) * PF < rhi) {
                issueGroup(grp + ringGroups);
            }
        }
    }
    while (curStart < i1) { // sums that no further row reaches, and the zeros of empty windows
        if (curStart >= i0) {
            flush(curStart);
        }
        shift();
        ++curStart;
    }
    if (pending > 0) {
        runBatch();
    }
}

// ---- backward, gather (direct) --------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads)
    AABwdGatherKernel(const T* __restrict__ go, T* __restrict__ gi, int32_t hin, int32_t win, int32_t hout,
                      int32_t wout, AAAxis th, AAAxis tw, RangeAxis rh, RangeAxis rw, int64_t total)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int64_t row = idx / win;
        const int32_t x = static_cast<int32_t>(idx - row * win);
        const int64_t p = row / hin;
        const int32_t y = static_cast<int32_t>(row - p * hin);
        const int32_t is = __ldg(rh.start + y), ie = __ldg(rh.end + y);
        const int32_t js = __ldg(rw.start + x), je = __ldg(rw.end + x);
        const T* gp = go + p * hout * static_cast<int64_t>(wout);
        float value = 0.0f;
        for (int32_t i = is; i < ie; ++i) {
            const int32_t ty = y - __ldg(th.xmin + i);
            if (ty < 0 || ty >= __ldg(th.xsize + i)) {
                continue;
            }
            const float weightH = __ldg(th.w + static_cast<int64_t>(i) * th.taps + ty);
            if (weightH == 0.0f) {
                continue;
            }
            const T* gr = gp + static_cast<int64_t>(i) * wout;
            for (int32_t j = js; j < je; ++j) {
                const int32_t tx = x - __ldg(tw.xmin + j);
                if (tx < 0 || tx >= __ldg(tw.xsize + j)) {
                    continue;
                }
                const float weightW = __ldg(tw.w + static_cast<int64_t>(j) * tw.taps + tx);
                if (weightW == 0.0f) {
                    continue;
                }
                value = Add(value, Mul(Mul(DType<T>::Load(gr + j), weightH), weightW));
            }
        }
        gi[idx] = DType<T>::FromF(value);
    }
}

// ---- backward, band-tiled (down-scaling forward) ----------------------------------------------------------------
// gi[y][x] = sum_i wH(i,y) * sum_j wW(j,x) * go[i][j]. For scale >= 1 only a few outputs cover any input row or
// column, so the sum is done separably per block: the grads rows feeding a band of grad_input rows are staged in
// shared memory (fp32); for kBwdRows grad_input rows at a time the block first reduces vertically
// (t[y][j] = sum_i wH * go[i][j]: a thread takes one grads column for the rows of the step, reads each grads row that
// reaches any of them once and adds it to two packed pairs of sums, the four weights of a grads row being one 16-byte
// word of a table that the block builds first), then every thread expands horizontally for its four grad_input columns
// with the column weights it keeps in registers as packed pairs. Weights come from the slot records of both axes; a
// weight that does not exist is 0 and its product changes nothing while the grads are finite.
// What bounds it is instruction issue: 125 instructions per warp and row (photographs, fp32) while every row walked its
// own grads rows and sums were single, 68 % of the issue slots busy. 64x3x1024x1024 <-> 224x224 fp32, both directions: 529 -> 463 us.
constexpr int kBwdRows = 4;     // grad_input rows per synchronisation
constexpr int kBwdRowSlots = kAABwdRowSlots;
constexpr int kBwdGroupBytes = (kBwdRowSlots + 1) * 16; // weights of a step, its first grads row and their count

// Rows parked by the VEC = false variant: [kBwdRows][OutPitch] of T.
__host__ __device__ __forceinline__ int32_t OutPitch(int32_t win) { return (win + 7) & ~7; }
// Staged grads rows, the step's vertical sums and the zeros behind them that the last columns' slots may read.
__host__ __device__ __forceinline__ int64_t BwdStagedFloats(int32_t stageRows, int32_t wout)
{
    return ((static_cast<int64_t>(stageRows) + kBwdRows) * wout + kBwdRowSlots + 3) & ~3LL;
}

// VEC: every row of grad_input is aligned for the four-column store of a thread. Otherwise (odd widths, an odd base) the
// rows of a step are parked in shared memory and written from there, adjacent lanes to adjacent words: four scalar
// stores per thread would touch every sector of the row four times.
// CS: grads columns that may reach a thread's four columns.
template <typename T, bool VEC, int CS>
__global__ void __launch_bounds__(1024)
    AABwdBandKernel(const T* __restrict__ go, T* __restrict__ gi, int32_t hin, int32_t win, int32_t hout,
                    int32_t wout, RangeAxis rh, RangeAxis rw, const float* __restrict__ wrowH,
                    const float* __restrict__ wrowW, int32_t bandRows, int32_t stageRows)
{
    extern __shared__ __align__(16) float smemF[];
    const int32_t groups = bandRows / kBwdRows;
    float4* gw = reinterpret_cast<float4*>(smemF);                   // [groups][kBwdRowSlots] weights of the step's rows
    int4* gmeta = reinterpret_cast<int4*>(gw + groups * kBwdRowSlots); // [groups] first grads row (relative), count
    float* gos = reinterpret_cast<float*>(gmeta + groups);           // [stageRows][wout] grads rows of the band
    float* tbuf = gos + static_cast<int64_t>(stageRows) * wout;      // [kBwdRows][wout], then zeros
    T* obuf = reinterpret_cast<T*>(gos + BwdStagedFloats(stageRows, wout));
    const int64_t p = blockIdx.x;
    const int32_t y0 = blockIdx.y * bandRows, y1 = min(hin, y0 + bandRows);
    const int32_t i0 = __ldg(rh.start + y0);
    const int32_t i1 = min(max(i0, __ldg(rh.end + y1 - 1)), i0 + stageRows);
    for (int32_t e = threadIdx.x; e < groups * kBwdRowSlots; e += blockDim.x) {
        const int32_t grp = e / kBwdRowSlots, u = e - grp * kBwdRowSlots;
        const int32_t yb = y0 + grp * kBwdRows;
        if (yb >= y1) {
            break;
        }
        const int32_t first = __ldg(rh.start + yb), last = min(yb + kBwdRows, y1) - 1;
        float w[kBwdRows];
#pragma unroll
        for (int ry = 0; ry < kBwdRows; ++ry) {
            w[ry] = 0.0f;
            if (yb + ry < y1) {
                const float* rec = wrowH + static_cast<int64_t>(yb + ry) * kSlotStride;
                const int32_t a = first + u - __float_as_int(__ldg(rec + kSlots));
                if (a >= 0 && a < __float_as_int(__ldg(rec + kSlots + 1))) {
                    w[ry] = __ldg(rec + a);
                }
            }
        }
        gw[e] = make_float4(w[0], w[1], w[2], w[3]);
        if (u == 0) {
            gmeta[grp] = make_int4(first - i0, max(0, min(min(__ldg(rh.end + last), i1) - first, kBwdRowSlots)), 0, 0);
        }
    }
    for (int32_t e = threadIdx.x; e < kBwdRowSlots; e += blockDim.x) {
        tbuf[kBwdRows * wout + e] = 0.0f;
    }
    const T* gp = go + (p * hout + i0) * static_cast<int64_t>(wout);
    // While staging, note whether the band's grads rows hold an Inf / NaN: then both steps take a path that only touches
    // the sources with a weight of their own (the gather kernel skips zero weights), so that a non-finite value reaches
    // exactly the elements it reaches in the reference.
    bool sawNonFinite = false;
    for (int32_t e = threadIdx.x; e < (i1 - i0) * wout; e += blockDim.x) {
        const float v = DType<T>::Load(gp + e);
        gos[e] = v;
        sawNonFinite |= !(fabsf(v) <= 3.402823466e38f);
    }
    // horizontal weights of my four columns: slot u <-> grads column j0 + u
    const int32_t x = threadIdx.x * 4;
    const bool hasCols = x < win;
    int32_t j0 = 0;
    F2 wreg[CS][2];
    if (hasCols) {
        j0 = __ldg(rw.start + x);
        float w[4][CS];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool in = VEC || x + k < win;
            const int32_t sk = in ? __ldg(rw.start + x + k) : 0, ek = in ? __ldg(rw.end + x + k) : 0;
#pragma unroll
            for (int u = 0; u < CS; ++u) {
                const int32_t a = j0 + u - sk; // slot of grads column j0 + u in column x + k's own table
                w[k][u] = (a >= 0 && a < kSlots && j0 + u < ek)
                              ? __ldg(wrowW + static_cast<int64_t>(x + k) * kSlotStride + a)
                              : 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < CS; ++u) {
            wreg[u][0] = MakeF2(w[0][u], w[1][u]);
            wreg[u][1] = MakeF2(w[2][u], w[3][u]);
        }
        j0 = min(j0, wout); // a user scale can leave columns without any source
    }
    const bool masked = __syncthreads_or(sawNonFinite) != 0; // also: the staged rows and tables are visible
    T* op = gi + p * hin * static_cast<int64_t>(win);
    for (int32_t yb = y0; yb < y1; yb += kBwdRows) {
        const int32_t grp = (yb - y0) / kBwdRows;
        const int4 meta = gmeta[grp];
        const ulonglong2* wg = reinterpret_cast<const ulonglong2*>(gw + grp * kBwdRowSlots);
        for (int32_t j = threadIdx.x; j < wout; j += blockDim.x) {
            F2 v01 = MakeF2(0.0f, 0.0f), v23 = v01;
            const float* gcol = gos + meta.x * wout + j;
#pragma unroll
            for (int u = 0; u < kBwdRowSlots; ++u) {
                if (u >= meta.y) { // the same for every thread of the block
                    break;
                }
                const float g = gcol[u * wout];
                const ulonglong2 w = wg[u];
                if (!masked) {
                    const F2 gg = MakeF2(g, g);
                    v01 = Fma2(F2{w.x}, gg, v01);
                    v23 = Fma2(F2{w.y}, gg, v23);
                } else {
                    float ws[4], vs[4];
                    SplitF2(F2{w.x}, ws[0], ws[1]);
                    SplitF2(F2{w.y}, ws[2], ws[3]);
                    SplitF2(v01, vs[0], vs[1]);
                    SplitF2(v23, vs[2], vs[3]);
#pragma unroll
                    for (int ry = 0; ry < kBwdRows; ++ry) {
                        vs[ry] = ws[ry] != 0.0f ? fmaf(ws[ry], g, vs[ry]) : vs[ry];
                    }
                    v01 = MakeF2(vs[0], vs[1]);
                    v23 = MakeF2(vs[2], vs[3]);
                }
            }
            float v[kBwdRows];
            SplitF2(v01, v[0], v[1]);
            SplitF2(v23, v[2], v[3]);
#pragma unroll
            for (int ry = 0; ry < kBwdRows; ++ry) {
                tbuf[ry * wout + j] = v[ry];
            }
        }
        __syncthreads();
        if (hasCols) {
            T* dst = op + static_cast<int64_t>(yb) * win + x;
            const float* tr = tbuf + j0;
#pragma unroll
            for (int ry = 0; ry < kBwdRows; ++ry) {
                if (yb + ry < y1) {
                    F2 o01 = MakeF2(0.0f, 0.0f), o23 = o01;
                    float out[4];
                    if (!masked) {
#pragma unroll
                        for (int u = 0; u < CS; ++u) {
                            const F2 tt = MakeF2(tr[u], tr[u]);
                            o01 = Fma2(wreg[u][0], tt, o01);
                            o23 = Fma2(wreg[u][1], tt, o23);
                        }
                        SplitF2(o01, out[0], out[1]);
                        SplitF2(o23, out[2], out[3]);
                    } else {
                        out[0] = out[1] = out[2] = out[3] = 0.0f;
#pragma unroll
                        for (int u = 0; u < CS; ++u) {
                            float w[4];
                            SplitF2(wreg[u][0], w[0], w[1]);
                            SplitF2(wreg[u][1], w[2], w[3]);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                out[k] = w[k] != 0.0f ? fmaf(w[k], tr[u], out[k]) : out[k];
                            }
                        }
                    }
                    StorePack<T, 4>(VEC ? dst : obuf + ry * OutPitch(win) + x, out);
                }
                dst += win;
                tr += wout;
            }
        }
        __syncthreads();
        if (!VEC) { // the next writes to obuf come after the barrier behind the next vertical step
            const int32_t rows = min(kBwdRows, y1 - yb);
            for (int32_t ry = 0; ry < rows; ++ry) {
                const T* src = obuf + ry * OutPitch(win);
                T* row = op + static_cast<int64_t>(yb + ry) * win;
                if constexpr (sizeof(T) == 2) {
                    const int32_t lead = static_cast<int32_t>(reinterpret_cast<uintptr_t>(row) >> 1) & 1; // elements before a word
                    for (int32_t e = 2 * static_cast<int32_t>(threadIdx.x) - lead; e < win; e += 2 * blockDim.x) {
                        if (e >= 0 && e + 1 < win) {
                            const Pack<T, 2> w{{src[e], src[e + 1]}};
                            *reinterpret_cast<Pack<T, 2>*>(row + e) = w;
                        } else {
                            const int32_t one = e < 0 ? 0 : e;
                            row[one] = src[one];
                        }
                    }
                } else {
                    for (int32_t e = threadIdx.x; e < win; e += blockDim.x) {
                        row[e] = src[e];
                    }
                }
            }
        }
    }
}

// ---- backward, atomic -------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads)
    AABwdAtomicKernel(const T* __restrict__ go, float* __restrict__ acc, int32_t hin, int32_t win, int32_t hout,
                      int32_t wout, AAAxis th, AAAxis tw, int64_t total)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int64_t row = idx / wout;
        const int32_t w = static_cast<int32_t>(idx - row * wout);
        const int64_t p = row / hout;
        const int32_t h = static_cast<int32_t>(row - p * hout);
        const int32_t hmin = __ldg(th.xmin + h), hsz = __ldg(th.xsize + h);
        const int32_t wmin = __ldg(tw.xmin + w), wsz = __ldg(tw.xsize + w);
        const float* wh = th.w + static_cast<int64_t>(h) * th.taps;
        const float* ww = tw.w + static_cast<int64_t>(w) * tw.taps;
        const float v = DType<T>::Load(go + idx);
        float* ap = acc + p * hin * static_cast<int64_t>(win);
        for (int32_t m = 0; m < hsz; ++m) {
            const float weightH = __ldg(wh + m);
            if (weightH == 0.0f) {
                continue;
            }
            float* ar = ap + static_cast<int64_t>(hmin + m) * win + wmin;
            for (int32_t n = 0; n < wsz; ++n) {
                const float weightW = __ldg(ww + n);
                if (weightW == 0.0f) {
                    continue;
                }
                atomicAdd(ar + n, Mul(Mul(v, weightH), weightW));
            }
        }
    }
}

} // namespace

// The streaming and the band kernel own whole rows with 64 or 128 threads at least: little work and narrow rows (planes of a few
// columns) are done sooner by a thread per element. Both sides beyond the fixed part of a call (tables, launches), in
// microseconds, from sweeps of 2 to 63 columns by 256 rows, 3 to 300 planes, scales of 1.4 and 4, both filters:
//   forward, thread per output: 0.6 to 1 ns per thousand taps, and the chain of one window; streaming: its start, and its rows.
//   300 planes of 3 columns 256 -> 182 rows, cubic: 10 us against 45; 31 columns 43 against 47; 63 columns 79 against 49.
//   48 planes 240x248 -> 72x77, triangle: 27 us against 17.
static bool StreamPays(const Shape4& sh, int32_t tapsH, int32_t tapsW, int filter)
{
    const double planes = static_cast<double>(sh.n) * sh.c, taps = static_cast<double>(tapsH) * tapsW;
    const double outputs = planes * sh.hout * sh.wout;
    const double elements = std::max(1e-6 * outputs * taps * (0.6 + 0.0012 * taps) * (filter == 0 ? 1.0 : 1.4), 0.06 * taps);
    return elements > 4.5 + 3.0 * std::min(1.0, sh.hin / 256.0) + 0.3e-3 * planes * sh.hin;
}
//   backward, thread per grad_input element: 40 (cubic) or 16 ns per thousand elements and the chain of its taps; band: as above.
//   300 planes of 3 columns: 19 us against 47 (cubic); 13 columns 62 against 49; triangle 25 columns 41 against 39.
static bool BandPays(const Shape4& sh, int filter)
{
    const double planes = static_cast<double>(sh.n) * sh.c;
    const double inputs = planes * sh.hin * sh.win;
    const double elements = std::max(1e-6 * inputs * (filter == 0 ? 40.0 : 16.0), filter == 0 ? std::min(5.0, 1.0 * sh.wout) : 1.0);
    return elements > 3.0 + 0.3e-3 * planes * sh.hin;
}

AAFwdPlan MakeAAFwdPlan(Dt dt, Shape4 sh, float scaleH, int32_t tapsH, int32_t tapsW, int filter)
{
    AAFwdPlan plan{};
    // Streaming needs every input row covered by at most NS outputs (true for scale >= 1) and rows that one block can own
    // (four columns per thread). Wider rows and up-scales take a thread per output element.
    const int es = DtSize(dt);
    if (!(scaleH >= 1.0f) || sh.win > 4 * kStreamThreads || sh.hin > kAAMostRows || !StreamPays(sh, tapsH, tapsW, filter)) {
        return plan;
    }
    plan.slots = filter == 0 ? 5 : 3;
    plan.threads = std::max(64, static_cast<int32_t>((CeilDiv(sh.win, 4) + 31) & ~31));
    const size_t recBytes = static_cast<size_t>(plan.slots + 1) * 8;
    const size_t rowBufs = kFlushBatch * static_cast<size_t>(ParkedRowFloats(sh.win)) * sizeof(float);
    const size_t wBytes = static_cast<size_t>(tapsW) * sh.wout * sizeof(float);
    auto metaRows = [&](int64_t bandRows) { // a band's windows span bandRows * scale + 2 * support (+ rounding) rows
        return static_cast<int32_t>(std::min<double>(
            sh.hin, std::ceil(static_cast<double>(bandRows) * scaleH + 4.0 * scaleH + 4.0)));
    };
    constexpr size_t kMostSmem = 96 * 1024; // row buffers and records, beside the horizontal weights where those fit too
    auto restBytes = [&](int64_t bandRows) { return rowBufs + static_cast<size_t>(metaRows(bandRows)) * recBytes + 32; };
    // Bands per plane, of those whose records fit: least time by a model of the walk. A block alone takes a load latency per step (about 0.3 us a
    // row with the rows in flight that its registers hold); the blocks of an SM share its issue slots (about 50
    // instructions per warp and row). Every band re-reads the rows of its first window and pays a fixed start.
    const int64_t planes = std::max<int64_t>(sh.n * sh.c, 1);
    const double warps = plan.threads / 32;
    double bestTime = 0.0;
    for (int64_t b = 1; b == 1 || sh.hout / b >= 4; b += b < 256 ? 1 : b / 16) {
        const int64_t band = CeilDiv(sh.hout, b);
        if (restBytes(band) > kMostSmem) {
            continue;
        }
        const size_t smem = restBytes(band) + 32 + (wBytes <= 48 * 1024 ? wBytes : 0);
        const int64_t perSm = std::max<int64_t>(
            1, std::min<int64_t>(1024 / plan.threads, static_cast<int64_t>((225 * 1024) / (smem + 1024))));
        const int64_t blocks = planes * CeilDiv(sh.hout, band);
        const double k = static_cast<double>(CeilDiv(blocks, NumSMs()));
        const double rows = static_cast<double>(metaRows(band)) + 10.0;
        const double time = rows * std::max(0.3 * std::ceil(k / static_cast<double>(perSm)), 0.0065 * k * warps);
        if (plan.bandRows == 0 || time < bestTime * 0.98) {
            bestTime = time;
            plan.bandRows = static_cast<int32_t>(band);
        }
    }
    if (plan.bandRows == 0) {
        return plan;
    }
    plan.stream = true;
    plan.metaRows = metaRows(plan.bandRows);
    // Horizontal weights in shared memory if they fit beside the row buffer and the records, of which 32 bytes each count: that
    // is what a record takes without its weights twice, and 48 bytes must not drive the weights out.
    const size_t rest = restBytes(plan.bandRows);
    plan.regWeights = wBytes + rest - static_cast<size_t>(plan.metaRows) * (recBytes - 32) <= kMostSmem;
    plan.wrowBytes = static_cast<uint64_t>(sh.hin) * kSlotStride * sizeof(float);
    // The bulk-copy row ring is off by default: on B200 it measured 15-25 % slower than register prefetch for this
    // kernel (the limiter is the shared-memory data pipe of the horizontal pass, not load latency, and the ring adds
    // shared-memory traffic and two block barriers per four rows). OPSCV_AA_RING=<groups> (2..4) selects it.
    plan.ringGroups = 0;
    if (const char* o = getenv("OPSCV_AA_RING")) {
        const int groups = atoi(o);
        const int32_t cols = (es == 4 && sh.win <= 4 * kRingThreads) ? 4 : 8;
        const size_t ring = static_cast<size_t>(groups) * 4 * sh.win * es + 64;
        const size_t used = rest + (plan.regWeights ? wBytes : 0);
        if (groups >= 2 && groups <= 4 && used + ring <= 200 * 1024 && sh.win % 8 == 0 && sh.win <= 8 * kRingThreads) {
            plan.ringGroups = groups;
            plan.cols = cols;
            plan.threads = std::max(64, static_cast<int32_t>((CeilDiv(sh.win, cols) + 31) & ~31));
        }
    }
    return plan;
}

uint32_t AsyncCopyTimeouts()
{
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_asyncCopyTimeouts, sizeof(v)) != cudaSuccess) {
        return 0xffffffffu;
    }
    return v;
}

cudaError_t BicubicAAFwd(Dt dt, const void* x, void* y, Shape4 sh, AAAxis th, AAAxis tw, const float* wrow,
                         const AAFwdPlan& plan, cudaStream_t s)
{
    const int64_t planes = sh.n * sh.c;
    const bool stream = plan.stream && (plan.ringGroups == 0 || Aligned(x, 16)) && planes < (1LL << 31) &&
                        CeilDiv(sh.hout, plan.bandRows) <= 65535;
    if (stream) {
        const dim3 grid(static_cast<unsigned>(planes), static_cast<unsigned>(CeilDiv(sh.hout, plan.bandRows)));
        const int32_t wTaps = plan.regWeights ? tw.taps : 0;
        const size_t base = (kFlushBatch * static_cast<size_t>(ParkedRowFloats(sh.win)) +
                             static_cast<size_t>(plan.metaRows) * 2 * (plan.slots + 1) +
                             static_cast<size_t>(wTaps) * sh.wout) * sizeof(float);
        cudaError_t e = cudaSuccess;
        OPSCV_DISPATCH_DT(dt, T, {
            const T* px = static_cast<const T*>(x);
            T* py = static_cast<T*>(y);
            const int32_t slots = plan.ringGroups * 4;
            const size_t smem = base + (plan.ringGroups > 0 ? static_cast<size_t>(slots) * sh.win * sizeof(T) +
                                                                  static_cast<size_t>((slots + 1) & ~1) * 8
                                                            : 0);
            auto launch = [&](auto kernel) {
                if (smem > 48 * 1024) {
                    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
                }
                if (e == cudaSuccess) {
                    kernel<<<grid, plan.threads, smem, s>>>(px, py, sh.hin, sh.win, sh.hout, sh.wout, th, tw, wrow,
                                                            plan.bandRows, plan.metaRows, wTaps, plan.ringGroups);
                }
            };
            constexpr int kVec = 16 / sizeof(T);
            auto pick = [&](auto slots) {
                constexpr int NS = decltype(slots)::value;
                if (plan.ringGroups > 0) {
                    if (sizeof(T) == 4 && plan.cols == 4) {
                        launch(AAFwdStreamKernel<T, NS, kVec, kVec, kRingThreads, true>);
                    } else {
                        launch(AAFwdStreamKernel<T, NS, 8, kVec, kRingThreads, true>);
                    }
                    return;
                }
                const int v = std::min(4, PickVec(static_cast<int>(sizeof(T)), sh.win, {x}));
                if (v == 4) {
                    launch(AAFwdStreamKernel<T, NS, 4, 4, kStreamThreads, false>);
                } else if (v == 2) {
                    launch(AAFwdStreamKernel<T, NS, 4, 2, kStreamThreads, false>);
                } else {
                    launch(AAFwdStreamKernel<T, NS, 4, 1, kStreamThreads, false>);
                }
            };
            if (plan.slots == 5) {
                pick(std::integral_constant<int, 5>{});
            } else {
                pick(std::integral_constant<int, 3>{});
            }
        });
        CountLaunch();
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    const int64_t total = planes * sh.hout * static_cast<int64_t>(sh.wout);
    OPSCV_DISPATCH_DT(dt, T, {
        AAFwdDirectKernel<T><<<GridFor(total, kThreads), kThreads, 0, s>>>(
            static_cast<const T*>(x), static_cast<T*>(y), sh.hin, sh.win, sh.hout, sh.wout, th, tw, total);
    });
    CountLaunch();
    return cudaGetLastError();
}

// Shared memory of one block of the band kernel: slot records of the band's rows, staged grads rows, step buffer.
// and, for rows that are parked before they are written, those rows.
static size_t AABwdSmem(int32_t bandRows, int32_t stageRows, int32_t wout, int32_t win, int es, bool parked)
{
    const size_t groups = static_cast<size_t>(bandRows) / kBwdRows;
    return groups * kBwdGroupBytes + static_cast<size_t>(BwdStagedFloats(stageRows, wout)) * sizeof(float) +
           (parked ? static_cast<size_t>(kBwdRows) * OutPitch(win) * es : 0);
}

AABwdPlan MakeAABwdPlan(Dt dt, Shape4 sh, float scaleH, float scaleW, int filter)
{
    AABwdPlan plan{};
    const int es = DtSize(dt);
    // Same covering bound as the forward streaming kernel, on both axes; one block owns whole grad_input rows.
    plan.band = scaleH >= 1.0f && scaleW >= 1.0f && sh.win <= 4096 && sh.hin <= kAAMostRows && BandPays(sh, filter);
    if (!plan.band) {
        return plan;
    }
    // grads columns that reach four adjacent columns: centres in a span of 2 * support + 3, one more through rounding
    plan.colSlots = (filter == 1 || scaleW >= 3.0f) ? 6 : 8;
    plan.threads = std::min(1024, std::max(128, static_cast<int32_t>((CeilDiv(sh.win, 4) + 31) & ~31)));
    // Bands per plane: the split whose blocks fill whole waves of resident blocks best (up to four 256-thread
    // blocks per SM, fewer if the staged grads rows need more shared memory). t grad_input rows are fed by at most
    // t / scale + kSlots + 2 grads rows.
    const int64_t planes = std::max<int64_t>(sh.n * sh.c, 1);
    double bestScore = 0.0;
    for (int32_t b = 1; b <= 256 && (b == 1 || sh.hin / b >= 4 * kBwdRows); ++b) {
        int32_t band = static_cast<int32_t>(CeilDiv(sh.hin, b));
        band = (band + kBwdRows - 1) / kBwdRows * kBwdRows;
        const int32_t stage = static_cast<int32_t>(
            std::min<int64_t>(static_cast<int64_t>(band / static_cast<double>(scaleH)) + kSlots + 2, sh.hout));
        const size_t smem = AABwdSmem(band, stage, sh.wout, sh.win, es, sh.win % 4 != 0);
        // (an unaligned grad_input parks its rows too)
        if (smem > 200 * 1024 || AABwdSmem(band, stage, sh.wout, sh.win, es, true) > 224 * 1024) {
            continue;
        }
        const int64_t perSm = std::min<int64_t>({4, 2048 / plan.threads, static_cast<int64_t>((225 * 1024) / (smem + 1024))});
        const int64_t slots = static_cast<int64_t>(NumSMs()) * std::max<int64_t>(perSm, 1);
        const int64_t blocks = planes * CeilDiv(sh.hin, band);
        // waves filled, times the residency reached, with a slight preference for fewer (taller) bands
        const double score = static_cast<double>(blocks) / (static_cast<double>(CeilDiv(blocks, slots)) * slots) *
                             (0.5 + 0.125 * static_cast<double>(perSm)) - 0.001 * b;
        if (score > bestScore) {
            bestScore = score;
            plan.bandRows = band;
            plan.stageRows = stage;
        }
    }
    if (bestScore <= 0.0) {
        plan.band = false;
        return plan;
    }
    plan.wrowBytesH = static_cast<uint64_t>(sh.hin) * kSlotStride * sizeof(float);
    plan.wrowBytesW = static_cast<uint64_t>(sh.win) * kSlotStride * sizeof(float);
    return plan;
}

cudaError_t BicubicAABwdGather(Dt dt, const void* go, void* gi, Shape4 sh, AAAxis th, AAAxis tw, RangeAxis rh,
                               RangeAxis rw, const float* wrowH, const float* wrowW, const AABwdPlan& plan,
                               cudaStream_t s)
{
    const int64_t planes = sh.n * sh.c;
    const bool band = plan.band && planes < (1LL << 31) && CeilDiv(sh.hin, plan.bandRows) <= 65535;
    if (band) {
        const dim3 grid(static_cast<unsigned>(planes), static_cast<unsigned>(CeilDiv(sh.hin, plan.bandRows)));
        const bool vec = sh.win % 4 == 0 && Aligned(gi, 16);
        const size_t smem = AABwdSmem(plan.bandRows, plan.stageRows, sh.wout, sh.win, DtSize(dt), !vec);
        cudaError_t e = cudaSuccess;
        OPSCV_DISPATCH_DT(dt, T, {
            auto launch = [&](auto kernel) {
                if (smem > 48 * 1024) {
                    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
                }
                if (e == cudaSuccess) {
                    kernel<<<grid, plan.threads, smem, s>>>(static_cast<const T*>(go), static_cast<T*>(gi), sh.hin, sh.win,
                                                            sh.hout, sh.wout, rh, rw, wrowH, wrowW, plan.bandRows,
                                                            plan.stageRows);
                }
            };
            if (plan.colSlots == 6) {
                launch(vec ? AABwdBandKernel<T, true, 6> : AABwdBandKernel<T, false, 6>);
            } else {
                launch(vec ? AABwdBandKernel<T, true, 8> : AABwdBandKernel<T, false, 8>);
            }
        });
        CountLaunch();
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    const int64_t total = planes * sh.hin * static_cast<int64_t>(sh.win);
    OPSCV_DISPATCH_DT(dt, T, {
        AABwdGatherKernel<T><<<GridFor(total, kThreads), kThreads, 0, s>>>(
            static_cast<const T*>(go), static_cast<T*>(gi), sh.hin, sh.win, sh.hout, sh.wout, th, tw, rh, rw, total);
    });
    CountLaunch();
    return cudaGetLastError();
}

cudaError_t BicubicAABwdAtomic(Dt dt, const void* go, void* gi, float* acc, Shape4 sh, AAAxis th, AAAxis tw,
                               cudaStream_t s)
{
    const int64_t outElems = sh.n * sh.c * sh.hin * static_cast<int64_t>(sh.win);
    const int64_t total = sh.n * sh.c * sh.hout * static_cast<int64_t>(sh.wout);
    cudaError_t e = cudaMemsetAsync(acc, 0, static_cast<size_t>(outElems) * sizeof(float), s);
    if (e != cudaSuccess) {
        return e;
    }
    OPSCV_DISPATCH_DT(dt, T, {
        AABwdAtomicKernel<T><<<GridFor(total, kThreads), kThreads, 0, s>>>(static_cast<const T*>(go), acc, sh.hin,
                                                                           sh.win, sh.hout, sh.wout, th, tw, total);
    });
    CountLaunch(2);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        return e;
    }
    if (dt != Dt::F32 || static_cast<void*>(acc) != gi) {
        return CastFromF32(dt, gi, acc, outElems, s);
    }
    return cudaSuccess;
}

} // namespace opscv
