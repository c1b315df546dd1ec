// Batched lens-parameter sweep: hundreds of samples with uneven image sizes and visibility
// counts go through deflection, degridding and gridding in one CUDA graph.
//
// Every sample brings its own plan (binned visibilities; tile, KB width and chunk chosen per
// sample), its lens model and its pixel grid. The host flattens all of the samples' work into
// lists of items, ordered longest first:
//   grid    -- one plan work item of a sample into the sample's half-plane grid;
//   degrid  -- one plan work item of a sample into plan-order visibilities;
//   deflect -- kDeflectChunk pixels of a sample's grid: beta = theta - sum_l alpha_l(theta).
//
// The default form launches one kernel per kind and Kaiser-Bessel table, one CTA per item over
// all samples, on three branches of the graph (grids: zeroing, then gridding; degridding;
// deflection), so that big samples spread over the whole GPU and small ones fill the gaps. Each
// kernel is the single-plan one's item function with the registers it wants and its table in
// constant memory. One persistent kernel for all kinds (forms 1 and 2, and what samples with more
// than kMaxGroups tables fall back to) has to hold every path at once: under 80 registers, the
// limit for three CTAs per SM, the faster item functions spill, and each item stages its table
// in shared memory. 20 samples, 1.7e7 visibilities: 840 us persistent, 570 us split.
#include <algorithm>
#include <climits>
#include <new>
#include <vector>

#include "common.cuh"
#include "deflect_device.cuh"
#include "gridding_items.cuh"

namespace lentils {

constexpr int kDeflectChunk = 2048;  // pixels per deflection item
constexpr int kSweepMaxLenses = 8;   // lenses per sample

enum SweepKind { kSweepGrid = 0, kSweepDegrid = 1, kSweepDeflect = 2 };

struct SweepWork {
    int sample, kind, index, pad;
};

struct SweepSampleDev {
    GridGeom g;
    KBPoly kb;
    int w2;
    int nitems;
    const uint2 *coords;
    const WorkItem *items;
    const int *chunk_begin;   // same-cell chunks (null: not built)
    const int2 *item_chunks;
    const float2 *grid_in;
    float2 *vis_out;
    const float2 *vis_in;
    float2 *grid_out;
    int lens0, nlenses;
    int nx, ny;
    double x0, y0, dx, dy;
    float2 *beta_out;
};

static __device__ __noinline__ float2 pixel_tail(const DevLens &L, const SweepSampleDev &s, int i,
                                                 int j)
{
    return series_tail(L, (s.x0 - L.x0) + i * s.dx, (s.y0 - L.y0) + j * s.dy);
}

// not inlined: its registers would otherwise push the gridding path into spills
static __device__ __noinline__ void deflect_chunk(const SweepSampleDev &s,
                                                  const DevLens *__restrict__ lenses, int chunk)
{
    const long long npix = (long long)s.nx * s.ny;
    const long long p0 = (long long)chunk * kDeflectChunk;
    const long long p1 = min(npix, p0 + kDeflectChunk);
    // positions x0 + i dx in FP32 pairs (hi + lo), so the pixel loop stays off the FP64 units:
    // the offset from a lens centre, (x0 - xc) + i dx with x0 - xc a pair made on the host, is
    // formed with an exact product error (fma) and a two-sum, rounded once
    const float dxh = (float)s.dx, dxl = (float)(s.dx - (double)dxh);
    const float dyh = (float)s.dy, dyl = (float)(s.dy - (double)dyh);
    const float xh = (float)s.x0, xl = (float)(s.x0 - (double)xh);
    const float yh = (float)s.y0, yl = (float)(s.y0 - (double)yh);
    auto pair_sum = [](float ch, float cl, float2 k, float dh, float dl) {  // (ch+cl) + k(dh+dl)
        const float2 c = splat(ch), d = splat(dh);
        const float2 pr = __fmul2_rn(k, d);
        const float2 pe = __ffma2_rn(k, d, neg2(pr));
        const float2 sm = __fadd2_rn(c, pr);
        const float2 bp = sub2(sm, c);
        const float2 e = __fadd2_rn(sub2(c, sub2(sm, bp)), sub2(pr, bp));
        return __fadd2_rn(sm, __fadd2_rn(__fadd2_rn(e, pe), __ffma2_rn(k, splat(dl), splat(cl))));
    };
    // two pixels per thread and step, blockDim.x apart: each store is coalesced
    for (long long p = p0 + threadIdx.x; p < p1; p += 2 * blockDim.x) {
        const long long pb = min(p + blockDim.x, npix - 1);
        const int i = (int)(p / s.ny), j = (int)(p - (long long)i * s.ny);
        const int ib = (int)(pb / s.ny), jb = (int)(pb - (long long)ib * s.ny);
        const float2 ki = make_float2((float)i, (float)ib), kj = make_float2((float)j, (float)jb);
        float2 axs = splat(0.f), ays = splat(0.f), sx[1], sy[1];
        for (int l = 0; l < s.nlenses; ++l) {
            const DevLens &L = lenses[s.lens0 + l];
            float2 ax[1], ay[1];
            if (!L.same_centre) {
                sx[0] = pair_sum(L.gxh, L.gxl, ki, dxh, dxl);
                sy[0] = pair_sum(L.gyh, L.gyl, kj, dyh, dyl);
            }
            lens_alpha<1>(L, sx, sy, [&](const DevLens &T, int, int h) {
                return pixel_tail(T, s, h ? ib : i, h ? jb : j);
            }, ax, ay);
            axs = __fadd2_rn(axs, ax[0]);
            ays = __fadd2_rn(ays, ay[0]);
        }
        const float2 bx = sub2(pair_sum(xh, xl, ki, dxh, dxl), axs);
        const float2 by = sub2(pair_sum(yh, yl, kj, dyh, dyl), ays);
        s.beta_out[p] = make_float2(bx.x, by.x);
        if (p + blockDim.x < p1) s.beta_out[p + blockDim.x] = make_float2(bx.y, by.y);
    }
}

// -- the split form -------------------------------------------------------------------------
constexpr int kMaxGroups = 4;  // Kaiser-Bessel tables with kernels of their own

// A plan work item of a sample, with all that locates it.
struct SweepItem {
    int sample, pad;
    WorkItem it;
    int2 chunks;  // its same-cell chunks
};

template <int W2>
__global__ void __launch_bounds__(128)
    sweep_grid_kernel(const SweepSampleDev *__restrict__ samples,
                      const SweepItem *__restrict__ items, const __grid_constant__ KBPoly kb)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const SweepItem d = items[blockIdx.x];
    const SweepSampleDev &s = samples[d.sample];
    const GridGeom g = s.g;
    grid_rows_item_pairs<W2, 4>(s.vis_in, s.coords, s.grid_out, d.it, kb, g, smraw);
}

template <int W2>
__global__ void __launch_bounds__(128, 4)
    sweep_degrid_kernel(const SweepSampleDev *__restrict__ samples,
                        const SweepItem *__restrict__ items, const __grid_constant__ KBPoly kb)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const SweepItem d = items[blockIdx.x];
    const SweepSampleDev &s = samples[d.sample];
    const GridGeom g = s.g;
    degrid_item_chunks<W2, 4>(s.grid_in, s.coords, s.vis_out, d.it, d.chunks, s.chunk_begin, kb,
                              g, smraw);
}

// work: (sample, chunk) pairs
__global__ void __launch_bounds__(256)
    sweep_deflect_kernel(const SweepSampleDev *__restrict__ samples,
                         const int2 *__restrict__ work, const DevLens *__restrict__ lenses)
{
    const int2 w = work[blockIdx.x];
    deflect_chunk(samples[w.x], lenses, w.y);
}

// All samples' output grids, kZeroBlocks CTAs each (one launch instead of a memset per sample).
constexpr int kZeroBlocks = 16;
__global__ void __launch_bounds__(256) sweep_zero_kernel(const SweepSampleDev *__restrict__ samples)
{
    const SweepSampleDev &s = samples[blockIdx.x / kZeroBlocks];
    if (!s.grid_out) return;
    const long long n = (long long)s.g.nu * s.g.half_nv;
    const long long first = (blockIdx.x % kZeroBlocks) * 256LL + threadIdx.x;
    if (reinterpret_cast<uintptr_t>(s.grid_out) & 15) {
        for (long long e = first; e < n; e += kZeroBlocks * 256) s.grid_out[e] = make_float2(0.f, 0.f);
        return;
    }
    float4 *p = reinterpret_cast<float4 *>(s.grid_out);
    for (long long e = first; e < n / 2; e += kZeroBlocks * 256) p[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((n & 1) && first == 0) s.grid_out[n - 1] = make_float2(0.f, 0.f);
}

// -- the persistent forms -------------------------------------------------------------------
// FORM 0: the ballot gridder and one visibility per degridding thread, three CTAs per SM (80
// registers, a few bytes of spill). FORM 1: the column-pair gridder and same-cell chunk
// degridding, two CTAs per SM (128 registers). FORM 2: the column-pair gridder and one
// visibility per degridding thread, two CTAs per SM.
template <int FORM>
__global__ void __launch_bounds__(kGridBatch, FORM == 0 ? 3 : 2)
    sweep_kernel(const SweepSampleDev *__restrict__ samples, const SweepWork *__restrict__ work,
                 int nwork, const DevLens *__restrict__ lenses, int *__restrict__ counter)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int next;
    __shared__ KBPoly kb;
    __shared__ GridGeom g;
    for (;;) {
        __syncthreads();  // the previous item is done with shared memory
        if (threadIdx.x == 0) next = atomicAdd(counter, 1);
        __syncthreads();
        const int w = next;
        if (w >= nwork) break;
        const SweepWork d = work[w];
        const SweepSampleDev &s = samples[d.sample];
        if (d.kind == kSweepDeflect) {
            deflect_chunk(s, lenses, d.index);
            continue;
        }
        // the sample's KB table and geometry, staged once per item
        {
            const int *src = reinterpret_cast<const int *>(&s.kb);
            int *dst = reinterpret_cast<int *>(&kb);
            for (int k = threadIdx.x; k < (int)(sizeof(KBPoly) / 4); k += blockDim.x) dst[k] = src[k];
            if (threadIdx.x == 0) g = s.g;
        }
        __syncthreads();
        const WorkItem it = s.items[d.index];
        if constexpr (FORM != 0) {
            if (d.kind == kSweepGrid) {
                if (s.w2 == 8)
                    grid_rows_item_pairs<8, 8>(s.vis_in, s.coords, s.grid_out, it, kb, g, smraw);
                else
                    grid_rows_item_pairs<6, 8>(s.vis_in, s.coords, s.grid_out, it, kb, g, smraw);
            } else if constexpr (FORM == 1) {
                const int2 cr = s.item_chunks[d.index];
                if (s.w2 == 8)
                    degrid_item_chunks<8, 4>(s.grid_in, s.coords, s.vis_out, it, cr,
                                             s.chunk_begin, kb, g, smraw);
                else
                    degrid_item_chunks<6, 4>(s.grid_in, s.coords, s.vis_out, it, cr,
                                             s.chunk_begin, kb, g, smraw);
            } else {
                if (s.w2 == 8) degrid_item<8, float>(s.grid_in, s.coords, s.vis_out, it, kb, g, nullptr, smraw);
                else degrid_item<6, float>(s.grid_in, s.coords, s.vis_out, it, kb, g, nullptr, smraw);
            }
        } else {
            if (d.kind == kSweepGrid) {
                if (s.w2 == 8)
                    grid_rows_item_ballot<8>(s.vis_in, s.coords, s.grid_out, it, kb, g, smraw);
                else
                    grid_rows_item_ballot<6>(s.vis_in, s.coords, s.grid_out, it, kb, g, smraw);
            } else {
                if (s.w2 == 8) degrid_item<8, float>(s.grid_in, s.coords, s.vis_out, it, kb, g, nullptr, smraw);
                else degrid_item<6, float>(s.grid_in, s.coords, s.vis_out, it, kb, g, nullptr, smraw);
            }
        }
    }
}

}  // namespace lentils

struct SweepGroup {  // items of one Kaiser-Bessel table
    lentils::KBPoly kb;
    int w2, nitems;
    size_t grid_smem, degrid_smem;
    lentils::SweepItem *items;
};

struct lentils_sweep {
    bool split;  // the split form; else the persistent kernel
    std::vector<SweepGroup> groups;
    int2 *chunks;  // deflection work of the split form
    int nchunks;
    cudaStream_t side[2];  // its degridding and deflection branches
    cudaEvent_t fork, join[2];
    int nsamples;
    int nwork;
    int blocks;
    int form;  // sweep_kernel<form>
    size_t smem;
    long long total_vis, total_pixels;
    double algorithmic_bytes;
    lentils::SweepSampleDev *samples;
    lentils::SweepWork *work;
    lentils::DevLens *lenses;
    int *counter;
    std::vector<std::pair<float2 *, size_t>> zero;  // output grids to clear per run
    cudaGraph_t graph;
    cudaGraphExec_t gexec;
};

using namespace lentils;

static void sweep_free(lentils_sweep *sw)
{
    if (sw->gexec) cudaGraphExecDestroy(sw->gexec);
    if (sw->graph) cudaGraphDestroy(sw->graph);
    cudaFree(sw->samples);
    cudaFree(sw->work);
    cudaFree(sw->lenses);
    cudaFree(sw->counter);
    for (auto &g : sw->groups) cudaFree(g.items);
    cudaFree(sw->chunks);
    for (int k = 0; k < 2; ++k) {
        if (sw->side[k]) cudaStreamDestroy(sw->side[k]);
        if (sw->join[k]) cudaEventDestroy(sw->join[k]);
    }
    if (sw->fork) cudaEventDestroy(sw->fork);
}

constexpr size_t kMaxSweepSmem = 200 * 1024;

// The limit, not one group's need: groups and sweeps share the kernels.
template <typename K>
static cudaError_t sweep_smem_attr(K kern)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kMaxSweepSmem);
}

// The split form's launches, forked from s and joined to it again.
static int sweep_enqueue_split(lentils_sweep *sw, cudaStream_t s)
{
    LENTILS_CUDA_TRY(cudaEventRecord(sw->fork, s));
    for (int k = 0; k < 2; ++k) LENTILS_CUDA_TRY(cudaStreamWaitEvent(sw->side[k], sw->fork, 0));
    if (sw->nsamples > 0) {
        sweep_zero_kernel<<<sw->nsamples * kZeroBlocks, 256, 0, s>>>(sw->samples);
        LENTILS_CHECK_LAUNCH("sweep_zero_kernel");
    }
    for (const SweepGroup &g : sw->groups) {
        if (g.nitems == 0) continue;
        if (g.w2 == 8) {
            sweep_grid_kernel<8><<<g.nitems, 128, g.grid_smem, s>>>(sw->samples, g.items, g.kb);
            sweep_degrid_kernel<8><<<g.nitems, 128, g.degrid_smem, sw->side[0]>>>(sw->samples,
                                                                                g.items, g.kb);
        } else {
            sweep_grid_kernel<6><<<g.nitems, 128, g.grid_smem, s>>>(sw->samples, g.items, g.kb);
            sweep_degrid_kernel<6><<<g.nitems, 128, g.degrid_smem, sw->side[0]>>>(sw->samples,
                                                                                g.items, g.kb);
        }
        LENTILS_CHECK_LAUNCH("sweep grid / degrid kernel");
    }
    if (sw->nchunks > 0) {
        sweep_deflect_kernel<<<sw->nchunks, 256, 0, sw->side[1]>>>(sw->samples, sw->chunks,
                                                                  sw->lenses);
        LENTILS_CHECK_LAUNCH("sweep_deflect_kernel");
    }
    for (int k = 0; k < 2; ++k) {
        LENTILS_CUDA_TRY(cudaEventRecord(sw->join[k], sw->side[k]));
        LENTILS_CUDA_TRY(cudaStreamWaitEvent(s, sw->join[k], 0));
    }
    return LENTILS_OK;
}

static cudaError_t sweep_set_smem(int form, int smem)
{
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (form == 1) return cudaFuncSetAttribute(sweep_kernel<1>, a, smem);
    if (form == 2) return cudaFuncSetAttribute(sweep_kernel<2>, a, smem);
    return cudaFuncSetAttribute(sweep_kernel<0>, a, smem);
}

static cudaError_t sweep_occupancy(int form, int *per_sm, size_t smem)
{
    if (form == 1)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, sweep_kernel<1>, kGridBatch, smem);
    if (form == 2)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, sweep_kernel<2>, kGridBatch, smem);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, sweep_kernel<0>, kGridBatch, smem);
}

static int sweep_enqueue(lentils_sweep *sw, cudaStream_t s)
{
    if (sw->split) return sweep_enqueue_split(sw, s);
    LENTILS_CUDA_TRY(cudaMemsetAsync(sw->counter, 0, sizeof(int), s));
    for (auto &z : sw->zero) LENTILS_CUDA_TRY(cudaMemsetAsync(z.first, 0, z.second, s));
    if (sw->nwork > 0) {
        if (sw->form == 1)
            sweep_kernel<1><<<sw->blocks, kGridBatch, sw->smem, s>>>(
                sw->samples, sw->work, sw->nwork, sw->lenses, sw->counter);
        else if (sw->form == 2)
            sweep_kernel<2><<<sw->blocks, kGridBatch, sw->smem, s>>>(
                sw->samples, sw->work, sw->nwork, sw->lenses, sw->counter);
        else
            sweep_kernel<0><<<sw->blocks, kGridBatch, sw->smem, s>>>(
                sw->samples, sw->work, sw->nwork, sw->lenses, sw->counter);
        LENTILS_CHECK_LAUNCH("sweep_kernel");
    }
    return LENTILS_OK;
}

extern "C" {

int lentils_sweep_create(lentils_sweep **out, const lentils_sweep_sample *in, int n, int flags,
                         void *stream)
{
    clear_error();
    if (!out || (!in && n > 0) || n < 0) return set_error(LENTILS_ERR_INVALID, "sweep_create: bad arguments");
    *out = nullptr;
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<SweepSampleDev> hs(n);
    std::vector<DevLens> hl;
    std::vector<std::pair<double, SweepWork>> items;
    lentils_sweep *sw = new (std::nothrow) lentils_sweep();
    if (!sw) return set_error(LENTILS_ERR_ALLOC, "sweep_create: host allocation");
    sw->form = flags & LENTILS_SWEEP_FORM_MASK;
    if (sw->form > 2) {
        delete sw;
        return set_error(LENTILS_ERR_INVALID, "sweep_create: kernel form %d (0 to 2)", flags & 3);
    }
    sw->split = sw->form == 0;
    std::vector<std::vector<std::pair<double, SweepItem>>> gitems;  // per group
    std::vector<std::pair<double, int2>> chunks;
    size_t smem = 0;
    int st = LENTILS_OK;
    for (int k = 0; k < n && !st; ++k) {
        const lentils_sweep_sample &a = in[k];
        const lentils_plan *p = a.plan;
        SweepSampleDev &d = hs[k];
        memset(&d, 0, sizeof(d));
        d.lens0 = (int)hl.size();
        d.nlenses = a.nlenses;
        d.nx = a.nx;
        d.ny = a.ny;
        d.x0 = a.x0;
        d.y0 = a.y0;
        d.dx = a.dx;
        d.dy = a.dy;
        d.beta_out = reinterpret_cast<float2 *>(a.beta_out);
        if (a.nlenses < 0 || a.nlenses > kSweepMaxLenses || (a.nlenses > 0 && !a.lenses) ||
            a.nx < 0 || a.ny < 0 || ((long long)a.nx * a.ny > 0 && !a.beta_out)) {
            st = set_error(LENTILS_ERR_INVALID, "sweep_create: sample %d: lenses or pixel grid", k);
            break;
        }
        for (int l = 0; l < a.nlenses && !st; ++l) {
            DevLens L;
            st = build_lens(a.lenses[l], L);
            const double gx = a.x0 - L.x0, gy = a.y0 - L.y0;
            L.gxh = (float)gx;
            L.gxl = (float)(gx - (double)L.gxh);
            L.gyh = (float)gy;
            L.gyl = (float)(gy - (double)L.gyh);
            L.same_centre = l > 0 && L.x0 == hl.back().x0 && L.y0 == hl.back().y0;
            hl.push_back(L);
        }
        if (st) break;
        const long long npix = (long long)a.nx * a.ny;
        sw->total_pixels += npix;
        for (long long c = 0; c * kDeflectChunk < npix; ++c) {
            const double cost = (double)std::min<long long>(kDeflectChunk, npix - c * kDeflectChunk) *
                                (0.6 + 0.3 * a.nlenses);
            items.push_back({cost, SweepWork{k, kSweepDeflect, (int)c, 0}});
            chunks.push_back({cost, make_int2(k, (int)c)});
        }
        if (!p) continue;
        const int w2 = 2 * p->geom.w;
        if (w2 != 6 && w2 != 8) {
            st = set_error(LENTILS_ERR_UNSUPPORTED, "sweep_create: sample %d: KB width %d (6 or 8)", k, w2);
            break;
        }
        if (!a.grid_in || !a.vis_out || !a.vis_in || !a.grid_out) {
            st = set_error(LENTILS_ERR_INVALID, "sweep_create: sample %d: null grid/vis buffer", k);
            break;
        }
        d.g = p->geom;
        d.kb = p->kb;
        d.w2 = w2;
        d.nitems = p->nitems;
        d.coords = p->coords;
        d.items = p->items;
        d.chunk_begin = p->chunk_begin;
        d.item_chunks = p->item_chunks;
        if (sw->form == 1 && p->nitems > 0 && (!p->chunk_begin || p->chunk_k != 4)) {
            st = set_error(LENTILS_ERR_UNSUPPORTED, "sweep_create: sample %d: no chunks", k);
            break;
        }
        d.grid_in = reinterpret_cast<const float2 *>(a.grid_in);
        d.vis_out = reinterpret_cast<float2 *>(a.vis_out);
        d.vis_in = reinterpret_cast<const float2 *>(a.vis_in);
        d.grid_out = reinterpret_cast<float2 *>(a.grid_out);
        const size_t gbytes = sizeof(float2) * (size_t)p->geom.nu * p->geom.half_nv;
        sw->zero.push_back({d.grid_out, gbytes});
        sw->total_vis += p->nvis;
        sw->algorithmic_bytes += 2.0 * (16.0 * (double)p->nvis + (double)gbytes);
        if (sw->form != 0)
            smem = std::max(smem, w2 == 8 ? grid_pairs_smem_bytes<8, 8>(p->geom)
                                          : grid_pairs_smem_bytes<6, 8>(p->geom));
        else
            smem = std::max(smem, w2 == 8 ? grid_ballot_smem_bytes<8>(p->geom)
                                          : grid_ballot_smem_bytes<6>(p->geom));
        smem = std::max(smem, degrid_smem_bytes<float>(p->geom));
        std::vector<WorkItem> hitems(p->nitems);
        if (p->nitems > 0) {
            cudaError_t e = cudaMemcpy(hitems.data(), p->items, sizeof(WorkItem) * p->nitems,
                                       cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) {
                st = cuda_status(e, "sweep_create items");
                break;
            }
        }
        // the split form: this sample's items join the group of its table
        std::vector<int2> hchunks(p->nitems);
        if (p->nitems > 0 && (!p->chunk_begin || p->chunk_k != 4)) sw->split = false;
        if (sw->split) {
            size_t q = 0;
            while (q < sw->groups.size() &&
                   (sw->groups[q].w2 != w2 || memcmp(&sw->groups[q].kb, &p->kb, sizeof(KBPoly))))
                ++q;
            if (q == sw->groups.size()) {
                if (q == kMaxGroups) {
                    sw->split = false;
                } else {
                    sw->groups.push_back(SweepGroup{p->kb, w2, 0, 0, 0, nullptr});
                    gitems.emplace_back();
                }
            }
            if (sw->split) {
                SweepGroup *grp = &sw->groups[q];
                grp->grid_smem = std::max(grp->grid_smem, w2 == 8
                                                              ? grid_pairs_smem_bytes<8, 4>(p->geom)
                                                              : grid_pairs_smem_bytes<6, 4>(p->geom));
                grp->degrid_smem = std::max(grp->degrid_smem, degrid_smem_bytes<float>(p->geom));
                if (std::max(grp->grid_smem, grp->degrid_smem) > kMaxSweepSmem) sw->split = false;
                if (p->nitems > 0) {
                    const cudaError_t e =
                        cudaMemcpy(hchunks.data(), p->item_chunks, sizeof(int2) * p->nitems,
                                   cudaMemcpyDeviceToHost);
                    if (e != cudaSuccess) {
                        st = cuda_status(e, "sweep_create chunks");
                        break;
                    }
                    for (int i = 0; i < p->nitems; ++i)
                        gitems[q].push_back({(double)hitems[i].count +
                                                 0.5 * p->geom.E * p->geom.E,
                                             SweepItem{k, 0, hitems[i], hchunks[i]}});
                }
            }
        }
        const double tile_cost = (double)p->geom.E * p->geom.E;
        const double taps = (double)w2 * w2;
        for (int i = 0; i < p->nitems; ++i) {
            const double c = (double)hitems[i].count;
            items.push_back({2.0 * tile_cost + c * taps * 0.35, SweepWork{k, kSweepGrid, i, 0}});
            items.push_back({tile_cost + c * taps * 0.2, SweepWork{k, kSweepDegrid, i, 0}});
        }
    }
    sw->algorithmic_bytes += 8.0 * (double)sw->total_pixels;
    if (!st && smem > kMaxSweepSmem)
        st = set_error(LENTILS_ERR_UNSUPPORTED, "sweep_create: %zu bytes of shared memory per item", smem);
    if (st) {
        delete sw;
        return st;
    }
    sw->nsamples = n;
    sw->nwork = (int)items.size();
    cudaError_t e = cudaMalloc(&sw->samples, sizeof(SweepSampleDev) * std::max(1, n));
    if (e == cudaSuccess) e = cudaMalloc(&sw->lenses, sizeof(DevLens) * std::max<size_t>(1, hl.size()));
    if (e == cudaSuccess && n > 0)
        e = cudaMemcpyAsync(sw->samples, hs.data(), sizeof(SweepSampleDev) * n, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !hl.empty())
        e = cudaMemcpyAsync(sw->lenses, hl.data(), sizeof(DevLens) * hl.size(), cudaMemcpyHostToDevice, s);
    // sources of copies on s, as hs and hl: until the wait below
    std::vector<std::vector<SweepItem>> hgroups(sw->groups.size());
    std::vector<int2> hchunk;
    std::vector<SweepWork> hw;
    const auto longest = [](const auto &x, const auto &y) { return x.first > y.first; };
    if (sw->split) {
        long long ctas = (long long)n * kZeroBlocks + (long long)chunks.size();
        sw->smem = 0;
        for (size_t q = 0; q < sw->groups.size() && e == cudaSuccess; ++q) {
            SweepGroup &g = sw->groups[q];
            std::stable_sort(gitems[q].begin(), gitems[q].end(), longest);
            std::vector<SweepItem> &h = hgroups[q];
            for (const auto &x : gitems[q]) h.push_back(x.second);
            g.nitems = (int)h.size();
            ctas += 2LL * g.nitems;
            sw->smem = std::max(sw->smem, std::max(g.grid_smem, g.degrid_smem));
            e = cudaMalloc(&g.items, sizeof(SweepItem) * std::max<size_t>(1, h.size()));
            if (e == cudaSuccess && !h.empty())
                e = cudaMemcpyAsync(g.items, h.data(), sizeof(SweepItem) * h.size(),
                                    cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess)
                e = g.w2 == 8 ? sweep_smem_attr(sweep_grid_kernel<8>)
                              : sweep_smem_attr(sweep_grid_kernel<6>);
            if (e == cudaSuccess)
                e = g.w2 == 8 ? sweep_smem_attr(sweep_degrid_kernel<8>)
                              : sweep_smem_attr(sweep_degrid_kernel<6>);
        }
        std::stable_sort(chunks.begin(), chunks.end(), longest);
        for (const auto &x : chunks) hchunk.push_back(x.second);
        sw->nchunks = (int)hchunk.size();
        if (e == cudaSuccess)
            e = cudaMalloc(&sw->chunks, sizeof(int2) * std::max<size_t>(1, hchunk.size()));
        if (e == cudaSuccess && !hchunk.empty())
            e = cudaMemcpyAsync(sw->chunks, hchunk.data(), sizeof(int2) * hchunk.size(),
                                cudaMemcpyHostToDevice, s);
        for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
            e = cudaStreamCreateWithFlags(&sw->side[k], cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sw->join[k], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sw->fork, cudaEventDisableTiming);
        sw->blocks = (int)std::min<long long>(INT_MAX, ctas);
    } else {
        std::stable_sort(items.begin(), items.end(), longest);
        for (const auto &x : items) hw.push_back(x.second);
        sw->smem = std::max<size_t>(smem, 16);
        if (e == cudaSuccess) e = cudaMalloc(&sw->counter, sizeof(int));
        if (e == cudaSuccess)
            e = cudaMalloc(&sw->work, sizeof(SweepWork) * std::max<size_t>(1, hw.size()));
        if (e == cudaSuccess && !hw.empty())
            e = cudaMemcpyAsync(sw->work, hw.data(), sizeof(SweepWork) * hw.size(),
                                cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = sweep_set_smem(sw->form, (int)sw->smem);
        int per_sm = 0, nsm = 0, dev = 0;
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = sweep_occupancy(sw->form, &per_sm, sw->smem);
        sw->blocks = std::max(1, std::min(sw->nwork, std::max(1, per_sm) * nsm));
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        st = cuda_status(e, "sweep_create");
        sweep_free(sw);
        delete sw;
        return st;
    }
    *out = sw;
    return LENTILS_OK;
}

int lentils_sweep_destroy(lentils_sweep *sw)
{
    clear_error();
    if (!sw) return LENTILS_OK;
    sweep_free(sw);
    delete sw;
    return LENTILS_OK;
}

int lentils_sweep_run(lentils_sweep *sw, int use_graph, void *stream)
{
    clear_error();
    if (!sw) return set_error(LENTILS_ERR_INVALID, "sweep_run: null");
    cudaStream_t s = (cudaStream_t)stream;
    if (!use_graph) return sweep_enqueue(sw, s);
    if (!s) return set_error(LENTILS_ERR_INVALID, "sweep_run: graph capture needs a non-default stream");
    if (!sw->gexec) {
        cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return cuda_status(e, "sweep capture");
        const int q = sweep_enqueue(sw, s);
        e = cudaStreamEndCapture(s, &sw->graph);
        if (q) return q;
        if (e != cudaSuccess) return cuda_status(e, "sweep capture end");
        e = cudaGraphInstantiate(&sw->gexec, sw->graph, 0);
        if (e != cudaSuccess) return cuda_status(e, "sweep graph instantiate");
    }
    LENTILS_CUDA_TRY(cudaGraphLaunch(sw->gexec, s));
    return LENTILS_OK;
}

int lentils_sweep_get_stats(const lentils_sweep *sw, lentils_sweep_stats *st)
{
    clear_error();
    if (!sw || !st) return set_error(LENTILS_ERR_INVALID, "sweep_get_stats: null");
    st->nsamples = sw->nsamples;
    st->nwork = sw->nwork;
    st->blocks = sw->blocks;
    st->smem_bytes = (long long)sw->smem;
    st->total_vis = sw->total_vis;
    st->total_pixels = sw->total_pixels;
    st->algorithmic_bytes = sw->algorithmic_bytes;
    return LENTILS_OK;
}

}  // extern "C"
