// Interaction lists ("takes"): point-in-box count/fill over a uniform cell
// grid, prefix scans, compaction, the stable subdomain-major pair sort and the
// work queue.  All integer work; results are bit-exact with the reference's
// inside_points / get_inputs (fbpinns/decompositions_base.py:24-84,
// fbpinns/trainers.py:332-419).
#include <algorithm>

#include "common.cuh"

namespace fbp {

// ---------------------------------------------------------------------------
// cell lookup (must match fbpinns_gb300/decompositions.py:build_cell_grid)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cell_coord(float v, double lo, double inv_h, int nc) {
    const double t = __dmul_rn(__dsub_rn((double)v, lo), inv_h);
    double f = floor(t);
    if (!(f >= 0.0)) f = 0.0;  // also maps NaN to cell 0
    if (f > (double)(nc - 1)) f = (double)(nc - 1);
    return (int)f;
}

template <int XD>
__device__ __forceinline__ int cell_of(const float* xp, const fbp_boxes& b) {
    int c = cell_coord(xp[XD - 1], b.lo[XD - 1], b.inv_h[XD - 1], b.ncell[XD - 1]);
#pragma unroll
    for (int d = XD - 2; d >= 0; --d) c = c * b.ncell[d] + cell_coord(xp[d], b.lo[d], b.inv_h[d], b.ncell[d]);
    return c;
}

template <int XD>
__device__ __forceinline__ bool inside_box(const float* xp, const float* __restrict__ xmins,
                                           const float* __restrict__ xmaxs, int j) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < XD; ++d) {
        const float v = xp[d];
        in = in && (v >= xmins[j * XD + d]) && (v <= xmaxs[j * XD + d]);
    }
    return in;
}

// Boxes up to which the count pass keeps its points-per-box counts in shared
// memory (48 KB of int32, what a CTA gets without opting in).  A box of the
// coarsest level holds every point, and one global atomic per hit then queues
// up on that one word: 1365 boxes of six levels and 150001 points took 1195 us,
// 27 us without the counts.  A CTA's counts are added to the global ones at
// its end, so with them the launch is one resident wave of at most
// COUNT_CTAS CTAs per SM.
constexpr int64_t COUNT_MAX_M = 12288;
constexpr int COUNT_CTAS = 2, COUNT_T = 512;

// Points per chunk of the list build: the count pass leaves the pairs and
// slots of each chunk (the CTA's points), and the fill pass, which works on the
// same chunks, adds those of the chunks before its own and scans within the
// chunk -- two launches for the lists, where separate scans take four more
// (with the work queues in one launch each and the sort's starts in its scatter,
// 16381 points in 85 boxes redrawn every step: 161 -> 150.5 us a step).
constexpr int LIST_CHUNK = 256;

// SHIST: model_count through the CTA's table in shared memory (m words).
// sums (nullable): per chunk its pairs and slots; with SHIST added by the warps
// (sums zeroed before), else written by CTAs of LIST_CHUNK threads.
template <int XD, bool SHIST>
__global__ void inside_count_kernel(const float* __restrict__ x, int64_t n, fbp_boxes b,
                                    int32_t* __restrict__ pt_count, int32_t* __restrict__ pt_nlvl,
                                    uint64_t* __restrict__ pt_lvl, int32_t* __restrict__ model_count,
                                    uint64_t* __restrict__ pt_hit, int32_t* __restrict__ pt_cand,
                                    int2* __restrict__ sums) {
    pdl_wait();
    extern __shared__ int32_t box_count[];
    if constexpr (SHIST) {
        for (int64_t j = threadIdx.x; j < b.m; j += blockDim.x) box_count[j] = 0;
        __syncthreads();
    }
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x; p0 < n; p0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = p0 + threadIdx.x;
        float xp[XD];
#pragma unroll
        for (int d = 0; d < XD; ++d) xp[d] = p < n ? x[p * XD + d] : 0.f;
        const int c = cell_of<XD>(xp, b);
        const int e0 = b.cell_start[c], e1 = p < n ? b.cell_start[c + 1] : e0;
        int cnt = 0;
        uint64_t lvl = 0, hit = 0;
        for (int e = e0; e < e1; ++e) {
            const int j = b.cell_boxes[e];
            if (b.select && !b.select[j]) continue;
            if (inside_box<XD>(xp, b.xmins, b.xmaxs, j)) {
                ++cnt;
                lvl |= 1ull << (b.pou[j] & 63);
                if (e - e0 < 64) hit |= 1ull << (e - e0);
                if constexpr (SHIST)
                    atomicAdd(&box_count[j], 1);
                else if (model_count)
                    atomicAdd(&model_count[j], 1);
            }
        }
        if (p < n) {
            pt_count[p] = cnt;
            if (pt_nlvl) pt_nlvl[p] = __popcll(lvl);
            if (pt_lvl) pt_lvl[p] = lvl;
            // hits as a mask over the cell's candidate list (cells of <= 64 candidates)
            if (pt_hit) pt_hit[p] = hit;
            if (pt_cand) pt_cand[p] = e1 - e0 <= 64 ? e0 : -1;
        }
        if (sums) {
            const int ws = __reduce_add_sync(0xffffffffu, cnt), wu = __reduce_add_sync(0xffffffffu, __popcll(lvl));
            if constexpr (SHIST) {
                int2* t = &sums[(p0 + threadIdx.x) / LIST_CHUNK];
                if ((threadIdx.x & 31) == 0 && ws) {
                    atomicAdd(&t->x, ws);
                    atomicAdd(&t->y, wu);
                }
            } else {
                __shared__ int2 warp_sums[LIST_CHUNK / 32];
                if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = make_int2(ws, wu);
                __syncthreads();
                if (threadIdx.x == 0) {
                    int2 t = make_int2(0, 0);
#pragma unroll
                    for (int w = 0; w < LIST_CHUNK / 32; ++w) t = make_int2(t.x + warp_sums[w].x, t.y + warp_sums[w].y);
                    sums[p0 / LIST_CHUNK] = t;
                }
                __syncthreads();
            }
        }
    }
    if constexpr (SHIST) {
        __syncthreads();
        for (int64_t j = threadIdx.x; j < b.m; j += blockDim.x)
            if (box_count[j]) atomicAdd(&model_count[j], box_count[j]);
    }
}

// Fill: one thread per point takes its hits from the count pass's candidate
// mask (or, for cells of more than 64 candidates or without the mask, tests
// the candidates again; the box arrays are small and stay in L1); a warp's 32
// consecutive points own one contiguous
// range of the point-major pair arrays, so their hits are staged in shared
// memory and the warp writes the range out coalesced.  A warp whose range
// exceeds its staging space writes its points' pairs directly.  A staged pair
// is one int32: box id << 11 | POU level << 5 | point within the warp
// (box ids below 2^21, checked by the caller).
constexpr int FILL_WARPS = 8;     // warps per CTA
constexpr int FILL_STAGE = 1280;  // staged pairs per warp
constexpr int64_t FILL_MAX_M = int64_t(1) << 21;

// OFFS: pt_off and np_off are made here, from pt_count, the levels and the
// count pass's chunk sums; else they are read.
template <int XD, bool OFFS>
__global__ void __launch_bounds__(FILL_WARPS * 32)
    inside_fill_kernel(const float* __restrict__ x, int64_t n, fbp_boxes b, int32_t* __restrict__ pt_off,
                       int32_t* __restrict__ np_off, const int32_t* __restrict__ pt_count,
                       const int2* __restrict__ sums, const uint64_t* __restrict__ pt_lvl,
                       const uint64_t* __restrict__ pt_hit, const int32_t* __restrict__ pt_cand,
                       int32_t* __restrict__ n_take, int32_t* __restrict__ m_take, int32_t* __restrict__ p_take,
                       int32_t* __restrict__ np_take, int64_t s_cap, int64_t u_cap, int32_t* __restrict__ status) {
    pdl_wait();
    __shared__ int32_t stage[FILL_WARPS][FILL_STAGE];
    __shared__ uint64_t s_lvl[FILL_WARPS][32];
    __shared__ int32_t s_ubase[FILL_WARPS][32];
    __shared__ int2 s_part[FILL_WARPS], s_pre[FILL_WARPS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert(FILL_WARPS * 32 == LIST_CHUNK, "a CTA fills a chunk at a time");
    int64_t done = 0;               // chunks whose sums are in pre
    int2 pre = make_int2(0, 0);     // this thread's part of the sums of the chunks before
    const int64_t nchunk = (n + LIST_CHUNK - 1) / LIST_CHUNK;
    for (int64_t chunk = blockIdx.x; chunk < nchunk; chunk += gridDim.x) {
        const int64_t p0 = chunk * LIST_CHUNK + w * 32;
        const int64_t p = p0 + lane;
        const bool valid = p < n;
        const int np = (int)max((int64_t)0, min((int64_t)32, n - p0));
        int64_t base = 0, wb = 0, we = 0;
        int32_t ubase = 0;
        uint64_t lvl = 0;
        if (valid) lvl = pt_lvl[p];
        if constexpr (OFFS) {
            for (int64_t c = done + threadIdx.x; c < chunk; c += LIST_CHUNK) {
                const int2 t = sums[c];
                pre.x += t.x;
                pre.y += t.y;
            }
            done = chunk;
            const int cnt = valid ? pt_count[p] : 0, nl = __popcll(lvl);
            int a = cnt, u = nl;  // inclusive scans over the warp
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int ta = __shfl_up_sync(0xffffffffu, a, o), tu = __shfl_up_sync(0xffffffffu, u, o);
                if (lane >= o) a += ta, u += tu;
            }
            const int wa = __shfl_sync(0xffffffffu, a, 31), wu = __shfl_sync(0xffffffffu, u, 31);
            const int pa = __reduce_add_sync(0xffffffffu, pre.x), pu = __reduce_add_sync(0xffffffffu, pre.y);
            __syncthreads();  // the previous chunk's s_part and s_pre have been read
            if (lane == 0) s_part[w] = make_int2(wa, wu), s_pre[w] = make_int2(pa, pu);
            __syncthreads();
            int2 o = make_int2(0, 0);
#pragma unroll
            for (int v = 0; v < FILL_WARPS; ++v) {
                o.x += s_pre[v].x + (v < w ? s_part[v].x : 0);
                o.y += s_pre[v].y + (v < w ? s_part[v].y : 0);
            }
            base = o.x + a - cnt;
            ubase = o.y + u - nl;
            wb = o.x;
            we = o.x + wa;
            if (valid) {
                pt_off[p] = (int32_t)base;
                np_off[p] = ubase;
                if (p == n - 1) pt_off[n] = (int32_t)base + cnt, np_off[n] = ubase + nl;
            }
        } else if (np > 0) {
            wb = pt_off[p0];
            we = pt_off[p0 + np];
            if (valid) {
                base = pt_off[p];
                ubase = np_off[p];
            }
        }
        const int64_t total = we - wb;
        const bool staged = total <= FILL_STAGE && b.m <= FILL_MAX_M;
        s_lvl[w][lane] = lvl;
        s_ubase[w][lane] = ubase;
        if (valid) {
            int cand = -1;
            uint64_t hit = 0;
            if (pt_hit && pt_cand) {
                cand = pt_cand[p];
                hit = pt_hit[p];
            }
            int e = 0, e1 = 0;
            float xp[XD];
            if (cand < 0) {
#pragma unroll
                for (int d = 0; d < XD; ++d) xp[d] = x[p * XD + d];
                const int c = cell_of<XD>(xp, b);
                e = b.cell_start[c];
                e1 = b.cell_start[c + 1];
            }
            int64_t k = 0;
            // the point's k-th pair (box j at POU level lv): staged or written directly
            auto emit = [&](int j, int lv) {
                const int64_t q = base + k - wb;
                if (staged) {
                    if (q >= 0 && q < total)
                        stage[w][q] = (int32_t)(((uint32_t)j << 11) | (uint32_t)(lv << 5) | (uint32_t)lane);
                    else
                        atomicOr(status, FBP_STATUS_BAD_INDEX);
                } else {
                    const int64_t o = base + k;
                    if (o < s_cap) {
                        const uint64_t below = lv ? (lvl & ((1ull << lv) - 1ull)) : 0ull;
                        n_take[o] = (int32_t)p;
                        m_take[o] = j;
                        p_take[o] = ubase + __popcll(below);
                    } else {
                        atomicOr(status, FBP_STATUS_PAIR_OVERFLOW);
                    }
                }
                ++k;
            };
            if (cand >= 0) {
                // hits from the mask, four at a time so that their loads overlap
                while (hit) {
                    int jj[4], ll[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        jj[u] = -1;
                        if (hit) {
                            jj[u] = b.cell_boxes[cand + __ffsll((long long)hit) - 1];
                            hit &= hit - 1;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) ll[u] = jj[u] >= 0 ? (b.pou[jj[u]] & 63) : 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (jj[u] >= 0) emit(jj[u], ll[u]);
                }
            } else {
                for (; e < e1; ++e) {
                    const int j = b.cell_boxes[e];
                    if ((!b.select || b.select[j]) && inside_box<XD>(xp, b.xmins, b.xmaxs, j)) emit(j, b.pou[j] & 63);
                }
            }
            // unique (point, level) slots in ascending level order
            const int nl = __popcll(lvl);
            for (int r = 0; r < nl; ++r) {
                const int64_t o = (int64_t)ubase + r;
                if (o < u_cap)
                    np_take[o] = (int32_t)p;
                else
                    atomicOr(status, FBP_STATUS_SLOT_OVERFLOW);
            }
        }
        __syncwarp();
        if (staged) {
            for (int64_t q = lane; q < total; q += 32) {
                const int32_t v = stage[w][q];
                const int idx = v & 31, lv = (v >> 5) & 63;
                const int64_t o = wb + q;
                if (o < s_cap) {
                    const uint64_t l = s_lvl[w][idx];
                    const uint64_t below = lv ? (l & ((1ull << lv) - 1ull)) : 0ull;
                    n_take[o] = (int32_t)(p0 + idx);
                    m_take[o] = (int32_t)((uint32_t)v >> 11);
                    p_take[o] = s_ubase[w][idx] + __popcll(below);
                } else {
                    atomicOr(status, FBP_STATUS_PAIR_OVERFLOW);
                }
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Exclusive scan of int32 (3 kernels, deterministic)
// ---------------------------------------------------------------------------
constexpr int SCAN_T = 256, SCAN_V = 8, SCAN_TILE = SCAN_T * SCAN_V;
static_assert(SCAN_TILE == kScanTile, "the scan tile is shared with the allocation-free scan");

__device__ __forceinline__ int block_exclusive_scan(int v, int* smem_warp, int& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) smem_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        int w = lane < nw ? smem_warp[lane] : 0;
        int wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nw) smem_warp[lane] = wi - w;
        if (lane == nw - 1) smem_warp[32] = wi;
    }
    __syncthreads();
    total = smem_warp[32];
    const int r = incl - v + smem_warp[wid];
    __syncthreads();
    return r;
}

__global__ void scan_reduce_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ sums) {
    pdl_wait();
    __shared__ int sw[33];
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int s = 0;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) {
        const int64_t i = base + (int64_t)v * SCAN_T + threadIdx.x;
        if (i < n) s += in[i];
    }
    int tot;
    block_exclusive_scan(s, sw, tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// single block: exclusive scan of the tile sums in place, total at sums[nb]
__global__ void scan_sums_kernel(int32_t* __restrict__ sums, int64_t nb) {
    pdl_wait();
    __shared__ int sw[33];
    int carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += blockDim.x) {
        const int64_t i = b0 + threadIdx.x;
        const int v = i < nb ? sums[i] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, sw, tot);
        if (i < nb) sums[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) sums[nb] = carry;
}

// Tiles up to which a down-sweep block adds the earlier tiles' sums itself
// (no scan of the sums in between: two launches per scan instead of three;
// the loads grow with the square of the tile count).
constexpr int64_t SCAN_FUSED_TILES = 4096;

// fused: the block's offset is the sum of sums[0 .. blockIdx.x) (tile totals,
// added here) and the last block writes the total; else sums holds the
// scanned offsets and the total at sums[nb].
__global__ void scan_down_kernel(const int32_t* __restrict__ in, int64_t n, const int32_t* __restrict__ sums,
                                 int64_t nb, int32_t* __restrict__ out, bool fused) {
    pdl_wait();
    __shared__ int sw[33];
    __shared__ int tile[SCAN_TILE];
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int prefix = 0;
    if (fused) {
        int a = 0;
        for (int64_t i = threadIdx.x; i < (int64_t)blockIdx.x; i += blockDim.x) a += sums[i];
        block_exclusive_scan(a, sw, prefix);  // prefix = the block total of a
    } else {
        prefix = sums[blockIdx.x];
    }
    // blocked arrangement: thread t owns items [t*V, t*V+V) of the tile
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) {
        const int64_t i = base + (int64_t)v * SCAN_T + threadIdx.x;
        tile[v * SCAN_T + threadIdx.x] = i < n ? in[i] : 0;
    }
    __syncthreads();
    int loc[SCAN_V];
    int s = 0;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) {
        loc[v] = s;
        s += tile[threadIdx.x * SCAN_V + v];
    }
    int tot;
    const int ex = block_exclusive_scan(s, sw, tot);
    const int off = prefix + ex;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) tile[threadIdx.x * SCAN_V + v] = off + loc[v];
    __syncthreads();
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) {
        const int64_t i = base + (int64_t)v * SCAN_T + threadIdx.x;
        if (i < n) out[i] = tile[v * SCAN_T + threadIdx.x];
    }
    if (threadIdx.x == 0) {
        if (fused && blockIdx.x == nb - 1) out[n] = prefix + tot;
        if (!fused && blockIdx.x == 0) out[n] = sums[nb];
    }
}

int scan_launch(const int32_t* in, int32_t* out, int64_t n, int32_t* sums, cudaStream_t st) {
    const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (nb == 0) {
        FBP_CUDA_CHECK(cudaMemsetAsync(out, 0, sizeof(int32_t), st));
        return FBP_OK;
    }
    const bool fused = nb <= SCAN_FUSED_TILES;
    FBP_CUDA_CHECK(launch_after(scan_reduce_kernel, (int)nb, SCAN_T, 0, st, in, n, sums));
    if (!fused) {
        FBP_CUDA_CHECK(launch_after(scan_sums_kernel, 1, 1024, 0, st, sums, nb));
    }
    FBP_CUDA_CHECK(launch_after(scan_down_kernel, (int)nb, SCAN_T, 0, st, in, n, sums, nb, out, fused));
    return FBP_OK;
}

size_t scan_scratch(int64_t n) { return (size_t)(((n + SCAN_TILE - 1) / SCAN_TILE) + 1) * sizeof(int32_t); }

// ---------------------------------------------------------------------------
// gather / compaction
// ---------------------------------------------------------------------------
__global__ void gather_i32_kernel(const int32_t* __restrict__ in, int64_t n, const int32_t* __restrict__ cnt,
                                  const int32_t* __restrict__ inv, int32_t* __restrict__ out) {
    const int64_t lim = cnt ? (int64_t)(*cnt) < n ? (int64_t)(*cnt) : n : n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < lim;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = inv[in[i]];
}

__global__ void flag_to_count_kernel(const int32_t* __restrict__ flag, int64_t n, int32_t* __restrict__ c) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        c[i] = flag[i] != 0;
}

__global__ void compact_kernel(const int32_t* __restrict__ flag, const int32_t* __restrict__ off, int64_t n,
                               int32_t* __restrict__ out, int32_t* __restrict__ count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        if (flag[i]) out[off[i]] = (int32_t)i;
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = off[n];
}

// ---------------------------------------------------------------------------
// Stable counting sort of pairs by subdomain.
// Pass 1 (one warp per chunk of CH pairs): per-chunk histogram, written
// bucket-major hist[j * nchunks + chunk].  Scan.  Pass 2: each warp re-reads
// its chunk in order and scatters with ranks from __match_any_sync, keeping
// per-bucket running counts in shared memory: stable and deterministic.
// ---------------------------------------------------------------------------
// Pairs per chunk of the subdomain sort, from the pair capacity: each chunk
// costs O(m) in bucket tables and histogram entries besides its pairs, so
// larger chunks pay while there are enough of them to fill the GPU (about
// four per SM of a GB300; measured with cell-ordered batches of 9.4e6 pairs:
// 4096 0.382 ms, 8192 0.364, 16384 0.33 for the whole list build; 2.3e6 pairs:
// 4096 33.6 us, 16384 55.4 us for the scatter).  A function of s_cap only, so
// that the scratch size and the launches agree; the order does not depend on it.
static int64_t sort_chunk(int64_t s_cap) {
    int64_t ch = 4096;
    while (ch < 16384 && s_cap / (2 * ch) >= 4 * kSM) ch *= 2;
    return ch;
}

// With pt_keep, a pair whose point has pt_keep[point] == 0 is left out (its
// key reads as -1, outside every bucket); the kept pairs keep their order.
__device__ __forceinline__ int kept_key(const int32_t* __restrict__ key, const int32_t* __restrict__ n_take,
                                        const uint8_t* __restrict__ pt_keep, int64_t i) {
    const int k = key[i];
    return (pt_keep && !pt_keep[n_take[i]]) ? -1 : k;
}

__global__ void sort_hist_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ n_take,
                                 const uint8_t* __restrict__ pt_keep, const int32_t* __restrict__ s_dev,
                                 int64_t s_cap, int64_t m, int64_t nchunks, int64_t chn,
                                 int32_t* __restrict__ hist) {
    pdl_wait();
    extern __shared__ int cnt[];
    const int64_t s = min((int64_t)*s_dev, s_cap);
    for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        for (int64_t j = threadIdx.x; j < m; j += blockDim.x) cnt[j] = 0;
        __syncthreads();
        const int64_t b0 = ch * chn, b1 = min(b0 + chn, s);
        for (int64_t i0 = b0; i0 < b1; i0 += (int64_t)blockDim.x * 8) {  // loads first, then the counts
            int kk[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t i = i0 + (int64_t)u * blockDim.x + threadIdx.x;
                kk[u] = i < b1 ? kept_key(key, n_take, pt_keep, i) : -1;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (kk[u] >= 0 && kk[u] < m) atomicAdd(&cnt[kk[u]], 1);
        }
        __syncthreads();
        for (int64_t j = threadIdx.x; j < m; j += blockDim.x) hist[j * nchunks + ch] = cnt[j];
        __syncthreads();
    }
}

constexpr int SCATTER_U = 16;  // 32-pair rows whose loads are issued together
#ifndef FBP_SCATTER_W
#define FBP_SCATTER_W 4
#endif
constexpr int SCATTER_W = FBP_SCATTER_W;  // warps per chunk (fewer when their bucket tables do not fit)

// One CTA of W <= SCATTER_W warps per chunk of chn pairs (point-major).
// Each warp first counts the buckets of its part of the chunk; the running
// offsets of warp w start at the chunk's bucket offset plus the counts of
// warps < w, so the warps then place their quarters independently and the
// result is the same stable order as one pass over the chunk.  A point's
// pairs have distinct boxes, so each row of 32 pairs is placed point by
// point: the lanes of one point read and advance distinct bucket counters,
// and the points of the row follow each other in order (no key matching).
__global__ void __launch_bounds__(SCATTER_W * 32)
    sort_scatter_kernel(const int32_t* __restrict__ key, const int32_t* __restrict__ n_take,
                        const int32_t* __restrict__ p_take, const uint8_t* __restrict__ pt_keep,
                        const int32_t* __restrict__ s_dev, int64_t s_cap, int64_t m, int64_t nchunks,
                        int64_t chn, const int32_t* __restrict__ hoff, int4* __restrict__ sd_rec,
                        int32_t* __restrict__ sd_start) {
    pdl_wait();
    extern __shared__ int run[];  // [W][m]: per-warp counts, then running offsets
    // sd_start[j] = hoff[j * nchunks] (start of bucket j), sd_start[m] = s
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j <= m; j += (int64_t)gridDim.x * blockDim.x)
        sd_start[j] = hoff[j * nchunks];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    int* myrun = run + (int64_t)w * m;
    const int64_t s = min((int64_t)*s_dev, s_cap);
    const int64_t SUB = (chn + W - 1) / W;
    for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        for (int64_t j = threadIdx.x; j < m * W; j += blockDim.x) run[j] = 0;
        __syncthreads();
        const int64_t c0 = ch * chn, c1 = min(c0 + chn, s);
        const int64_t b0 = min(c0 + (int64_t)w * SUB, c1), b1 = min(b0 + SUB, c1);
        for (int64_t i0 = b0; i0 < b1; i0 += 32 * 8) {  // loads of 8 rows first, then the counts
            int kk[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t i = i0 + u * 32 + lane;
                kk[u] = i < b1 ? kept_key(key, n_take, pt_keep, i) : -1;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (kk[u] >= 0 && kk[u] < m) atomicAdd(&myrun[kk[u]], 1);
        }
        __syncthreads();
        for (int64_t j0 = threadIdx.x; j0 < m; j0 += (int64_t)blockDim.x * 8) {
            int oo[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t j = j0 + (int64_t)u * blockDim.x;
                oo[u] = j < m ? hoff[j * nchunks + ch] : 0;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t j = j0 + (int64_t)u * blockDim.x;
                if (j >= m) break;
                int o = oo[u];
                for (int v = 0; v < W; ++v) {
                    const int c = run[(int64_t)v * m + j];
                    run[(int64_t)v * m + j] = o;
                    o += c;
                }
            }
        }
        __syncthreads();
        for (int64_t i0 = b0; i0 < b1; i0 += 32 * SCATTER_U) {
            int kk[SCATTER_U], nn[SCATTER_U], pp[SCATTER_U];
#pragma unroll
            for (int u = 0; u < SCATTER_U; ++u) {
                const int64_t i = i0 + u * 32 + lane;
                kk[u] = -1;
                nn[u] = -1;
                pp[u] = 0;
                if (i < b1) {
                    kk[u] = key[i];
                    nn[u] = n_take[i];
                    pp[u] = p_take[i];
                    if (pt_keep && !pt_keep[nn[u]]) kk[u] = -1;
                }
            }
#pragma unroll
            for (int u = 0; u < SCATTER_U; ++u) {
                const int64_t i = i0 + u * 32 + lane;
                const int k = kk[u];
                const bool ok = k >= 0 && k < m;
                unsigned todo = __ballot_sync(0xffffffffu, i < b1);
                while (todo) {
                    // the row's next point: the lanes holding it form one group
                    const int pt = __shfl_sync(0xffffffffu, nn[u], __ffs(todo) - 1);
                    const unsigned grp = __ballot_sync(0xffffffffu, (todo >> lane & 1u) && nn[u] == pt);
                    if ((grp >> lane & 1u) && ok) {
                        const int o = myrun[k];
                        myrun[k] = o + 1;
                        sd_rec[o] = make_int4((int32_t)i, pt, pp[u], 0);
                    }
                    todo &= ~grp;
                    __syncwarp();
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// work queue
// ---------------------------------------------------------------------------
// A CTA makes the items of WORK_T subdomains: it adds the item counts of the
// subdomains before its own (m reads, from L2), scans its own, and its warps
// write the items of one subdomain after the other (a subdomain holding all
// points has hundreds of them).  One launch; count, scan and fill apart take four.
constexpr int WORK_T = 256;

__global__ void __launch_bounds__(WORK_T) work_kernel(const int32_t* __restrict__ sd_start, int64_t m,
                                                      const uint8_t* __restrict__ sel, int chunk,
                                                      int32_t* __restrict__ items, int32_t* __restrict__ item_start,
                                                      int32_t* __restrict__ n_items, int64_t cap,
                                                      int32_t* __restrict__ status) {
    pdl_wait();
    __shared__ int sw[33];
    __shared__ int2 s_item[WORK_T];  // first item and number of items of the CTA's subdomains
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t j0 = (int64_t)blockIdx.x * WORK_T;
    auto count = [&](int64_t j) {
        return (sel && !sel[j]) ? 0 : (sd_start[j + 1] - sd_start[j] + chunk - 1) / chunk;
    };
    int before = 0, prefix, total;
    for (int64_t j = threadIdx.x; j < j0; j += WORK_T) before += count(j);
    block_exclusive_scan(before, sw, prefix);  // prefix = the sum over the CTA
    const int64_t j = j0 + threadIdx.x;
    const int c = j < m ? count(j) : 0;
    const int i0 = prefix + block_exclusive_scan(c, sw, total);
    s_item[threadIdx.x] = make_int2(i0, c);
    if (j < m) item_start[j] = (int32_t)min((int64_t)i0, cap);
    if (j == m - 1) {
        item_start[m] = (int32_t)min((int64_t)(i0 + c), cap);
        *n_items = (int32_t)min((int64_t)(i0 + c), cap);
    }
    __syncthreads();
    for (int q = w; q < WORK_T && j0 + q < m; q += WORK_T / 32) {
        const int2 it = s_item[q];
        const int b = sd_start[j0 + q], e = sd_start[j0 + q + 1];
        for (int k = lane; k < it.y; k += 32) {
            const int64_t i = (int64_t)it.x + k;
            if (i >= cap) {
                atomicOr(status, FBP_STATUS_ITEM_OVERFLOW);
                break;
            }
            const int beg = b + k * chunk;
            items[3 * i + 0] = (int32_t)(j0 + q);
            items[3 * i + 1] = beg;
            items[3 * i + 2] = min(chunk, e - beg);
        }
    }
}

// ---------------------------------------------------------------------------
// scheduled training: the points and subdomain states of one active mask
// ---------------------------------------------------------------------------
// Per point: kept when one of its boxes has raw state 1; the boxes of a kept
// point are marked in state[] (a store of 1 by any of its points); kept
// points are counted into *n_keep (warp sums, one atomic per warp).
__global__ void train_mark_kernel(const int32_t* __restrict__ pt_off, const int32_t* __restrict__ m_take, int64_t n,
                                  int64_t s_cap, const uint8_t* __restrict__ raw, uint8_t* __restrict__ pt_keep,
                                  uint8_t* __restrict__ state, int32_t* __restrict__ n_keep) {
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x; p0 < n; p0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = p0 + threadIdx.x;
        bool keep = false;
        if (p < n) {
            const int64_t e0 = min((int64_t)pt_off[p], s_cap), e1 = min((int64_t)pt_off[p + 1], s_cap);
            for (int64_t e = e0; e < e1 && !keep; ++e) keep = raw[m_take[e]] == 1;
            pt_keep[p] = keep ? 1 : 0;
            if (keep)
                for (int64_t e = e0; e < e1; ++e) state[m_take[e]] = 1;
        }
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if ((threadIdx.x & 31) == 0 && b) atomicAdd(n_keep, __popc(b));
    }
}

// Per box: 1 (trained) where it holds a kept point and its raw state is 0 or
// 1, 2 (fixed) where it holds one and its raw state is 2, else 0; active[j]
// = state[j] == 1 (the adjoint's selection and Adam's mask).
__global__ void train_state_kernel(const uint8_t* __restrict__ raw, int64_t m, uint8_t* __restrict__ state,
                                   uint8_t* __restrict__ active) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t v = state[j] ? (raw[j] == 2 ? 2 : 1) : 0;
        state[j] = v;
        active[j] = v == 1 ? 1 : 0;
    }
}

static int grid_for(int64_t n, int threads, int per_sm = 16) {
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

static int check_boxes(const fbp_boxes* b) {
    FBP_REQUIRE(b, FBP_ERR_INVALID, "boxes: null");
    FBP_REQUIRE(b->xd >= 1 && b->xd <= FBP_MAX_XD, FBP_ERR_UNSUPPORTED, "boxes: xd=%d not in 1..3", b->xd);
    FBP_REQUIRE(b->xmins && b->xmaxs && b->pou && b->cell_start && b->cell_boxes, FBP_ERR_INVALID,
                "boxes: null device pointer");
    for (int d = 0; d < b->xd; ++d)
        FBP_REQUIRE(b->ncell[d] >= 1, FBP_ERR_INVALID, "boxes: ncell[%d]=%d", d, b->ncell[d]);
    return FBP_OK;
}

}  // namespace fbp

using namespace fbp;

extern "C" size_t fbp_scan_scratch_bytes(int64_t n) { return scan_scratch(n); }

extern "C" int fbp_scan_i32(const int32_t* in, int32_t* out, int64_t n, void* scratch, size_t scratch_bytes,
                            void* stream) {
    FBP_REQUIRE(out && (in || n == 0), FBP_ERR_INVALID, "fbp_scan_i32: null pointer");
    FBP_REQUIRE(n >= 0 && n < (int64_t)1 << 31, FBP_ERR_INVALID, "fbp_scan_i32: n=%lld", (long long)n);
    FBP_REQUIRE(scratch && scratch_bytes >= scan_scratch(n), FBP_ERR_CAPACITY,
                "fbp_scan_i32: scratch %zu < %zu", scratch_bytes, scan_scratch(n));
    return scan_launch(in, out, n, (int32_t*)scratch, as_stream(stream));
}

// sums: see inside_count_kernel
static int launch_count(const float* x, int64_t n, const fbp_boxes* boxes, int32_t* pt_count, int32_t* pt_nlvl,
                        uint64_t* pt_lvl, int32_t* model_count, uint64_t* pt_hit, int32_t* pt_cand, int2* sums,
                        cudaStream_t st) {
    const bool shist = model_count && boxes->m <= COUNT_MAX_M;
    const int t = shist ? COUNT_T : LIST_CHUNK;
    const int g = shist ? grid_for(n, t, COUNT_CTAS) : grid_for(n, t);
    const size_t shm = shist ? (size_t)boxes->m * sizeof(int32_t) : 0;
#define X(D)                                                                                                        \
    if (boxes->xd == D) {                                                                                           \
        if (shist)                                                                                                  \
            FBP_CUDA_CHECK(launch_after(inside_count_kernel<D, true>, g, t, shm, st, x, n, *boxes, pt_count, pt_nlvl, \
                                        pt_lvl, model_count, pt_hit, pt_cand, sums));                               \
        else                                                                                                        \
            FBP_CUDA_CHECK(launch_after(inside_count_kernel<D, false>, g, t, 0, st, x, n, *boxes, pt_count, pt_nlvl, \
                                        pt_lvl, model_count, pt_hit, pt_cand, sums));                               \
    }
    X(1) X(2) X(3)
#undef X
    return FBP_OK;
}

static int launch_fill(const float* x, int64_t n, const fbp_boxes* boxes, int32_t* pt_off, int32_t* np_off,
                       const int32_t* pt_count, const int2* sums, const uint64_t* pt_lvl, const uint64_t* pt_hit,
                       const int32_t* pt_cand, int32_t* n_take, int32_t* m_take, int32_t* p_take, int32_t* np_take,
                       int64_t s_cap, int64_t u_cap, int32_t* status, cudaStream_t st) {
    const int g = grid_for(n, FILL_WARPS * 32, 8);  // 32 points per warp
#define X(D)                                                                                                        \
    if (boxes->xd == D) {                                                                                           \
        if (sums)                                                                                                   \
            FBP_CUDA_CHECK(launch_after(inside_fill_kernel<D, true>, g, FILL_WARPS * 32, 0, st, x, n, *boxes, pt_off, \
                                        np_off, pt_count, sums, pt_lvl, pt_hit, pt_cand, n_take, m_take, p_take,    \
                                        np_take, s_cap, u_cap, status));                                            \
        else                                                                                                        \
            FBP_CUDA_CHECK(launch_after(inside_fill_kernel<D, false>, g, FILL_WARPS * 32, 0, st, x, n, *boxes, pt_off, \
                                        np_off, nullptr, nullptr, pt_lvl, pt_hit, pt_cand, n_take, m_take, p_take,  \
                                        np_take, s_cap, u_cap, status));                                            \
    }
    X(1) X(2) X(3)
#undef X
    return FBP_OK;
}

extern "C" int fbp_inside_count(const float* x, int64_t n, const fbp_boxes* boxes, int32_t* pt_count,
                                int32_t* pt_nlvl, uint64_t* pt_lvl, int32_t* model_count, uint64_t* pt_hit,
                                int32_t* pt_cand, void* stream) {
    int rc = check_boxes(boxes);
    if (rc) return rc;
    FBP_REQUIRE(pt_count && (x || n == 0), FBP_ERR_INVALID, "fbp_inside_count: null pointer");
    if (n == 0) return FBP_OK;
    return launch_count(x, n, boxes, pt_count, pt_nlvl, pt_lvl, model_count, pt_hit, pt_cand, nullptr,
                        as_stream(stream));
}

extern "C" int fbp_inside_fill(const float* x, int64_t n, const fbp_boxes* boxes, const int32_t* pt_off,
                               const int32_t* np_off, const uint64_t* pt_lvl, const uint64_t* pt_hit,
                               const int32_t* pt_cand, int32_t* n_take, int32_t* m_take,
                               int32_t* p_take, int32_t* np_take, int64_t s_cap, int64_t u_cap, int32_t* status,
                               void* stream) {
    int rc = check_boxes(boxes);
    if (rc) return rc;
    FBP_REQUIRE(pt_off && np_off && pt_lvl && status && (x || n == 0), FBP_ERR_INVALID,
                "fbp_inside_fill: null pointer");
    FBP_REQUIRE((n_take && m_take && p_take) || s_cap == 0, FBP_ERR_INVALID, "fbp_inside_fill: null take");
    FBP_REQUIRE(np_take || u_cap == 0, FBP_ERR_INVALID, "fbp_inside_fill: null np_take");
    if (n == 0) return FBP_OK;
    return launch_fill(x, n, boxes, const_cast<int32_t*>(pt_off), const_cast<int32_t*>(np_off), nullptr, nullptr,
                       pt_lvl, pt_hit, pt_cand, n_take, m_take, p_take, np_take, s_cap, u_cap, status,
                       as_stream(stream));
}

extern "C" size_t fbp_inside_lists_scratch_bytes(int64_t n) {
    return (size_t)((n + LIST_CHUNK - 1) / LIST_CHUNK + 1) * sizeof(int2);
}

static int check_chunks(int64_t n, const void* sums, size_t sums_bytes) {
    FBP_REQUIRE(n >= 0 && n < (int64_t)1 << 31, FBP_ERR_INVALID, "inside lists: n=%lld", (long long)n);
    FBP_REQUIRE(sums && ((uintptr_t)sums & 7) == 0 && sums_bytes >= fbp_inside_lists_scratch_bytes(n),
                FBP_ERR_CAPACITY, "inside lists: chunk sums too small");
    return FBP_OK;
}

extern "C" int fbp_inside_count_chunks(const float* x, int64_t n, const fbp_boxes* boxes, int32_t* pt_count,
                                       uint64_t* pt_lvl, int32_t* model_count, uint64_t* pt_hit, int32_t* pt_cand,
                                       void* sums, size_t sums_bytes, void* stream) {
    int rc = check_boxes(boxes);
    if (rc) return rc;
    rc = check_chunks(n, sums, sums_bytes);
    if (rc) return rc;
    FBP_REQUIRE(n == 0 || (x && pt_count && pt_lvl), FBP_ERR_INVALID, "fbp_inside_count_chunks: null pointer");
    FBP_REQUIRE(!pt_hit == !pt_cand, FBP_ERR_INVALID, "fbp_inside_count_chunks: pt_hit and pt_cand go together");
    if (n == 0) return FBP_OK;
    return launch_count(x, n, boxes, pt_count, nullptr, pt_lvl, model_count, pt_hit, pt_cand, static_cast<int2*>(sums),
                        as_stream(stream));
}

extern "C" int fbp_inside_fill_chunks(const float* x, int64_t n, const fbp_boxes* boxes, const int32_t* pt_count,
                                      const uint64_t* pt_lvl, const uint64_t* pt_hit, const int32_t* pt_cand,
                                      const void* sums, size_t sums_bytes, int32_t* pt_off, int32_t* np_off,
                                      int32_t* n_take, int32_t* m_take, int32_t* p_take, int32_t* np_take,
                                      int64_t s_cap, int64_t u_cap, int32_t* status, void* stream) {
    int rc = check_boxes(boxes);
    if (rc) return rc;
    rc = check_chunks(n, sums, sums_bytes);
    if (rc) return rc;
    FBP_REQUIRE(pt_off && np_off && status, FBP_ERR_INVALID, "fbp_inside_fill_chunks: null pointer");
    FBP_REQUIRE(n == 0 || (x && pt_count && pt_lvl), FBP_ERR_INVALID, "fbp_inside_fill_chunks: null pointer");
    FBP_REQUIRE(!pt_hit == !pt_cand, FBP_ERR_INVALID, "fbp_inside_fill_chunks: pt_hit and pt_cand go together");
    FBP_REQUIRE((n_take && m_take && p_take) || s_cap == 0, FBP_ERR_INVALID, "fbp_inside_fill_chunks: null take");
    FBP_REQUIRE(np_take || u_cap == 0, FBP_ERR_INVALID, "fbp_inside_fill_chunks: null np_take");
    cudaStream_t st = as_stream(stream);
    if (n == 0) {
        FBP_CUDA_CHECK(cudaMemsetAsync(pt_off, 0, sizeof(int32_t), st));
        FBP_CUDA_CHECK(cudaMemsetAsync(np_off, 0, sizeof(int32_t), st));
        return FBP_OK;
    }
    return launch_fill(x, n, boxes, pt_off, np_off, pt_count, static_cast<const int2*>(sums), pt_lvl, pt_hit, pt_cand,
                       n_take, m_take, p_take, np_take, s_cap, u_cap, status, st);
}

extern "C" int fbp_gather_i32(const int32_t* in, int64_t n, const int32_t* count_dev, const int32_t* inv,
                              int32_t* out, void* stream) {
    FBP_REQUIRE(inv && out && (in || n == 0), FBP_ERR_INVALID, "fbp_gather_i32: null pointer");
    if (n == 0) return FBP_OK;
    gather_i32_kernel<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(in, n, count_dev, inv, out);
    FBP_LAUNCH_CHECK();
    return FBP_OK;
}

extern "C" size_t fbp_compact_scratch_bytes(int64_t n) {
    return (size_t)(n + 1) * sizeof(int32_t) * 2 + scan_scratch(n) + 256;
}

extern "C" int fbp_compact_flags(const int32_t* flag, int64_t n, int32_t* out, int32_t* count_dev, void* scratch,
                                 size_t scratch_bytes, void* stream) {
    FBP_REQUIRE(out && count_dev && (flag || n == 0), FBP_ERR_INVALID, "fbp_compact_flags: null pointer");
    FBP_REQUIRE(scratch && scratch_bytes >= fbp_compact_scratch_bytes(n), FBP_ERR_CAPACITY,
                "fbp_compact_flags: scratch too small");
    cudaStream_t st = as_stream(stream);
    int32_t* c = (int32_t*)scratch;
    int32_t* off = c + (n + 1);
    int32_t* sums = off + (n + 1);
    if (n == 0) {
        FBP_CUDA_CHECK(cudaMemsetAsync(count_dev, 0, sizeof(int32_t), st));
        return FBP_OK;
    }
    flag_to_count_kernel<<<grid_for(n, 256), 256, 0, st>>>(flag, n, c);
    FBP_LAUNCH_CHECK();
    int rc = scan_launch(c, off, n, sums, st);
    if (rc) return rc;
    compact_kernel<<<grid_for(n, 256), 256, 0, st>>>(flag, off, n, out, count_dev);
    FBP_LAUNCH_CHECK();
    return FBP_OK;
}

extern "C" size_t fbp_sort_scratch_bytes(int64_t s_cap, int64_t m) {
    const int64_t chn = sort_chunk(s_cap);
    const int64_t nch = (s_cap + chn - 1) / chn;
    const int64_t hn = m * nch + 1;
    return (size_t)hn * sizeof(int32_t) * 2 + scan_scratch(hn) + 256;
}

static int sort_pairs(const int32_t* m_take, const int32_t* n_take, const int32_t* p_take, const uint8_t* pt_keep,
                      const int32_t* s_dev, int64_t s_cap, int64_t m, int32_t* sd_start, int32_t* sd_rec,
                      void* scratch, size_t scratch_bytes, void* stream) {
    FBP_REQUIRE(s_dev && sd_start && m > 0, FBP_ERR_INVALID, "fbp_sort_pairs: bad args");
    FBP_REQUIRE(((uintptr_t)sd_rec & 15) == 0, FBP_ERR_INVALID, "fbp_sort_pairs: sd_rec must be 16-byte aligned");
    FBP_REQUIRE(s_cap == 0 || (m_take && n_take && p_take && sd_rec), FBP_ERR_INVALID,
                "fbp_sort_pairs: null pointer");
    FBP_REQUIRE(m * 4 <= 200 * 1024, FBP_ERR_UNSUPPORTED, "fbp_sort_pairs: m=%lld exceeds the shared-memory histogram",
                (long long)m);
    FBP_REQUIRE(scratch && scratch_bytes >= fbp_sort_scratch_bytes(s_cap, m), FBP_ERR_CAPACITY,
                "fbp_sort_pairs: scratch too small");
    cudaStream_t st = as_stream(stream);
    const int64_t chn = sort_chunk(s_cap);
    const int64_t nch = (s_cap + chn - 1) / chn;
    const int64_t hn = m * nch;
    int32_t* hist = (int32_t*)scratch;
    int32_t* hoff = hist + (hn + 1);
    int32_t* sums = hoff + (hn + 1);
    const size_t shm = (size_t)m * sizeof(int);
    int sw = SCATTER_W;  // warps per chunk in the scatter: one bucket table each
    while (sw > 1 && shm * sw > 200 * 1024) sw >>= 1;
    if (shm > 48 * 1024)
        FBP_CUDA_CHECK(cudaFuncSetAttribute(sort_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
    if (shm * sw > 48 * 1024)
        FBP_CUDA_CHECK(
            cudaFuncSetAttribute(sort_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(shm * sw)));
    if (nch > 0) {
        const int g = (int)std::min<int64_t>(nch, (int64_t)sm_count() * 8);
        FBP_CUDA_CHECK(launch_after(sort_hist_kernel, g, 256, shm, st, m_take, n_take, pt_keep, s_dev, s_cap, m, nch, chn,
                                    hist));
    }
    int rc = scan_launch(hist, hoff, hn, sums, st);
    if (rc) return rc;
    if (nch > 0) {
        const int g = (int)std::min<int64_t>(nch, (int64_t)sm_count() * 32 / sw);
        FBP_CUDA_CHECK(launch_after(sort_scatter_kernel, g, 32 * sw, shm * sw, st, m_take, n_take, p_take, pt_keep, s_dev,
                                    s_cap, m, nch, chn, hoff, reinterpret_cast<int4*>(sd_rec), sd_start));
    } else {
        FBP_CUDA_CHECK(cudaMemsetAsync(sd_start, 0, (size_t)(m + 1) * sizeof(int32_t), st));
    }
    return FBP_OK;
}

extern "C" int fbp_sort_pairs(const int32_t* m_take, const int32_t* n_take, const int32_t* p_take,
                              const int32_t* s_dev, int64_t s_cap, int64_t m, int32_t* sd_start, int32_t* sd_rec,
                              void* scratch, size_t scratch_bytes, void* stream) {
    return sort_pairs(m_take, n_take, p_take, nullptr, s_dev, s_cap, m, sd_start, sd_rec, scratch, scratch_bytes,
                      stream);
}

extern "C" int fbp_sort_pairs_kept(const int32_t* m_take, const int32_t* n_take, const int32_t* p_take,
                                   const uint8_t* pt_keep, const int32_t* s_dev, int64_t s_cap, int64_t m,
                                   int32_t* sd_start, int32_t* sd_rec, void* scratch, size_t scratch_bytes,
                                   void* stream) {
    FBP_REQUIRE(pt_keep, FBP_ERR_INVALID, "fbp_sort_pairs_kept: null pt_keep");
    return sort_pairs(m_take, n_take, p_take, pt_keep, s_dev, s_cap, m, sd_start, sd_rec, scratch, scratch_bytes,
                      stream);
}

extern "C" int fbp_train_mask(const int32_t* pt_off, const int32_t* m_take, int64_t n, int64_t s_cap,
                              const uint8_t* raw, int64_t m, uint8_t* pt_keep, int32_t* n_keep, uint8_t* state,
                              uint8_t* active, void* stream) {
    FBP_REQUIRE(pt_off && raw && pt_keep && n_keep && state && active && m > 0 && n >= 0, FBP_ERR_INVALID,
                "fbp_train_mask: bad args");
    FBP_REQUIRE(s_cap == 0 || m_take, FBP_ERR_INVALID, "fbp_train_mask: null m_take");
    cudaStream_t st = as_stream(stream);
    FBP_CUDA_CHECK(cudaMemsetAsync(state, 0, (size_t)m, st));
    FBP_CUDA_CHECK(cudaMemsetAsync(n_keep, 0, sizeof(int32_t), st));
    if (n > 0) {
        train_mark_kernel<<<grid_for(n, 256), 256, 0, st>>>(pt_off, m_take, n, s_cap, raw, pt_keep, state, n_keep);
        FBP_LAUNCH_CHECK();
    }
    train_state_kernel<<<grid_for(m, 256), 256, 0, st>>>(raw, m, state, active);
    FBP_LAUNCH_CHECK();
    return FBP_OK;
}

extern "C" size_t fbp_work_scratch_bytes(int64_t) { return 0; }

extern "C" int fbp_build_work(const int32_t* sd_start, int64_t m, const uint8_t* select, int32_t chunk,
                              int32_t* items, int32_t* item_start, int32_t* n_items, int64_t items_cap,
                              int32_t* status, void*, size_t, void* stream) {
    FBP_REQUIRE(sd_start && items && item_start && n_items && status && m > 0 && chunk > 0, FBP_ERR_INVALID,
                "fbp_build_work: bad args");
    cudaStream_t st = as_stream(stream);
    FBP_CUDA_CHECK(launch_after(work_kernel, (int)((m + WORK_T - 1) / WORK_T), WORK_T, 0, st, sd_start, m, select, chunk,
                                items, item_start, n_items, items_cap, status));
    return FBP_OK;
}
