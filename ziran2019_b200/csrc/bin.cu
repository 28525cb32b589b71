// Particle binning onto SPGrid pages, bit-exact with
// MpmSimulationBase::sortParticlesAndPolluteGrid (Lib/MPM/MpmSimulationBase.cpp:1032-1103).
//
//  1. key   = ((Linear_Offset(baseNode(x/dx)) >> data_bits) << (32 - block_bits)) + index
//             = page_index << 32 | element << index_bits | index        (k_keys)
//  2. sort  : the keys are unique, so any correct sort gives the reference's
//             order.  LSD: pass 0 places each key at its particle index
//             (k_keys), then 8-bit radix passes over the page/element bits.
//  3. groups: runs of equal page index (key >> 32), in sorted order.
//  4. pages : the reference calls Set_Page on each group's page and its 7
//             upper neighbours, in group order, and appends a page the first
//             time it is seen (SPGrid_Page_Map.h:61-70).  Emission e = 8g + t;
//             a page's block index is its rank among first emissions, found by
//             atomicMin(first[page], e) then a stable compaction of the
//             emissions that won.  This reproduces the first-touch order.
//  5. permutation of all particle state into sorted slots (coalesced passes).
//
// Two ways to the same order.  The usual one bins by page first: the groups
// are few (a page holds about 500 particles), so their order and starts come
// from comparing their page indices pairwise, and each group's particles are
// ordered in shared memory by one CTA (k_count, k_pages, one host read of the
// counts, k_rank, k_place, k_order, k_emit, k_number): 9 launches.  Scenes with
// more than RANK_MAX groups (see there) or with a
// group of more than ORDER_CAP particles (shared memory, and one cell may hold
// them all) take the radix sort over particle keys of steps 1-4 above: about 40
// launches.  A context stays on the radix way until a pass on it finds a scene
// for the other (counting the pages first cost such scenes 0.06 ms a pass).
// Measured at 60k particles in FP64 the radix way's kernels took 0.19 of a 0.37 ms
// explicit substep.
#include <algorithm>

#include "internal.cuh"
#include "xfer.cuh"

namespace zmpm {

constexpr int BIN_THREADS = 256;

static inline unsigned nblk(int64_t n, int t = BIN_THREADS) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ int int_floor_d(double u)
{
    int i = (int)u;
    return i - (i > u);
}
__device__ __forceinline__ int int_floor_f(float u)
{
    int i = (int)u;
    return i - (i > u);
}

struct PageDims {
    int px, py, pz;
    __device__ __forceinline__ int64_t index(int x, int y, int z) const { return ((int64_t)x * py + y) * pz + z; }
};

// The dense page table.  Between passes every word is PAGE_CLEAN.  Binning by page
// subtracts the page's particles (fewer than 2^27, so PAGE_BIT stays set), clears
// PAGE_BIT in every page that gets a block and puts PAGE_CURSOR plus the next free
// slot into the groups' pages; both ways then take the smallest emission that touches
// the page, which is below all of these (below 8 RANK_MAX by page; below 2^30 by
// radix sort, which starts from clean words).
constexpr int32_t PAGE_CLEAN = 0x7f7f7f7f, PAGE_BIT = 0x40000000, PAGE_CURSOR = 0x40000000;

// Base node of the particle in slot s, or node 0 and false when its stencil
// leaves the grid.  KT: precision of the key arithmetic (double for FP64 runs, float for the
// mixed runs whose grid mirrors the reference's T=float build).
template <class L, class KT>
__device__ __forceinline__ bool base_node(const double* __restrict__ x, int64_t cap, int64_t s, double inv_dx_d, float inv_dx_f, PageDims pd, int b[3])
{
    bool finite = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        finite = finite && isfinite(x[d * cap + s]);
        if constexpr (sizeof(KT) == 8) {
            double t = __dmul_rn(x[d * cap + s], inv_dx_d);
            b[d] = int_floor_d(__dsub_rn(t, 0.5));
        }
        else {
            float t = __fmul_rn((float)x[d * cap + s], inv_dx_f);
            b[d] = int_floor_f(__fsub_rn(t, 0.5f));
        }
    }
    // a non-finite position converts to an arbitrary integer: it is out of the grid
    if (!finite || b[0] < 0 || b[1] < 0 || b[2] < 0 || (b[0] >> L::XB) + 1 >= pd.px || (b[1] >> L::YB) + 1 >= pd.py
        || (b[2] >> L::ZB) + 1 >= pd.pz) {
        b[0] = b[1] = b[2] = 0;
        return false;
    }
    return true;
}

template <class L, class KT>
__global__ void k_keys(const double* __restrict__ x, int64_t cap, int64_t P, double inv_dx_d, float inv_dx_f, const int32_t* __restrict__ orig_id,
    uint64_t* __restrict__ keys_by_id, short4* __restrict__ base_by_id, PageDims pd, int32_t* __restrict__ flags)
{
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P) return;
    int b[3];
    if (!base_node<L, KT>(x, cap, s, inv_dx_d, inv_dx_f, pd, b)) atomicOr(flags, (int32_t)FLAG_OUT_OF_GRID);
    const int p0 = b[0] >> L::XB, p1 = b[1] >> L::YB, p2 = b[2] >> L::ZB;
    const int e = L::elem(b[0] & (L::BX - 1), b[1] & (L::BY - 1), b[2] & (L::BZ - 1));
    const uint64_t page = L::page_index(p0, p1, p2);
    const int32_t id = orig_id[s];
    keys_by_id[id] = (page << 32) | ((uint64_t)e << L::INDEX_BITS) | (uint64_t)id;
    base_by_id[id] = make_short4((short)b[0], (short)b[1], (short)b[2], 0);
}

__global__ void k_group_heads(const uint64_t* __restrict__ keys, int64_t P, int32_t* __restrict__ flag)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    flag[i] = (i == 0 || (keys[i] >> 32) != (keys[i - 1] >> 32)) ? 1 : 0;
}

// New slot i receives particle keys[i] & idmask: gather every field from its
// old slot.  Also writes group starts and each group's page coordinates.
template <class L>
__global__ void k_permute(const uint64_t* __restrict__ keys, int64_t P, int64_t cap, int npd, const double* __restrict__ pd_src,
    double* __restrict__ pd_dst, const int32_t* __restrict__ pi_src, int32_t* __restrict__ pi_dst, int32_t* __restrict__ slot_of_id,
    const short4* __restrict__ base_by_id, short4* __restrict__ base, const int32_t* __restrict__ head, const int32_t* __restrict__ gidx,
    int32_t* __restrict__ group_start, int4* __restrict__ group_page)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const uint64_t k = keys[i];
    const int32_t id = (int32_t)(k & ((1ull << L::INDEX_BITS) - 1));
    const int32_t old = slot_of_id[id];
#pragma unroll 4
    for (int f = 0; f < npd; ++f) pd_dst[f * cap + i] = pd_src[f * cap + old];
#pragma unroll
    for (int f = 0; f < PI_FIELDS; ++f) pi_dst[f * cap + i] = pi_src[f * cap + old];
    pi_dst[PI_ID * cap + i] = id;
    slot_of_id[id] = (int32_t)i;
    short4 b = base_by_id[id];
    base[i] = b;
    if (head[i]) {
        int g = gidx[i];
        group_start[g] = (int32_t)i;
        group_page[g] = make_int4(b.x >> L::XB, b.y >> L::YB, b.z >> L::ZB, 0);
    }
}

__global__ void k_set_last(int32_t* __restrict__ group_start, const int32_t* __restrict__ G, int64_t P)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) group_start[*G] = (int32_t)P;
}

// Emission e = 8 g + t visits page (group page + (t>>2, (t>>1)&1, t&1)),
// the loop order of MpmSimulationBase.cpp:1081-1088.
__global__ void k_emit(const int4* __restrict__ group_page, int64_t G, PageDims pd, int32_t* __restrict__ first)
{
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 8 * G) return;
    int4 gp = group_page[e >> 3];
    int t = (int)(e & 7);
    int64_t idx = pd.index(gp.x + (t >> 2), gp.y + ((t >> 1) & 1), gp.z + (t & 1));
    atomicMin(&first[idx], (int32_t)e);
}

__global__ void k_mark_first(const int4* __restrict__ group_page, int64_t G, PageDims pd, const int32_t* __restrict__ first, int32_t* __restrict__ flag)
{
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 8 * G) return;
    int4 gp = group_page[e >> 3];
    int t = (int)(e & 7);
    int64_t idx = pd.index(gp.x + (t >> 2), gp.y + ((t >> 1) & 1), gp.z + (t & 1));
    flag[e] = (first[idx] == (int32_t)e) ? 1 : 0;
}

template <class L>
__global__ void k_blocks(const int4* __restrict__ group_page, int64_t G, PageDims pd, const int32_t* __restrict__ flag,
    const int32_t* __restrict__ pos, int32_t* __restrict__ page_block, int4* __restrict__ block_page, uint64_t* __restrict__ block_index)
{
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 8 * G || !flag[e]) return;
    int4 gp = group_page[e >> 3];
    int t = (int)(e & 7);
    int x = gp.x + (t >> 2), y = gp.y + ((t >> 1) & 1), z = gp.z + (t & 1);
    int b = pos[e];
    page_block[pd.index(x, y, z)] = b;
    block_page[b] = make_int4(x, y, z, 0);
    block_index[b] = L::page_index(x, y, z);
}

__global__ void k_group_nbr(const int4* __restrict__ group_page, int64_t G, PageDims pd, const int32_t* __restrict__ page_block,
    int32_t* __restrict__ first, int32_t* __restrict__ nbr)
{
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 8 * G) return;
    int4 gp = group_page[e >> 3];
    int t = (int)(e & 7);
    int64_t idx = pd.index(gp.x + (t >> 2), gp.y + ((t >> 1) & 1), gp.z + (t & 1));
    nbr[e] = page_block[idx];
    first[idx] = PAGE_CLEAN; // for the next pass
}

// ------------------------------------------------------ binning by page ----
// Groups up to which binning by page is worth it: k_rank compares all pairs (40 us
// at 7500 groups) and k_number numbers the pages in one CTA (132 us).  A pass by
// page and by radix sort, 2 particles per group: 5000 groups 0.122 ms by page, 7000
// 0.214 and 0.231, 8000 0.258 and 0.226, 16000 0.545 and 0.267; 128 per group: 7000
// 0.325 and 0.38, 8000 0.383 and 0.40, 16000 0.79 and 0.59.  In a substep, where the
// radix way's 30 launches more also leave gaps, the two meet between 8400 and
// 10700 groups.
constexpr int RANK_MAX = 8192;
constexpr int ORDER_CAP = 2048;       // particles of one group: 16 KB of shared memory

// Base node of every slot, particles per page; the particle that finds its
// page clean appends the page to the list.  Slots are in the last
// pass's order, so the lanes of a warp mostly share a page and count as one.
template <class L, class KT>
__global__ void __launch_bounds__(BIN_THREADS) k_count(const double* __restrict__ x, int64_t cap, int64_t P, double inv_dx_d, float inv_dx_f,
    short4* __restrict__ base, int32_t* __restrict__ first, int4* __restrict__ list, PageDims pd, DevCounters* __restrict__ dc)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = s < P;
    int b[3] = { 0, 0, 0 };
    if (in) {
        if (!base_node<L, KT>(x, cap, s, inv_dx_d, inv_dx_f, pd, b)) atomicOr(&dc->flags, (int32_t)FLAG_OUT_OF_GRID);
        base[s] = make_short4((short)b[0], (short)b[1], (short)b[2], 0);
    }
    const int p0 = b[0] >> L::XB, p1 = b[1] >> L::YB, p2 = b[2] >> L::ZB;
    const int64_t page = in ? pd.index(p0, p1, p2) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, page);
    if (!in || (threadIdx.x & 31) != __ffs(peers) - 1) return;
    if (atomicSub(&first[page], __popc(peers)) == PAGE_CLEAN) {
        const unsigned long long g = atomicAdd(reinterpret_cast<unsigned long long*>(&dc->G), 1ull);
        list[g] = make_int4(p0, p1, p2, (int)(uint32_t)L::page_index(p0, p1, p2));
    }
}

// Per listed page: its particle count, the largest count, and the number of
// distinct pages among it and its 7 upper neighbours.
__global__ void __launch_bounds__(BIN_THREADS) k_pages(const int4* __restrict__ list, PageDims pd, int32_t* __restrict__ list_cnt,
    int32_t* __restrict__ first, DevCounters* __restrict__ dc)
{
    const int64_t G = dc->G;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < 8 * G; e += (int64_t)gridDim.x * blockDim.x) {
        const int4 p = list[e >> 3];
        const int t = (int)(e & 7);
        const int64_t idx = pd.index(p.x + (t >> 2), p.y + ((t >> 1) & 1), p.z + (t & 1));
        const int32_t was = atomicAnd(&first[idx], ~PAGE_BIT);
        if (was & PAGE_BIT) atomicAdd(reinterpret_cast<unsigned long long*>(&dc->B), 1ull);
        if (t == 0) {
            const int c = PAGE_CLEAN - (was | PAGE_BIT);
            list_cnt[e >> 3] = c;
            atomicMax(&dc->max_group, c);
        }
    }
}

// Leaves the page table clean when the pass stops after k_pages.
__global__ void __launch_bounds__(BIN_THREADS) k_unmark(const int4* __restrict__ list, int64_t G, PageDims pd, int32_t* __restrict__ first)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 8 * G) return;
    const int4 p = list[e >> 3];
    const int t = (int)(e & 7);
    const int64_t idx = pd.index(p.x + (t >> 2), p.y + ((t >> 1) & 1), p.z + (t & 1));
    first[idx] = PAGE_CLEAN;
}

// One warp per listed page: its rank among the page indices and its first slot
// (the particles of the smaller ones); the page's word becomes the cursor of
// k_place.
__global__ void __launch_bounds__(BIN_THREADS) k_rank(const int4* __restrict__ list, const int32_t* __restrict__ list_cnt, int G, int64_t P,
    PageDims pd, int32_t* __restrict__ group_start, int4* __restrict__ group_page, int32_t* __restrict__ first)
{
    const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= G) return;
    const int4 p = list[i];
    const uint32_t mine = (uint32_t)p.w;
    int rank = 0, start = 0;
#pragma unroll 4
    for (int j = lane; j < G; j += 32) {
        const bool below = (uint32_t)list[j].w < mine;
        rank += below ? 1 : 0;
        start += below ? list_cnt[j] : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rank += __shfl_xor_sync(0xffffffffu, rank, o);
        start += __shfl_xor_sync(0xffffffffu, start, o);
    }
    if (lane != 0) return;
    group_start[rank] = start;
    group_page[rank] = make_int4(p.x, p.y, p.z, p.w);
    first[pd.index(p.x, p.y, p.z)] = PAGE_CURSOR + start;
    if (i == 0) group_start[G] = (int32_t)P;
}

// Every particle into its group's range, in any order: (element, index) of its
// key above its old slot.
template <class L>
__global__ void __launch_bounds__(BIN_THREADS) k_place(const short4* __restrict__ base, int64_t P, const int32_t* __restrict__ orig_id,
    PageDims pd, int32_t* __restrict__ first, uint64_t* __restrict__ pairs)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = s < P;
    const short4 b = in ? base[s] : make_short4(0, 0, 0, 0);
    const int64_t page = in ? pd.index(b.x >> L::XB, b.y >> L::YB, b.z >> L::ZB) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, page);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    int at = 0;
    if (in && lane == leader) at = atomicAdd(&first[page], __popc(peers)) - PAGE_CURSOR;
    at = __shfl_sync(0xffffffffu, at, leader);
    if (!in) return;
    at += __popc(peers & ((1u << lane) - 1u));
    const uint32_t e = (uint32_t)L::elem(b.x & (L::BX - 1), b.y & (L::BY - 1), b.z & (L::BZ - 1));
    pairs[at] = ((uint64_t)((e << L::INDEX_BITS) | (uint32_t)orig_id[s]) << 32) | (uint32_t)s;
}

// One CTA per group: its particles ordered by (element, index): placed by
// element, then by the number of smaller indices in their cell.
template <class L>
__global__ void __launch_bounds__(BIN_THREADS) k_order(const int32_t* __restrict__ group_start, const int4* __restrict__ group_page,
    const uint64_t* __restrict__ pairs, uint64_t* __restrict__ keys, int32_t* __restrict__ old_slot, short4* __restrict__ base,
    int32_t* __restrict__ cells)
{
    __shared__ uint64_t cell[ORDER_CAP];
    __shared__ int32_t start[L::NPB + 1], fill[L::NPB];
    const int g = blockIdx.x, s0 = group_start[g], n = group_start[g + 1] - s0;
    for (int e = threadIdx.x; e < L::NPB; e += blockDim.x) fill[e] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&fill[pairs[s0 + i] >> (32 + L::INDEX_BITS)], 1);
    __syncthreads();
    if (threadIdx.x < 32) { // exclusive prefix over the elements
        constexpr int PER = L::NPB / 32;
        int c[PER], local = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            c[k] = fill[threadIdx.x * PER + k];
            local += c[k];
        }
        int incl = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)threadIdx.x >= o) incl += v;
        }
        int run = incl - local;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            start[threadIdx.x * PER + k] = run;
            fill[threadIdx.x * PER + k] = run;
            run += c[k];
        }
        if (threadIdx.x == 31) start[L::NPB] = run;
        __syncwarp();
        write_cells<L>(start, g, cells);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const uint64_t v = pairs[s0 + i];
        cell[atomicAdd(&fill[v >> (32 + L::INDEX_BITS)], 1)] = v;
    }
    __syncthreads();
    const int4 gp = group_page[g];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const uint64_t v = cell[i];
        const int e = (int)(v >> (32 + L::INDEX_BITS)), a = start[e], b = start[e + 1];
        int r = a;
        for (int j = a; j < b; ++j) r += cell[j] < v ? 1 : 0;
        const int64_t at = s0 + r;
        keys[at] = ((uint64_t)(uint32_t)gp.w << 32) | (v >> 32);
        old_slot[at] = (int32_t)(uint32_t)v;
        base[at] = make_short4((short)((gp.x << L::XB) | (e >> (L::YB + L::ZB))), (short)((gp.y << L::YB) | ((e >> L::ZB) & (L::BY - 1))),
            (short)((gp.z << L::ZB) | (e & (L::BZ - 1))), 0);
    }
}

// The cell records of sorted groups (the radix way): one warp per group, cell
// starts by the heads of equal elements.
template <class L>
__global__ void __launch_bounds__(32) k_cells(const int32_t* __restrict__ group_start, const short4* __restrict__ base, int32_t* __restrict__ cells,
    DevCounters* __restrict__ dc)
{
    __shared__ int32_t start[L::NPB + 1];
    const int g = blockIdx.x, lane = threadIdx.x, s0 = group_start[g], n = group_start[g + 1] - s0;
    if (lane == 0) atomicMax(&dc->max_group, n);
    for (int e = lane; e <= L::NPB; e += 32) start[e] = n;
    __syncwarp();
#pragma unroll 4
    for (int i = lane; i < n; i += 32) {
        const short4 b = base[s0 + i];
        const int e = (int)L::elem(b.x & (L::BX - 1), b.y & (L::BY - 1), b.z & (L::BZ - 1));
        atomicMin(&start[e], i);
    }
    __syncwarp();
    // an empty cell starts where the next one does: the smallest start from each cell on
    constexpr int PER = L::NPB / 32;
    int c[PER], m = n;
#pragma unroll
    for (int k = PER - 1; k >= 0; --k) {
        m = min(m, start[lane * PER + k]);
        c[k] = m;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) m = min(m, __shfl_down_sync(0xffffffffu, m, o)); // of this lane's cells and all after
    int after = __shfl_down_sync(0xffffffffu, m, 1);
    if (lane == 31) after = n;
#pragma unroll
    for (int k = 0; k < PER; ++k) start[lane * PER + k] = min(c[k], after);
    __syncwarp();
    write_cells<L>(start, g, cells);
}

// New slot i receives the particle of old_slot[i]: every field gathered.
template <class L>
__global__ void __launch_bounds__(BIN_THREADS) k_move(const uint64_t* __restrict__ keys, const int32_t* __restrict__ old_slot, int64_t P, int64_t cap,
    int npd, const double* __restrict__ pd_src, double* __restrict__ pd_dst, const int32_t* __restrict__ pi_src, int32_t* __restrict__ pi_dst,
    int32_t* __restrict__ slot_of_id)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const int32_t id = (int32_t)(keys[i] & ((1ull << L::INDEX_BITS) - 1)), old = old_slot[i];
#pragma unroll 8
    for (int f = 0; f < npd; ++f) pd_dst[f * cap + i] = pd_src[f * cap + old];
#pragma unroll
    for (int f = 0; f < PI_FIELDS; ++f)
        if (f != PI_ID) pi_dst[f * cap + i] = pi_src[f * cap + old];
    pi_dst[PI_ID * cap + i] = id;
    slot_of_id[id] = (int32_t)i;
}

// Page numbering by one CTA: a page's block index is its rank among the first
// emissions (k_emit), each thread numbering a run of consecutive emissions.
template <class L>
__global__ void __launch_bounds__(1024) k_number(const int4* __restrict__ group_page, int G, PageDims pd, const int32_t* __restrict__ first,
    int32_t* __restrict__ page_block, int4* __restrict__ block_page, uint64_t* __restrict__ block_index)
{
    __shared__ int warp_tot[32];
    const int n = 8 * G, per = (n + 1023) / 1024, e0 = (int)threadIdx.x * per, e1 = e0 + per < n ? e0 + per : n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int mine = 0;
#pragma unroll 4
    for (int e = e0; e < e1; ++e) {
        const int4 gp = group_page[e >> 3];
        const int t = e & 7;
        mine += first[pd.index(gp.x + (t >> 2), gp.y + ((t >> 1) & 1), gp.z + (t & 1))] == e ? 1 : 0;
    }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int b = incl - mine;
    for (int w = 0; w < warp; ++w) b += warp_tot[w];
    for (int e = e0; e < e1; ++e) {
        const int4 gp = group_page[e >> 3];
        const int t = e & 7, x = gp.x + (t >> 2), y = gp.y + ((t >> 1) & 1), z = gp.z + (t & 1);
        if (first[pd.index(x, y, z)] != e) continue;
        page_block[pd.index(x, y, z)] = b;
        block_page[b] = make_int4(x, y, z, 0);
        block_index[b] = L::page_index(x, y, z);
        ++b;
    }
}

// The radix way (see the top of the file); dc is zeroed and the page table is
// clean, but counts as dirty until the pass is complete.
template <class L, class KT>
static int binning_radix(Ctx* ctx)
{
    cudaStream_t st = ctx->stream;
    const int64_t P = ctx->P, cap = ctx->Pcap;
    PageDims pdims{ ctx->pages[0], ctx->pages[1], ctx->pages[2] };
    DevCounters* dc = ctx->counters.as<DevCounters>();
    ZMPM_CUDA(ctx->scan_i32.ensure((P + 1) * sizeof(int32_t)));
    ZMPM_CUDA(ctx->scan_scr.ensure((scan_scratch_elems(8 * P + 8) + 8) * sizeof(int32_t)));
    ZMPM_CUDA(ctx->radix_scr.ensure((radix_scratch_elems(P) + 8) * sizeof(int32_t)));

    k_keys<L, KT><<<nblk(P), BIN_THREADS, 0, st>>>(ctx->pdf(PD_X), cap, P, 1.0 / ctx->cfg.dx, 1.0f / (float)ctx->cfg.dx, ctx->pif(PI_ID), ctx->keys.as<uint64_t>(),
        ctx->base_by_id.as<short4>(), pdims, &dc->flags);
    ++g_kernel_launches;
    uint64_t* sorted = radix_sort(ctx->keys.as<uint64_t>(), ctx->keys_alt.as<uint64_t>(), P, L::INDEX_BITS, ctx->key_bits,
        ctx->radix_scr.as<int32_t>(), st);
    if (sorted != ctx->keys.as<uint64_t>()) std::swap(ctx->keys, ctx->keys_alt);
    const uint64_t* keys = ctx->keys.as<uint64_t>();

    int32_t* head = ctx->flags_i32.as<int32_t>();
    int32_t* gidx = ctx->scan_i32.as<int32_t>();
    int32_t* tot = ctx->scan_scr.as<int32_t>();
    int32_t* sscr = tot + 8;
    k_group_heads<<<nblk(P), BIN_THREADS, 0, st>>>(keys, P, head);
    ++g_kernel_launches;
    exclusive_scan<int32_t>(head, gidx, P, tot, sscr, st);
    k_permute<L><<<nblk(P), BIN_THREADS, 0, st>>>(keys, P, cap, ctx->pd_active, ctx->pd.as<double>(), ctx->pd_alt.as<double>(), ctx->pi.as<int32_t>(),
        ctx->pi_alt.as<int32_t>(), ctx->slot_of_id.as<int32_t>(), ctx->base_by_id.as<short4>(), ctx->base.as<short4>(), head, gidx,
        ctx->group_start.as<int32_t>(), ctx->group_page.as<int4>());
    ++g_kernel_launches;
    std::swap(ctx->pd, ctx->pd_alt);
    std::swap(ctx->pi, ctx->pi_alt);
    k_set_last<<<1, 32, 0, st>>>(ctx->group_start.as<int32_t>(), tot, P);
    ++g_kernel_launches;

    int32_t hG = 0;
    ZMPM_CUDA(cudaMemcpyAsync(&hG, tot, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    ZMPM_CUDA(cudaMemcpyAsync(&ctx->hcounters, dc, sizeof(DevCounters), cudaMemcpyDeviceToHost, st));
    ZMPM_CUDA(cudaStreamSynchronize(st));
    if (ctx->hcounters.flags & FLAG_OUT_OF_GRID) {
        ctx->err = "a particle's stencil leaves the grid (raise grid_log2 or move the scene)";
        return ZMPM_OUT_OF_GRID;
    }
    const int64_t G = hG;
    ctx->G = G;

    ZMPM_CUDA(ctx->group_nbr.ensure(8 * G * sizeof(int32_t)));
    ZMPM_CUDA(ctx->group_cells.ensure(G * GroupCells<L>::WORDS * sizeof(int32_t)));
    k_cells<L><<<(unsigned)G, 32, 0, st>>>(ctx->group_start.as<int32_t>(), ctx->base.as<short4>(), ctx->group_cells.as<int32_t>(), dc);
    ++g_kernel_launches;
    ZMPM_CUDA(ctx->emit_flag.ensure(8 * G * sizeof(int32_t)));
    ZMPM_CUDA(ctx->emit_scan.ensure(8 * G * sizeof(int32_t)));
    const int4* gpage = ctx->group_page.as<int4>();
    int32_t* first = ctx->page_first.as<int32_t>();
    k_emit<<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, first);
    ++g_kernel_launches;
    k_mark_first<<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, first, ctx->emit_flag.as<int32_t>());
    ++g_kernel_launches;
    exclusive_scan<int32_t>(ctx->emit_flag.as<int32_t>(), ctx->emit_scan.as<int32_t>(), 8 * G, tot, sscr, st);
    int32_t hB = 0;
    ZMPM_CUDA(cudaMemcpyAsync(&hB, tot, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    ZMPM_CUDA(cudaMemcpyAsync(&ctx->hcounters, dc, sizeof(DevCounters), cudaMemcpyDeviceToHost, st));
    ZMPM_CUDA(cudaStreamSynchronize(st));
    const int64_t B = hB;
    ctx->B = B;
    ctx->bin_radix = G > RANK_MAX || ctx->hcounters.max_group > ORDER_CAP;
    ZMPM_CUDA(ctx->block_page.ensure(B * sizeof(int4)));
    ZMPM_CUDA(ctx->block_index.ensure(B * sizeof(uint64_t)));
    k_blocks<L><<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, ctx->emit_flag.as<int32_t>(), ctx->emit_scan.as<int32_t>(),
        ctx->page_block.as<int32_t>(), ctx->block_page.as<int4>(), ctx->block_index.as<uint64_t>());
    ++g_kernel_launches;
    k_group_nbr<<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, ctx->page_block.as<int32_t>(), first, ctx->group_nbr.as<int32_t>());
    ++g_kernel_launches;
    ZMPM_CUDA(cudaGetLastError());
    ctx->table_dirty = false;
    ctx->binned = true;
    return ZMPM_OK;
}

template <class L, class KT>
static int binning_impl(Ctx* ctx)
{
    cudaStream_t st = ctx->stream;
    const int64_t P = ctx->P, cap = ctx->Pcap;
    PageDims pdims{ ctx->pages[0], ctx->pages[1], ctx->pages[2] };
    DevCounters* dc = ctx->counters.as<DevCounters>();
    ctx->binned = false;
    ZMPM_CUDA(cudaMemsetAsync(dc, 0, sizeof(DevCounters), st));
    if (P == 0) {
        ctx->G = ctx->B = 0;
        ctx->binned = true;
        return ZMPM_OK;
    }
    ZMPM_CUDA(ctx->keys.ensure(P * sizeof(uint64_t)));
    ZMPM_CUDA(ctx->keys_alt.ensure(P * sizeof(uint64_t)));
    ZMPM_CUDA(ctx->flags_i32.ensure(P * sizeof(int32_t)));
    ZMPM_CUDA(ctx->group_start.ensure((P + 1) * sizeof(int32_t)));
    ZMPM_CUDA(ctx->group_page.ensure(P * sizeof(int4)));
    ZMPM_CUDA(ctx->page_list.ensure(P * (sizeof(int4) + sizeof(int32_t))));

    int4* list = ctx->page_list.as<int4>();
    int32_t* list_cnt = reinterpret_cast<int32_t*>(list + P);
    int32_t* first = ctx->page_first.as<int32_t>();
    short4* base_old = ctx->base_by_id.as<short4>(); // here by old slot
    // A pass marks the page table and clears the marks at its end; one that
    // stopped in between (a failed allocation) left them, and a pass over such a
    // table would miss pages and place particles out of range.
    if (ctx->table_dirty) ZMPM_CUDA(cudaMemsetAsync(first, PAGE_CLEAN & 0xff, ctx->table_size * sizeof(int32_t), st));
    ctx->table_dirty = true;
    if (ctx->bin_radix) return binning_radix<L, KT>(ctx);
    k_count<L, KT><<<nblk(P), BIN_THREADS, 0, st>>>(ctx->pdf(PD_X), cap, P, 1.0 / ctx->cfg.dx, 1.0f / (float)ctx->cfg.dx, base_old, first, list,
        pdims, dc);
    k_pages<<<std::min(nblk(8 * P), 1024u), BIN_THREADS, 0, st>>>(list, pdims, list_cnt, first, dc);
    g_kernel_launches += 2;
    ZMPM_CUDA(cudaMemcpyAsync(&ctx->hcounters, dc, sizeof(DevCounters), cudaMemcpyDeviceToHost, st));
    ZMPM_CUDA(cudaStreamSynchronize(st));
    const int64_t G = ctx->hcounters.G, B = ctx->hcounters.B;
    const bool out = (ctx->hcounters.flags & FLAG_OUT_OF_GRID) != 0;
    if (out || G > RANK_MAX || ctx->hcounters.max_group > ORDER_CAP) {
        k_unmark<<<nblk(8 * G), BIN_THREADS, 0, st>>>(list, G, pdims, first);
        ++g_kernel_launches;
        ZMPM_CUDA(cudaGetLastError());
        if (out) {
            ctx->table_dirty = false;
            ctx->err = "a particle's stencil leaves the grid (raise grid_log2 or move the scene)";
            return ZMPM_OUT_OF_GRID;
        }
        ZMPM_CUDA(cudaMemsetAsync(dc, 0, sizeof(DevCounters), st));
        ctx->bin_radix = true;
        return binning_radix<L, KT>(ctx);
    }
    ctx->G = G;
    ctx->B = B;
    ZMPM_CUDA(ctx->group_nbr.ensure(8 * G * sizeof(int32_t)));
    ZMPM_CUDA(ctx->group_cells.ensure(G * GroupCells<L>::WORDS * sizeof(int32_t)));
    ZMPM_CUDA(ctx->block_page.ensure(B * sizeof(int4)));
    ZMPM_CUDA(ctx->block_index.ensure(B * sizeof(uint64_t)));
    int32_t* gstart = ctx->group_start.as<int32_t>();
    int4* gpage = ctx->group_page.as<int4>();
    int32_t* old_slot = ctx->flags_i32.as<int32_t>();
    k_rank<<<nblk(32 * G), BIN_THREADS, 0, st>>>(list, list_cnt, (int)G, P, pdims, gstart, gpage, first);
    k_place<L><<<nblk(P), BIN_THREADS, 0, st>>>(base_old, P, ctx->pif(PI_ID), pdims, first, ctx->keys_alt.as<uint64_t>());
    k_order<L><<<(unsigned)G, BIN_THREADS, 0, st>>>(gstart, gpage, ctx->keys_alt.as<uint64_t>(), ctx->keys.as<uint64_t>(), old_slot,
        ctx->base.as<short4>(), ctx->group_cells.as<int32_t>());
    k_move<L><<<nblk(P), BIN_THREADS, 0, st>>>(ctx->keys.as<uint64_t>(), old_slot, P, cap, ctx->pd_active, ctx->pd.as<double>(),
        ctx->pd_alt.as<double>(), ctx->pi.as<int32_t>(), ctx->pi_alt.as<int32_t>(), ctx->slot_of_id.as<int32_t>());
    std::swap(ctx->pd, ctx->pd_alt);
    std::swap(ctx->pi, ctx->pi_alt);
    k_emit<<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, first);
    k_number<L><<<1, 1024, 0, st>>>(gpage, (int)G, pdims, first, ctx->page_block.as<int32_t>(), ctx->block_page.as<int4>(),
        ctx->block_index.as<uint64_t>());
    k_group_nbr<<<nblk(8 * G), BIN_THREADS, 0, st>>>(gpage, G, pdims, ctx->page_block.as<int32_t>(), first, ctx->group_nbr.as<int32_t>());
    g_kernel_launches += 7;
    ZMPM_CUDA(cudaGetLastError());
    ctx->table_dirty = false;
    ctx->binned = true;
    return ZMPM_OK;
}

int run_binning(Ctx* ctx)
{
    if (ctx->layout == 1) return ctx->mixed ? binning_impl<Layout244, float>(ctx) : binning_impl<Layout244, double>(ctx);
    return ctx->mixed ? binning_impl<Layout444, float>(ctx) : binning_impl<Layout444, double>(ctx);
}

} // namespace zmpm
