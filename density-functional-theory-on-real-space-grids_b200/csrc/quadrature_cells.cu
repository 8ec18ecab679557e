// (d4) L^T of the cusp-aware quadrature over nodes sorted by their base cell.
//
// A node at base cell (bx, by, bz) reaches the 8 x 8 x 8 grid points bx-3 .. bx+4 (and so on), so the
// nodes that reach a block of grid points are those of a box of cells: with the nodes sorted by
// cell (x, y, z, z fastest) they are one contiguous run per (bx, by), found from a table of each
// cell's first node. L^T therefore needs no list of its 512 m entries (12 bytes each: 260 MB at He
// 65^3, and a radix sort of that many keys to build): a block gathers from the runs around it, with
// weights formed from each node's 24 one-dimensional ones (src/cdft/operators/quadrature.py:506-650).
//
// The blocks are very uneven (one next to a nucleus is reached by a quarter of all nodes), so the
// concatenated runs of a block are cut into items of equal length, one CTA each; an item leaves the
// sums of its nodes and a second kernel adds a block's items in order. Everything is summed in a fixed
// order, so the results do not depend on scheduling.

#include "common.cuh"
#include "per_device.cuh"

namespace cdftb {
namespace {

constexpr int KTAP = 8;
constexpr int HALFD = 3;
constexpr int kRow = 24;   // doubles per node: x, y, z weights
constexpr int kChunk = 8;  // nodes a warp stages at a time

// A few fields: blocks of 4 x 8 x 8 points, items of 512 nodes on 4 warps. Many: 2 x 2 x 8, 1024 on 8.
// The items make the launch even: with a cluster of 8 CTAs per block instead, the warps of the blocks next
// to the nucleus had 1100 nodes where the mean is 100, and the few-field lift took 171 us.
struct FewShape {
    static constexpr int BX = 4, BY = 8, BZ = 8, WARPS = 4, NODES = 512;
    static constexpr int RX = BX + KTAP - 1, RY = BY + KTAP - 1, RUNS = RX * RY, POINTS = BX * BY * BZ;
};
struct ManyShape {
    static constexpr int BX = 2, BY = 2, BZ = 8, WARPS = 8, NODES = 1024;
    static constexpr int RX = BX + KTAP - 1, RY = BY + KTAP - 1, RUNS = RX * RY, POINTS = BX * BY * BZ;
};
constexpr int MANY = 32;  // fields per pass of the many-field kernels

// The blocks of one shape: those covering the points reached from the cells lo .. hi.
struct Blocks {
    int p0[3], n[3];
    int64_t count, items;  // items: at most this many (a block of b points takes ceil(7 / b) + 1 per axis at most)
};

// The plan, in one device buffer.
struct CellPlan {
    int nx, ny, nz;
    int lo[3], hi[3];  // the box of cells that may hold nodes (inclusive)
    int64_t m;
    Blocks few, many;
    int* cell_ptr;       // first sorted node of every cell, n_points + 1
    int* order;          // node of every sorted position
    int* z_sorted;       // z cell per sorted node
    double* w_sorted;    // 24 weights per sorted node
    int *few_ptr, *few_block, *many_ptr, *many_block;  // a block's first item; an item's block
    int64_t bytes;
    // The plan's first words: how many of its nodes failed the build's check (none in a plan that may be used),
    // and the key of the sizes and box it was built for. The kernels compare the key with their call's before they
    // follow anything in the plan, so that a plan that failed, or another call's, is never followed out of range.
    unsigned long long *bad, *built;
    unsigned long long key;
};

__device__ __forceinline__ bool usable(const CellPlan& p) { return *p.built == p.key; }

// A key of the sizes and the box (FNV-1a over them, never zero).
unsigned long long plan_key(const CellPlan& p) {
    const int64_t words[] = {p.m, p.nx, p.ny, p.nz, p.lo[0], p.lo[1], p.lo[2], p.hi[0], p.hi[1], p.hi[2]};
    unsigned long long h = 14695981039346656037ull;
    for (const int64_t w : words)
        for (int byte = 0; byte < 8; ++byte) h = (h ^ ((static_cast<unsigned long long>(w) >> (8 * byte)) & 255)) * 1099511628211ull;
    return h | 1;
}

template <typename S>
Blocks blocks_of(const CellPlan& p) {
    const int b[3] = {S::BX, S::BY, S::BZ};
    const int dims[3] = {p.nx, p.ny, p.nz};
    Blocks r{};
    r.count = 1;
    int64_t reach = 1;
    for (int d = 0; d < 3; ++d) {
        r.p0[d] = p.lo[d] - HALFD > 0 ? p.lo[d] - HALFD : 0;
        const int top = p.hi[d] + KTAP - HALFD < dims[d] ? p.hi[d] + KTAP - HALFD : dims[d];
        r.n[d] = static_cast<int>(ceil_div(top - r.p0[d], b[d]));
        r.count *= r.n[d];
        reach *= ceil_div(KTAP - 1, b[d]) + 1;
    }
    r.items = ceil_div(p.m * reach, S::NODES) + r.count;
    return r;
}

// False if the sizes are not ones a plan can have.
bool plan_layout(int64_t m, int nx, int ny, int nz, const int* cell_box, void* base, CellPlan* out) {
    const int64_t cells = int64_t(nx) * ny * nz;
    if (m <= 0 || nx <= 0 || ny <= 0 || nz <= 0 || !cell_box) return false;
    if (m >= (1ll << 31) / kRow || cells >= (1ll << 31) - 1) return false;
    CellPlan p{};
    p.nx = nx;
    p.ny = ny;
    p.nz = nz;
    p.m = m;
    const int dims[3] = {nx, ny, nz};
    for (int d = 0; d < 3; ++d) {
        p.lo[d] = cell_box[d];
        p.hi[d] = cell_box[3 + d];
        if (p.lo[d] < 0 || p.hi[d] >= dims[d] || p.lo[d] > p.hi[d]) return false;
    }
    p.few = blocks_of<FewShape>(p);
    p.many = blocks_of<ManyShape>(p);
    char* at = static_cast<char*>(base);
    auto take = [&](int64_t bytes) {
        char* r = at;
        at += (bytes + 255) / 256 * 256;
        return r;
    };
    p.bad = reinterpret_cast<unsigned long long*>(take(16));
    p.built = p.bad + 1;
    p.key = plan_key(p);
    p.w_sorted = reinterpret_cast<double*>(take(m * kRow * 8));
    p.cell_ptr = reinterpret_cast<int*>(take((cells + 1) * 4));
    p.order = reinterpret_cast<int*>(take(m * 4));
    p.z_sorted = reinterpret_cast<int*>(take(m * 4));
    p.few_ptr = reinterpret_cast<int*>(take((p.few.count + 1) * 4));
    p.few_block = reinterpret_cast<int*>(take(p.few.items * 4));
    p.many_ptr = reinterpret_cast<int*>(take((p.many.count + 1) * 4));
    p.many_block = reinterpret_cast<int*>(take(p.many.items * 4));
    p.bytes = at - static_cast<char*>(base);
    *out = p;
    return true;
}

// cell_ptr[c] = the first sorted node whose cell key is at least c (keys: (x ny + y) nz + z).
__global__ void cell_starts_kernel(const int64_t* __restrict__ keys, int64_t m, int64_t cells,
                                   int* __restrict__ cell_ptr) {
    const int64_t c = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (c > cells) return;
    int64_t lo = 0, hi = m;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (keys[mid] < c) lo = mid + 1;
        else hi = mid;
    }
    cell_ptr[c] = static_cast<int>(lo);
}

// The weights, node and z cell of every sorted node, which is checked on the way: the runs and items take for
// granted that the keys ascend, that each is its node's cell, and that no cell lies outside the box.
__global__ void sort_nodes_kernel(const int* __restrict__ base, const double* __restrict__ w1d,
                                  const int* __restrict__ order, const int64_t* __restrict__ keys, const CellPlan p) {
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= p.m * kRow) return;
    const int64_t i = k / kRow;
    const int c = static_cast<int>(k - i * kRow);
    const int node = order[i];
    if (node < 0 || node >= p.m) {
        if (c == 0) atomicAdd(p.bad, 1ull);
        return;
    }
    p.w_sorted[k] = w1d[int64_t(node) * kRow + c];
    if (c == 0) {
        const int x = base[int64_t(node) * 3], y = base[int64_t(node) * 3 + 1], z = base[int64_t(node) * 3 + 2];
        const bool inside = x >= p.lo[0] && x <= p.hi[0] && y >= p.lo[1] && y <= p.hi[1] && z >= p.lo[2] && z <= p.hi[2];
        if (!inside || keys[i] != (int64_t(x) * p.ny + y) * p.nz + z || (i > 0 && keys[i - 1] > keys[i]))
            atomicAdd(p.bad, 1ull);
        p.order[i] = node;
        p.z_sorted[i] = z;
    }
}

template <typename S>
__device__ __forceinline__ void block_origin(const Blocks& b, int block, int& x0, int& y0, int& z0) {
    z0 = b.p0[2] + (block % b.n[2]) * S::BZ;
    y0 = b.p0[1] + (block / b.n[2] % b.n[1]) * S::BY;
    x0 = b.p0[0] + block / (b.n[2] * b.n[1]) * S::BX;
}

// The sorted nodes of run r of the block at (x0, y0, z0): the cells (x0 - 4 + r / RY, y0 - 4 + r % RY)
// that reach z points z0 .. z0 + BZ - 1.
template <typename S>
__device__ __forceinline__ void run_range(const CellPlan& p, int x0, int y0, int z0, int r, int& first, int& count) {
    first = count = 0;
    const int bx = x0 - 4 + r / S::RY, by = y0 - 4 + r % S::RY;
    if (bx < p.lo[0] || bx > p.hi[0] || by < p.lo[1] || by > p.hi[1]) return;
    const int za = max(z0 - (KTAP - HALFD - 1), p.lo[2]), zb = min(z0 + S::BZ - 1 + HALFD, p.hi[2]);
    if (za > zb) return;
    const int64_t row = (int64_t(bx) * p.ny + by) * p.nz;
    first = p.cell_ptr[row + za];
    count = p.cell_ptr[row + zb + 1] - first;
}

// Items per block (into ptr[block]; none in a plan that failed the check), one warp per block.
template <typename S>
__global__ void item_counts_kernel(const CellPlan p, const Blocks b, int* __restrict__ ptr) {
    const int64_t block = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (block >= b.count) return;
    int x0, y0, z0, nodes = 0;
    block_origin<S>(b, static_cast<int>(block), x0, y0, z0);
    for (int r = *p.bad ? S::RUNS : lane; r < S::RUNS; r += 32) {
        int first, count;
        run_range<S>(p, x0, y0, z0, r, first, count);
        nodes += count;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) nodes += __shfl_down_sync(0xffffffffu, nodes, off);
    if (lane == 0) ptr[block] = (nodes + S::NODES - 1) / S::NODES;
}

// ptr[block] := the items of the blocks before it, ptr[count] := all items; item_block: by one CTA, which
// then marks the plan as built if its nodes passed the check.
__global__ void __launch_bounds__(1024) item_scan_kernel(const CellPlan p, int* __restrict__ ptr, int64_t count,
                                                         int* __restrict__ item_block) {
    __shared__ int warp_sum[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int64_t b0 = 0; b0 < count; b0 += blockDim.x) {
        const int64_t b = b0 + threadIdx.x;
        const int own = b < count ? ptr[b] : 0;
        int sum = own;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, off);
            if (lane >= off) sum += v;
        }
        if (lane == 31) warp_sum[warp] = sum;
        __syncthreads();
        int before = carry;
        for (int w = 0; w < warp; ++w) before += warp_sum[w];
        const int first = before + sum - own;
        if (b < count) {
            ptr[b] = first;
            for (int k = 0; k < own; ++k) item_block[first + k] = static_cast<int>(b);
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = first + own;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        ptr[count] = carry;
        *p.built = *p.bad ? 0 : p.key;
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The runs of an item's block, in shared memory: run r's first sorted node and the nodes before it.
template <typename S>
struct Runs {
    int first[S::RUNS];
    int before[S::RUNS + 1];

    // by every thread of the CTA
    __device__ __forceinline__ void load(const CellPlan& p, int x0, int y0, int z0) {
        for (int r = threadIdx.x; r < S::RUNS; r += S::WARPS * 32) run_range<S>(p, x0, y0, z0, r, first[r], before[r + 1]);
        __syncthreads();
        if (threadIdx.x < 32) {
            constexpr int PER = (S::RUNS + 31) / 32;
            const int lane = threadIdx.x;
            int own[PER], total = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int r = lane * PER + k;
                own[k] = total;
                total += r < S::RUNS ? before[r + 1] : 0;
            }
            int sum = total;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, off);
                if (lane >= off) sum += v;
            }
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (lane * PER + k < S::RUNS) before[lane * PER + k] = sum - total + own[k];
            if (lane == 31) before[S::RUNS] = sum;
        }
        __syncthreads();
    }
};

// A warp's share of a block's concatenated runs, in chunks of at most kChunk nodes of one run.
template <typename S>
struct ChunkWalk {
    const Runs<S>& runs;
    int r, n0, end, left, count = 0;

    __device__ __forceinline__ ChunkWalk(const Runs<S>& all, int from, int nodes) : runs(all) {
        left = min(nodes, all.before[S::RUNS] - from);
        int lo = 0, hi = S::RUNS - 1;  // the last run that starts at or before `from`
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (all.before[mid] <= from) lo = mid;
            else hi = mid - 1;
        }
        r = lo;
        n0 = all.first[r] + from - all.before[r];
        end = all.first[r] + all.before[r + 1] - all.before[r];
    }
    __device__ __forceinline__ bool next() {
        left -= count;
        n0 += count;
        count = 0;
        if (left <= 0) return false;
        while (n0 >= end) {
            ++r;
            n0 = runs.first[r];
            end = n0 + runs.before[r + 1] - runs.before[r];
        }
        count = min(min(kChunk, end - n0), left);
        return true;
    }
};

template <int BYTES>
__device__ __forceinline__ void copy_nodes(void* dst, const void* src, int count, int lane) {
    constexpr int kUnits = BYTES / 16;
#pragma unroll
    for (int u = 0; u < kChunk * kUnits / 32; ++u) {
        const int k = u * 32 + lane;
        if (k < count * kUnits) cp_async16(static_cast<char*>(dst) + k * 16, static_cast<const char*>(src) + k * 16);
    }
}

// ---- L^T, a few fields. Lanes are 4 x by 8 z points, each with 8 y points of every field in
// registers: which y points a node reaches depends on its run alone, so the node loop is compiled for
// each of the 15 cases and does no test on y; a lane outside the node's reach in x or z adds zeros (a
// product is formed only within the reach, so a node's infinity or NaN stays its own). Instruction issue
// bounds it (55% of cycles, FP64 pipe 23%). He 65^3, two fields: 43 us and 5 us for the sums, where a
// warp per point over the list of entries took 271 us (260 MB of entries read).

// The nodes of one chunk of a run J - 4 cells from the block's first y point.
template <int NF, int J>
__device__ __forceinline__ void few_nodes(const double* stage, const double* xs, const int* zs, int count, int ai,
                                          bool okx, int cz, double (&acc)[NF][FewShape::BY]) {
#pragma unroll 2
    for (int n = 0; n < count; ++n) {
        const double* row = stage + n * kRow;
        const int c = cz - zs[n];
        const bool ok = okx && static_cast<unsigned>(c) < KTAP;
        const double wxz = row[ai] * row[16 + (ok ? c : 0)];
        double t[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const double v = wxz * xs[n * NF + f];
            t[f] = ok ? v : 0.0;
        }
#pragma unroll
        for (int ly = 0; ly < FewShape::BY; ++ly) {
            constexpr int kTop = KTAP - 1;
            if (ly + kTop - J < 0 || ly + kTop - J > kTop) continue;
            const double w = row[8 + ((ly + kTop - J) & 7)];
#pragma unroll
            for (int f = 0; f < NF; ++f) acc[f][ly] = fma(t[f], w, acc[f][ly]);
        }
    }
}

// partial[item][f][x lane, z lane, y] of the item's nodes.
template <int NF>
__global__ void __launch_bounds__(FewShape::WARPS * 32)
    lift_cells_few_kernel(const CellPlan p, const double* __restrict__ x, int64_t x_stride,
                          double* __restrict__ partial) {
    using S = FewShape;
    __shared__ __align__(16) double stage[S::WARPS][2][kChunk * kRow];
    __shared__ __align__(16) double xs[S::WARPS][kChunk * NF];
    __shared__ int zs[S::WARPS][kChunk];
    __shared__ double red[S::WARPS][NF][S::POINTS];
    __shared__ Runs<S> runs;
    const int item = blockIdx.x;
    const int items = p.few_ptr[p.few.count], block = p.few_block[item];
    if (!usable(p) || item >= items) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x0, y0, z0;
    block_origin<S>(p.few, block, x0, y0, z0);
    runs.load(p, x0, y0, z0);

    const int lx = lane >> 3, lz = lane & 7;
    double acc[NF][S::BY];
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int k = 0; k < S::BY; ++k) acc[f][k] = 0.0;

    ChunkWalk<S> walk(runs, (item - p.few_ptr[block]) * S::NODES + warp * (S::NODES / S::WARPS), S::NODES / S::WARPS);
    // lane f * 8 + n holds field f of the chunk's node n; lane n its z cell
    double xr = 0.0;
    int zr = 0;
    auto issue = [&](int slot) {
        copy_nodes<kRow * 8>(stage[warp][slot], p.w_sorted + int64_t(walk.n0) * kRow, walk.count, lane);
        const int n = lane & 7, f = lane >> 3;
        if (f < NF && n < walk.count) {
            xr = x[f * x_stride + p.order[walk.n0 + n]];
            if (f == 0) zr = p.z_sorted[walk.n0 + n];
        }
    };
    bool more = walk.next();
    if (more) issue(0);
    cp_async_commit();
    for (int slot = 0; more; slot ^= 1) {
        const int count = walk.count, r = walk.r;
        if ((lane >> 3) < NF) xs[warp][(lane & 7) * NF + (lane >> 3)] = xr;
        if (lane < kChunk) zs[warp][lane] = zr;
        more = walk.next();
        if (more) issue(slot ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncwarp();
        // x0 + lx = bx - 3 + a, z0 + lz = bz - 3 + c
        const int a = lx + KTAP - 1 - r / S::RY;
        const bool okx = static_cast<unsigned>(a) < KTAP;
        const int ai = okx ? a : 0, cz = z0 + lz + HALFD;
        const double* st = stage[warp][slot];
        switch (r % S::RY) {
#define CDFTB_FEW(J_) \
    case J_: few_nodes<NF, J_>(st, xs[warp], zs[warp], count, ai, okx, cz, acc); break;
            CDFTB_FEW(0) CDFTB_FEW(1) CDFTB_FEW(2) CDFTB_FEW(3) CDFTB_FEW(4) CDFTB_FEW(5) CDFTB_FEW(6) CDFTB_FEW(7)
            CDFTB_FEW(8) CDFTB_FEW(9) CDFTB_FEW(10) CDFTB_FEW(11) CDFTB_FEW(12) CDFTB_FEW(13)
            default: few_nodes<NF, 14>(st, xs[warp], zs[warp], count, ai, okx, cz, acc); break;
#undef CDFTB_FEW
        }
        __syncwarp();
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int k = 0; k < S::BY; ++k) red[warp][f][k * 32 + lane] = acc[f][k];
    __syncthreads();
    double* dst = partial + int64_t(item) * (NF * S::POINTS);
    for (int k = threadIdx.x; k < NF * S::POINTS; k += S::WARPS * 32) {
        double sum = red[0][0][k];
#pragma unroll
        for (int w = 1; w < S::WARPS; ++w) sum += red[w][0][k];
        dst[k] = sum;
    }
}

// out[f] at the block's points: the block's items in order (none: zero; NaN for a plan that is not this
// call's). One CTA per block and field.
template <int NF>
__global__ void __launch_bounds__(FewShape::POINTS) lift_cells_few_sum_kernel(const CellPlan p,
                                                                              const double* __restrict__ partial,
                                                                              double* __restrict__ out,
                                                                              int64_t out_stride) {
    using S = FewShape;
    const int block = blockIdx.x, f = blockIdx.y, k = threadIdx.x;
    int x0, y0, z0;
    block_origin<S>(p.few, block, x0, y0, z0);
    const int px = x0 + ((k & 31) >> 3), py = y0 + (k >> 5), pz = z0 + (k & 7);
    const double* src = partial + f * S::POINTS + k;
    const int first = p.few_ptr[block], end = p.few_ptr[block + 1];
    const bool ok = usable(p);
    const int last = ok ? end : first;
    double sum = ok ? 0.0 : nan("");
#pragma unroll 4
    for (int item = first; item < last; ++item) sum += src[int64_t(item) * (NF * S::POINTS)];
    if (px < p.nx && py < p.ny && pz < p.nz) out[f * out_stride + (int64_t(px) * p.ny + py) * p.nz + pz] = sum;
}

// ---- L^T, up to 32 fields per pass, lanes are the fields. A warp holds a 2 x 2 x 8 block of all
// fields in registers; per node it reads the 256-byte row of the node's field values, the four products
// of its x and y weights (formed once per chunk, one per lane) and its z weights, and does 4 multiplies
// and up to 32 multiply-adds: only the z points within the node's reach (the node loop jumps on the
// node's z cell; 17 of 32 on average). He 65^3, 32 fields: 268 us and 9 us for the sums; segments of the
// list of entries took 518 + 33 us (each entry a 256-byte row from L2, 5.5 GB).

// acc[..][k] += t w_z for the z points k that a node at z cell z0 + D reaches.
template <int D>
__device__ __forceinline__ void many_node(const double* row, const double (&t)[4], double (&acc)[4][ManyShape::BZ]) {
#pragma unroll
    for (int k = 0; k < ManyShape::BZ; ++k) {
        if (k < D - HALFD || k > D + KTAP - HALFD - 1) continue;
        const double w = row[16 + ((HALFD - D + k) & 7)];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][k] = fma(t[i], w, acc[i][k]);
    }
}

constexpr int kManyStage = kChunk * (kRow + MANY);  // doubles of a stage: weights, then field values
constexpr int kManyWxy = kChunk * 4;
constexpr size_t kManyRed = size_t(ManyShape::WARPS) * ManyShape::POINTS * MANY * 8;
constexpr size_t kManyStaged = size_t(ManyShape::WARPS) * (2 * kManyStage + kManyWxy) * 8;
constexpr size_t kManySmem = kManyRed > kManyStaged ? kManyRed : kManyStaged;

// partial[item][point][field] of the item's nodes.
__global__ void __launch_bounds__(ManyShape::WARPS * 32, 2)
    lift_cells_many_kernel(const CellPlan p, const double* __restrict__ rows, double* __restrict__ partial) {
    using S = ManyShape;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Runs<S> runs;
    double* red = reinterpret_cast<double*>(smem_raw);  // the sums reuse the stages' memory
    const int item = blockIdx.x;
    const int items = p.many_ptr[p.many.count], block = p.many_block[item];
    if (!usable(p) || item >= items) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* stage = red + warp * (2 * kManyStage + kManyWxy);
    double* wxy = stage + 2 * kManyStage;
    int x0, y0, z0;
    block_origin<S>(p.many, block, x0, y0, z0);
    runs.load(p, x0, y0, z0);

    double acc[4][S::BZ];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < S::BZ; ++k) acc[i][k] = 0.0;

    ChunkWalk<S> walk(runs, (item - p.many_ptr[block]) * S::NODES + warp * (S::NODES / S::WARPS), S::NODES / S::WARPS);
    int zr = 0;
    auto issue = [&](int slot) {
        double* st = stage + slot * kManyStage;
        copy_nodes<kRow * 8>(st, p.w_sorted + int64_t(walk.n0) * kRow, walk.count, lane);
        copy_nodes<MANY * 8>(st + kChunk * kRow, rows + int64_t(walk.n0) * MANY, walk.count, lane);
        if (lane < walk.count) zr = p.z_sorted[walk.n0 + lane];
    };
    bool more = walk.next();
    if (more) issue(0);
    cp_async_commit();
    for (int slot = 0; more; slot ^= 1) {
        const int count = walk.count, r = walk.r;
        const int z_now = zr;
        more = walk.next();
        if (more) issue(slot ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncwarp();
        // column i = 2 dx + dy of the block has taps a = 7 - r / RY + dx and b = 7 - r % RY + dy, of 0 .. 7
        const double* st = stage + slot * kManyStage;
        const int a0 = KTAP - 1 - r / S::RY, b0 = KTAP - 1 - r % S::RY;
        const bool whole = a0 >= 0 && a0 + 1 < KTAP && b0 >= 0 && b0 + 1 < KTAP;
        {
            const int a = a0 + ((lane >> 1) & 1), b = b0 + (lane & 1);
            const double* row = st + (lane >> 2) * kRow;
            wxy[lane] = row[a & 7] * row[8 + (b & 7)];
        }
        __syncwarp();
        for (int n = 0; n < count; ++n) {
            const double* row = st + n * kRow;
            const double xv = st[kChunk * kRow + n * MANY + lane];
            const double2 w0 = *reinterpret_cast<const double2*>(wxy + 4 * n);
            const double2 w1 = *reinterpret_cast<const double2*>(wxy + 4 * n + 2);
            double t[4] = {w0.x * xv, w0.y * xv, w1.x * xv, w1.y * xv};
            if (!whole) {  // a column out of the node's reach adds zeros
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (static_cast<unsigned>(a0 + (i >> 1)) >= KTAP || static_cast<unsigned>(b0 + (i & 1)) >= KTAP)
                        t[i] = 0.0;
            }
            switch (__shfl_sync(0xffffffffu, z_now, n) - z0) {
#define CDFTB_MANY(D_) \
    case D_: many_node<D_>(row, t, acc); break;
                CDFTB_MANY(-4) CDFTB_MANY(-3) CDFTB_MANY(-2) CDFTB_MANY(-1) CDFTB_MANY(0) CDFTB_MANY(1) CDFTB_MANY(2)
                CDFTB_MANY(3) CDFTB_MANY(4) CDFTB_MANY(5) CDFTB_MANY(6) CDFTB_MANY(7) CDFTB_MANY(8) CDFTB_MANY(9)
                CDFTB_MANY(10)
                default: break;
#undef CDFTB_MANY
            }
        }
        __syncwarp();
    }
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < S::BZ; ++k) red[(warp * S::POINTS + i * S::BZ + k) * MANY + lane] = acc[i][k];
    __syncthreads();
    double* dst = partial + int64_t(item) * (S::POINTS * MANY);
#pragma unroll
    for (int u = 0; u < S::POINTS / S::WARPS; ++u) {
        const int k = u * (S::WARPS * 32) + threadIdx.x;
        double sum = red[k];
#pragma unroll
        for (int w = 1; w < S::WARPS; ++w) sum += red[w * (S::POINTS * MANY) + k];
        dst[k] = sum;
    }
}

// out[f] at the block's 32 points: the block's items in order (NaN for a plan that is not this call's).
// One CTA per block; the sums pass through a shared tile so that the field-major stores run along z.
__global__ void __launch_bounds__(256) lift_cells_many_sum_kernel(const CellPlan p, const double* __restrict__ partial,
                                                                  int nf, double* __restrict__ out,
                                                                  int64_t out_stride) {
    using S = ManyShape;
    static_assert(S::POINTS == 32, "a tile of 32 points by 32 fields");
    __shared__ double tile[S::POINTS][MANY + 1];
    const int block = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = p.many_ptr[block], end = p.many_ptr[block + 1];
    const bool ok = usable(p);
    const int last = ok ? end : first;
    for (int pt = warp; pt < S::POINTS; pt += 8) {
        double sum = ok ? 0.0 : nan("");
#pragma unroll 4
        for (int item = first; item < last; ++item) sum += partial[(int64_t(item) * S::POINTS + pt) * MANY + lane];
        tile[pt][lane] = sum;
    }
    __syncthreads();
    int x0, y0, z0;
    block_origin<S>(p.many, block, x0, y0, z0);
    const int px = x0 + (lane >> 4), py = y0 + ((lane >> 3) & 1), pz = z0 + (lane & 7);
    if (px >= p.nx || py >= p.ny || pz >= p.nz) return;
    for (int f = warp; f < nf; f += 8) out[f * out_stride + (int64_t(px) * p.ny + py) * p.nz + pz] = tile[lane][f];
}

// x[f][order[i]] (f < nf) -> rows[i][f], zero for f >= nf: the field values of a sorted node as one row.
__global__ void __launch_bounds__(256) sorted_rows_kernel(const CellPlan p, const double* __restrict__ x, int nf,
                                                          int64_t stride, double* __restrict__ rows) {
    __shared__ double tile[MANY][MANY + 1];
    const int64_t m = p.m;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t i0 = int64_t(blockIdx.x) * MANY;
    const int64_t node = i0 + tx < m ? p.order[i0 + tx] : 0;
    if (!usable(p)) return;
    for (int f = ty; f < MANY; f += 8) tile[f][tx] = (f < nf && i0 + tx < m) ? x[f * stride + node] : 0.0;
    __syncthreads();
    for (int r = ty; r < MANY; r += 8)
        if (i0 + r < m) rows[(i0 + r) * MANY + tx] = tile[tx][r];
}

template <typename S>
int build_items(const CellPlan& p, const Blocks& b, int* ptr, int* item_block, cudaStream_t s) {
    item_counts_kernel<S><<<static_cast<unsigned>(ceil_div(b.count * 32, 256)), 256, 0, s>>>(p, b, ptr);
    int st = check_launch();
    if (st != CDFTB_OK) return st;
    item_scan_kernel<<<1, 1024, 0, s>>>(p, ptr, b.count, item_block);
    return check_launch();
}

template <int NF>
int lift_few(const CellPlan& p, const double* x, int64_t x_stride, double* out, int64_t out_stride, double* partial,
             cudaStream_t s) {
    lift_cells_few_kernel<NF><<<static_cast<unsigned>(p.few.items), FewShape::WARPS * 32, 0, s>>>(p, x, x_stride, partial);
    int st = check_launch();
    if (st != CDFTB_OK) return st;
    lift_cells_few_sum_kernel<NF><<<dim3(static_cast<unsigned>(p.few.count), NF), FewShape::POINTS, 0, s>>>(
        p, partial, out, out_stride);
    return check_launch();
}

int64_t few_scratch(const CellPlan& p, int nf) { return p.few.items * (nf < 4 ? nf : 4) * FewShape::POINTS * 8; }
int64_t many_scratch(const CellPlan& p) { return (p.m + p.many.items * ManyShape::POINTS) * MANY * 8; }

}  // namespace
}  // namespace cdftb

using namespace cdftb;

extern "C" int64_t cdftb_cell_plan_bytes(int64_t m, int nx, int ny, int nz, const int* cell_box) {
    CellPlan p;
    return plan_layout(m, nx, ny, nz, cell_box, nullptr, &p) ? p.bytes : 0;
}

extern "C" int cdftb_cell_plan_build(const int* base, const double* w1d, const int* order, const int64_t* keys,
                                     int64_t m, int nx, int ny, int nz, const int* cell_box, void* plan,
                                     int64_t plan_bytes, cdftb_stream_t stream) {
    CellPlan p;
    if (!base || !w1d || !order || !keys || !plan || reinterpret_cast<uintptr_t>(plan) % 16 != 0 ||
        !plan_layout(m, nx, ny, nz, cell_box, plan, &p) || plan_bytes < p.bytes)
        return CDFTB_ERR_ARGUMENT;
    const int64_t cells = int64_t(nx) * ny * nz;
    cudaStream_t s = as_stream(stream);
    int st = check(cudaMemsetAsync(p.bad, 0, 16, s));
    if (st != CDFTB_OK) return st;
    cell_starts_kernel<<<static_cast<unsigned>(ceil_div(cells + 1, 256)), 256, 0, s>>>(keys, m, cells, p.cell_ptr);
    if ((st = check_launch()) != CDFTB_OK) return st;
    sort_nodes_kernel<<<static_cast<unsigned>(ceil_div(m * kRow, 256)), 256, 0, s>>>(base, w1d, order, keys, p);
    if ((st = check_launch()) != CDFTB_OK) return st;
    if ((st = build_items<FewShape>(p, p.few, p.few_ptr, p.few_block, s)) != CDFTB_OK) return st;
    return build_items<ManyShape>(p, p.many, p.many_ptr, p.many_block, s);
}

extern "C" int64_t cdftb_lift_cells_scratch_bytes(int64_t m, int nx, int ny, int nz, const int* cell_box, int nf) {
    CellPlan p;
    if (nf < 1 || !plan_layout(m, nx, ny, nz, cell_box, nullptr, &p)) return 0;
    const int64_t few = few_scratch(p, nf);
    return nf < CDFTB_LIFT_CELLS_MANY || many_scratch(p) < few ? few : many_scratch(p);
}

extern "C" int cdftb_quadrature_lift_cells_f64(const void* plan, int64_t plan_bytes, int64_t m, int nx, int ny, int nz,
                                               const int* cell_box, const double* node_values, int nf,
                                               int64_t x_stride, double* out, int64_t out_stride, void* scratch,
                                               int64_t scratch_bytes, cdftb_stream_t stream) {
    CellPlan p;
    const int64_t n_points = int64_t(nx) * ny * nz;
    if (!plan || !node_values || !out || !scratch || nf < 1 || out_stride < n_points ||
        reinterpret_cast<uintptr_t>(plan) % 16 != 0 || reinterpret_cast<uintptr_t>(scratch) % 16 != 0 ||
        !plan_layout(m, nx, ny, nz, cell_box, const_cast<void*>(plan), &p) || plan_bytes < p.bytes ||
        scratch_bytes < cdftb_lift_cells_scratch_bytes(m, nx, ny, nz, cell_box, nf))
        return CDFTB_ERR_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    // points that no node reaches are zero
    int st = out_stride == n_points
                 ? check(cudaMemsetAsync(out, 0, size_t(nf) * n_points * 8, s))
                 : check(cudaMemset2DAsync(out, size_t(out_stride) * 8, 0, size_t(n_points) * 8, nf, s));
    if (st != CDFTB_OK) return st;
    int f0 = 0;
    if (nf >= CDFTB_LIFT_CELLS_MANY) {
        static OncePerDevice configured;
        st = configured.run([] {
            return check(cudaFuncSetAttribute(lift_cells_many_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              static_cast<int>(kManySmem)));
        });
        if (st != CDFTB_OK) return st;
        double* rows = static_cast<double*>(scratch);
        double* partial = rows + m * MANY;
        for (; nf - f0 >= CDFTB_LIFT_CELLS_MANY; f0 += MANY) {
            const int count = nf - f0 < MANY ? nf - f0 : MANY;
            sorted_rows_kernel<<<static_cast<unsigned>(ceil_div(m, MANY)), 256, 0, s>>>(
                p, node_values + f0 * x_stride, count, x_stride, rows);
            if ((st = check_launch()) != CDFTB_OK) return st;
            lift_cells_many_kernel<<<static_cast<unsigned>(p.many.items), ManyShape::WARPS * 32, kManySmem, s>>>(
                p, rows, partial);
            if ((st = check_launch()) != CDFTB_OK) return st;
            lift_cells_many_sum_kernel<<<static_cast<unsigned>(p.many.count), 256, 0, s>>>(
                p, partial, count, out + f0 * out_stride, out_stride);
            if ((st = check_launch()) != CDFTB_OK) return st;
        }
    }
    double* partial = static_cast<double*>(scratch);
    for (; f0 < nf; f0 += 4) {
        const double* x = node_values + f0 * x_stride;
        double* o = out + f0 * out_stride;
        switch (nf - f0) {
            case 1: st = lift_few<1>(p, x, x_stride, o, out_stride, partial, s); break;
            case 2: st = lift_few<2>(p, x, x_stride, o, out_stride, partial, s); break;
            case 3: st = lift_few<3>(p, x, x_stride, o, out_stride, partial, s); break;
            default: st = lift_few<4>(p, x, x_stride, o, out_stride, partial, s); break;
        }
        if (st != CDFTB_OK) return st;
    }
    return CDFTB_OK;
}
