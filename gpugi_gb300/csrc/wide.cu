// Four-wide copy of an axis-aligned-box hierarchy for the ray walkers.
//
// The binary escape tree stays the scene's hierarchy (export, importance,
// oracle parity); this is a second, derived layout of the same tree in which
// every second level is left out: a wide node holds the boxes of the (two to
// four) grandchildren, or children that are leaves, of a binary node at even
// depth, in preorder, as structure-of-arrays in one 128-B line:
//   {lo.x[4]} {hi.x[4]} {lo.y[4]} {hi.y[4]} {lo.z[4]} {hi.z[4]} {ref[4]} {unused}
// ref: a wide node index, or the binary tree's leaf word (LEAF_FLAG | count |
// block), or kWideEmpty. Boxes are the binary nodes' own floats.
//
// Which walks may use it (wide_walks, trace.cuh) rests on the tree being what
// bvhmake and the LBVH builder write; gpugi_scene_upload accepts any forward
// escape graph, so it is checked here, edge by edge, on the device: every
// inner node has exactly two children, the right one is the left one's escape
// and shares its parent's escape, no node has two parents, and every child's
// box lies inside its parent's (and is not empty or NaN). A scene that fails
// any of it keeps the binary walkers.
//
// Bound by launch latency for small trees (5 us a kernel at 34k nodes; nodes
// are numbered with one atomic per block instead of a scan) and by the parent
// climb of k_wide_mark for large ones; once per scene.
#include "ctx.cuh"

namespace gpugi {
namespace {

constexpr uint32_t kNoParent = 0xFFFFFFFFu, kNoIndex = 0xFFFFFFFFu;

GPUGI_D uint32_t child_word(const float4* nodes, uint32_t i) { return __float_as_uint(__ldg(nodes + 2 * (size_t)i).w); }
GPUGI_D uint32_t escape_word(const float4* nodes, uint32_t i) {
    return __float_as_uint(__ldg(nodes + 2 * (size_t)i + 1).w);
}

// parent[] of every child (kNoParent before), and the structure checks (*bad
// becomes 0 where one fails).
__global__ void k_wide_parents(const float4* __restrict__ nodes, uint32_t n, uint32_t* parent, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = child_word(nodes, i);
    if (c & LEAF_FLAG) {
        if (i == 0) *bad = 0u;  // a leaf root with nodes behind it
        return;
    }
    const uint32_t r = c < n ? escape_word(nodes, c) : 0u;
    bool ok = c > i && c < n && r > c && r < n && escape_word(nodes, r) == escape_word(nodes, i);
    if (ok) ok = atomicExch(parent + c, i) == kNoParent && atomicExch(parent + r, i) == kNoParent;
    if (!ok || (i == 0 && escape_word(nodes, 0) != 0u)) *bad = 0u;
}

// index[i] = number of the wide node of inner node i at even depth below the
// root (blocks of nodes take consecutive ranges in the order they finish, the
// root's block the first one, so that the root is 0), kNoIndex for the other
// nodes; *minNotDepth = ~(depth of the deepest inner node). Parents have
// smaller indexes than their children, so the climb ends.
__global__ void k_wide_mark(const float4* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ parent,
                            uint32_t* __restrict__ index, uint32_t* minNotDepth, uint32_t* count) {
    __shared__ uint32_t s_warp[8], s_base;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t depth = 0;
    bool mark = false;
    if (i < n && !(child_word(nodes, i) & LEAF_FLAG)) {
        uint32_t v = i;
        while (v != 0 && parent[v] < v) {
            v = parent[v];
            ++depth;
        }
        mark = v == 0 && (depth & 1u) == 0;
        if (v != 0) depth = 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, mark), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) s_warp[warp] = __popc(m);
    depth = __reduce_max_sync(0xffffffffu, depth);
    if (lane == 0 && depth) atomicMin(minNotDepth, ~depth);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = s_warp[w];
            s_warp[w] = sum;
            sum += c;
        }
        // *count starts at ~0: ~*count numbers are taken. Block 0 owns the numbers from 0 on, as many as
        // a block can need; the others start behind them.
        s_base = blockIdx.x == 0 ? 0u : 256u + ~atomicSub(count, sum);
    }
    __syncthreads();
    if (i < n) index[i] = mark ? s_base + s_warp[warp] + __popc(m & ((1u << lane) - 1u)) : kNoIndex;
}

__global__ void k_wide_fill(const float4* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ index,
                            uint32_t capacity, float4* __restrict__ wide,
                            uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || index[i] >= capacity) return;
    uint32_t kid[4], count = 0;
    bool ok = true;
    auto inside = [&](uint32_t outer, uint32_t inner) {
        const float4 a = __ldg(nodes + 2 * (size_t)outer), b = __ldg(nodes + 2 * (size_t)outer + 1);
        const float4 c = __ldg(nodes + 2 * (size_t)inner), d = __ldg(nodes + 2 * (size_t)inner + 1);
        return a.x <= c.x && a.y <= c.y && a.z <= c.z && d.x <= b.x && d.y <= b.y && d.z <= b.z && c.x <= d.x &&
               c.y <= d.y && c.z <= d.z;
    };
    auto kids = [&](uint32_t p, uint32_t& l, uint32_t& r) {
        l = child_word(nodes, p);
        r = l < n ? escape_word(nodes, l) : n;
        if (l >= n || r >= n) return false;
        return inside(p, l) && inside(p, r);
    };
    uint32_t c[2];
    ok = kids(i, c[0], c[1]);
    for (int s = 0; s < 2 && ok; ++s) {
        if (child_word(nodes, c[s]) & LEAF_FLAG) {
            kid[count++] = c[s];
        } else {
            ok = kids(c[s], kid[count], kid[count + 1]);
            count += 2;
        }
    }
    if (!ok) {
        *bad = 0u;
        return;
    }
    float* w = reinterpret_cast<float*>(wide + 8 * (size_t)index[i]);
    for (uint32_t k = 0; k < 4; ++k) {
        uint32_t ref = kWideEmpty;
        float4 a = make_float4(0, 0, 0, 0), b = a;
        if (k < count) {
            a = __ldg(nodes + 2 * (size_t)kid[k]);
            b = __ldg(nodes + 2 * (size_t)kid[k] + 1);
            ref = __float_as_uint(a.w);
            if (!(ref & LEAF_FLAG)) {
                ref = index[kid[k]];
                if (ref >= capacity) *bad = 0u;
            }
        }
        w[k] = a.x, w[4 + k] = b.x;
        w[8 + k] = a.y, w[12 + k] = b.y;
        w[16 + k] = a.z, w[20 + k] = b.z;
        w[24 + k] = __uint_as_float(ref);
        w[28 + k] = 0.0f;
    }
}

}  // namespace

gpugi_status build_wide(gpugi_ctx* ctx, gpugi_scene* sc) {
    sc->dev.wide = nullptr;
    sc->dev.numWide = 0;
    const uint32_t n = sc->dev.numNodes;
    if (sc->dev.boundsKind != GPUGI_BOUNDS_AABB || sc->dev.topNodes || n < 3) return GPUGI_OK;
    cudaStream_t st = ctx->stream;
    // scratch in the context's staging buffer (kept between calls; every user of it finishes before it
    // returns): parent and {checks passed, ~depth, ~nodes behind block 0's}, index
    const size_t col = (4 * (size_t)n + 16 + 255) & ~size_t(255);
    if (gpugi_status gs = ensure_stage(ctx, 2 * col)) {
        cudaGetLastError();
        return gs == GPUGI_ERROR_OUT_OF_MEMORY ? GPUGI_OK : gs;  // the binary walkers need no extra memory
    }
    uint32_t* parent = static_cast<uint32_t*>(ctx->stageDev);
    uint32_t* word = parent + n;
    uint32_t* index = reinterpret_cast<uint32_t*>(static_cast<char*>(ctx->stageDev) + col);
    const unsigned grid = (n + 255) / 256;
    GPUGI_CUDA_TRY(ctx, cudaMemsetAsync(parent, 0xFF, 4 * ((size_t)n + 3), st));
    k_wide_parents<<<grid, 256, 0, st>>>(sc->dev.nodes, n, parent, word);
    k_wide_mark<<<grid, 256, 0, st>>>(sc->dev.nodes, n, parent, index, word + 1, word + 2);
    // At most every inner node is a wide one: small trees allocate for that (64 B a node), so that the
    // host waits once; large ones read the count first.
    uint32_t got[3], count = 256 + (n - 1) / 2;
    if (n > (1u << 20)) {
        GPUGI_CUDA_TRY(ctx, cudaMemcpyAsync(got, word, 12, cudaMemcpyDeviceToHost, st));
        GPUGI_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        if (~got[2] > (n - 1) / 2) return GPUGI_OK;
        count = 256 + ~got[2];
    }
    float4* wide = nullptr;
    if (cudaMalloc(&wide, 128 * (size_t)count) != cudaSuccess) {
        cudaGetLastError();
        return GPUGI_OK;
    }
    sc->allocations.push_back(wide);
    k_wide_fill<<<grid, 256, 0, st>>>(sc->dev.nodes, n, index, count, wide, word);
    GPUGI_CUDA_TRY(ctx, cudaGetLastError());
    GPUGI_CUDA_TRY(ctx, cudaMemcpyAsync(got, word, 12, cudaMemcpyDeviceToHost, st));
    GPUGI_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    // a walk's stack holds at most three entries per wide level, and its node offsets are 32-bit bytes
    const uint32_t numbers = 256 + ~got[2];  // the root's block leaves some of its numbers unused
    const bool fits = 3 * (~got[1] / 2 + 1) <= kWideStack && numbers < (1u << 25);
    if (got[0] == 0 || !fits || numbers > count) return GPUGI_OK;
    sc->wide = sc->dev.wide = wide;
    sc->dev.numWide = numbers;
    return GPUGI_OK;
}

}  // namespace gpugi
