// Four-wide copy of an axis-aligned-box hierarchy for the ray walkers.
//
// The binary escape tree stays the scene's hierarchy (export, importance,
// oracle parity); this is a second, derived layout of the same tree that
// leaves most inner levels out: a wide node holds the boxes of up to four
// descendants of a binary node, in preorder, as structure-of-arrays in one
// 128-B line:
//   {lo.x[4]} {hi.x[4]} {lo.y[4]} {hi.y[4]} {lo.z[4]} {hi.z[4]} {ref[4]} {unused}
// ref: a wide node index, or the binary tree's leaf word (LEAF_FLAG | count |
// block), or kWideEmpty. Boxes are the binary nodes' own floats. A node starts
// from its two children and replaces the inner one with the largest surface by
// its two children until it has four (taking every second level instead cost
// 4-8 %: path-traced room 9.30 / 8.90 ms, light tracing 5.37 / 4.96, any-hit
// terrain 0.84 / 0.80).
//
// Which walks may use it (wide_walks, trace.cuh) rests on the tree being what
// bvhmake and the LBVH builder write; gpugi_scene_upload accepts any forward
// escape graph, so it is checked here, edge by edge, on the device: nodes lie
// in preorder, every inner node has exactly two children (the next node and
// its escape, which shares the parent's escape and lies before it), and every
// child's box lies inside its parent's (and is not empty or NaN). A scene that
// fails any of it keeps the binary walkers.
//
// Level by level the choice of wide nodes is a chain of dependent launches or
// barriers (120-220 us for 34k nodes). Instead every inner node finds the
// children it would have as a wide node (k_wide_kids), and every node looks
// itself up from the root through those (preorder intervals tell which child
// contains it), which takes one fetch per wide level (k_wide_mark). Bound by
// launch latency for small trees; once per scene.
#include "ctx.cuh"

namespace gpugi {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;  // no child, no index
constexpr size_t kKeptScratch = 16u << 20;  // 838,000 nodes
constexpr uint32_t kMaxLevels = kWideStack / 3;  // a walk's stack holds at most three entries per wide level

// kids[i]: the children (binary node indexes, increasing, kNone behind the
// last) of node i as a wide node, none for a leaf; *ok becomes 0 where a check
// fails.
__global__ void k_wide_kids(const float4* __restrict__ nodes, uint32_t n, uint4* __restrict__ kids, uint32_t* ok) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    struct Node {
        float4 a, b;  // {lo, child}, {hi, escape}
        uint32_t at;
    };
    auto fetch = [&](uint32_t k) { return Node{__ldg(nodes + 2 * (size_t)k), __ldg(nodes + 2 * (size_t)k + 1), k}; };
    auto leaf = [](const Node& p) { return (__float_as_uint(p.a.w) & LEAF_FLAG) != 0; };
    auto children = [&](const Node& p, Node& l, Node& r) {
        const uint32_t c = __float_as_uint(p.a.w), e = __float_as_uint(p.b.w), end = e ? e : n;
        if (c != p.at + 1 || c >= n) return false;
        l = fetch(c);
        const uint32_t s = __float_as_uint(l.b.w);
        if (s <= c || s >= end) return false;
        r = fetch(s);
        auto inside = [&](const Node& q) {
            return p.a.x <= q.a.x && p.a.y <= q.a.y && p.a.z <= q.a.z && q.b.x <= p.b.x && q.b.y <= p.b.y &&
                   q.b.z <= p.b.z && q.a.x <= q.b.x && q.a.y <= q.b.y && q.a.z <= q.b.z;
        };
        return __float_as_uint(r.b.w) == e && inside(l) && inside(r);
    };
    auto surface = [&](const Node& p) {  // of an inner node; below any for a leaf
        if (leaf(p)) return -1.0f;
        const float x = p.b.x - p.a.x, y = p.b.y - p.a.y, z = p.b.z - p.a.z;
        return fmaxf(x * y + y * z + z * x, 0.0f);
    };
    const Node self = fetch(i);
    uint32_t k0 = kNone, k1 = kNone, k2 = kNone, k3 = kNone;
    bool good = true;
    if (leaf(self)) {
        good = i != 0;  // a leaf root has no wide hierarchy
    } else {
        Node l, r;
        good = children(self, l, r) && (i != 0 || __float_as_uint(self.b.w) == 0u);
        k0 = l.at;
        k1 = r.at;
        const float sl = surface(l), sr = surface(r);
        if (good && fmaxf(sl, sr) >= 0.0f) {  // the larger one becomes its children x, y
            const bool first = sl >= sr;
            Node x, y;
            good = children(first ? l : r, x, y);
            const Node other = first ? r : l;
            if (good) {
                const float so = surface(other), sx = surface(x), sy = surface(y), most = fmaxf(so, fmaxf(sx, sy));
                const uint32_t a0 = first ? x.at : other.at, a1 = first ? y.at : x.at, a2 = first ? other.at : y.at;
                k0 = a0;
                k1 = a1;
                k2 = a2;
                if (most >= 0.0f) {
                    const Node from = so == most ? other : sx == most ? x : y;
                    Node p, q;
                    good = children(from, p, q);
                    if (good) {
                        if (from.at == a0) k0 = p.at, k1 = q.at, k2 = a1, k3 = a2;
                        else if (from.at == a1) k1 = p.at, k2 = q.at, k3 = a2;
                        else k2 = p.at, k3 = q.at;
                    }
                }
            }
        }
    }
    if (!good) *ok = 0u;
    kids[i] = make_uint4(k0, k1, k2, k3);
}

// index[i] = number of the wide node of binary node i if the wide tree has
// one (blocks of nodes take consecutive ranges in the order they finish, the
// root's block the first one, so that the root is 0), else kNone; *minNotLevel
// = ~(deepest wide level).
__global__ void k_wide_mark(const uint4* __restrict__ kids, uint32_t n, uint32_t* __restrict__ index,
                            uint32_t* minNotLevel, uint32_t* count) {
    __shared__ uint32_t s_warp[8], s_base;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t depth = 0;
    bool mark = false;
    if (i < n && __ldg(&kids[i].x) != kNone) {
        // from the root down to the child that contains i, until that is i itself; a node that was
        // replaced by its children ends in a leaf or before every child
        uint32_t v = 0;
        while (v != i && depth <= kMaxLevels) {
            const uint4 k = __ldg(kids + v);
            const uint32_t c = k.w <= i ? k.w : k.z <= i ? k.z : k.y <= i ? k.y : k.x;
            if (c > i || c <= v) break;
            v = c;
            ++depth;
        }
        mark = v == i;
        if (!mark && depth <= kMaxLevels) depth = 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, mark), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) s_warp[warp] = __popc(m);
    depth = __reduce_max_sync(0xffffffffu, depth);
    if (lane == 0 && depth) atomicMin(minNotLevel, ~depth);
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
    if (i < n) index[i] = mark ? s_base + s_warp[warp] + __popc(m & ((1u << lane) - 1u)) : kNone;
}

__global__ void k_wide_fill(const float4* __restrict__ nodes, uint32_t n, const uint4* __restrict__ kids,
                            const uint32_t* __restrict__ index, uint32_t capacity, float4* __restrict__ wide,
                            uint32_t* ok) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || index[i] >= capacity || *ok == 0u) return;
    const uint4 four = __ldg(kids + i);
    const uint32_t kid[4] = {four.x, four.y, four.z, four.w};
    float* w = reinterpret_cast<float*>(wide + 8 * (size_t)index[i]);
    for (uint32_t k = 0; k < 4; ++k) {
        uint32_t ref = kWideEmpty;
        float4 a = make_float4(0, 0, 0, 0), b = a;
        if (kid[k] < n) {
            a = __ldg(nodes + 2 * (size_t)kid[k]);
            b = __ldg(nodes + 2 * (size_t)kid[k] + 1);
            ref = __float_as_uint(a.w);
            if (!(ref & LEAF_FLAG)) {
                ref = index[kid[k]];
                if (ref >= capacity) *ok = 0u;
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
    sc->numWide = sc->dev.numWide = 0;
    const uint32_t n = sc->dev.numNodes;
    if (sc->dev.boundsKind != GPUGI_BOUNDS_AABB || sc->dev.topNodes || n < 3) return GPUGI_OK;
    cudaStream_t st = ctx->stream;
    // Scratch: {checks passed, ~deepest level, ~nodes behind block 0's}, children, index. Up to
    // kKeptScratch it is the context's staging buffer, which is kept between calls (every user of it
    // finishes before it returns) and which host-array queries make as large; above, it goes again with
    // this call. No memory for it or for the copy: the binary walkers need none.
    const size_t scratchBytes = 256 + 20 * (size_t)n;
    void *own = nullptr, *wide = nullptr;
    if (scratchBytes <= kKeptScratch) {
        if (gpugi_status gs = ensure_stage(ctx, scratchBytes)) {
            cudaGetLastError();
            return gs == GPUGI_ERROR_OUT_OF_MEMORY ? GPUGI_OK : gs;
        }
    } else if (cudaMalloc(&own, scratchBytes) != cudaSuccess) {
        cudaGetLastError();
        return GPUGI_OK;
    }
    char* scratch = static_cast<char*>(own ? own : ctx->stageDev);
    uint32_t* word = reinterpret_cast<uint32_t*>(scratch);
    uint4* kids = reinterpret_cast<uint4*>(scratch + 256);
    uint32_t* index = reinterpret_cast<uint32_t*>(kids + n);
    auto leave = [&](gpugi_status gs) {  // what the scene does not keep (its stream has been waited for, or failed)
        if (own) cudaFree(own);
        if (wide && !sc->dev.wide) cudaFree(wide);
        return gs;
    };
    auto check = [&](cudaError_t e) { return e == cudaSuccess ? GPUGI_OK : cuda_fail(ctx, e, "wide hierarchy"); };
    const unsigned grid = (n + 255) / 256;
    gpugi_status gs = check(cudaMemsetAsync(word, 0xFF, 12, st));
    if (gs) return leave(gs);
    k_wide_kids<<<grid, 256, 0, st>>>(sc->dev.nodes, n, kids, word);
    k_wide_mark<<<grid, 256, 0, st>>>(kids, n, index, word + 1, word + 2);
    uint32_t got[3];
    auto read = [&]() {
        if (gpugi_status e = check(cudaMemcpyAsync(got, word, 12, cudaMemcpyDeviceToHost, st))) return e;
        return check(cudaStreamSynchronize(st));
    };
    // At most every inner node is a wide one: small trees allocate for that (64 B a node, 4 MiB), so that
    // the host waits once; large ones read the count first.
    uint32_t count = 256 + (n - 1) / 2;
    if (n > (1u << 16)) {
        if ((gs = read())) return leave(gs);
        if (got[0] == 0 || ~got[2] > (n - 1) / 2) return leave(GPUGI_OK);
        count = 256 + ~got[2];
    }
    if (cudaMalloc(&wide, 128 * (size_t)count) != cudaSuccess) {
        cudaGetLastError();
        wide = nullptr;
        cudaStreamSynchronize(st);
        return leave(GPUGI_OK);
    }
    k_wide_fill<<<grid, 256, 0, st>>>(sc->dev.nodes, n, kids, index, count, static_cast<float4*>(wide), word);
    if ((gs = check(cudaGetLastError())) || (gs = read())) return leave(gs);
    // a walk's stack holds at most three entries per wide level, and its node offsets are 32-bit bytes
    const uint32_t numbers = 256 + ~got[2];  // the root's block leaves some of its numbers unused
    const bool fits = ~got[1] + 1 <= kMaxLevels && numbers < (1u << 25);
    if (got[0] == 0 || !fits || numbers > count) return leave(GPUGI_OK);
    sc->allocations.push_back(wide);
    sc->dev.wide = static_cast<const float4*>(wide);
    sc->numWide = sc->dev.numWide = numbers;
    return leave(GPUGI_OK);
}

}  // namespace gpugi
