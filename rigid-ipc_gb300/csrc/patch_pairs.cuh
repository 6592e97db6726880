// Element pairs by patches (part of broad_phase.cu).
//
// The elements of a body move together, so which of them are neighbours is
// known from the rest shape: at set-up each body's vertices, edges and faces
// are ordered along a Morton curve of their rest centroids and cut into patches
// of 32.  A call boxes the patches, pairs the bodies whose element boxes
// overlap, their patches, then the elements of those, a warp per pair of
// patches.  Nothing is sorted and nothing is sized on the host before the
// pairs are known.
//
// The grid (statistics, cell filter, items, their radix sort, the cells' pairs: 22
// launches and a read-back) is bound by its items, some of every element near
// another body, in memory's order of cells: 1000 icospheres, a discrete and a
// continuous call, 2.5 ms of kernels, here 0.7 ms, half of them the element
// tests (single-precision issue: 32 x 32 per pair of patches), the rest the
// boxes (gathers of the vertices' boxes) and the patch tests.

constexpr int kPatch = 32;
constexpr int kPatchTests = 2048;  // patch tests of a work item (a block of 128: 16 each)

constexpr int kPatchBlocks = 152 * 16;            // blocks over the lists, whose lengths are on the device
constexpr int kPatchPairsPerPatch = 32;           // overlapping patches a patch may have on average
constexpr int64_t kMaxBodyTests = int64_t(1) << 31;  // pairs of bodies up to which all are tested

struct Patch {
    int first;  // position of its first element in the order
    int count, body, type;
};

// The order's sort keys: type and body (so that the elements of a body's type
// keep their range), then the Morton code of the rest centroid in the cube of
// the body's radius
__global__ void k_patch_keys(const double* __restrict__ rest, const int* __restrict__ Ed,
                             const int* __restrict__ Fa, const int* __restrict__ vbody,
                             const int* __restrict__ ebody, const int* __restrict__ fbody,
                             const double* __restrict__ rmax, int nv, int ne, int nf, int nb,
                             uint64_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)nv + ne + nf) return;
    const int t = e < nv ? 0 : (e < (int64_t)nv + ne ? 1 : 2);
    const int i = (int)(t == 0 ? e : (t == 1 ? e - nv : e - nv - ne));
    int v[3] = { i, i, i };
    for (int k = 0; k < 2 && t == 1; k++) v[k] = Ed[2 * i + k];
    for (int k = 0; k < 3 && t == 2; k++) v[k] = Fa[3 * i + k];
    const int b = (t == 0 ? vbody : (t == 1 ? ebody : fbody))[i];
    const float scale = 1024.0f / (2 * (t + 1) * (float)rmax[b]);
    uint64_t code = 0;
    for (int j = 0; j < 3; j++) {
        float s = (t + 1) * (float)rmax[b];
        for (int k = 0; k <= t; k++) s += (float)rest[3 * (size_t)v[k] + j];
        const int q = (int)fminf(fmaxf(s * scale, 0.0f), 1023.0f);
        for (int k = 0; k < 10; k++) code |= (uint64_t)((q >> k) & 1) << (3 * k + j);
    }
    keys[e] = ((uint64_t)t * nb + b) << 30 | code;
    vals[e] = (uint32_t)i;
}

// a float as an integer of the same order
__device__ __forceinline__ int ordered_int(float x)
{
    const int b = __float_as_int(x);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float ordered_float(int b)
{
    return __int_as_float(b ^ ((b >> 31) & 0x7fffffff));
}

// the double box of an element, from its vertices (as k_edge_face_boxes)
__device__ __forceinline__ void element_box(const Elems& E, const int* __restrict__ Ed,
                                            const int* __restrict__ Fa, int t, int i, double* box)
{
    const int a = t == 0 ? i : (t == 1 ? Ed[2 * i] : Fa[3 * i]);
    for (int j = 0; j < 6; j++) box[j] = E.vb[6 * (size_t)a + j];
    for (int k = 1; k <= t; k++) {
        const int v = t == 1 ? Ed[2 * i + k] : Fa[3 * i + k];
        for (int j = 0; j < 3; j++) {
            box[j] = smin(box[j], E.vb[6 * (size_t)v + j]);
            box[3 + j] = smax(box[3 + j], E.vb[6 * (size_t)v + 3 + j]);
        }
    }
}

// A warp per patch: its elements' float boxes (rounded outward; empty where
// there is no element or it is not included) by components, its own box, and
// the body's (bounds: ordered ints of lo and -hi, all minima)
__global__ void __launch_bounds__(128) k_patch_boxes(
    const Patch* __restrict__ patches, int np, const uint32_t* __restrict__ order,
    const int* __restrict__ Ed, const int* __restrict__ Fa, Elems E, const int* __restrict__ body_in,
    float* __restrict__ ebox, float* __restrict__ pbox, int* __restrict__ bounds)
{
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (p >= np) return;
    const Patch q = patches[p];
    if (!body_in[q.body]) return;  // in no pair of bodies
    float b[6] = { INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY };  // lo, -hi
    if (lane < q.count) {
        const int i = (int)order[q.first + lane];
        bool in = E.vin[q.type == 0 ? i : (q.type == 1 ? Ed[2 * i] : Fa[3 * i])];
        for (int k = 1; k <= q.type; k++) in = in && E.vin[q.type == 1 ? Ed[2 * i + k] : Fa[3 * i + k]];
        if (in) {
            double box[6];
            element_box(E, Ed, Fa, q.type, i, box);
            for (int j = 0; j < 3; j++) {
                b[j] = __double2float_rd(box[j]);
                b[3 + j] = -__double2float_ru(box[3 + j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 6; j++) {
        ebox[((size_t)p * 6 + j) * kPatch + lane] = b[j];
        for (int o = 16; o > 0; o >>= 1) b[j] = fminf(b[j], __shfl_xor_sync(0xffffffffu, b[j], o));
    }
    float x = b[0];
#pragma unroll
    for (int j = 1; j < 6; j++)
        if (lane == j) x = b[j];
    if (lane < 6) {
        pbox[(size_t)p * 6 + lane] = x;
        atomicMin(bounds + (size_t)q.body * 6 + lane, ordered_int(x));
    }
}

// boxes as lo, -hi: apart on an axis where one's lo is above the other's hi
__device__ __forceinline__ bool neg_disjoint(const float* a, const float* b)
{
#pragma unroll
    for (int j = 0; j < 3; j++)
        if (a[j] > -b[3 + j] || b[j] > -a[3 + j]) return true;
    return false;
}

// patches of a body's type: [start[t * (nb + 1) + b], ... + 1)
struct PatchRange {
    int first[3], n[3];
};
__device__ __forceinline__ PatchRange patch_range(const int* __restrict__ start, int nb, int b)
{
    PatchRange r;
    for (int t = 0; t < 3; t++) {
        r.first[t] = start[t * (nb + 1) + b];
        r.n[t] = start[t * (nb + 1) + b + 1] - r.first[t];
    }
    return r;
}

struct PatchLists {
    int4* items;  // (body, body, part, tests of the pair of bodies)
    int2* pairs;  // overlapping patches
    unsigned long long cap_items, cap_pairs;
    unsigned long long* n_items;
    unsigned long long* n_pairs;
};

// A warp per body: the later bodies of its scene, of another group, whose
// bounds overlap; a pair's patch tests are cut into items of kPatchTests.
__global__ void __launch_bounds__(128) k_body_pairs(const int* __restrict__ bounds,
                                                    const int* __restrict__ body_in,
                                                    const int* __restrict__ grank,
                                                    const int* __restrict__ bscene,
                                                    const int* __restrict__ scene_bstart, int nb,
                                                    const int* __restrict__ start, int kind, PatchLists o)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= nb || !body_in[i]) return;
    float a[6];
    for (int j = 0; j < 6; j++) a[j] = ordered_float(bounds[6 * (size_t)i + j]);
    const PatchRange ra = patch_range(start, nb, i);
    const int end = scene_bstart[bscene[i] + 1];
    for (int j = i + 1 + lane; j < end; j += 32) {
        if (!body_in[j] || grank[j] == grank[i]) continue;
        float b[6];
        for (int k = 0; k < 6; k++) b[k] = ordered_float(bounds[6 * (size_t)j + k]);
        if (neg_disjoint(a, b)) continue;
        const PatchRange rb = patch_range(start, nb, j);
        long long tests = (long long)ra.n[2] * rb.n[kind == kPairsEF ? 1 : 0]
            + (long long)ra.n[kind == kPairsEF ? 1 : 0] * rb.n[2];
        if (kind != kPairsEF) tests += (long long)ra.n[1] * rb.n[1];
        if (tests == 0) continue;
        unsigned long long parts = (unsigned long long)(tests + kPatchTests - 1) / kPatchTests;
        if (tests > INT32_MAX - 2 * kPatchTests) parts = o.cap_items + 1;
        // more than the list takes: the count says so, nothing is written
        unsigned long long at = atomicAdd(o.n_items, parts);
        if (at + parts > o.cap_items) continue;
        for (unsigned long long k = 0; k < parts; k++) o.items[at + k] = make_int4(i, j, (int)k, (int)tests);
    }
}

__global__ void __launch_bounds__(128) k_patch_pairs(const int* __restrict__ start, int nb, int kind,
                                                     const float* __restrict__ pbox, PatchLists o)
{
    const unsigned long long n = *o.n_items;
    if (n > o.cap_items) return;
    const int lane = threadIdx.x & 31;
    for (unsigned long long k = blockIdx.x; k < n; k += gridDim.x) {
        const int4 it = o.items[k];
        const PatchRange ra = patch_range(start, nb, it.x), rb = patch_range(start, nb, it.y);
        // the pair's tests: edges by edges, faces by vertices (or edges), and
        // vertices (or edges) by faces
        const int other = kind == kPairsEF ? 1 : 0;
        const int n0 = kind == kPairsEF ? 0 : ra.n[1] * rb.n[1], n1 = ra.n[2] * rb.n[other];
        for (int s = 0; s < kPatchTests; s += 128) {
            const int t = it.z * kPatchTests + s + (int)threadIdx.x;
            if (t - (int)threadIdx.x >= it.w) break;
            bool hit = false;
            int pa = 0, pb = 0;
            if (t < it.w) {
                const int ta = t < n0 ? 1 : (t < n0 + n1 ? 2 : other), tb = t < n0 ? 1 : (t < n0 + n1 ? other : 2);
                const int u = t < n0 ? t : (t < n0 + n1 ? t - n0 : t - n0 - n1);
                pa = ra.first[ta] + u / rb.n[tb];
                pb = rb.first[tb] + u % rb.n[tb];
                hit = !neg_disjoint(pbox + 6 * (size_t)pa, pbox + 6 * (size_t)pb);
            }
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (!m) continue;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(o.n_pairs, (unsigned long long)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (hit && at < o.cap_pairs) o.pairs[at] = make_int2(pa, pb);
        }
    }
}

// Intervals rounded outward to floats that overlap by more than 2^-20 of their
// ends' magnitudes: the rounding of the ends (2^-23) and of the exact test's
// doubles cannot have made that, the exact test accepts the axis too.
__device__ __forceinline__ bool surely_overlap(float al, float ah, float bl, float bh)
{
    const float size = (fabsf(al) + fabsf(ah)) + (fabsf(bl) + fabsf(bh));
    return fminf(ah, bh) - fmaxf(al, bl) > 9.5367431640625e-07f * size && size < 1e30f && size > 1e-30f;
}

// A warp per pair of patches: an element of the first per lane, all of the
// second from shared memory; the float tests as a mask, then the exact ones
__global__ void __launch_bounds__(128) k_patch_elements(
    const Patch* __restrict__ patches, const uint32_t* __restrict__ order, const int* __restrict__ Ed,
    const int* __restrict__ Fa, Elems E, const float* __restrict__ ebox, PatchLists l, PairOut o)
{
    __shared__ float4 sh[4][kPatch][2];
    const unsigned long long n = *l.n_pairs;
    if (n > l.cap_pairs || *l.n_items > l.cap_items) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (unsigned long long k = blockIdx.x * 4ull + w; k < n; k += gridDim.x * 4ull) {
        const int2 pr = l.pairs[k];
        const Patch pa = patches[pr.x], pb = patches[pr.y];
        float a[6], b[6];
        for (int j = 0; j < 6; j++) {
            a[j] = ebox[((size_t)pr.x * 6 + j) * kPatch + lane];
            b[j] = ebox[((size_t)pr.y * 6 + j) * kPatch + lane];
        }
        __syncwarp();
        sh[w][lane][0] = make_float4(b[0], b[1], b[2], -b[3]);
        sh[w][lane][1] = make_float4(-b[4], -b[5], 0, 0);
        __syncwarp();
        const float h0 = -a[3], h1 = -a[4], h2 = -a[5];
        unsigned m = 0;
#pragma unroll 8
        for (int j = 0; j < kPatch; j++) {
            const float4 x = sh[w][j][0];
            const float2 y = *reinterpret_cast<const float2*>(&sh[w][j][1]);
            const bool apart = a[0] > x.w || a[1] > y.x || a[2] > y.y || x.x > h0 || x.y > h1 || x.z > h2;
            if (!apart) m |= 1u << j;
        }
        if (lane >= pa.count || a[0] == INFINITY) m = 0;
        if (pb.count < kPatch) m &= (1u << pb.count) - 1u;
        // hits that the floats do not prove: the exact test
        const int ia = m ? (int)order[pa.first + lane] : 0;
        for (unsigned r = m; r; r &= r - 1) {
            const int j = __ffs(r) - 1;
            const float4 x = sh[w][j][0];
            const float2 y = *reinterpret_cast<const float2*>(&sh[w][j][1]);
            const bool sure = surely_overlap(a[0], h0, x.x, x.w) && surely_overlap(a[1], h1, x.y, y.x)
                && surely_overlap(a[2], h2, x.z, y.y);
            if (sure) continue;
            double xa[6], xb[6];
            element_box(E, Ed, Fa, pa.type, ia, xa);
            element_box(E, Ed, Fa, pb.type, (int)order[pb.first + j], xb);
            if (!boxes_overlap(xa, xb)) m &= ~(1u << j);
        }
        // the pair's hits in one range of the output
        const int c = __popc(m);
        int incl = c;
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        if (total == 0) continue;
        const bool ee = pa.type == 1 && pb.type == 1;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(ee ? o.n_ee : o.n_fv, (unsigned long long)total);
        at = __shfl_sync(0xffffffffu, at, 0) + (incl - c);
        for (; m; m &= m - 1, at++) {
            const unsigned long long key = element_pair_key(E, pa.type, ia, pb.type, (int)order[pb.first + __ffs(m) - 1]);
            if (at < (ee ? o.cap_ee : o.cap_fv)) (ee ? o.ee : o.fv)[at] = key;
        }
    }
}
