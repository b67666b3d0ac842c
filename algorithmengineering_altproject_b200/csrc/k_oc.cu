// Optimality-criteria update (driver.cpp:160-189): dc scaling, the lambda bisection with its volume
// sum, change and sharpness.  Two summation orders are provided:
//   fp64_sum = 1  canonical deterministic FP64 sums over cells (the throughput path);
//   fp64_sum = 0  the float summation order of the reference build's vectorised std::accumulate over
//                 the Morton-ordered element vector (8 lane sums, folded, remainder), which keeps the
//                 bisection bit-identical to the reference; evaluated in parallel (k_oc_vec8).
// A pass does not store the candidate densities: k_oc_finish evaluates the last pass's multiplier again.
#include "kernels.hpp"
#include "red.cuh"

namespace t3d {

namespace {

// dc = dcf / max(1e-3, x) (driver.cpp:166)
__global__ void k_dc_scale(Grid g, const uint8_t* __restrict__ solid, const float* __restrict__ dcf,
                           const float* __restrict__ x, float* __restrict__ dc) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.NE || !solid[i]) return;
    const float xv = x[i];
    dc[i] = dcf[i] / (1.0e-3f < xv ? xv : 1.0e-3f);
}

__global__ void k_oc_init(OcState* st) {
    st->l1 = 0.0f;
    st->l2 = 1e9f;
    st->lmid = 0.0f;
    st->vol = 0.0f;
    st->passes = 0;
    st->done = 0;
}

// xnew = max(1e-3, clamp(clamp(x*sqrt(max(1e-30,-dc*(2/(l1+l2)))), x-0.2, x+0.2), 0, 1))
// (driver.cpp:174-180; -dc/lmid is evaluated as -dc*(2/(l1+l2)) as in the reference build)
__device__ __forceinline__ float oc_candidate(float xv, float d, float rl) {
    float q = -(d * rl);
    if (q < 1e-30f) q = 1e-30f;
    const float val = sqrtf(q);
    const float lo = xv - 0.2f, hi = xv + 0.2f;
    float xe = xv * val;
    xe = xe < lo ? lo : (hi < xe ? hi : xe);
    xe = xe < 0.0f ? 0.0f : (1.0f < xe ? 1.0f : xe);
    return 1.0e-3f < xe ? xe : 1.0e-3f;
}

__device__ __forceinline__ bool oc_continue(const OcState* st) {
    const float l1 = st->l1, l2 = st->l2;
    return (double)((l2 - l1) / (l1 + l2)) > 1e-6;
}

// the bisection step after a pass at l1, l2 gave `vol` (driver.cpp:181-183); rl: the pass's multiplier
__device__ __forceinline__ void oc_step(OcState* st, float l1, float l2, float vol, float V0) {
    const float lmid = 0.5f * (l1 + l2);
    st->vol = vol;
    st->lmid = lmid;
    st->rl = 2.0f / (l1 + l2);
    if (vol - V0 > 0) st->l1 = lmid;
    else st->l2 = lmid;
    st->passes = st->passes + 1;
}

// Cell coordinates of a grid-stride walk over the cells: one division at the start, then additions with carry.
struct CellWalk {
    int cx, cy, cz, dx, dy, dz;
    __device__ CellWalk(const Grid& g, int k, int stride)
        : cx(k % g.nx), cy((k / g.nx) % g.ny), cz(k / (g.nx * g.ny)), dx(stride % g.nx), dy((stride / g.nx) % g.ny),
          dz(stride / (g.nx * g.ny)) {}
    __device__ void next(const Grid& g) {
        cx += dx;
        const int kx = cx >= g.nx ? 1 : 0;
        cx -= kx ? g.nx : 0;
        cy += dy + kx;
        const int ky = cy >= g.ny ? 1 : 0;
        cy -= ky ? g.ny : 0;
        cz += dz + ky;
    }
};

// One bisection pass with the canonical FP64 volume sum.
__global__ void __launch_bounds__(RED_THREADS) k_oc_pass(Grid g, const uint8_t* __restrict__ solid,
                                                         const float* __restrict__ x, const float* __restrict__ dc,
                                                         OcState* st, float V0, int64_t ne, RedSlot red) {
    __shared__ double sh[32];
    if (st->done) return;
    if (!oc_continue(st)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
        return;
    }
    const float l1 = st->l1, l2 = st->l2;
    const float rl = 2.0f / (l1 + l2);
    const int ncell = g.nx * g.ny * g.nz, stride = gridDim.x * blockDim.x;
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    CellWalk w(g, k, stride);
    double part = 0.0;
    for (; k < ncell; k += stride, w.next(g)) {
        const int64_t ci = g.cell(w.cx, w.cy, w.cz);
        const uint8_t sc = solid[ci];
        if (!sc) continue;
        // passive solid elements of an external model (solid = 2) stay at 1 (TOP3D_XL.m:152,166)
        const float xn = sc == 2 ? 1.0f : oc_candidate(x[ci], dc[ci], rl);
        part = part + (double)xn;
    }
    double tot;
    if (grid_fold(part, red, sh, &tot) && threadIdx.x == 0) oc_step(st, l1, l2, (float)tot / (float)ne, V0);
}

// ---------------------------------------------------------------- the reference's float summation order
// Sum over the n Morton-ordered elements as the reference build evaluates it (see the oracle's vec8_sum): 8 lane
// sums over 8*floor(n/8) values (lane j adds value(8b+j), b = 0, 1, ... one after the other in float), folded
// ((l0+l4)+(l2+l6)) + ((l1+l5)+(l3+l7)); 4..7 remaining values added lane-wise to (l0+l4, ..) and folded
// (m1+m3)+(m0+m2); the last 0..3 added in sequence.
//
// The lane sums are chains of n/8 rounded additions, but they can be evaluated in parallel without changing a
// bit.  While the running sum l = m u stays in one binade (u = 2^(e-23), 2^23 <= m <= 2^24), adding v >= 0 adds
// an integer to m that depends on v / u and, when v / u lies halfway between two integers (ties go to even), on
// the parity of m -- on nothing else.  So a run of elements is, for each binade e, a function "parity of m ->
// integer added", and runs compose.  One block per group of 32 chunks of 32 elements per lane tabulates that
// function for every chunk and for the whole group, in the 16 binades below the largest one the group can reach
// (l never exceeds the number of elements added, since values are <= 1 and u <= 1 divides 1).  The last block
// to finish walks each lane's sum with one warp: 32 groups at a time by a prefix composition, up to the group in
// which the sum would leave its binade (m > 2^24; m = 2^24 is the next binade's first value); there 32 chunks
// at a time, and the crossing chunk's elements one by one, as the float additions they are.  A sum outside the
// tabulated binades (and 0, the start) also takes the element path, so the result never depends on the window.
//
// The first V8_HEAD chunks of a lane always go element by element, from values loaded together: the sum crosses a
// binade every few chunks there.  Sums of at most that many elements need no table.
//
// Latency bounds it (dependent loads of the last block: three per binade crossed).  Before, one warp gathered 4
// values per lane and step: 0.28 ms a pass at 54,000 elements, 2.7 ms at 524,000; now 29 and 37 us.
constexpr int V8_CHUNK = 32, V8_CHUNKS = 32, V8_CAND = 16;
constexpr int V8_RUN = V8_CHUNK * V8_CHUNKS;       // elements per lane and group
constexpr int V8_HEAD = 8;                         // chunks at a lane's start taken element by element
constexpr unsigned V8_BIG = 1u << 25;              // "leaves the binade" (sums of 32 of them fit 32 bits)
constexpr int V8_PAD = 8 * V8_CHUNK + 1;           // chunk stride in shared memory: lanes of a warp hit 32 banks

__device__ __forceinline__ int v8_top_binade(int64_t g) {   // floor(log2(elements per lane up to the group's end))
    return 63 - __clzll((g + 1) * V8_RUN);
}

// what a run adds to m when m starts even (x) and odd (y); a, then b
__device__ __forceinline__ uint2 v8_then(uint2 a, uint2 b) {
    const unsigned x = a.x + ((a.x & 1u) ? b.y : b.x), y = a.y + ((a.y & 1u) ? b.x : b.y);
    return make_uint2(min(x, V8_BIG), min(y, V8_BIG));
}

// Advances the lane sum l over up to 32 consecutive runs, run i's function t in thread i (all of a warp), l in
// every thread.  Returns how many runs were taken: the first one not taken leaves l's binade.
__device__ __forceinline__ int v8_advance(float& l, int e, uint2 t) {
    const int lane = threadIdx.x & 31;
    const unsigned m = (__float_as_uint(l) & 0x7fffffu) | 0x800000u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint2 q = make_uint2(__shfl_up_sync(0xffffffffu, t.x, off), __shfl_up_sync(0xffffffffu, t.y, off));
        if (lane >= off) t = v8_then(q, t);
    }
    const unsigned end = m + ((m & 1u) ? t.y : t.x);
    const unsigned fit = __ballot_sync(0xffffffffu, end <= (1u << 24));
    const int k = __popc(fit);                     // `end` grows with the lane: the fitting ones come first
    if (k > 0) {
        const unsigned mk = __shfl_sync(0xffffffffu, end, k - 1);
        // m = 2^24 is 1.0 x 2^(e+1): adding to the exponent field carries over
        l = __uint_as_float(((unsigned)(e + 127) << 23) + (mk - (1u << 23)));
    }
    return k;
}

// MODE 0: volume of the candidate at the current multiplier, then the bisection step; 1: volume fraction of x;
// 2: sharpness sum x(1-x).  xm, dm: the elements' densities and scaled sensitivities in Morton order (MODE 0);
// perm, x: cell order (MODE 1, 2).  tab: chunk functions [group][lane][binade][chunk], run: [lane][group][binade].
template <int MODE>
__global__ void __launch_bounds__(256) k_oc_vec8(int64_t ne, const float* __restrict__ xm,
                                                 const float* __restrict__ dm, const int32_t* __restrict__ perm,
                                                 const float* __restrict__ x, uint2* __restrict__ tab,
                                                 uint2* __restrict__ run, unsigned int* __restrict__ counter,
                                                 OcState* st, float V0) {
    __shared__ float v[V8_CHUNKS * V8_PAD];
    __shared__ float lsum[8];
    __shared__ int last;
    float l1 = 0.0f, l2 = 0.0f, rl = 0.0f;
    if (MODE == 0) {
        if (st->done) return;
        if (!oc_continue(st)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
            return;
        }
        l1 = st->l1;
        l2 = st->l2;
        rl = 2.0f / (l1 + l2);
    }
    auto value = [&](int64_t i) -> float {
        if (MODE == 0) return oc_candidate(xm[i], dm[i], rl);
        const float w = x[perm[i]];
        return MODE == 1 ? w : w * (1.0f - w);
    };
    const int64_t nb = ne / 8, groups = (nb + V8_RUN - 1) / V8_RUN;
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;   // warp j works on lane sum j
    const int64_t g0 = blockIdx.x;
    if (nb > V8_HEAD * V8_CHUNK && g0 < groups) {
        const int64_t i0 = g0 * 8 * V8_RUN;
        for (int t = threadIdx.x; t < 8 * V8_RUN; t += 256)   // elements past the last whole block of 8 add 0
            v[(t >> 8) * V8_PAD + (t & 255)] = i0 + t < 8 * nb ? value(i0 + t) : 0.0f;
        __syncthreads();
        // thread (j, chunk): the chunk's additions from m = 2^23 (even) and 2^23 + 1 (odd), in units of u
        float even[V8_CAND], odd[V8_CAND];
#pragma unroll
        for (int k = 0; k < V8_CAND; ++k) {
            even[k] = 8388608.0f;
            odd[k] = 8388609.0f;
        }
        const int top = v8_top_binade(g0);
        const float inv_u = __int_as_float((127 + 23 - (top - V8_CAND + 1)) << 23);   // 1/u of the lowest binade
#pragma unroll 2
        for (int b = 0; b < V8_CHUNK; ++b) {
            const float f = v[lane * V8_PAD + 8 * b + j] * inv_u;
#pragma unroll
            for (int k = 0; k < V8_CAND; ++k) {   // f 2^-k, exact, each from f: no chain from binade to binade
                const float fk = f * __int_as_float((127 - k) << 23);
                even[k] = even[k] + fk;
                odd[k] = odd[k] + fk;
            }
        }
        uint2* out = tab + ((g0 * 8 + j) * V8_CAND) * V8_CHUNKS + lane;
        uint2* rout = run + ((int64_t)j * groups + g0) * V8_CAND;
#pragma unroll
        for (int k = 0; k < V8_CAND; ++k) {
            uint2 t;   // past 2^24 the float no longer counts in units of u
            t.x = even[k] <= 16777216.0f ? (unsigned)even[k] - 8388608u : V8_BIG;
            t.y = odd[k] <= 16777216.0f ? (unsigned)odd[k] - 8388609u : V8_BIG;
            out[k * V8_CHUNKS] = t;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {   // the 32 chunks in order: thread 0 ends with all of them
                const uint2 q = make_uint2(__shfl_down_sync(0xffffffffu, t.x, off),
                                           __shfl_down_sync(0xffffffffu, t.y, off));
                t = v8_then(t, q);
            }
            if (lane == 0) rout[k] = t;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1 ? 1 : 0;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) *counter = 0u;
    float l = 0.0f;
    float head[V8_HEAD];
#pragma unroll
    for (int c = 0; c < V8_HEAD; ++c) {
        const int64_t i = 8 * (c * V8_CHUNK + lane) + j;
        head[c] = i < 8 * nb ? value(i) : 0.0f;
    }
#pragma unroll
    for (int c = 0; c < V8_HEAD; ++c) {
        if (c * V8_CHUNK >= nb) break;
#pragma unroll
        for (int b = 0; b < V8_CHUNK; ++b) l = l + __shfl_sync(0xffffffffu, head[c], b);
    }
    for (int64_t g = 0; g < groups && nb > V8_HEAD * V8_CHUNK;) {
        const int e = (int)(__float_as_uint(l) >> 23) - 127;
        if (g > 0) {
            const int k = e - (v8_top_binade(g + lane) - V8_CAND + 1);
            uint2 t = make_uint2(V8_BIG, V8_BIG);
            if (g + lane < groups && k >= 0 && k < V8_CAND)
                t = __ldcg(run + ((int64_t)j * groups + g + lane) * V8_CAND + k);
            g += v8_advance(l, e, t);
        }
        if (g >= groups) break;
        // group g may leave the binade: its chunks, then the crossing chunk's elements, until a whole run of 32
        // groups fits again
        const int low = v8_top_binade(g) - V8_CAND + 1;
        for (int c = g == 0 ? V8_HEAD : 0; c < V8_CHUNKS;) {
            const int ec = (int)(__float_as_uint(l) >> 23) - 127, k = ec - low;
            uint2 t = make_uint2(V8_BIG, V8_BIG);
            if (c + lane < V8_CHUNKS && k >= 0 && k < V8_CAND)
                t = __ldcg(tab + ((g * 8 + j) * V8_CAND + k) * V8_CHUNKS + c + lane);
            c += v8_advance(l, ec, t);
            if (c >= V8_CHUNKS) break;
            const int64_t i = 8 * (g * V8_RUN + c * V8_CHUNK + lane) + j;
            const float w = i < 8 * nb ? value(i) : 0.0f;
#pragma unroll
            for (int b = 0; b < V8_CHUNK; ++b) l = l + __shfl_sync(0xffffffffu, w, b);
            ++c;
        }
        ++g;
    }
    if (lane == 0) lsum[j] = l;
    __syncthreads();
    if (threadIdx.x != 0) return;
    float s = 0.0f, h[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (nb > 0) {
        for (int k = 0; k < 4; ++k) h[k] = lsum[k + 4] + lsum[k];
        s = (h[1] + h[3]) + (h[0] + h[2]);
    }
    int64_t i = 8 * nb;
    if (ne - i >= 4) {
        const float m0 = h[0] + value(i), m1 = h[1] + value(i + 1);
        const float m2 = h[2] + value(i + 2), m3 = h[3] + value(i + 3);
        s = (m1 + m3) + (m0 + m2);
        i += 4;
    }
    for (; i < ne; ++i) s = s + value(i);
    if (MODE == 0) {
        const float vol = s * (1.0f / (float)ne);
        oc_step(st, l1, l2, vol, V0);
    } else if (MODE == 1) {
        st->volfrac = s / (float)ne;
    } else {
        st->sharp = 4.0f * s / (float)ne;
    }
}

// Morton-ordered copies of the densities and scaled sensitivities, read by every pass.  A passive element
// (solid = 2, candidate 1 at any multiplier) becomes x = 1 with an infinite sensitivity, which the candidate
// formula clamps to exactly 1.
__global__ void k_oc_gather(int64_t ne, const int32_t* __restrict__ perm, const uint8_t* __restrict__ solid,
                            const float* __restrict__ x, const float* __restrict__ dc, float* __restrict__ xm,
                            float* __restrict__ dm) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ne) return;
    const int32_t c = perm[i];
    const bool passive = solid[c] == 2;
    xm[i] = passive ? 1.0f : x[c];
    dm[i] = passive ? __int_as_float(0xff800000) : dc[c];
}

// xnew of the last pass's multiplier; change = max|xnew-x| (order-free), x = xnew; FP64 sums of x and x(1-x) for the fp64 path
__global__ void __launch_bounds__(RED_THREADS) k_oc_finish(Grid g, const uint8_t* __restrict__ solid,
                                                           float* __restrict__ x, const float* __restrict__ dc,
                                                           OcState* st, int fp64_sum, int64_t ne, RedSlot r1,
                                                           RedSlot r2) {
    __shared__ double sh[32];
    __shared__ float shm[32];
    const int ncell = g.nx * g.ny * g.nz, stride = gridDim.x * blockDim.x;
    const float rl = st->rl;
    float ch = 0.0f;
    double sv = 0.0, sp = 0.0;
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    CellWalk w(g, k, stride);
    for (; k < ncell; k += stride, w.next(g)) {
        const int64_t ci = g.cell(w.cx, w.cy, w.cz);
        const uint8_t sc = solid[ci];
        if (!sc) continue;
        const float xv = x[ci];
        const float xn = sc == 2 ? 1.0f : oc_candidate(xv, dc[ci], rl);
        ch = fmaxf(ch, fabsf(xn - xv));
        x[ci] = xn;
        sv = sv + (double)xn;
        sp = sp + (double)(xn * (1.0f - xn));
    }
    // max-reduction: order does not matter; non-negative floats compare as their bit patterns
    ch = warp_fold_max(ch);
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = ch;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, shm[w]);
        atomicMax(reinterpret_cast<int*>(&st->change), __float_as_int(m));
    }
    if (!fp64_sum) return;
    double tv, tp;
    if (grid_fold(sv, r1, sh, &tv) && threadIdx.x == 0) st->volfrac = (float)tv / (float)ne;
    __syncthreads();
    if (grid_fold(sp, r2, sh, &tp) && threadIdx.x == 0) st->sharp = 4.0f * (float)tp / (float)ne;
}

__global__ void k_oc_reset_change(OcState* st) { st->change = 0.0f; }

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_dc_scale(const Grid& g, const uint8_t* solid, const float* dcf, const float* x, float* dc,
                     cudaStream_t s) {
    k_dc_scale<<<blocks_for(g.NE, 256), 256, 0, s>>>(g, solid, dcf, x, dc);
}
void launch_oc_init(OcState* st, cudaStream_t s) { k_oc_init<<<1, 1, 0, s>>>(st); }
void launch_oc_pass(const Grid& g, const uint8_t* solid, const float* x, const float* dc, OcState* st, float V0,
                    int64_t ne, RedSlot red, cudaStream_t s) {
    k_oc_pass<<<red_blocks((int64_t)g.nx * g.ny * g.nz), RED_THREADS, 0, s>>>(g, solid, x, dc, st, V0, ne, red);
}
static int64_t oc_vec8_groups(int64_t ne) { return (ne / 8 + V8_RUN - 1) / V8_RUN; }
int64_t oc_vec8_bytes(int64_t ne) {
    const int64_t g = oc_vec8_groups(ne);
    return (g * 8 * V8_CAND * (V8_CHUNKS + 1)) * (int64_t)sizeof(uint2) + 2 * ne * (int64_t)sizeof(float);
}
namespace {
struct Vec8Buf {   // the scratch block of oc_vec8_bytes(ne): tables first (8-byte aligned), then the copies
    uint2 *tab, *run;
    float *xm, *dm;
    Vec8Buf(int64_t ne, void* scratch) {
        const int64_t g = oc_vec8_groups(ne);
        tab = static_cast<uint2*>(scratch);
        run = tab + g * 8 * V8_CAND * V8_CHUNKS;
        xm = reinterpret_cast<float*>(run + g * 8 * V8_CAND);
        dm = xm + ne;
    }
};
inline unsigned vec8_blocks(int64_t ne) { return (unsigned)(ne >= 8 ? oc_vec8_groups(ne) : 1); }
}  // namespace
void launch_oc_vec8_begin(int64_t ne, const int32_t* morton_cells, const uint8_t* solid, const float* x,
                          const float* dc, void* scratch, cudaStream_t s) {
    const Vec8Buf b(ne, scratch);
    k_oc_gather<<<blocks_for(ne, 256), 256, 0, s>>>(ne, morton_cells, solid, x, dc, b.xm, b.dm);
}
void launch_oc_vec8_pass(int64_t ne, void* scratch, OcState* st, float V0, RedSlot red, cudaStream_t s) {
    const Vec8Buf b(ne, scratch);
    k_oc_vec8<0><<<vec8_blocks(ne), 256, 0, s>>>(ne, b.xm, b.dm, nullptr, nullptr, b.tab, b.run, red.counter, st, V0);
}
void launch_oc_finish(const Grid& g, const uint8_t* solid, float* x, const float* dc, OcState* st, int fp64_sum,
                      int64_t ne, RedSlot r1, RedSlot r2, cudaStream_t s) {
    k_oc_reset_change<<<1, 1, 0, s>>>(st);
    k_oc_finish<<<red_blocks((int64_t)g.nx * g.ny * g.nz), RED_THREADS, 0, s>>>(g, solid, x, dc, st, fp64_sum, ne, r1, r2);
}
void launch_oc_vec8_stats(int64_t ne, const int32_t* morton_cells, const float* x, void* scratch, OcState* st,
                          RedSlot red, cudaStream_t s) {
    const Vec8Buf b(ne, scratch);
    k_oc_vec8<1><<<vec8_blocks(ne), 256, 0, s>>>(ne, nullptr, nullptr, morton_cells, x, b.tab, b.run, red.counter, st,
                                                 0.0f);
    k_oc_vec8<2><<<vec8_blocks(ne), 256, 0, s>>>(ne, nullptr, nullptr, morton_cells, x, b.tab, b.run, red.counter, st,
                                                 0.0f);
}

}  // namespace t3d
