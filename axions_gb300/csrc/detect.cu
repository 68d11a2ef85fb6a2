// String detection on the "now" level of one scalar.
//
// 1. Bilinear face crossings (mpi_evolution.cpp:536-789, evolution.cpp:749-1004):
//    each site checks its three positive faces; each face's bilinear
//    interpolation of (Re phi, Im phi) is inverted through a quadratic.  The
//    reference appends roots to per-rank vectors; here a pass that finds and
//    counts them, a scan of block totals and a pass that places them put every
//    crossing at its position in the reference's order (sites in linear order;
//    z-, y-, x-directed face; "+" root before "-" root) with no sort.  A face's
//    roots are found in double precision in the reference's order of operations
//    and this file is compiled with -fmad=false, so the output is bit-identical
//    to the reference on identical fields; faces that provably have none are
//    left out of that by an FP32 test.
// 2. Plaquette winding (new, defined in include/lattice_gpu.h).
#include "detect_face.cuh"
#include "lattice_internal.cuh"

namespace lat {

namespace {

constexpr int DB = 256;           // threads per detection block
constexpr int DR_MOST = 4;        // sites per thread: 4, or 1 (detect_rounds)
constexpr int DWARPS = DB / 32;
constexpr int DCHUNKS = 3 * DR_MOST;   // most chunks of DB candidate faces in a block

// Sites per thread: four, so that the faces left by the FP32 test fill the lanes
// of the FP64 root search, unless that leaves fewer than two blocks for each SM.
// us for counting FP64 levels, noise and 60 steps later, with one and with four:
// 16^3 41, 29 and 78, 33; 32^3 41, 30 and 78, 34; 48^3 66, 29 and 77, 32; 64^3 115, 41
// and 116, 42; 80^3 177, 54 and 201, 43; 128^3 606, 127 and 601, 102.
inline int detect_rounds(int64_t sites) { return sites < 2 * 152 * DB * DR_MOST ? 1 : DR_MOST; }

// Offsets to the forward neighbours of site s, and whether it is examined.
struct Site {
    int i, j, k, xp, yp, zp;
};

__device__ __forceinline__ bool site_at(const DetectArgs& a, long long sl, Site& o)
{
    if (sl >= (long long)a.nx * a.syz) return false;
    const int s = (int)sl;
    o.i = s / a.syz;
    const int rem = s - o.i * a.syz;
    o.j = rem / a.nz;
    o.k = rem - o.j * a.nz;
    o.xp = (o.i + 1 == a.nx) ? -(a.nx - 1) * a.syz : a.syz;
    o.yp = (o.j + 1 == a.ny) ? -(a.ny - 1) * a.nz : a.nz;
    o.zp = (o.k + 1 == a.nz) ? -(a.nz - 1) : 1;
    return o.i >= a.lox && o.i < a.hix && o.j >= a.loy && o.j < a.hiy && o.k >= a.loz && o.k < a.hiz;
}

// Roots found by the count pass, so that the write pass need not evaluate the
// faces again: chunk c of block b put `count` triples at `base` of the stash.
struct StashChunk {
    unsigned base, count;
};

// a stash: 16 bytes (the counter), the blocks' chunk records, the triples
inline StashChunk* stash_chunks(const DetectStash& sh) { return (StashChunk*)((char*)sh.buf + 16); }
inline double* stash_xyz(const DetectStash& sh, int nb)
{
    return (double*)((char*)sh.buf + 16 + sizeof(StashChunk) * DCHUNKS * (size_t)nb);
}

enum DetectMode { DETECT_COUNT, DETECT_STASH, DETECT_WRITE };

// Sites [blockIdx.x*DB*DR, +DB*DR): candidate faces are listed in the
// reference's order (sites in linear order; z-, y-, x-directed face), then
// evaluated DB at a time.  COUNT: the block's number of crossings to totals;
// STASH: the same, and the crossings to the stash (`used` counts them, beyond
// `cap` they are not stored); WRITE: the crossings to xyz at totals (scanned).
template <class T, int MODE, int DR>
__global__ void __launch_bounds__(DB) detect_kernel(const DetectArgs a, const T* __restrict__ re,
                                                    const T* __restrict__ im, const float eref, long long* totals,
                                                    double* __restrict__ xyz, long long cap, unsigned* used,
                                                    StashChunk* __restrict__ chunks)
{
    constexpr int DSITES = DB * DR;
    __shared__ unsigned short list[3 * DSITES];   // site within the block * 4 + face
    __shared__ int wsum[DR * DWARPS];             // candidates of warp w, round r at [r*DWARPS + w]
    __shared__ int csum[DWARPS];                  // crossings of a warp in the current chunk
    __shared__ unsigned s_base;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const long long first = (long long)blockIdx.x * DSITES;

    unsigned mask[DR];
#pragma unroll
    for (int r = 0; r < DR; ++r) {
        Site o;
        const long long sl = first + r * DB + tid;
        mask[r] = 0;
        if (site_at(a, sl, o)) {
            const int s = (int)sl;
            auto at = [&](int off) { return Corner{corner_float(re[s + off]), corner_float(im[s + off])}; };
            const Corner v0 = at(0), vx = at(o.xp), vy = at(o.yp), vz = at(o.zp);
            if (face_maybe(v0, vx, vy, at(o.xp + o.yp), eref)) mask[r] |= 1u;   // z-directed face (x,y)
            if (face_maybe(v0, vx, vz, at(o.xp + o.zp), eref)) mask[r] |= 2u;   // y-directed face (x,z)
            if (face_maybe(v0, vy, vz, at(o.yp + o.zp), eref)) mask[r] |= 4u;   // x-directed face (y,z)
        }
        int n = 0;
#pragma unroll
        for (int f = 0; f < 3; ++f) n += __popc(__ballot_sync(0xffffffffu, (mask[r] >> f) & 1u));
        if (lane == 0) wsum[r * DWARPS + wid] = n;
    }
    __syncthreads();
    constexpr int NSUM = DR * DWARPS;
    static_assert(NSUM <= 32, "one warp scans the warps' candidate counts");
    if (wid == 0) {
        const int own = lane < NSUM ? wsum[lane] : 0;
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane < NSUM) wsum[lane] = incl - own;
        if (lane == 31) s_base = (unsigned)incl;
    }
    __syncthreads();
    const int m = (int)s_base;
#pragma unroll
    for (int r = 0; r < DR; ++r) {
        int pos = wsum[r * DWARPS + wid];
        const unsigned below = (1u << lane) - 1u;
#pragma unroll
        for (int f = 0; f < 3; ++f) pos += __popc(__ballot_sync(0xffffffffu, (mask[r] >> f) & 1u) & below);
#pragma unroll
        for (int f = 0; f < 3; ++f)
            if (mask[r] >> f & 1u) list[pos++] = (unsigned short)((r * DB + tid) * 4 + f);
    }
    __syncthreads();

    long long run = MODE == DETECT_WRITE ? totals[blockIdx.x] : 0;   // crossings before the chunk
    int mine = 0;
    for (int c0 = 0; c0 < m; c0 += DB) {
        Roots q;
        q.n = 0;
        int face = 0;
        double x = 0, y = 0, z = 0;
        if (c0 + tid < m) {
            const int item = list[c0 + tid];
            face = item & 3;
            Site o;
            const long long sl = first + (item >> 2);
            site_at(a, sl, o);
            const int s = (int)sl;
            // physical coordinates (mpi_evolution.cpp:547-549)
            x = (double)(o.i - a.x0) * a.dx;
            y = (double)(o.j - a.y0) * a.dy;
            z = (double)(o.k - a.z0) * a.dz;
            const int d1 = face == 2 ? o.yp : o.xp, d2 = face == 0 ? o.yp : o.zp;
            const double v00[2] = {(double)re[s], (double)im[s]};
            const double v10[2] = {(double)re[s + d1], (double)im[s + d1]};
            const double v01[2] = {(double)re[s + d2], (double)im[s + d2]};
            const double v11[2] = {(double)re[s + d1 + d2], (double)im[s + d1 + d2]};
            q = face_roots(v00, v10, v01, v11, face == 2 ? y : x, face == 0 ? y : z, face == 2 ? a.dy : a.dx,
                           face == 0 ? a.dy : a.dz);
        }
        if constexpr (MODE == DETECT_COUNT) {
            mine += q.n;
        } else {
            const unsigned one = __ballot_sync(0xffffffffu, q.n & 1), two = __ballot_sync(0xffffffffu, q.n & 2);
            if (lane == 0) csum[wid] = __popc(one) + 2 * __popc(two);
            __syncthreads();
            int before = 0, all = 0;
#pragma unroll
            for (int w = 0; w < DWARPS; ++w) {
                if (w < wid) before += csum[w];
                all += csum[w];
            }
            const unsigned below = (1u << lane) - 1u;
            before += __popc(one & below) + 2 * __popc(two & below);
            long long pos;
            if constexpr (MODE == DETECT_STASH) {
                if (tid == 0) {
                    s_base = all ? atomicAdd(used, (unsigned)all) : 0u;
                    chunks[(size_t)blockIdx.x * DCHUNKS + c0 / DB] = StashChunk{s_base, (unsigned)all};
                }
                __syncthreads();
                pos = (long long)s_base + before;
            } else {
                pos = run + before;
            }
            for (int t = 0; t < q.n; ++t, ++pos) {
                if (pos >= cap) break;
                xyz[3 * pos + 0] = face == 2 ? x : q.s1[t];
                xyz[3 * pos + 1] = face == 0 ? q.s2[t] : (face == 1 ? y : q.s1[t]);
                xyz[3 * pos + 2] = face == 0 ? z : q.s2[t];
            }
            run += all;
            __syncthreads();  // csum and s_base are rewritten by the next chunk
        }
    }
    if constexpr (MODE == DETECT_STASH) {
        for (int c = (m + DB - 1) / DB + tid; c < DCHUNKS; c += DB)
            chunks[(size_t)blockIdx.x * DCHUNKS + c] = StashChunk{0u, 0u};
        if (tid == 0) totals[blockIdx.x] = run;
    }
    if constexpr (MODE == DETECT_COUNT) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
        if (lane == 0) csum[wid] = mine;
        __syncthreads();
        if (tid == 0) {
            int all = 0;
            for (int w = 0; w < DWARPS; ++w) all += csum[w];
            totals[blockIdx.x] = all;
        }
    }
}

// The stashed crossings of every block to their places (offsets: the scanned
// totals); those at `cap` and beyond are left out.
__global__ void __launch_bounds__(DB) detect_place_kernel(const double* __restrict__ stash,
                                                          const StashChunk* __restrict__ chunks,
                                                          const long long* __restrict__ offsets, double* __restrict__ xyz,
                                                          long long cap)
{
    long long pos = offsets[blockIdx.x];
    for (int c = 0; c < DCHUNKS; ++c) {
        const StashChunk k = chunks[(size_t)blockIdx.x * DCHUNKS + c];
        if (k.count == 0) continue;
        const long long room = cap - pos;
        const int n = 3 * (int)(room < (long long)k.count ? (room > 0 ? room : 0) : (long long)k.count);
        for (int t = threadIdx.x; t < n; t += DB) xyz[3 * pos + t] = stash[3 * (size_t)k.base + t];
        pos += k.count;
    }
}

// Exclusive scan of block totals in place (one block); *total = grand total.
// Tiles of 4096, four consecutive values a thread.
__global__ void __launch_bounds__(1024) scan_totals_kernel(long long* v, int n, long long* total)
{
    __shared__ long long ws[32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    long long carry = 0;
    for (int base = 0; base < n; base += 4096) {
        long long own[4], sum = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int q = base + 4 * t + r;
            own[r] = q < n ? v[q] : 0;
            sum += own[r];
        }
        long long incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) ws[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            const long long w = ws[lane];
            long long wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long u = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += u;
            }
            ws[lane] = wi;  // inclusive over warps
        }
        __syncthreads();
        long long run = carry + (wid ? ws[wid - 1] : 0) + incl - sum;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int q = base + 4 * t + r;
            if (q < n) v[q] = run;
            run += own[r];
        }
        carry += ws[31];
        __syncthreads();  // ws is rewritten by the next tile
    }
    if (t == 0) *total = carry;
}

// ---------------------------------------------------------------------------
// plaquette winding
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ int edge_cross(T ax, T ay, T bx, T by)
{
    T cr;
    if constexpr (sizeof(T) == 8) cr = __dsub_rn(__dmul_rn(ax, by), __dmul_rn(ay, bx));
    else cr = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
    if (ay <= 0) {
        if (by > 0 && cr > 0) return 1;
    } else {
        if (by <= 0 && cr < 0) return -1;
    }
    return 0;
}

template <class T>
__global__ void __launch_bounds__(DB) winding_kernel(const DetectArgs a, int open_axes, const T* __restrict__ re,
                                                     const T* __restrict__ im, int8_t* out,
                                                     unsigned long long* abs_sum)
{
    const long long N = (long long)a.nx * a.syz;
    const long long sl = (long long)blockIdx.x * DB + threadIdx.x;
    int tot = 0;
    if (sl < N) {
        const int s = (int)sl;
        const int i = s / a.syz;
        const int rem = s - i * a.syz;
        const int j = rem / a.nz;
        const int k = rem - j * a.nz;
        const int oxp = (i + 1 == a.nx) ? -(a.nx - 1) * a.syz : a.syz;
        const int oyp = (j + 1 == a.ny) ? -(a.ny - 1) * a.nz : a.nz;
        const int ozp = (k + 1 == a.nz) ? -(a.nz - 1) : 1;
        // corners counter-clockwise about +d (include/lattice_gpu.h)
        const int cs[3][4] = {{s, s + oyp, s + oyp + ozp, s + ozp},
                              {s, s + ozp, s + ozp + oxp, s + oxp},
                              {s, s + oxp, s + oxp + oyp, s + oyp}};
        // a face is valid unless it wraps around a non-periodic axis (bit 0: x/y, bit 1: z)
        const bool xin = !(open_axes & 1) || i + 1 < a.nx, yin = !(open_axes & 1) || j + 1 < a.ny;
        const bool zin = !(open_axes & 2) || k + 1 < a.nz;
        const bool valid[3] = {yin && zin, zin && xin, xin && yin};
        T vr[3][4], vi[3][4];
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                vr[d][e] = re[cs[d][e]];
                vi[d][e] = im[cs[d][e]];
            }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            int w = 0;
            if (valid[d]) {
#pragma unroll
                for (int e = 0; e < 4; ++e) w += edge_cross<T>(vr[d][e], vi[d][e], vr[d][(e + 1) & 3], vi[d][(e + 1) & 3]);
            }
            if (out) out[(long long)d * N + s] = (int8_t)w;
            tot += w < 0 ? -w : w;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(0xffffffffu, tot, o);
    __shared__ int ws[DB / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = tot;
    __syncthreads();
    if (threadIdx.x == 0) {
        int b = 0;
        for (int w = 0; w < DB / 32; ++w) b += ws[w];
        if (b) atomicAdd(abs_sum, (unsigned long long)b);
    }
}

inline unsigned nblocks_of(const DetectArgs& a) { return (unsigned)(((long long)a.nx * a.syz + DB - 1) / DB); }

}  // namespace

namespace {

// 16 eps N^3 with N = the largest distance from the origin in spacings (see face_maybe)
inline float reference_error(const DetectArgs& a)
{
    const double n = 1 + 0.5 * (a.nx > a.ny ? (a.nx > a.nz ? a.nx : a.nz) : (a.ny > a.nz ? a.ny : a.nz));
    const double e = 16 * 1.1102230246251565e-16 * n * n * n;
    return (float)(e < 1 ? e : 1);
}

template <class T, int DR>
cudaError_t detect_launch_t(const DetectArgs& a, const T* re, const T* im, long long* bt, int nb, const DetectStash& sh,
                            double* xyz, long long cap, cudaStream_t st)
{
    const float e = reference_error(a);
    if (xyz) {
        detect_kernel<T, DETECT_WRITE, DR><<<nb, DB, 0, st>>>(a, re, im, e, bt, xyz, cap, nullptr, nullptr);
    } else if (sh.cap > 0) {
        const cudaError_t m = cudaMemsetAsync(sh.buf, 0, 16, st);
        if (m != cudaSuccess) return m;
        detect_kernel<T, DETECT_STASH, DR><<<nb, DB, 0, st>>>(a, re, im, e, bt, stash_xyz(sh, nb), sh.cap,
                                                              (unsigned*)sh.buf, stash_chunks(sh));
    } else {
        detect_kernel<T, DETECT_COUNT, DR><<<nb, DB, 0, st>>>(a, re, im, e, bt, nullptr, 0, nullptr, nullptr);
    }
    return cudaGetLastError();
}

template <class T>
cudaError_t detect_launch(const DetectArgs& a, const T* re, const T* im, long long* bt, int nb, const DetectStash& sh,
                          double* xyz, long long cap, cudaStream_t st)
{
    return detect_rounds((int64_t)a.nx * a.syz) == 1 ? detect_launch_t<T, 1>(a, re, im, bt, nb, sh, xyz, cap, st)
                                                     : detect_launch_t<T, DR_MOST>(a, re, im, bt, nb, sh, xyz, cap, st);
}

}  // namespace

int detect_blocks(int64_t sites)
{
    const int64_t per = (int64_t)DB * detect_rounds(sites);
    return (int)((sites + per - 1) / per);
}

size_t detect_stash_bytes(int nb, int64_t cap)
{
    return 16 + sizeof(StashChunk) * DCHUNKS * (size_t)nb + 24 * (size_t)cap;
}

cudaError_t launch_detect_count(const DetectArgs& a, int elem, const void* re, const void* im, long long* bt, int nb,
                                const DetectStash& sh, cudaStream_t st)
{
    return elem == 8 ? detect_launch(a, (const double*)re, (const double*)im, bt, nb, sh, nullptr, 0, st)
                     : detect_launch(a, (const float*)re, (const float*)im, bt, nb, sh, nullptr, 0, st);
}

cudaError_t launch_detect_write(const DetectArgs& a, int elem, const void* re, const void* im, long long* bo, int nb,
                                double* xyz, long long cap, cudaStream_t st)
{
    return elem == 8 ? detect_launch(a, (const double*)re, (const double*)im, bo, nb, DetectStash{}, xyz, cap, st)
                     : detect_launch(a, (const float*)re, (const float*)im, bo, nb, DetectStash{}, xyz, cap, st);
}

cudaError_t launch_detect_place(const DetectStash& sh, const long long* bo, int nb, double* xyz, long long cap,
                                cudaStream_t st)
{
    detect_place_kernel<<<nb, DB, 0, st>>>(stash_xyz(sh, nb), stash_chunks(sh), bo, xyz, cap);
    return cudaGetLastError();
}

cudaError_t launch_scan_totals(long long* bt, int nb, long long* total, cudaStream_t st)
{
    scan_totals_kernel<<<1, 1024, 0, st>>>(bt, nb, total);
    return cudaGetLastError();
}
cudaError_t launch_winding_f64(const DetectArgs& a, int open_axes, const double* re, const double* im, int8_t* out,
                               unsigned long long* abs_sum, cudaStream_t st)
{
    winding_kernel<double><<<nblocks_of(a), DB, 0, st>>>(a, open_axes, re, im, out, abs_sum);
    return cudaGetLastError();
}
cudaError_t launch_winding_f32(const DetectArgs& a, int open_axes, const float* re, const float* im, int8_t* out,
                               unsigned long long* abs_sum, cudaStream_t st)
{
    winding_kernel<float><<<nblocks_of(a), DB, 0, st>>>(a, open_axes, re, im, out, abs_sum);
    return cudaGetLastError();
}

}  // namespace lat
