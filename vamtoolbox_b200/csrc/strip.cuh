// strip.cuh -- the rotate-and-sum forward by detector strips.
//
// One warp owns M neighbouring detector bins (a strip) of one angle, or of an angle and the one 180
// degrees from it, over the slices of one z chunk.  The forward is linear in the pixels: bin j of an angle
// gets W(j, p) x(p) from pixel p with
//     W(j, p) = sum over samples k of hat(row(j, k) - row_p) hat(col(j, k) - col_p),  hat(d) = max(0, 1 - |d|),
// the bilinear weights of all samples of the bin that touch the pixel (Projector3DParallel.py:137-156 via
// skimage.warp).  Going through the pixels under the strip instead of through its samples loads every
// pixel's row of slices once for all M bins and all their samples: 1.63 rows per sample for two bins, 1.42 for
// three, against four taps per sample.  The rows' loads are what bounds the forward (L1 data path), so this is
// where its time goes down.
//
// The warp lists the pixels in batches: the 32 lanes take R rows (or columns, whichever the rays run across)
// of S candidate pixels, form each pixel's position in the rotated lattice and, from its fractions, its M
// weights; pixels with any nonzero weight go through a ring in shared memory (pixel, M weights) that the same
// warp then works off, U pixels at a time, the next U pixels' rows in flight meanwhile.
//
// Measured (B200): 256^3 x 360 angles 1.39 -> 0.83 ms, 512^2 x 128 x 720 7.30 -> 4.37 ms, 201^2 x 117 x 240 3.92 ->
// 0.25 ms against the sample kernels before.  At 256^3 the L1 data path is
// 79 % busy (a pixel is eight cycles of row and three or four of weights, which are written to every lane's
// registers), issue 50 %; the rest is what 16 warps leave uncovered.
#pragma once

#include "vam_internal.cuh"

namespace vam {
namespace {

// Bins per strip: two with eight slices per lane, three with four.  A strip's pixel costs its row's loads and
// one broadcast load of its weights; three bins share the row better (4.30 against 4.86 ms at 512^2 x 128 x 720,
// four slices per lane) until their accumulators take the registers that keep rows in flight (0.93 against
// 0.82 ms at 256^3 x 360, eight slices per lane).
__host__ __device__ constexpr int strip_bins(int q) { return q == 2 ? 2 : 3; }
constexpr int kStripRing = 128;  // ring entries per warp (the whole groups of them): a group short of one entry and a batch of 32 fit

// The strip's geometry, read back by every batch (registers are what the rows in flight need).  A pixel is
// (main, other): (row, column) when the rays run across rows, (column, row) otherwise.  Its lattice position
// is J = jc.x main + jc.y other + j0, K = kc.x main + kc.y other + k0; the fractions come from the same sums
// in 32-bit fixed point, whose overflow drops the whole part, with the coefficients' rounding added back in
// float32, so they are good to float32 rounding at any size.
struct StripGeo {
    float4 coef;   // J and K per step of main and other
    float4 res;    // what the fixed-point coefficients leave out
    uint4 fix;     // the coefficients times 2^32, modulo 2^32 (unsigned: the sums wrap)
    float4 org;    // J and K at the origin; least other of the strip = slope * main + base
    uint2 fixorg;  // the origin in fixed point
    float4 cs;     // cos and sin, and what their float32 values leave out
};

struct StripRing {
    float4 e[kWarpsPerBlock][kStripRing];  // M weights and the pixel
    StripGeo geo[kWarpsPerBlock];
};

__device__ __forceinline__ StripRing& strip_ring() {
    __shared__ __align__(16) StripRing r;
    return r;
}

struct FastArgs {
    const float* vol;
    float* sino;
    const double4* trig;
    const int2* tasks;
    const float* mask;  // per-pixel factor of the volume, or null
    int nY, nX, nZ, nA, C;
    int vs;          // floats from one pixel's row to the next (nZ, or nZ rounded up to four: padded rows)
    int ntasks;
    int zchunks;
    int lz_shift;    // log2 of the lanes along z (a warp's other lanes take other pixels)
    int ashift;      // log2 of the angle tasks per block
    int even;        // N even
    float alpha, R;  // per-ray absorption (tasks are unpaired then)
};

// A lane's 4 Q slices of one pixel's row as slice pairs, p pointing at its first.  VEC: float4s 4 LZ apart
// (LZ = 32 when Q = 2), the first n of them inside the volume.  Otherwise single slices LZ apart, any slice
// count and any alignment.  Slices past the volume are not read; their values are undefined.
template <int Q, bool VEC>
__device__ __forceinline__ void strip_load(const float* __restrict__ p, unsigned long long (&v)[2 * Q], int n, int lz) {
    if constexpr (VEC) {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            asm volatile("{ .reg .pred p; setp.gt.s32 p, %3, %4; @p ld.global.nc.v2.u64 {%0, %1}, [%2]; }"
                : "=l"(v[2 * q]), "=l"(v[2 * q + 1]) : "l"(p + 128 * q), "r"(n), "r"(q));
    } else {
        const int st = Q == 2 ? 32 : lz;
#pragma unroll
        for (int e = 0; e < 2 * Q; ++e) {
            float lo, hi;
            asm volatile("{ .reg .pred p; setp.gt.s32 p, %2, %3; @p ld.global.nc.f32 %0, [%1]; }"
                : "=f"(lo) : "l"(p + st * 2 * e), "r"(n), "r"(2 * e));
            asm volatile("{ .reg .pred p; setp.gt.s32 p, %2, %3; @p ld.global.nc.f32 %0, [%1]; }"
                : "=f"(hi) : "l"(p + st * (2 * e + 1)), "r"(n), "r"(2 * e + 1));
            v[e] = pk_pair(lo, hi);
        }
    }
}

__device__ __forceinline__ void fma_pairs(unsigned long long& acc, unsigned long long w2, unsigned long long v2) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w2), "l"(v2));
}

// what the rounding of t = s + x drops (s the larger)
__device__ __forceinline__ unsigned long long dropped(unsigned long long s, unsigned long long t, unsigned long long x) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(t), "l"(s));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(d));
    return d;
}

__device__ __forceinline__ unsigned long long add_pairs(unsigned long long s, unsigned long long x) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s) : "l"(x));
    return s;
}

// s + x into s; what the rounding drops, whichever is larger
__device__ __forceinline__ unsigned long long two_sum(unsigned long long& s, unsigned long long x) {
    const unsigned long long t = add_pairs(s, x);
    unsigned long long d, e;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(t), "l"(s));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(e) : "l"(t), "l"(d));
    asm("sub.rn.f32x2 %0, %1, %0;" : "+l"(e) : "l"(s));
    asm("sub.rn.f32x2 %0, %1, %0;" : "+l"(d) : "l"(x));
    s = t;
    return add_pairs(e, d);
}

// s + x, but s where that is no number (s infinite: what its rounding dropped is none)
__device__ __forceinline__ unsigned long long add_finite(unsigned long long s, unsigned long long x) {
    float s0, s1, t0, t1;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(s));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(t0), "=f"(t1) : "l"(add_pairs(s, x)));
    return pk_pair(t0 == t0 ? t0 : s0, t1 == t1 ? t1 : s1);
}

// whole: the float4s may be stored as such; otherwise (padded rows) slice by slice, the first `left` of them
// (those the output has: a padded row holds up to three more)
template <int Q, bool VEC>
__device__ __forceinline__ void strip_store(float* __restrict__ p, const unsigned long long (&v)[2 * Q], int n, int lz,
                                            int whole, int left) {
    if constexpr (VEC) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if (q >= n) break;
            if (whole) {
                *reinterpret_cast<ulonglong2*>(p + 128 * q) = make_ulonglong2(v[2 * q], v[2 * q + 1]);
                continue;
            }
            float x[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(x[0]), "=f"(x[1]) : "l"(v[2 * q]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(x[2]), "=f"(x[3]) : "l"(v[2 * q + 1]));
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (128 * q + e < left) p[128 * q + e] = x[e];
        }
    } else {
        const int st = Q == 2 ? 32 : lz;
#pragma unroll
        for (int e = 0; e < 2 * Q; ++e) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[e]));
            if (2 * e < n) p[st * 2 * e] = lo;
            if (2 * e + 1 < n) p[st * (2 * e + 1)] = hi;
        }
    }
}

// One bilinear sample (every tap checked against the image) times f added into acc: the end samples k = 0 and
// k = N of a paired strip, which belong to one of its two angles only.
template <int Q, bool VEC>
__device__ __forceinline__ void strip_sample(const FastArgs& a, const float* __restrict__ volz, double row, double col,
                                             unsigned long long (&acc)[2 * Q], int n, int lz, float f = 1.f) {
    const double fr = floor(row), fc = floor(col);
    const int r0 = (int)fr, c0 = (int)fc;
    const float dr = (float)(row - fr), dc = (float)(col - fc);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int r = r0 + (t >> 1), c = c0 + (t & 1);
        if ((unsigned)r >= (unsigned)a.nY || (unsigned)c >= (unsigned)a.nX) continue;
        if (((t >> 1) && !(row > fr)) || ((t & 1) && !(col > fc))) continue;
        float w = ((t >> 1) ? dr : 1.f - dr) * ((t & 1) ? dc : 1.f - dc) * f;
        const unsigned p = (unsigned)r * (unsigned)a.nX + (unsigned)c;
        if (a.mask) w *= __ldg(a.mask + p);
        unsigned long long v[2 * Q];
        strip_load<Q, VEC>(volz + (size_t)p * a.vs, v, n, lz);
#pragma unroll
        for (int e = 0; e < 2 * Q; ++e) fma_pairs(acc[e], pk_pair(w, w), v[e]);
    }
}

// Blocks: 2^ashift angle tasks times 8 / 2^ashift neighbouring strips, which read the same pixels at about
// the same time.
//
// Stores lattice row j's sum: both angles' bins, for even N with the end sample of each (angle a sums k =
// 0 .. N - 1 of rows 0 .. N - 1, its partner k = 1 .. N of rows 1 .. N).
template <int Q, bool VEC>
__device__ __forceinline__ void strip_finish(const FastArgs& a, int2 task, bool ext, int j, const float* __restrict__ volz,
                                             int z0, int n, int lz, unsigned long long (&sum)[2 * Q]) {
    float* const here = a.sino + ((size_t)j * a.nA + task.x) * a.nZ + z0;
    float* const there = a.sino + ((size_t)(2 * a.C - j) * a.nA + task.y) * a.nZ + z0;
    if (!ext) {
        strip_store<Q, VEC>(here, sum, n, lz, a.vs == a.nZ, a.nZ - z0);
        if (task.y >= 0) strip_store<Q, VEC>(there, sum, n, lz, a.vs == a.nZ, a.nZ - z0);
        return;
    }
    const double4 tr = a.trig[task.x];
    const double rowb = fma(-tr.y, (double)j, tr.w), colb = fma(tr.x, (double)j, tr.z);
    const int N = a.nY;
    // (an end sample is formed by itself: its four taps would otherwise round the whole sum four times)
    for (int end = 0; end < 2; ++end) {
        if (end ? j == 0 : j == N) continue;
        unsigned long long o[2 * Q] = {};
        strip_sample<Q, VEC>(a, volz, fma(tr.x, (double)(end * N), rowb), fma(tr.y, (double)(end * N), colb), o, n, lz);
#pragma unroll
        for (int e = 0; e < 2 * Q; ++e) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(o[e]) : "l"(sum[e]));
        strip_store<Q, VEC>(end ? there : here, o, n, lz, a.vs == a.nZ, a.nZ - z0);
    }
}

// The sums run over all M bins of every listed pixel; a zero weight then spreads an infinity or a NaN to
// bins that do not sample it.  A strip with a non-finite sum is therefore done again sample by sample.
template <int Q, bool VEC, bool RAY>
__device__ __noinline__ void forward_strip_samples(const FastArgs& a, unsigned bx, unsigned by);

// The warp's place: angle task, first bin, lane's first slice and number of slices (float4s), false when idle.
template <int Q, bool VEC>
__device__ __forceinline__ bool strip_place(const FastArgs& a, unsigned bx, unsigned by, int2& task, bool& ext, int& j0,
                                            int& z0, int& n) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, sshift = 3 - a.ashift, LZ = 1 << a.lz_shift;
    const int ti = (int)((by << a.ashift) + (wp >> sshift));
    j0 = (int)(((bx / (unsigned)a.zchunks) << sshift) + (wp & ((1 << sshift) - 1))) * strip_bins(Q);
    if (ti >= a.ntasks) return false;
    task = a.tasks[ti];
    ext = task.y >= 0 && a.even;  // lattice row and sample N belong to the partner angle
    if (j0 > (ext ? a.nY : a.nY - 1)) return false;
    constexpr int per = VEC ? 4 : 1;
    z0 = (int)(bx % (unsigned)a.zchunks) * LZ * 4 * Q + per * (lane & (LZ - 1));
    n = 0;
#pragma unroll
    for (int e = 0; e < 4 * Q / per; ++e) n += z0 + per * LZ * e < a.nZ ? 1 : 0;
    if (n == 0) z0 = 0;
    return true;
}

// (param: the arguments where the launch left them, for the call at the end; a copy's address would keep it in memory)
//
// EXACT: the running sum takes up the current one after every group of pixels and keeps what its rounding drops, to
// the end.  For slice counts that the generic kernel gives more lanes per bin, or of which the strips have several
// groups (Sums in describe()): its lanes' partial sums are otherwise the more exact ones, the more so for volumes of
// zeros and ones, whose samples it adds without rounding (64^2 x 40 x 90 angles, relative to float64: generic 4.3e-8,
// 3.2e-8 for zeros and ones; strips 5.9e-8 and 4.4e-8, so 3.1e-8 and 2.7e-8; 17.3 -> 18.1 us, generic 32).
template <int Q, bool VEC, bool RAY, bool EXACT = false>
__device__ __forceinline__ void forward_strip_body(const FastArgs& a, const FastArgs& param, unsigned bx, unsigned by) {
    constexpr int M = strip_bins(Q), U = Q == 2 ? 3 : 4, VZ = 4 * Q;
    StripRing& ring = strip_ring();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    int2 task;
    bool ext;
    int j0, z0, n;
    if (!strip_place<Q, VEC>(a, bx, by, task, ext, j0, z0, n)) return;  // uniform per warp
    const int N = a.nY, jmax = ext ? N : N - 1;
    const int LZ = 1 << a.lz_shift, g = lane >> a.lz_shift, G = 32 >> a.lz_shift;
    const float* __restrict__ volz = a.vol + z0;

    const double4 tr = a.trig[task.x];
    const double c = tr.x, s = tr.y;
    const double B = fabs(c) + fabs(s);  // a bin touches pixels nearer than this along the detector
    const bool rmain = fabs(c) >= fabs(s);  // the rays run across rows (else across columns)
    const bool on_axis = fmin(fabs(c), fabs(s)) < 1e-12;
    const int kfirst = ext ? 1 : 0, klast = N - 1;

    // rows (columns) the strip's samples inside the image touch
    int mlo = INT_MAX, mhi = INT_MIN;
    if (lane < M && j0 + lane <= jmax) {
        const double rowb = fma(-s, (double)(j0 + lane), tr.w), colb = fma(c, (double)(j0 + lane), tr.z);
        int klo, khi;
        sample_range(rowb, colb, c, s, a.nY, a.nX, klast, klo, khi);
        klo = max(klo, kfirst);
        if (klo <= khi) {
            const double p0 = rmain ? fma(c, (double)klo, rowb) : fma(s, (double)klo, colb);
            const double p1 = rmain ? fma(c, (double)khi, rowb) : fma(s, (double)khi, colb);
            mlo = (int)floor(fmin(p0, p1));
            mhi = (int)floor(fmax(p0, p1)) + 1;
        }
    }
    mlo = max(__reduce_min_sync(kFull, mlo), 0);
    mhi = min(__reduce_max_sync(kFull, mhi), (rmain ? a.nY : a.nX) - 1);

    // sum: the batches finished so far; acc: the current one.  Adding batch by batch keeps the rounding of a
    // long ray's sum at well below a running sum's (64^2 x 40 x 90: 1.1e-7 -> 6.8e-8 relative to float64; 256^3 x 360: 3.8e-7 -> 1.0e-7).
    unsigned long long sum[M][VZ / 2], acc[M][VZ / 2];
    // U * G entries from head on: their rows into flight, and the bins' sums once the rows are there
    auto entries = [&](const float4* ep, float4 (&t)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = ep[u];
    };
    auto rows = [&](const float4 (&t)[U], unsigned long long (&v)[U][VZ / 2]) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            strip_load<Q, VEC>(volz + (size_t)__float_as_uint(t[u].w) * (unsigned)a.vs, v[u], n, LZ);
    };
    auto add1 = [&](const float4& t, const unsigned long long (&v)[VZ / 2]) {
        const float w[3] = {t.x, t.y, t.z};
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[m][e]) : "l"(pk_pair(w[m], w[m])), "l"(v[e]));
    };
    // one step: the next group's entries, one pixel of the waiting group while they arrive, the next
    // group's rows into flight, the rest of the waiting group
    auto step = [&](const float4* ep, float4 (&tn)[U], unsigned long long (&vn)[U][VZ / 2], const float4 (&tc)[U],
                    const unsigned long long (&vc)[U][VZ / 2]) {
        entries(ep, tn);
        add1(tc[0], vc[0]);
        rows(tn, vn);
#pragma unroll
        for (int u = 1; u < U; ++u) add1(tc[u], vc[u]);
    };

    const bool some = mlo <= mhi;
    int R = 1, lr = 0, slot = 0;
    if (some) {
        const double inv = 1.0 / (rmain ? c : s);
        const double slack = 1e-3 + 2e-6 * N;  // covers the float32 rounding of the edge
        const int S = (int)(((double)(M - 1) + 2.0 * B) * fabs(inv) + 2.0 * slack) + 1;  // pixels of one row under the strip
        R = 32 / S;
        lr = lane / S;
        slot = lane - lr * S;
        if (lane == 0) {
            StripGeo& q = ring.geo[wp];
            // the edge of the strip (widened by B) that has its least column (row)
            const double jlo = (rmain ? c > 0.0 : s < 0.0) ? (double)j0 - B : (double)(j0 + M - 1) + B;
            const double jo = fma(s, tr.w, -c * tr.z), ko = -fma(c, tr.w, s * tr.z);
            const double x = rmain ? -s : c, y = rmain ? c : -s, z = rmain ? c : s, w = rmain ? s : c;
            const double two32 = 4294967296.0, qx = rint(x * two32), qy = rint(y * two32), qz = rint(z * two32),
                         qw = rint(w * two32);
            q.coef = make_float4((float)x, (float)y, (float)z, (float)w);
            q.res = make_float4((float)(x - qx / two32), (float)(y - qy / two32), (float)(z - qz / two32), (float)(w - qw / two32));
            q.fix = make_uint4((unsigned)(long long)qx, (unsigned)(long long)qy, (unsigned)(long long)qz, (unsigned)(long long)qw);
            q.org = make_float4((float)jo, (float)ko, (float)((rmain ? s : c) * inv),
                                (float)((rmain ? (jlo - s * tr.w) * inv + tr.z : tr.w - (c * tr.z + jlo) * inv) - slack));
            q.fixorg = make_uint2((unsigned)(long long)rint(jo * two32), (unsigned)(long long)rint(ko * two32));
            q.cs = make_float4((float)c, (float)s, (float)(c - (double)(float)c), (float)(s - (double)(float)s));
        }
        __syncwarp();
    }

#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int e = 0; e < VZ / 2; ++e) sum[m][e] = acc[m][e] = 0ull;
    auto carry = [&]() {
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) {
                const unsigned long long was = sum[m][e];
                asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[m][e]) : "l"(acc[m][e]));
                acc[m][e] = EXACT ? dropped(was, sum[m][e], acc[m][e]) : 0ull;
            }
    };
    if (some) {
        float4 t0[U], t1[U];
        unsigned long long v0[U][VZ / 2], v1[U][VZ / 2];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            t0[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) v0[u][e] = 0ull;
        }
        // the ring holds whole rounds of two groups, so a group never wraps
        const int round = 2 * U * G, size = kStripRing - kStripRing % round;
        const float4* const first = &ring.e[wp][g * U];
        int head = 0, tail = 0, wait = 0;  // next to work off, next free, number between them
        for (int m0 = mlo; m0 <= mhi; m0 += R) {
            const StripGeo& q = ring.geo[wp];
            const int mi = m0 + lr;
            const float fm = (float)mi;
            const int ot = (int)ceilf(fmaf(fm, q.org.z, q.org.w)) + slot;
            const unsigned pix = rmain ? (unsigned)mi * (unsigned)a.nX + (unsigned)ot : (unsigned)ot * (unsigned)a.nX + (unsigned)mi;
            float W[3] = {0.f, 0.f, 0.f};
            bool listed = false;
            if (lr < R && mi <= mhi && (unsigned)ot < (unsigned)N) {
                const float fo = (float)ot;
                // nearest lattice point (Jn, Kn) and the pixel's offset from it
                const float4 co = q.coef, re = q.res;
                const uint4 fx = q.fix;
                const unsigned um = (unsigned)mi, uo = (unsigned)ot;
                const float dj = fmaf((float)(int)(fx.x * um + fx.y * uo + q.fixorg.x), 2.3283064e-10f, fmaf(re.x, fm, re.y * fo));
                const float dk = fmaf((float)(int)(fx.z * um + fx.w * uo + q.fixorg.y), 2.3283064e-10f, fmaf(re.z, fm, re.w * fo));
                const float Jn = rintf(fmaf(co.x, fm, fmaf(co.y, fo, q.org.x)) - dj);
                const float Kn = rintf(fmaf(co.z, fm, fmaf(co.w, fo, q.org.y)) - dk);
                // cos and sin to more than float32: their rounding would scale every weight of the angle
                const float4 cs = q.cs;
                // samples Kn - 1 .. Kn + 1; one outside the ray is moved away, where its weight is zero
                float ck[3], sk[3];
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float kb = Kn + (float)(b - 1);
                    const float kk = (kb >= (float)kfirst && kb <= (float)klast) ? (float)(b - 1) - dk : 1e9f;
                    ck[b] = fmaf(cs.x, kk, cs.z * kk);
                    sk[b] = fmaf(cs.y, kk, cs.w * kk);
                }
                const float jn = (float)j0 - Jn;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float d = (jn + (float)m) - dj;
                    float sent = 0.f;
                    bool dark = j0 + m > jmax;
                    if (RAY) {
                        const float t = (float)(j0 + m - a.C);
                        if (fabsf(t) > a.R) dark = true;
                        else sent = -sqrtf(a.R * a.R - t * t);
                    }
                    const float sd = -fmaf(cs.y, d, cs.w * d), cd = fmaf(cs.x, d, cs.z * d);
                    float w = 0.f;
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        float h = __saturatef(1.f - fabsf(ck[b] + sd)) * __saturatef(1.f - fabsf(sk[b] + cd));
                        if (RAY && h != 0.f) h *= ray_factor(Kn + (float)(b - 1 - a.C), sent, a.alpha);
                        w += h;
                    }
                    W[m] = dark ? 0.f : w;
                    listed |= W[m] != 0.f;
                }
                // on an axis the samples' float64 rounding may touch the next row or column with a weight that is
                // zero here; listing those pixels too lets an infinity in them through
                listed |= on_axis;
                if (a.mask) {
                    const float f = __ldg(a.mask + pix);
#pragma unroll
                    for (int m = 0; m < M; ++m) W[m] *= f;
                }
            }
            const unsigned has = __ballot_sync(kFull, listed);
            if (listed) {
                const int at = tail + __popc(has & ((1u << lane) - 1u));
                ring.e[wp][at < size ? at : at - size] = make_float4(W[0], W[1], W[2], __uint_as_float(pix));
            }
            const int cnt = __popc(has);
            tail = tail + cnt < size ? tail + cnt : tail + cnt - size;
            wait += cnt;
            __syncwarp();
            for (; wait >= round; wait -= round) {
                step(first + head, t1, v1, t0, v0);
                if (EXACT) carry();
                step(first + head + U * G, t0, v0, t1, v1);
                if (EXACT) carry();
                head = head + round < size ? head + round : 0;
            }
            if (!EXACT) carry();
            __syncwarp();  // the entries worked off are free again
        }
        if (wait > 0) {  // the rest, filled up with entries of no weight (and the first pixel's row)
            for (int k = wait + lane; k < round; k += 32) ring.e[wp][head + k] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
            step(first + head, t1, v1, t0, v0);
            if (EXACT) carry();
            step(first + head + U * G, t0, v0, t1, v1);
            if (EXACT) carry();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) add1(t0[u], v0[u]);
        carry();
        __syncwarp();
        float bad = 0.f;
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) {
                float lo, hi;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(sum[m][e]));
                // (slices past the volume hold anything)
                if (VEC ? e / 2 < n : 2 * e < n) bad = fmaf(lo, 0.f, bad);
                if (VEC ? e / 2 < n : 2 * e + 1 < n) bad = fmaf(hi, 0.f, bad);
            }
        if (__any_sync(kFull, bad != 0.f)) {
            forward_strip_samples<Q, VEC, RAY>(param, bx, by);
            return;
        }
    }

    if constexpr (Q == 1)  // the groups' parts
        for (int off = LZ; off < 32; off <<= 1)
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int e = 0; e < VZ / 2; ++e) {
                    const unsigned long long t = __shfl_xor_sync(kFull, sum[m][e], off);
                    if constexpr (EXACT) {
                        acc[m][e] = add_pairs(acc[m][e], __shfl_xor_sync(kFull, acc[m][e], off));
                        acc[m][e] = add_pairs(acc[m][e], two_sum(sum[m][e], t));
                    } else {
                        sum[m][e] = add_pairs(sum[m][e], t);
                    }
                }
    if constexpr (EXACT)
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) sum[m][e] = add_finite(sum[m][e], acc[m][e]);
    if (n == 0 || g != 0) return;
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (j0 + m <= jmax) strip_finish<Q, VEC>(a, task, ext, j0 + m, volz, z0, n, LZ, sum[m]);
}

template <int Q, bool VEC, bool RAY>
__device__ __noinline__ void forward_strip_samples(const FastArgs& a, unsigned bx, unsigned by) {
    int2 task;
    bool ext;
    int j0, z0, n;
    if (!strip_place<Q, VEC>(a, bx, by, task, ext, j0, z0, n)) return;
    const int LZ = 1 << a.lz_shift, N = a.nY;
    if (n == 0 || (threadIdx.x & 31) >> a.lz_shift) return;
    const float* __restrict__ volz = a.vol + z0;
    const double4 tr = a.trig[task.x];
    for (int m = 0; m < strip_bins(Q) && j0 + m <= (ext ? N : N - 1); ++m) {
        const int j = j0 + m;
        const double rowb = fma(-tr.y, (double)j, tr.w), colb = fma(tr.x, (double)j, tr.z);
        unsigned long long acc[2 * Q] = {};
        int klo, khi;
        sample_range(rowb, colb, tr.x, tr.y, a.nY, a.nX, N - 1, klo, khi);
        float sent = 0.f;
        if (RAY) {
            const float t = (float)(j - a.C);
            if (fabsf(t) > a.R) khi = -1;
            else sent = -sqrtf(a.R * a.R - t * t);
        }
        for (int k = max(klo, ext ? 1 : 0); k <= khi; ++k)
            strip_sample<Q, VEC>(a, volz, fma(tr.x, (double)k, rowb), fma(tr.y, (double)k, colb), acc, n, LZ,
                                 RAY ? ray_factor((float)(k - a.C), sent, a.alpha) : 1.f);
        strip_finish<Q, VEC>(a, task, ext, j, volz, z0, n, LZ, acc);
    }
}

// 128 registers, two blocks per SM: rows in flight per warp hide more than a third block does (three at 80
// registers: 0.88 against 0.82 ms at 256^3 x 360)
template <int Q, bool VEC, bool RAY, bool EXACT = false>
__global__ void __launch_bounds__(256, 2) k_forward_strip(const __grid_constant__ FastArgs a) {
    forward_strip_body<Q, VEC, RAY, EXACT>(a, a, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------------------
// Matched transpose by pixel blocks.
//
// One warp owns a 2 x 2 block of pixels over the slices of one z chunk.  Detector bin j of an angle gives
// pixel p W(j, p) times its row, W the strip forward's weights (every sample k of the bin with the pixel under
// its bilinear kernel), so the block needs the at most five bins within 1.5 (|cos| + |sin|) of its centre, 3.6
// on average, where a pixel alone needs 2.3: 0.9 rows per pixel and angle.  The warp lists the rows of six
// angles at a time (lanes: angle x bin), weights for the four pixels, and works the ring off like the strips.
// ---------------------------------------------------------------------------
constexpr int kBlockBins = 5;

struct BlockRing {
    float4 w[kWarpsPerBlock][kStripRing];    // the four pixels' weights
    unsigned o[kWarpsPerBlock][kStripRing];  // the row: bin * angles + angle
};

__device__ __forceinline__ BlockRing& block_ring() {
    __shared__ __align__(16) BlockRing r;
    return r;
}

// The warp's block (its first pixel), lane's first slice and number of slices (float4s), false when idle.  A
// thread block covers 4 x 2 blocks of one z chunk, whose warps read the same rows at about the same time.
template <int Q, bool VEC>
__device__ __forceinline__ bool block_place(const Args& a, unsigned bx, int& i, int& j, int& z0, int& n) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, LZ = 1 << a.lz_shift;
    const unsigned tile = bx / (unsigned)a.zchunks, ntx = (unsigned)((a.nX + 7) >> 3);
    i = 2 * (int)(tile / ntx * 2 + (wp >> 2));
    j = 2 * (int)(tile % ntx * 4 + (wp & 3));
    if (i >= a.nY || j >= a.nX) return false;
    constexpr int per = VEC ? 4 : 1;
    z0 = (int)(bx % (unsigned)a.zchunks) * LZ * 4 * Q + per * (lane & (LZ - 1));
    n = 0;
#pragma unroll
    for (int e = 0; e < 4 * Q / per; ++e) n += z0 + per * LZ * e < a.nZ ? 1 : 0;
    if (n == 0) z0 = 0;
    return true;
}

// Weight of bin J for the pixel at lattice position (J0 + dj, K0 + dk): its samples within one pixel of it.
// cs: cos and sin and (EXACT) what their float32 values leave out.
template <bool RAY, bool EXACT>
__device__ __forceinline__ float bin_weight(const Args& a, float4 cs, float d, float dk, float K0, float sent) {
    const float kc = rintf(dk);
    const float sd = EXACT ? fmaf(cs.y, d, cs.w * d) : cs.y * d, cd = EXACT ? fmaf(cs.x, d, cs.z * d) : cs.x * d;
    float w = 0.f;
#pragma unroll
    for (int b = -1; b <= 1; ++b) {
        const float k = K0 + (kc + (float)b);
        const float kk = (k >= 0.f && k <= (float)(a.nY - 1)) ? (kc + (float)b) - dk : 1e9f;  // outside: no weight
        float h = __saturatef(1.f - fabsf(fmaf(cs.x, kk, EXACT ? fmaf(cs.z, kk, -sd) : -sd))) *
                  __saturatef(1.f - fabsf(fmaf(cs.y, kk, EXACT ? fmaf(cs.w, kk, cd) : cd)));
        if (RAY && h != 0.f) h *= ray_factor(k - (float)a.C, sent, a.alpha);
        w += h;
    }
    return w;
}

template <int Q, bool VEC, bool RAY>
__device__ __noinline__ void adjoint_block_rows(const Args& a, unsigned bx);

// EXACT: as for the strips, summing every six angles' rows on their own, with cos and sin to more than float32 (the
// generic kernel forms its weights in float64): 64^2 x 40 x 90 1.0e-7 -> 4.0e-8 (generic 4.2e-8), 18.6 -> 20.4 us.
template <int Q, bool VEC, bool RAY, bool EXACT = false>
__device__ __forceinline__ void adjoint_block_body(const Args& a, const Args& param, unsigned bx) {
    constexpr int U = Q == 2 ? 2 : 4, VZ = 4 * Q, R = 32 / kBlockBins;
    BlockRing& ring = block_ring();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    int i0, j0, z0, n;
    if (!block_place<Q, VEC>(a, bx, i0, j0, z0, n)) return;  // uniform per warp
    const int LZ = 1 << a.lz_shift, g = lane >> a.lz_shift, G = 32 >> a.lz_shift;
    const float* __restrict__ bz = a.in + z0;

    unsigned long long acc[4][VZ / 2], sum[4][EXACT ? VZ / 2 : 1];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < VZ / 2; ++e) acc[q][e] = sum[q][EXACT ? e : 0] = 0ull;
    auto carry = [&]() {
        if constexpr (EXACT) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int e = 0; e < VZ / 2; ++e) {
                    const unsigned long long was = sum[q][e];
                    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[q][e]) : "l"(acc[q][e]));
                    acc[q][e] = dropped(was, sum[q][e], acc[q][e]);
                }
        }
    };
    auto entries = [&](int at, float4 (&t)[U], unsigned (&o)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            t[u] = ring.w[wp][at + u];
            o[u] = ring.o[wp][at + u];
        }
    };
    auto rows = [&](const unsigned (&o)[U], unsigned long long (&v)[U][VZ / 2]) {
#pragma unroll
        for (int u = 0; u < U; ++u) strip_load<Q, VEC>(bz + (size_t)o[u] * (unsigned)a.zs, v[u], n, LZ);
    };
    auto add1 = [&](const float4& t, const unsigned long long (&v)[VZ / 2]) {
        const float w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) fma_pairs(acc[q][e], pk_pair(w[q], w[q]), v[e]);
    };
    auto step = [&](int at, float4 (&tn)[U], unsigned long long (&vn)[U][VZ / 2], const float4 (&tc)[U],
                    const unsigned long long (&vc)[U][VZ / 2]) {
        unsigned o[U];
        entries(at, tn, o);
        add1(tc[0], vc[0]);
        rows(o, vn);
#pragma unroll
        for (int u = 1; u < U; ++u) add1(tc[u], vc[u]);
    };
    float4 t0[U], t1[U];
    unsigned long long v0[U][VZ / 2], v1[U][VZ / 2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        t0[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int e = 0; e < VZ / 2; ++e) v0[u][e] = 0ull;
    }
    const int round = 2 * U * G, size = kStripRing - kStripRing % round;  // whole rounds: a group never wraps
    int head = 0, tail = 0, wait = 0;
    const int la = lane / kBlockBins, slot = lane - la * kBlockBins;
    for (int th0 = 0; th0 < a.nA; th0 += R) {
        const int th = th0 + la;
        float W[4] = {0.f, 0.f, 0.f, 0.f};
        unsigned row = 0;
        bool listed = false;
        if (la < R && th < a.nA) {
            const double4 tr = a.trig[th];
            const double ri = (double)i0 - tr.w, ci = (double)j0 - tr.z;
            const double Jf = fma(-tr.y, ri, tr.x * ci), Kf = fma(tr.x, ri, tr.y * ci);
            const double Jn = rint(Jf), Kn = rint(Kf);
            const float cf = (float)tr.x, sf = (float)tr.y;
            const float4 cs = make_float4(cf, sf, EXACT ? (float)(tr.x - (double)cf) : 0.f, EXACT ? (float)(tr.y - (double)sf) : 0.f);
            const float dj = (float)(Jf - Jn), dk = (float)(Kf - Kn);
            // bins from 1.5 (|cos| + |sin|) below the block's centre on
            const float lo = dj + 0.5f * (cf - sf) - 1.5f * (fabsf(cf) + fabsf(sf));
            const float jr = ceilf(lo - 1e-5f) + (float)slot;  // the bin, from Jn
            const int J = (int)Jn + (int)jr;
            float sent = 0.f;
            bool lit = (unsigned)J < (unsigned)a.nX;
            if (RAY) {
                const float t = (float)(J - a.C);
                if (fabsf(t) > a.R) lit = false;
                else sent = -sqrtf(a.R * a.R - t * t);
            }
            if (lit) {
                row = (unsigned)J * (unsigned)a.nA + (unsigned)th;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float pr = (float)(q >> 1), pc = (float)(q & 1);  // the pixel, from the block's first
                    const float d = jr - (dj + (pc * cf - pr * sf)), k = dk + (pr * cf + pc * sf);
                    W[q] = bin_weight<RAY, EXACT>(a, cs, d, k, (float)Kn, sent);
                    listed |= W[q] != 0.f;
                }
            }
        }
        const unsigned has = __ballot_sync(kFull, listed);
        if (listed) {
            int at = tail + __popc(has & ((1u << lane) - 1u));
            at = at < size ? at : at - size;
            ring.w[wp][at] = make_float4(W[0], W[1], W[2], W[3]);
            ring.o[wp][at] = row;
        }
        const int cnt = __popc(has);
        tail = tail + cnt < size ? tail + cnt : tail + cnt - size;
        wait += cnt;
        __syncwarp();
        for (; wait >= round; wait -= round) {
            step(head + g * U, t1, v1, t0, v0);
            step(head + U * G + g * U, t0, v0, t1, v1);
            head = head + round < size ? head + round : 0;
        }
        carry();
        __syncwarp();  // the entries worked off are free again
    }
    if (wait > 0) {  // the rest, filled up with entries of no weight (and the first row)
        for (int k = wait + lane; k < round; k += 32) {
            ring.w[wp][head + k] = make_float4(0.f, 0.f, 0.f, 0.f);
            ring.o[wp][head + k] = 0u;
        }
        __syncwarp();
        step(head + g * U, t1, v1, t0, v0);
        step(head + U * G + g * U, t0, v0, t1, v1);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) add1(t0[u], v0[u]);
    carry();
    if constexpr (EXACT) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) acc[q][e] = sum[q][e];
    }
    __syncwarp();  // (the next call of a persistent block refills the ring)
    float bad = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < VZ / 2; ++e) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[q][e]));
            if (VEC ? e / 2 < n : 2 * e < n) bad = fmaf(lo, 0.f, bad);
            if (VEC ? e / 2 < n : 2 * e + 1 < n) bad = fmaf(hi, 0.f, bad);
        }
    if (__any_sync(kFull, bad != 0.f)) {  // as in the strips: an infinity only where it is sampled
        adjoint_block_rows<Q, VEC, RAY>(param, bx);
        return;
    }
    if constexpr (Q == 1)
        for (int off = LZ; off < 32; off <<= 1)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int e = 0; e < VZ / 2; ++e) {
                    const unsigned long long t = __shfl_xor_sync(kFull, acc[q][e], off);
                    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc[q][e]) : "l"(t));
                }
    if (n == 0 || g != 0) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = i0 + (q >> 1), j = j0 + (q & 1);
        if (i >= a.nY || j >= a.nX) continue;
        const size_t p = (size_t)i * a.nX + j;
        if (a.mask) {
            const float m = __ldg(a.mask + p);
            const unsigned long long mm = pk_pair(m, m);
#pragma unroll
            for (int e = 0; e < VZ / 2; ++e) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[q][e]) : "l"(mm));
        }
        strip_store<Q, VEC>(a.out + p * a.nZ + z0, acc[q], n, LZ, a.zs == a.nZ, a.nZ - z0);
    }
}

// The block pixel by pixel, reading only the rows whose samples have the pixel among their taps (decided on
// the forward's float64 coordinates).
template <int Q, bool VEC, bool RAY>
__device__ __noinline__ void adjoint_block_rows(const Args& a, unsigned bx) {
    int i0, j0, z0, n;
    if (!block_place<Q, VEC>(a, bx, i0, j0, z0, n)) return;
    const int LZ = 1 << a.lz_shift;
    if (n == 0 || (threadIdx.x & 31) >> a.lz_shift) return;
    const float* __restrict__ bz = a.in + z0;
    for (int q = 0; q < 4; ++q) {
        const int i = i0 + (q >> 1), j = j0 + (q & 1);
        if (i >= a.nY || j >= a.nX) continue;
        unsigned long long acc[2 * Q] = {};
        for (int th = 0; th < a.nA; ++th) {
            const double4 tr = a.trig[th];
            const double c = tr.x, s = tr.y, ri = (double)i - tr.w, ci = (double)j - tr.z;
            const int Jn = __double2int_rn(fma(-s, ri, c * ci)), Kn = __double2int_rn(fma(c, ri, s * ci));
            for (int J = max(Jn - 1, 0); J <= min(Jn + 1, a.nX - 1); ++J) {
                const float t = (float)(J - a.C);
                if (RAY && fabsf(t) > a.R) continue;
                const float sent = RAY ? -sqrtf(a.R * a.R - t * t) : 0.f;
                const double rowb = fma(-s, (double)J, tr.w), colb = fma(c, (double)J, tr.z);
                float w = 0.f;
                for (int K = max(Kn - 2, 0); K <= min(Kn + 2, a.nY - 1); ++K) {
                    const double row = fma(c, (double)K, rowb), col = fma(s, (double)K, colb);
                    const double fr = floor(row), fc = floor(col);
                    const int r0 = (int)fr, c0 = (int)fc;
                    if (!(i == r0 || (row > fr && i == r0 + 1)) || !(j == c0 || (col > fc && j == c0 + 1))) continue;
                    const float dr = (float)(row - fr), dc = (float)(col - fc);
                    float h = (i == r0 ? 1.f - dr : dr) * (j == c0 ? 1.f - dc : dc);
                    if (RAY) h *= ray_factor((float)(K - a.C), sent, a.alpha);
                    w += h;
                }
                if (w == 0.f) continue;
                unsigned long long v[2 * Q];
                strip_load<Q, VEC>(bz + ((size_t)J * a.nA + th) * a.zs, v, n, LZ);
#pragma unroll
                for (int e = 0; e < 2 * Q; ++e) fma_pairs(acc[e], pk_pair(w, w), v[e]);
            }
        }
        const size_t p = (size_t)i * a.nX + j;
        if (a.mask) {
            const float m = __ldg(a.mask + p);
#pragma unroll
            for (int e = 0; e < 2 * Q; ++e) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[e]) : "l"(pk_pair(m, m)));
        }
        strip_store<Q, VEC>(a.out + p * a.nZ + z0, acc, n, LZ, a.zs == a.nZ, a.nZ - z0);
    }
}

template <int Q, bool VEC, bool RAY, bool EXACT = false>
__global__ void __launch_bounds__(256, 2) k_adjoint_block(const __grid_constant__ Args a) {
    adjoint_block_body<Q, VEC, RAY, EXACT>(a, a, blockIdx.x);
}

}  // namespace
}  // namespace vam
