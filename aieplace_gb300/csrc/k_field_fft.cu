// Electrostatic field solve by fast transforms, FP32.
//
// Restates replace::FFT::doFFT (python/AIEmath/fft_replace/fft.cpp:204-299)
// and Placer::compute_a_uv_DCT / compute_eField_DCT (vck5000/host/src/
// AIEplace.cpp:752-934): 2-D DCT-II of the density, halved edge rows,
// 4/(Mx My), phi = a/(wx^2+wy^2), Ex = S^T (phi wx) C, Ey = C^T (phi wy) S.
//
// Three passes over the map, each a launch of complex FFTs of length m in
// shared memory, two real lines (or a line's two fields) to a complex one:
//   P1  T[x][v] = sum_y d[x][y] cos(pi v (y+1/2)/m), rows x and x+1 together;
//   P2  per column v: a[u] = sum_x T[x][v] cos(pi u (x+1/2)/m) (columns v, v+1
//       together), the spectral step, then along x back
//       ux[x] = sum_u phi wx sin(..), uy[x] = sum_u phi wy cos(..) together;
//   P3  per row x: Ex[y] = sum_v ux cos(..), Ey[y] = sum_v uy sin(..) together.
// The cosine transforms run through a complex FFT of the same length after
// the reordering v[n] = x[2n], v[m-1-n] = x[2n+1] (J. Makhoul, "A fast cosine
// transform in one and two dimensions", 1980): X[k] = Re(h_k V[k]), h_k =
// exp(-i pi k / 2m), and back with W[k] = conj(h_k) (X[k] - i X[m-k]) / 2; a
// sine sum is the cosine sum of the reversed coefficients with alternating
// signs.  15 m^2 log2 m operations instead of the 12 m^3 of dense transform
// matrices, and a rounding error that grows with log m instead of sqrt(m)
// (2-norm against 64 bits at m = 1024: 2.0e-7; the matrices' 1.3e-6).
//
// Bound: latency (a chain of shared-memory exchanges per FFT, all maps in
// L2), so the lines are spread over as many blocks as there are: two FFTs a
// block from 256 points up.  T and U are kept in tiles of a few rows,
// T[x/4][v][x%4] and U[x/2][v][x%2] (ux, uy), so that the passes along y
// read and write whole rows of tiles and the pass along x whole 32-byte
// sectors; within 64 registers a thread, so that every block of a pass is
// resident at once (72: 15.1 us for P2, a second wave).  Measured (m = 1024, launches
// alone under ncu): 7.4 + 14.4 + 9.4 us, the first 15.0 with the density in it; shared
// memory 44-64% busy.  The solve alone in a loop of launches, against the dense
// contractions on the FP32 pipes: 18 and 460 us; at 512 11 and 125.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "../../include/aieplace.h"
#include "ap_density.cuh"
#include "ap_kernels.h"

namespace ap {

namespace {

// ---- plan of a length-m FFT ---------------------------------------------------
// m = 2^k (64..4096), or 2^k p with p = 3, 5, 7 (the sizes of the
// allocation-free entry point): radix-8 stages and a last one of 2 or 4, or
// radix-4 stages, one of 2 and one of p.  A thread holds E points, so m / E
// threads share an FFT.
__host__ __device__ constexpr int odd_part(int m) {
    while (m % 2 == 0) m /= 2;
    return m;
}
__host__ __device__ constexpr int fft_radix(int m, int s) {
    const int odd = odd_part(m), base = odd == 1 ? 8 : 4;
    int two = m / odd;
    for (; s > 0 && two > 1; --s) two /= two < base ? two : base;
    return two > 1 ? (two < base ? two : base) : (s == 0 ? odd : 1);
}
__host__ __device__ constexpr int fft_stages(int m) {
    int n = 0;
    for (int p = 1; p < m; p *= fft_radix(m, n), ++n) {
    }
    return n;
}
__host__ __device__ constexpr int fft_ns(int m, int s) {  // product of the radices before stage s
    int p = 1;
    for (int t = 0; t < s; ++t) p *= fft_radix(m, t);
    return p;
}
// twiddles of stage s >= 1, exp(-2 pi i k r / (R ns)), at [off + (r - 1) ns + k]
__host__ __device__ constexpr int fft_tw_off(int m, int s) {
    int off = 0;
    for (int t = 1; t < s; ++t) off += (fft_radix(m, t) - 1) * fft_ns(m, t);
    return off;
}
__host__ __device__ constexpr int fft_points(int m) {  // E
    return odd_part(m) > 1 ? 4 * odd_part(m) : (m > 2048 ? 16 : 8);
}
__host__ __device__ constexpr int fft_threads(int m) { return m / fft_points(m); }
// the grid small enough for one block (dense_solve)
constexpr int kDense = 32;
// float2 table: m entries of twiddles (fewer are used), then h_k, k < m; for
// kDense bins the cosine and the sine matrix instead
__host__ __device__ constexpr int field_table_len(int m) { return m == kDense ? m * m : 2 * m; }

__global__ void field_table_kernel(float2 *tab, float *wx, float *wy, int m, float ratio) {
    const double pi = 3.14159265358979323846;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double s, c;
    if (m == kDense && t < m * m) {  // C[k][i], then S[k][i]
        sincospi((double)(t / m) * (t % m + 0.5) / m, &s, &c);
        reinterpret_cast<float *>(tab)[t] = (float)c;
        reinterpret_cast<float *>(tab)[m * m + t] = (float)s;
    }
    if (t >= m) return;
    wx[t] = (float)(pi * t / m);
    wy[t] = (float)(pi * t / m * ratio);
    if (m == kDense) return;
    int st = 1;
    const int n = fft_stages(m);
    while (st < n && t >= fft_tw_off(m, st + 1)) ++st;
    if (st < n) {
        const int e = t - fft_tw_off(m, st), ns = fft_ns(m, st);
        sincospi(2.0 * (double)(e % ns) * (double)(e / ns + 1) / (double)(ns * fft_radix(m, st)), &s, &c);
        tab[t] = make_float2((float)c, (float)-s);
    }
    sincospi((double)t / (2.0 * m), &s, &c);
    tab[m + t] = make_float2((float)c, (float)-s);
}

// ---- butterflies --------------------------------------------------------------
// Products are fused by hand: left to the compiler, which of two products an
// FMA takes may differ between the kernels that share this code, and with it
// the last bit of a batch's result against the instance alone.
__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a w, or a conj(w) in the inverse transform
template <bool INV>
__device__ __forceinline__ float2 twiddle(float2 a, float2 w) {
    const float p = __fmul_rn(a.y, w.y), q = __fmul_rn(a.x, w.y);
    return INV ? make_float2(fmaf(a.x, w.x, p), fmaf(a.y, w.x, -q)) : make_float2(fmaf(a.x, w.x, -p), fmaf(a.y, w.x, q));
}
template <bool INV>
__device__ __forceinline__ float2 quarter(float2 a) {  // a (-i), inverse: a i
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3) {
    const float2 a = v0 + v2, b = v0 - v2, c = v1 + v3, d = quarter<INV>(v1 - v3);
    v0 = a + c;
    v2 = a - c;
    v1 = b + d;
    v3 = b - d;
}

// cos and sin of 2 pi k / p, p = 3, 5, 7 (folded at compile time)
__host__ __device__ constexpr float odd_cos(int p, int k) {
    k = k > p - k ? p - k : k;  // 0 .. (p - 1) / 2
    if (k == 0) return 1.f;
    if (p == 3) return -0.5f;
    if (p == 5) return k == 1 ? 0.309016994374947424f : -0.809016994374947424f;
    return k == 1 ? 0.623489801858733531f : k == 2 ? -0.222520933956314404f : -0.900968867902419126f;
}
__host__ __device__ constexpr float odd_sin(int p, int k) {
    if (k > p - k) return -odd_sin(p, p - k);
    if (k == 0) return 0.f;
    if (p == 3) return 0.866025403784438647f;
    if (p == 5) return k == 1 ? 0.951056516295153572f : 0.587785252292473129f;
    return k == 1 ? 0.781831482468029809f : k == 2 ? 0.974927912181823607f : 0.433883739117558120f;
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 2) {
        const float2 a = v[0];
        v[0] = a + v[1];
        v[1] = a - v[1];
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        constexpr float h = 0.707106781186547524f;
        dft4<INV>(v[0], v[2], v[4], v[6]);
        dft4<INV>(v[1], v[3], v[5], v[7]);
        const float2 o1 = v[3], o3 = v[7];
        // o1, o3 times exp(-+ i pi / 4), exp(-+ 3 i pi / 4): w1 h, w3 h
        const float2 w1 = INV ? make_float2(o1.x - o1.y, o1.x + o1.y) : make_float2(o1.x + o1.y, o1.y - o1.x);
        const float2 w2 = quarter<INV>(v[5]);
        const float2 w3 = INV ? make_float2(-(o3.x + o3.y), o3.x - o3.y) : make_float2(o3.y - o3.x, -(o3.x + o3.y));
        const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = e0 + o0;
        v[4] = e0 - o0;
        v[1] = make_float2(fmaf(h, w1.x, e1.x), fmaf(h, w1.y, e1.y));
        v[5] = make_float2(fmaf(-h, w1.x, e1.x), fmaf(-h, w1.y, e1.y));
        v[2] = e2 + w2;
        v[6] = e2 - w2;
        v[3] = make_float2(fmaf(h, w3.x, e3.x), fmaf(h, w3.y, e3.y));
        v[7] = make_float2(fmaf(-h, w3.x, e3.x), fmaf(-h, w3.y, e3.y));
    } else {
        // R odd prime: sums and differences of the pairs q, R - q
        constexpr int H = (R - 1) / 2;
        float2 p[H], m[H];
#pragma unroll
        for (int q = 0; q < H; ++q) {
            p[q] = v[q + 1] + v[R - 1 - q];
            m[q] = v[q + 1] - v[R - 1 - q];
        }
        const float2 v0 = v[0];
#pragma unroll
        for (int q = 0; q < H; ++q) v[0] = v[0] + p[q];
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            float2 a = v0, b = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < H; ++q) {
                const float c = odd_cos(R, (r * (q + 1)) % R), s = odd_sin(R, (r * (q + 1)) % R);
                a = make_float2(fmaf(c, p[q].x, a.x), fmaf(c, p[q].y, a.y));
                b = make_float2(fmaf(s, m[q].x, b.x), fmaf(s, m[q].y, b.y));
            }
            b = quarter<INV>(b);  // -i sum (inverse: +i)
            v[r] = a + b;
            v[R - r] = a - b;
        }
    }
}

// ---- FFT of a slot ------------------------------------------------------------
// A block of NT threads holds S = NT / (m / E) FFTs ("slots"), slot `slot`'s
// points at sm + slot * fft_slot(m), element i at fft_pad(i) (no bank
// conflicts at the stages' power-of-two strides).
// No sum of two indices below carries into bit 4 (one of them is a multiple of
// the stride that bounds the other), so fft_pad(i + c) = fft_pad(i) + fft_pad(c)
// and a constant c becomes an offset of the access.
__host__ __device__ constexpr int fft_pad(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int fft_slot(int m) { return m + m / 16; }
__host__ __device__ constexpr int fft_slots(int m, int nt) { return nt / fft_threads(m); }
__host__ __device__ constexpr int fft_smem(int m, int nt) {
    return fft_slots(m, nt) * fft_slot(m) * (int)sizeof(float2);
}

// barrier among the threads of a slot (of a warp, or of the block; every
// thread of the block takes part)
template <int M>
__device__ __forceinline__ void fft_sync() {
    if constexpr (fft_threads(M) <= 32)
        __syncwarp();
    else
        __syncthreads();
}

template <int M>
__device__ __forceinline__ void slot_load(float2 (&x)[fft_points(M)], const float2 *sm, int j) {
    sm += fft_pad(j);
#pragma unroll
    for (int q = 0; q < fft_points(M); ++q) x[q] = sm[fft_pad(q * fft_threads(M))];
}
template <int M>
__device__ __forceinline__ void slot_store(const float2 (&x)[fft_points(M)], float2 *sm, int j) {
    sm += fft_pad(j);
#pragma unroll
    for (int q = 0; q < fft_points(M); ++q) sm[fft_pad(q * fft_threads(M))] = x[q];
}

// Stage ST onwards of the FFT of x[q] = element j + q m/E; the result comes
// back in the same order.  Stockham: the output of butterfly jj, point r goes
// to (jj / ns) ns R + jj % ns + r ns.  `on`: false for the threads of a slot
// without work, which only meet the barriers.
template <int M, bool INV, int ST>
__device__ __forceinline__ void fft_stage(float2 (&x)[fft_points(M)], float2 *sm, int j, const float2 *tw,
                                          bool on = true) {
    constexpr int E = fft_points(M), TPF = M / E, R = fft_radix(M, ST), NS = fft_ns(M, ST), B = E / R;
    static_assert(E % R == 0, "whole butterflies per thread");
    if (on) {
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const float2 *w = tw + fft_tw_off(M, ST) + (j + b * TPF) % NS;
            float2 v[R];
            v[0] = x[b];
#pragma unroll
            for (int r = 1; r < R; ++r) {
                v[r] = x[b + r * B];
                if constexpr (NS > 1) v[r] = twiddle<INV>(v[r], __ldg(w + (r - 1) * NS));
            }
            dft<R, INV>(v);
#pragma unroll
            for (int r = 0; r < R; ++r) x[b + r * B] = v[r];
        }
    }
    if constexpr (NS * R < M) {
        fft_sync<M>();  // every earlier read of the slot is done
        if (on) {
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const int jj = j + b * TPF;
                float2 *o = sm + fft_pad((jj / NS) * (NS * R) + jj % NS);
#pragma unroll
                for (int r = 0; r < R; ++r) o[fft_pad(r * NS)] = x[b + r * B];
            }
        }
        fft_sync<M>();
        if (on) slot_load<M>(x, sm, j);
        fft_stage<M, INV, ST + 1>(x, sm, j, tw, on);
    }
}

// the two real lines a + i b behind one complex DFT: cosine coefficients of
// both at k from Z[k] and Zp = Z[m - k]
__device__ __forceinline__ float2 split_cos(float2 z, float2 zp, float2 h) {
    const float2 s = z + zp, d = z - zp;
    return make_float2(0.5f * fmaf(h.x, s.x, -__fmul_rn(h.y, d.y)), 0.5f * fmaf(h.x, s.y, __fmul_rn(h.y, d.x)));
}
// conj(h) (re + i im) / 2
__device__ __forceinline__ float2 merge_cos(float re, float im, float2 h) {
    return make_float2(0.5f * fmaf(h.x, re, __fmul_rn(h.y, im)), 0.5f * fmaf(h.x, im, -__fmul_rn(h.y, re)));
}

// The overflow sums of a block, through warp sums in `red`; the caller has a
// barrier between the two halves.
template <int NT>
__device__ __forceinline__ void put_overflow(long long over, long long over_abs, long long (*red)[2]) {
    over = warp_sum(over);
    over_abs = warp_sum(over_abs);
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5][0] = over;
        red[threadIdx.x >> 5][1] = over_abs;
    }
}
template <int NT>
__device__ __forceinline__ void get_overflow(const RhoArgs &rho, int vb, const long long (*red)[2]) {
    if (threadIdx.x < 2) {
        long long s = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) s += red[w][threadIdx.x];
        rho.partials[2 * vb + threadIdx.x] = s;
    }
}

// P1 from the fixed-point maps: the block's 2 S rows of densities into its
// slots (row 2 f of slot f the real part), the maps cleared, the overflow
// summed -- rho_kernel's work, without the map's round trip and its launch.
template <int M, int NT>
__device__ __forceinline__ void rows_density(const RhoArgs &rho, int vb, float2 *sm) {
    constexpr int S = fft_slots(M, NT), SL = fft_slot(M), N = fft_points(M);
    constexpr int B = M <= 1024 ? 4 : 2;  // pairs in flight
    static_assert(N * NT == 2 * S * (M / 2) && N % B == 0 && (M / 2) % S == 0, "the pairs fill the block");
    __shared__ long long red[NT / 32][2];
    float *d = reinterpret_cast<float *>(sm);
    long long over = 0, over_abs = 0;
#pragma unroll
    for (int it = 0; it < N; it += B) {
        BinPair b[B];
#pragma unroll
        for (int u = 0; u < B; ++u) b[u] = load_pair(rho, vb * (N * NT) + (it + u) * NT + (int)threadIdx.x);
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int at = (it + u) * NT + (int)threadIdx.x, row = at / (M / 2), c = at % (M / 2);
            const float2 v = take_pair(rho, vb * (N * NT) + at, b[u], over, over_abs);
            float *z = d + 2 * (row >> 1) * SL + (row & 1);  // bins 2 c, 2 c + 1: elements c, M - 1 - c
            z[2 * fft_pad(c)] = v.x;
            z[2 * fft_pad(M - 1 - c)] = v.y;
        }
    }
    put_overflow<NT>(over, over_abs, red);
    __syncthreads();
    get_overflow<NT>(rho, vb, red);
}

// P1: block vb transforms rows 2 f, 2 f + 1, f = vb S .. vb S + S - 1.  MAPS:
// from the fixed-point maps `rho`.
template <int M, int NT, bool MAPS = false>
__device__ __forceinline__ void fft_rows(const FieldRec &a, int vb, float2 *sm, const RhoArgs *rho = nullptr) {
    constexpr int TPF = fft_threads(M), E = fft_points(M), S = fft_slots(M, NT), SL = fft_slot(M);
    static_assert(S >= 2 && S % 2 == 0, "whole tiles of four rows per block");
    const int slot = (int)threadIdx.x / TPF, j = (int)threadIdx.x % TPF;
    const int f = vb * S + slot;
    float2 x[E];
    if constexpr (MAPS) {
        rows_density<M, NT>(*rho, vb, sm);
        slot_load<M>(x, sm + slot * SL, j);
    } else {
        const float *r0 = a.d + (size_t)(2 * f) * M, *r1 = r0 + M;
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int n = j + q * TPF, y = n < M / 2 ? 2 * n : 2 * (M - 1 - n) + 1;
            x[q] = f < M / 2 ? make_float2(__ldg(r0 + y), __ldg(r1 + y)) : make_float2(0.f, 0.f);
        }
    }
    fft_stage<M, false, 0>(x, sm + slot * SL, j, a.tab);
    __syncthreads();
    slot_store<M>(x, sm + slot * SL, j);
    __syncthreads();
    float4 *T = reinterpret_cast<float4 *>(a.t);
    for (int idx = threadIdx.x; idx < (S / 2) * M; idx += NT) {
        const int t = idx / M, k = idx % M, kk = k ? M - k : 0, tile = vb * (S / 2) + t;
        if (tile >= M / 4) continue;
        const float2 *z0 = sm + 2 * t * SL, *z1 = z0 + SL;
        const float2 h = __ldg(a.tab + M + k);
        const float2 c0 = split_cos(z0[fft_pad(k)], z0[fft_pad(kk)], h);
        const float2 c1 = split_cos(z1[fft_pad(k)], z1[fft_pad(kk)], h);
        __stcg(T + (size_t)tile * M + k, make_float4(c0.x, c0.y, c1.x, c1.y));
    }
}

// phi of coefficient c at frequencies (wx, wy) of indices (u, v), times them
__device__ __forceinline__ float2 spectral(float c, float scale, int u, int v, float wx, float wy) {
    if (u == 0 && v == 0) return make_float2(0.f, 0.f);
    c = __fmul_rn(c, scale);
    if (u == 0) c *= 0.5f;
    if (v == 0) c *= 0.5f;
    c = __fdiv_rn(c, fmaf(wx, wx, __fmul_rn(wy, wy)));
    return make_float2(__fmul_rn(c, wx), __fmul_rn(c, wy));
}

// P2: block vb takes column pairs p = vb P .. vb P + P - 1 (columns 2 p,
// 2 p + 1), P = S / 2: P forward FFTs, then 2 P back.
template <int M, int NT>
__device__ __forceinline__ void fft_columns(const FieldRec &a, int vb, float2 *sm) {
    constexpr int TPF = fft_threads(M), E = fft_points(M), S = fft_slots(M, NT), SL = fft_slot(M), P = S / 2;
    const int slot = (int)threadIdx.x / TPF, j = (int)threadIdx.x % TPF;
    const float4 *T = reinterpret_cast<const float4 *>(a.t);
    for (int idx = threadIdx.x; idx < P * (M / 4); idx += NT) {
        const int s = idx % P, xt = idx / P, p = vb * P + s;
        if (p >= M / 2) continue;
        const float4 c0 = __ldcg(T + (size_t)xt * M + 2 * p), c1 = __ldcg(T + (size_t)xt * M + 2 * p + 1);
        float2 *z = sm + s * SL;
        z[fft_pad(2 * xt)] = make_float2(c0.x, c1.x);  // x = 4 xt, 4 xt + 1, ...
        z[fft_pad(M - 1 - 2 * xt)] = make_float2(c0.y, c1.y);
        z[fft_pad(2 * xt + 1)] = make_float2(c0.z, c1.z);
        z[fft_pad(M - 2 - 2 * xt)] = make_float2(c0.w, c1.w);
    }
    __syncthreads();
    float2 x[E];
    const bool fwd = slot < P && vb * P + slot < M / 2;
    if (fwd) slot_load<M>(x, sm + slot * SL, j);
    fft_stage<M, false, 0>(x, sm + slot * SL, j, a.tab, fwd);
    __syncthreads();
    if (fwd) slot_store<M>(x, sm + slot * SL, j);
    __syncthreads();
    // items (s, i): coefficients k = i and m - i (i = 0: 0 and m/2, each its own partner)
    constexpr int IT = E / 4;
    static_assert(IT * NT == P * (M / 2), "the items fill the block");
    float2 w0[IT][2], w1[IT][2];
#pragma unroll
    for (int t = 0; t < IT; ++t) {
        const int item = (int)threadIdx.x + t * NT, s = item / (M / 2), i = item % (M / 2);
        const int k = i, kk = i ? M - i : M / 2, v = 2 * (vb * P + s);
        w0[t][0] = w0[t][1] = w1[t][0] = w1[t][1] = make_float2(0.f, 0.f);
        if (v >= M) continue;
        const float2 *z = sm + s * SL;
        const float2 z1 = z[fft_pad(k)], z2 = z[fft_pad(kk)];
        const float2 h1 = __ldg(a.tab + M + k), h2 = __ldg(a.tab + M + kk);
        const float2 a1 = split_cos(z1, i ? z2 : z1, h1), a2 = split_cos(z2, i ? z1 : z2, h2);
        const float wx1 = __ldg(a.wx + k), wx2 = __ldg(a.wx + kk);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float wy = __ldg(a.wy + v + c);
            const float2 p1 = spectral(c ? a1.y : a1.x, a.scale, k, v + c, wx1, wy);
            const float2 p2 = spectral(c ? a2.y : a2.x, a.scale, kk, v + c, wx2, wy);
            // sine sum of phi wx (reversed) and cosine sum of phi wy in one
            const float2 q1 = i ? p2 : p1, q2 = i ? p1 : p2;  // the partners' values
            float2 f1 = merge_cos(q1.x + q1.y, p1.y - p1.x, h1);
            if (i == 0) f1 = make_float2(0.f, p1.y);
            const float2 f2 = merge_cos(q2.x + q2.y, p2.y - p2.x, h2);
            (c ? w1 : w0)[t][0] = f1;
            (c ? w1 : w0)[t][1] = f2;
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < IT; ++t) {
        const int item = (int)threadIdx.x + t * NT, s = item / (M / 2), i = item % (M / 2);
        const int k = i, kk = i ? M - i : M / 2;
        float2 *y0 = sm + 2 * s * SL, *y1 = y0 + SL;
        y0[fft_pad(k)] = w0[t][0];
        y0[fft_pad(kk)] = w0[t][1];
        y1[fft_pad(k)] = w1[t][0];
        y1[fft_pad(kk)] = w1[t][1];
    }
    __syncthreads();
    slot_load<M>(x, sm + slot * SL, j);
    fft_stage<M, true, 0>(x, sm + slot * SL, j, a.tab);
    __syncthreads();
    slot_store<M>(x, sm + slot * SL, j);
    __syncthreads();
    float4 *U = reinterpret_cast<float4 *>(a.u);
    for (int idx = threadIdx.x; idx < S * (M / 2); idx += NT) {
        const int c = idx & 1, s = (idx >> 1) % P, t = (idx >> 1) / P, v = 2 * (vb * P + s) + c;
        if (v >= M) continue;
        const float2 *z = sm + (2 * s + c) * SL;
        const float2 e = z[fft_pad(t)], o = z[fft_pad(M - 1 - t)];  // rows 2 t, 2 t + 1
        __stcg(U + (size_t)t * M + v, make_float4(e.x, e.y, -o.x, o.y));
    }
}

// P3: block vb takes rows [row_lo + vb S, + S) of rows [row_lo, row_hi).
template <int M, int NT>
__device__ __forceinline__ void fft_fields(const FieldRec &a, int vb, float2 *sm) {
    constexpr int TPF = fft_threads(M), E = fft_points(M), S = fft_slots(M, NT), SL = fft_slot(M);
    const int slot = (int)threadIdx.x / TPF, j = (int)threadIdx.x % TPF;
    const int row0 = a.row_lo + vb * S;
    const float4 *U = reinterpret_cast<const float4 *>(a.u);
    constexpr int IT = E / 4;
#pragma unroll
    for (int t = 0; t < IT; ++t) {
        const int item = (int)threadIdx.x + t * NT, tl = item / (M / 2), i = item % (M / 2);
        const int k = i, kk = i ? M - i : M / 2, tile = row0 / 2 + tl;
        float4 u1 = make_float4(0.f, 0.f, 0.f, 0.f), u2 = u1;
        if (2 * tile < a.row_hi) {
            u1 = __ldcg(U + (size_t)tile * M + k);
            u2 = __ldcg(U + (size_t)tile * M + kk);
        }
        const float2 h1 = __ldg(a.tab + M + k), h2 = __ldg(a.tab + M + kk);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float2 p1 = r ? make_float2(u1.z, u1.w) : make_float2(u1.x, u1.y);
            const float2 p2 = r ? make_float2(u2.z, u2.w) : make_float2(u2.x, u2.y);
            const float2 q1 = i ? p2 : p1, q2 = i ? p1 : p2;
            float2 f1 = merge_cos(p1.x + p1.y, q1.y - q1.x, h1);
            if (i == 0) f1 = make_float2(p1.x, 0.f);
            const float2 f2 = merge_cos(p2.x + p2.y, q2.y - q2.x, h2);
            float2 *y = sm + (2 * tl + r) * SL;
            y[fft_pad(k)] = f1;
            y[fft_pad(kk)] = f2;
        }
    }
    __syncthreads();
    float2 x[E];
    slot_load<M>(x, sm + slot * SL, j);
    fft_stage<M, true, 0>(x, sm + slot * SL, j, a.tab);
    __syncthreads();
    slot_store<M>(x, sm + slot * SL, j);
    __syncthreads();
    for (int idx = threadIdx.x; idx < S * (M / 2); idx += NT) {
        const int s = idx / (M / 2), t = idx % (M / 2), row = row0 + s;
        if (row >= a.row_hi) continue;
        const float2 *z = sm + s * SL;
        const float2 e = z[fft_pad(t)], o = z[fft_pad(M - 1 - t)];  // y = 2 t, 2 t + 1
        const size_t at = (size_t)row * M + 2 * t;
        if (a.exy) {
            *reinterpret_cast<float4 *>(a.exy + at) = make_float4(e.x, e.y, o.x, -o.y);
        } else if (a.wide) {
            *reinterpret_cast<float2 *>(a.ex + at) = make_float2(e.x, o.x);
            *reinterpret_cast<float2 *>(a.ey + at) = make_float2(e.y, -o.y);
        } else {  // the caller's buffers, aligned to 4 bytes only
            a.ex[at] = e.x;
            a.ex[at + 1] = o.x;
            a.ey[at] = e.y;
            a.ey[at + 1] = -o.y;
        }
    }
}

// ---- kDense x kDense bins: the whole solve in one block -------------------------
// As four contractions with the dense transform matrices, D[i][j] = sum_k
// A[i][k] B[j][k], k ascending: a loop on a grid this small amplifies any
// change of rounding within some twenty iterations, and at 6 x 32^3 products
// the launches are what a solve costs (a 576-cell loop: 43.5 us an iteration
// with the four contractions as launches of their own, 39.0 in one block,
// 39.3 with the three passes above).
constexpr int kDenseLd = kDense + 4;  // row of a matrix in shared memory: 16-byte aligned, no bank conflicts
struct DenseSmem {
    float c[kDense][kDenseLd], ct[kDense][kDenseLd], st[kDense][kDenseLd];
    float b[4][kDense][kDenseLd];
};

// 2 x 2 outputs (i, i + 16) x (j, j + 16) of D by thread t of 256
__device__ __forceinline__ void dense_dot(const float (*A)[kDenseLd], const float (*B)[kDenseLd], int i, int j,
                                          float (&acc)[2][2]) {
#pragma unroll
    for (int r = 0; r < 2; ++r) acc[r][0] = acc[r][1] = 0.f;
#pragma unroll
    for (int k = 0; k < kDense; k += 4) {
        float4 a[2], b[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            a[r] = *reinterpret_cast<const float4 *>(&A[i + 16 * r][k]);
            b[r] = *reinterpret_cast<const float4 *>(&B[j + 16 * r][k]);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float v = acc[r][q];
                v = fmaf(a[r].x, b[q].x, v);
                v = fmaf(a[r].y, b[q].y, v);
                v = fmaf(a[r].z, b[q].z, v);
                acc[r][q] = fmaf(a[r].w, b[q].w, v);
            }
    }
}

// 256 or 512 threads; MAPS (512): from the fixed-point maps `rho`
template <int NT, bool MAPS = false>
__device__ __forceinline__ void dense_solve(const FieldRec &a, DenseSmem &sm, const RhoArgs *rho = nullptr) {
    constexpr int M = kDense;
    __shared__ long long red[NT / 32][2];
    // 256 threads a product; the two products of S3 and of S4 side by side
    // (512 threads) or in turn
    const int t = threadIdx.x & 255, z = threadIdx.x >> 8, i = t >> 4, j = t & 15;
    // every load up front (a 576-cell trial 21.0 -> 20.4 us)
    const float *tab = reinterpret_cast<const float *>(a.tab);
    constexpr int N = M * M / NT;
    float tc[N], ts[N], wx[2], wy[2];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        tc[n] = __ldg(tab + threadIdx.x + n * NT);
        ts[n] = __ldg(tab + M * M + threadIdx.x + n * NT);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        wx[r] = __ldg(a.wx + i + 16 * r);
        wy[r] = __ldg(a.wy + j + 16 * r);
    }
    if constexpr (MAPS) {
        static_assert(NT == M * M / 2, "a pair of bins per thread");
        long long over = 0, over_abs = 0;
        const int p = (int)threadIdx.x;
        const float2 d = take_pair(*rho, p, load_pair(*rho, p), over, over_abs);
        sm.b[0][2 * p / M][2 * p % M] = d.x;
        sm.b[0][2 * p / M][2 * p % M + 1] = d.y;
        put_overflow<NT>(over, over_abs, red);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int e = (int)threadIdx.x + n * NT, k = e / M, x = e % M;
        sm.c[k][x] = tc[n];
        sm.ct[x][k] = tc[n];
        sm.st[x][k] = ts[n];
        if constexpr (!MAPS) sm.b[0][k][x] = __ldg(a.d + e);
    }
    __syncthreads();
    if constexpr (MAPS) get_overflow<NT>(*rho, 0, red);
    float acc[2][2];
    auto put = [&](float (*D)[kDenseLd]) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) D[i + 16 * r][j + 16 * q] = acc[r][q];
    };
    if (z == 0) {  // S1: T[v][x]
        dense_dot(sm.c, sm.b[0], i, j, acc);
        put(sm.b[1]);
    }
    __syncthreads();
    if (z == 0) {  // S2: a[u][v] -> Px, Py
        dense_dot(sm.c, sm.b[1], i, j, acc);
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int u = i + 16 * r, v = j + 16 * q;
                const float2 p = spectral(acc[r][q], a.scale, u, v, wx[r], wy[q]);
                sm.b[2][u][v] = p.x;
                sm.b[3][u][v] = p.y;
            }
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 512 / NT; ++w) {  // S3: Ux[y][u], Uy[y][u]
        const int zz = z + w;
        dense_dot(zz ? sm.st : sm.ct, sm.b[2 + zz], i, j, acc);
        put(sm.b[zz]);
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 512 / NT; ++w) {  // S4: Ex[x][y], Ey[x][y]
        const int zz = z + w;
        dense_dot(zz ? sm.ct : sm.st, sm.b[zz], i, j, acc);
        float *e = a.exy ? reinterpret_cast<float *>(a.exy) + zz : zz ? a.ey : a.ex;
        const int step = a.exy ? 2 : 1;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) e[((i + 16 * r) * M + j + 16 * q) * step] = acc[r][q];
    }
}

// ---- launches of one solve ----------------------------------------------------
// The passes are programmatic dependents of the launch before (a solve in the
// caller's buffers 12.3 -> 9.8 us at 96 bins, 6.2 -> 4.0 at 32 against an
// ordinary first launch); a loop trial's first pass only at few bins.

// run only if gate is null or (1 << *gate) & mask
__device__ __forceinline__ bool gated_off(const int *gate, int mask) { return gate && !((1 << *gate) & mask); }

template <int M, int NT, int PASS>
__global__ void __launch_bounds__(NT, odd_part(M) == 1 && M <= 2048 ? 1024 / NT : 1) fft_kernel(FieldRec a, const int *gate, int mask) {
    extern __shared__ __align__(16) float2 fft_sm[];
    if (PASS < 2) grid_release();
    grid_wait();
    if (gated_off(gate, mask)) return;
    if (PASS == 0) fft_rows<M, NT>(a, blockIdx.x, fft_sm);
    if (PASS == 1) fft_columns<M, NT>(a, blockIdx.x, fft_sm);
    if (PASS == 2) fft_fields<M, NT>(a, blockIdx.x, fft_sm);
}

// (up to 1024 bins its blocks are resident at once with 512 threads an SM: 128 registers, no spills)
template <int M, int NT>
__global__ void __launch_bounds__(NT, (M <= 1024 ? 512 : 1024) / NT) fft_maps_kernel(FieldRec a, RhoArgs rho) {
    extern __shared__ __align__(16) float2 fft_sm[];
    grid_release();
    grid_wait();
    fft_rows<M, NT, true>(a, blockIdx.x, fft_sm, &rho);
}

__global__ void __launch_bounds__(512) dense_maps_kernel(FieldRec a, RhoArgs rho) {
    __shared__ __align__(16) DenseSmem sm;
    grid_wait();
    dense_solve<512, true>(a, sm, &rho);
}

__global__ void __launch_bounds__(512) dense_kernel(FieldRec a, const int *gate, int mask) {
    __shared__ __align__(16) DenseSmem sm;
    grid_wait();
    if (gated_off(gate, mask)) return;
    dense_solve<512>(a, sm);
}

// Blocks of a pass (over all m rows or columns; P3: of rows rows).
constexpr int fft_blocks(int m, int nt, int pass, int rows) {
    const int s = fft_slots(m, nt);
    return pass == 0 ? (m / 2 + s - 1) / s : pass == 1 ? (m / 2 + s / 2 - 1) / (s / 2) : (rows + s - 1) / s;
}

// Threads per block of a solve's own launches: two FFTs a block, but a warp
// at least.
constexpr int fft_block_threads(int m) { return std::max(32, 2 * fft_threads(m)); }

// rho: the first pass from the fixed-point maps (or null); returns its blocks
template <int M>
int launch_fft(const FieldRec &a, cudaStream_t st, const int *gate, int mask, const RhoArgs *rho = nullptr) {
    constexpr int NT = fft_block_threads(M), SM = fft_smem(M, NT);
    if constexpr (SM > 48 * 1024) {  // a no-op after the first call
        cudaFuncSetAttribute(fft_kernel<M, NT, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
        cudaFuncSetAttribute(fft_kernel<M, NT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
        cudaFuncSetAttribute(fft_kernel<M, NT, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
    }
    constexpr int blocks = fft_blocks(M, NT, 0, M);
    bool maps = false;
    if constexpr (odd_part(M) == 1) {
        if (rho) {
            maps = true;
            if constexpr (SM > 48 * 1024)
                cudaFuncSetAttribute(fft_maps_kernel<M, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
            // beyond 128 bins its blocks would take SMs while the WA launch is
            // still starting (an iteration without / with: 20k cells on 128
            // bins 25.0 / 24.5 us, 100k on 256 33.7 / 34.4)
            if constexpr (M <= 128)
                launch_dependent(fft_maps_kernel<M, NT>, blocks, NT, SM, st, a, *rho);
            else
                fft_maps_kernel<M, NT><<<blocks, NT, SM, st>>>(a, *rho);
        }
    }
    if (!maps) launch_dependent(fft_kernel<M, NT, 0>, blocks, NT, SM, st, a, gate, mask);
    launch_dependent(fft_kernel<M, NT, 1>, fft_blocks(M, NT, 1, M), NT, SM, st, a, gate, mask);
    launch_dependent(fft_kernel<M, NT, 2>, fft_blocks(M, NT, 2, M), NT, SM, st, a, gate, mask);
    return blocks;
}

// a solve's arguments: tables, scratch, all rows
FieldRec solve_rec(const FieldSolver &f, const float *d, float *ex, float *ey, float2 *exy) {
    FieldRec a{};
    a.m = f.m;
    a.d = d;
    a.t = f.t;
    a.u = f.u;
    a.ex = ex;
    a.ey = ey;
    a.exy = exy;
    a.tab = f.tab;
    a.wx = f.wx;
    a.wy = f.wy;
    a.scale = 4.0f / ((float)f.m * (float)f.m);
    a.row_lo = 0;
    a.row_hi = f.m;
    a.wide = (((uintptr_t)ex | (uintptr_t)ey) & 7u) == 0;
    return a;
}

void fill_tables(const FieldSolver &f, cudaStream_t st) {
    const int n = f.m == kDense ? f.m * f.m : f.m;
    field_table_kernel<<<(n + 127) / 128, 128, 0, st>>>(f.tab, f.wx, f.wy, f.m, f.bin_ratio);
}

__global__ void split_kernel(int n, const float *src, __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = src[i];
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        hi[i] = h;
        lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

template <typename T>
int dmalloc(T **p, size_t n) {
    return cudaMalloc((void **)p, sizeof(T) * (n ? n : 1)) == cudaSuccess ? 0 : -1;
}

}  // namespace

void launch_split_bf16(int n, const float *src, __nv_bfloat16 *hi, __nv_bfloat16 *lo, cudaStream_t st) {
    int blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    split_kernel<<<blocks, 256, 0, st>>>(n, src, hi, lo);
}

// The tensor-core solve's constant transform matrices as BF16 hi/lo pairs,
// and its scratch (field_solver_free_bf16 gives back what a failure leaves).
int field_solver_matrices(FieldSolver &f) {
    const int m = f.m;
    const size_t nn = (size_t)m * m;
    std::vector<float> C(nn), Ct(nn), St(nn);
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < m; ++k)
        for (int i = 0; i < m; ++i) {
            const double t = pi * k * (i + 0.5) / m;
            C[(size_t)k * m + i] = (float)cos(t);
            Ct[(size_t)i * m + k] = (float)cos(t);
            St[(size_t)i * m + k] = (float)sin(t);
        }
    int e = dmalloc(&f.C_hi, nn) | dmalloc(&f.C_lo, nn) | dmalloc(&f.Ct_hi, nn) | dmalloc(&f.Ct_lo, nn) |
            dmalloc(&f.St_hi, nn) | dmalloc(&f.St_lo, nn);
    e |= dmalloc(&f.b_t_hi, nn) | dmalloc(&f.b_t_lo, nn) | dmalloc(&f.b_px_hi, nn) | dmalloc(&f.b_px_lo, nn) |
         dmalloc(&f.b_py_hi, nn) | dmalloc(&f.b_py_lo, nn) | dmalloc(&f.b_ux_hi, nn) | dmalloc(&f.b_ux_lo, nn) |
         dmalloc(&f.b_uy_hi, nn) | dmalloc(&f.b_uy_lo, nn);
    if (e) return AP_ERR_CUDA;
    // staged through the solve's scratch
    struct {
        const float *src;
        __nv_bfloat16 *hi, *lo;
    } s[3] = {{C.data(), f.C_hi, f.C_lo}, {Ct.data(), f.Ct_hi, f.Ct_lo}, {St.data(), f.St_hi, f.St_lo}};
    for (auto &q : s) {
        if (cudaMemcpy(f.t, q.src, nn * 4, cudaMemcpyHostToDevice) != cudaSuccess) return AP_ERR_CUDA;
        launch_split_bf16((int)nn, f.t, q.hi, q.lo, 0);
        if (cudaGetLastError() != cudaSuccess) return AP_ERR_CUDA;
    }
    return AP_OK;
}

static bool field_fft_size(int m) {
    switch (m) {
    case 32: case 64: case 96: case 128: case 160: case 192: case 224: case 256: case 512: case 1024: case 2048:
    case 4096:
        return true;
    default:
        return false;
    }
}

void field_solve_fp32(FieldSolver &f, const float *d, float *ex, float *ey, cudaStream_t st, const int *gate,
                      int gate_mask, float2 *exy) {
    const FieldRec a = solve_rec(f, d, ex, ey, exy);
    switch (f.m) {
    case kDense: launch_dependent(dense_kernel, 1, 512, 0, st, a, gate, gate_mask); break;
    case 64: launch_fft<64>(a, st, gate, gate_mask); break;
    case 96: launch_fft<96>(a, st, gate, gate_mask); break;
    case 128: launch_fft<128>(a, st, gate, gate_mask); break;
    case 160: launch_fft<160>(a, st, gate, gate_mask); break;
    case 192: launch_fft<192>(a, st, gate, gate_mask); break;
    case 224: launch_fft<224>(a, st, gate, gate_mask); break;
    case 256: launch_fft<256>(a, st, gate, gate_mask); break;
    case 512: launch_fft<512>(a, st, gate, gate_mask); break;
    case 1024: launch_fft<1024>(a, st, gate, gate_mask); break;
    case 2048: launch_fft<2048>(a, st, gate, gate_mask); break;
    case 4096: launch_fft<4096>(a, st, gate, gate_mask); break;
    }
}

int field_solve_maps(FieldSolver &f, const RhoArgs &rho, float2 *exy, cudaStream_t st) {
    const FieldRec a = solve_rec(f, nullptr, nullptr, nullptr, exy);
    switch (f.m) {
    case kDense: launch_dependent(dense_maps_kernel, 1, 512, 0, st, a, rho); return 1;
    case 64: return launch_fft<64>(a, st, nullptr, 0, &rho);
    case 128: return launch_fft<128>(a, st, nullptr, 0, &rho);
    case 256: return launch_fft<256>(a, st, nullptr, 0, &rho);
    case 512: return launch_fft<512>(a, st, nullptr, 0, &rho);
    case 1024: return launch_fft<1024>(a, st, nullptr, 0, &rho);
    case 2048: return launch_fft<2048>(a, st, nullptr, 0, &rho);
    default: return launch_fft<4096>(a, st, nullptr, 0, &rho);
    }
}

int field_solver_init(FieldSolver &f, int m, float bin_ratio) {
    f = FieldSolver();
    if (!field_fft_size(m)) return AP_ERR_UNSUPPORTED;
    f.m = m;
    f.bin_ratio = bin_ratio;
    const size_t nn = (size_t)m * m;
    if (dmalloc(&f.tab, field_table_len(m)) | dmalloc(&f.wx, m) | dmalloc(&f.wy, m) | dmalloc(&f.t, nn) |
        dmalloc(&f.u, 2 * nn))
        return AP_ERR_CUDA;
    fill_tables(f, 0);
    // the solve's time for ap_solver_info (2 warm, 4 timed; the values do not
    // matter), on maps of its own
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess) return AP_ERR_CUDA;
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return AP_ERR_CUDA;
    }
    float *io = nullptr;
    int r = dmalloc(&io, 3 * nn) ? AP_ERR_CUDA : AP_OK;
    if (r == AP_OK && cudaMemset(io, 0, sizeof(float) * nn) != cudaSuccess) r = AP_ERR_CUDA;
    if (r == AP_OK) {
        for (int t = 0; t < 6; ++t) {
            if (t == 2) cudaEventRecord(e0, 0);
            field_solve_fp32(f, io, io + nn, io + 2 * nn, 0);
        }
        cudaEventRecord(e1, 0);
        if (cudaEventSynchronize(e1) != cudaSuccess || cudaGetLastError() != cudaSuccess) r = AP_ERR_CUDA;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        f.simt_tile = m == kDense || fft_block_threads(m) > 256 ? 64 : 32;
        f.simt_ms[0] = f.simt_ms[1] = -1.f;
        f.simt_ms[f.simt_tile == 64] = ms / 4;
    }
    cudaFree(io);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return r;
}

void field_solver_free_bf16(FieldSolver &f) {
    __nv_bfloat16 **maps[] = {&f.C_hi,   &f.C_lo,   &f.Ct_hi,   &f.Ct_lo,   &f.St_hi,   &f.St_lo,   &f.b_t_hi,  &f.b_t_lo,
                              &f.b_px_hi, &f.b_px_lo, &f.b_py_hi, &f.b_py_lo, &f.b_ux_hi, &f.b_ux_lo, &f.b_uy_hi, &f.b_uy_lo};
    for (__nv_bfloat16 **p : maps) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    void *ptrs[] = {f.tc_status, f.tc_sync, f.tc_part};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    f.tc_status = f.tc_sync = nullptr;
    f.tc_part = nullptr;
    free(f.tc_maps);  // host-side tensor-map table
    f.tc_maps = nullptr;
    f.tc_ready = f.tc_pinned = 0;
    for (float &ms : f.tc_tune_ms) ms = 0.f;
}

void field_solver_free(FieldSolver &f) {
    field_solver_free_bf16(f);
    void *ptrs[] = {f.tab, f.wx, f.wy, f.t, f.u};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    f = FieldSolver();
}

// ---- batched form ---------------------------------------------------------------
// The passes of every instance in one launch, record k + 1 of an instance
// waiting for the one before (the queue's dependencies): P1, P2, and P3 as two
// records of half the rows each.  A block of 8 tile threads (tile 32 or 64,
// the batch's choice) runs the passes of any grid; the bits do not depend on
// it (an FFT's arithmetic is its own).

bool field_records(const FieldSolver &f, const float *d, float2 *exy, int tile, FieldRec rec[4]) {
    if ((f.m != kDense && 2 * fft_threads(f.m) > 8 * tile) || odd_part(f.m) != 1) return false;
    for (int k = 0; k < 4; ++k) {
        rec[k] = solve_rec(f, d, nullptr, nullptr, exy);
        rec[k].pass = std::min(k, 2);
    }
    rec[2].row_hi = rec[3].row_lo = f.m / 2;
    return true;
}

int field_rec_blocks(const FieldRec &r, int tile) {
    if (r.m == kDense) return r.pass == 0;  // one block does it all
    return fft_blocks(r.m, 8 * tile, r.pass, r.row_hi - r.row_lo);
}

namespace {

template <int M, int NT>
__device__ __forceinline__ void fft_record(const FieldRec &r, int vb, float2 *sm) {
    if constexpr (2 * fft_threads(M) <= NT) {
        if (r.pass == 0) fft_rows<M, NT>(r, vb, sm);
        else if (r.pass == 1) fft_columns<M, NT>(r, vb, sm);
        else fft_fields<M, NT>(r, vb, sm);
    }
}

template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) persist_field_kernel(PersistQueue q, const FieldRec *recs) {
    extern __shared__ __align__(16) float2 persist_sm[];
    persist_loop(q, recs, [](const FieldRec &r, VBlock vb, int) {
        switch (r.m) {
        case kDense: dense_solve<NT>(r, *reinterpret_cast<DenseSmem *>(persist_sm)); break;
        case 64: fft_record<64, NT>(r, vb.id, persist_sm); break;
        case 128: fft_record<128, NT>(r, vb.id, persist_sm); break;
        case 256: fft_record<256, NT>(r, vb.id, persist_sm); break;
        case 512: fft_record<512, NT>(r, vb.id, persist_sm); break;
        case 1024: fft_record<1024, NT>(r, vb.id, persist_sm); break;
        case 2048: fft_record<2048, NT>(r, vb.id, persist_sm); break;
        case 4096: fft_record<4096, NT>(r, vb.id, persist_sm); break;
        }
    });
}

// dynamic shared memory of a persistent launch whose largest grid has m bins
// a side: every grid up to 2048 needs the same
constexpr int persist_field_smem(int tile, int m) {
    return std::max(fft_smem(m > 2048 ? 4096 : 512, 8 * tile), (int)sizeof(DenseSmem));
}

}  // namespace

int persist_field_wave(int tile, int m) {
    const int smem = persist_field_smem(tile, m);
    const void *k = tile == 64 ? (const void *)persist_field_kernel<512> : (const void *)persist_field_kernel<256>;
    // what the largest grid needs, whatever this launch's: the attribute is the
    // process's, and another thread's batch may be about to launch
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, persist_field_smem(tile, 4096));
    return wave_of(k, 8 * tile, 304, smem);
}

void launch_persist_field(const PersistQueue &q, int items, const FieldRec *recs, int tile, int m, cudaStream_t st) {
    const int w = persist_blocks(persist_field_wave(tile, m), items), smem = persist_field_smem(tile, m);
    if (tile == 64)
        persist_field_kernel<512><<<w, 512, smem, st>>>(q, recs);
    else
        persist_field_kernel<256><<<w, 256, smem, st>>>(q, recs);
}

// ---- field solve without allocation -------------------------------------------
// Some callers cannot allocate device memory at all: code that runs inside a
// host framework which owns every device allocation and hands out only the
// buffers it manages, or code on a path where a cudaMalloc would synchronise
// the device or fail under a fixed memory budget.  For them the FP32 solve
// also runs from one fixed scratch array in the library's static device
// memory.  The array holds the tables and the intermediate maps of one grid
// of up to kNoAllocMaxBins x kNoAllocMaxBins bins (3 m^2 + 6 m floats, 0.8 MB
// at the maximum); every GPU that loads the library keeps it until the process
// exits.

namespace {

constexpr int kNoAllocMaxBins = 256;
constexpr size_t kNoAllocFloats = 3ull * kNoAllocMaxBins * kNoAllocMaxBins + 6ull * kNoAllocMaxBins;
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) float g_field_scratch[kNoAllocFloats];

// Per device: which context's copy of g_field_scratch holds the tables of
// which grid.  A context that is destroyed and recreated (cudaDeviceReset)
// gets a fresh, zeroed copy of the array, so the key includes the context's
// unique id; without a way to read that id the tables are refilled on every
// call.
struct NoAllocState {
    unsigned long long ctx_id;  // 0: nothing cached
    float *base;
    int m;
    float ratio;
};
static NoAllocState g_noalloc_state[kNoAllocMaxDevices];

typedef int (*PfnCtxGetCurrent)(void **ctx);
typedef int (*PfnCtxGetId)(void *ctx, unsigned long long *id);

// Unique id of the calling thread's current context (driver entry points
// looked up through the runtime, so the library needs no libcuda link), or
// 0 if it cannot be read.
unsigned long long current_context_id() {
    static PfnCtxGetCurrent get_cur = nullptr;
    static PfnCtxGetId get_id = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_cur = (PfnCtxGetCurrent)p;
        p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (PfnCtxGetId)p;
        looked_up = true;
    }
    if (!get_cur || !get_id) return 0ull;
    void *ctx = nullptr;
    unsigned long long id = 0ull;
    if (get_cur(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0ull;
    return id;
}

}  // namespace

}  // namespace ap

// Same result as ap_field_solve with the FP32 solver, on caller-owned device
// buffers and without allocating.  Every call looks the scratch address up
// with cudaGetSymbolAddress (host code may not use the symbol as an address);
// the first call on a device, the first after the bin count or bin_ratio
// changes and the first in a new context fill the transform tables, so make
// that first call before any stream capture.  All calls share the one
// scratch array: calls whose GPU work overlaps (other streams, other threads)
// race on it.  density must start on a 16-byte boundary; ex and ey must be
// float-aligned.
extern "C" int ap_field_solve_noalloc(const float *density, float *ex, float *ey, int32_t bins, float bin_ratio,
                                      void *stream) {
    using namespace ap;
    if (!density || !ex || !ey) return AP_ERR_INVALID_ARG;
    if (((uintptr_t)density & 15u) != 0 || ((uintptr_t)ex & 3u) != 0 || ((uintptr_t)ey & 3u) != 0)
        return AP_ERR_INVALID_ARG;
    if (bins < 32 || bins > kNoAllocMaxBins || (bins % 32) != 0) return AP_ERR_INVALID_ARG;
    if (!(bin_ratio > 0.f) || !(bin_ratio < 1e30f)) return AP_ERR_INVALID_ARG;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return AP_ERR_NO_DEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_field_scratch) != cudaSuccess || !p) return AP_ERR_CUDA;
    const unsigned long long ctx = current_context_id();
    NoAllocState &s = g_noalloc_state[dev];
    const bool fresh = ctx == 0ull || s.ctx_id != ctx || s.base != (float *)p || s.m != bins || s.ratio != bin_ratio;
    const size_t mm = (size_t)bins * bins;
    FieldSolver f{};
    f.m = bins;
    f.bin_ratio = bin_ratio;
    f.t = (float *)p;  // 16-byte aligned: mm is a multiple of 1024
    f.u = f.t + mm;
    f.tab = (float2 *)(f.u + 2 * mm);
    f.wx = (float *)(f.tab + field_table_len(bins));
    f.wy = f.wx + bins;
    if (fresh) {
        s.ctx_id = 0ull;  // set again only once the fill is enqueued
        fill_tables(f, st);
        if (cudaGetLastError() != cudaSuccess) return AP_ERR_CUDA;
        s.ctx_id = ctx;
        s.base = (float *)p;
        s.m = bins;
        s.ratio = bin_ratio;
    }
    field_solve_fp32(f, density, ex, ey, st);  // writes every scratch element before reading it
    return cudaGetLastError() == cudaSuccess ? AP_OK : AP_ERR_CUDA;
}
