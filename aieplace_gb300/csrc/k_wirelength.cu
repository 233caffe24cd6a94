// Weighted-average wirelength gradient and HPWL over a net/pin CSR.
//
// Replaces Placer::computeAllPartials_CPU -> computeNetPartials_CPU ->
// compute_bc_terms_CPU -> compute_a_terms_CPU (vck5000/host/src/AIEplace.cpp:
// 574-673) and the AIE graph compute_abc + compute_partials
// (vck5000/aie/src/partials/compute_abc.cpp:23-125, compute_partials.cpp:
// 11-63).  Per net and axis the reference forms
//   a+_i = exp((x_i - x_max)/g), a-_i = exp((x_min - x_i)/g),
//   b+- = sum a+-, c+- = sum a+- x_i,
//   dWA/dx_i = ((1 + x_i/g) b+ - c+/g) a+_i / b+^2 - ((1 - x_i/g) b- + c-/g) a-_i / b-^2.
// The kernels evaluate the same expression in the algebraically equal
// shifted form
//   dWA/dx_i = a+_i/b+ (1 + (x_i - WA+)/g) - a-_i/b- (1 - (x_i - WA-)/g),
//   WA+ = x_max + sum a+ (x - x_max) / b+,  WA- = x_min + sum a- (x - x_min) / b-,
// which keeps FP32 exact where the reference form cancels (x_i/g ~ 1e4).
// Each pin's gradient is rounded to 2^-20 and accumulated per node in int64,
// so the sum over a node's nets is the same whatever order the atomics land in;
// both axes share one 64-bit atomic (pack_q) unless the node has more than
// kPackMaxPins pins.
#include <algorithm>

#include "ap_common.cuh"
#include "ap_kernels.h"

namespace ap {

namespace {

struct AxisTerms {
    float inv_bp, inv_bm, wp, wm;  // 1/b+, 1/b-, shifted WA+ - x_max, WA- - x_min
};

// 1/b for the sums b+- (1 <= b <= net degree: the extreme pin adds exp(0)):
// the 2-ulp reciprocal, well inside its range; IEEE division spent a dozen
// instructions and a branch per call here
__device__ __forceinline__ float rcp(float b) { return __fdividef(1.f, b); }

// Both axes at once: two IEEE FP32 operations an instruction (the WA kernels
// are bound by instruction issue).  exp(x) = 2^(x log2 e), results below 2^-126
// taken as 0: next to the extreme pin's 1 they change no sum, and no gradient
// in its fixed point.  The stage at 2M cells 108 -> 100.5 us, at 60k 31 -> 28.
__device__ __forceinline__ float2 exp2_pair(float2 a) {
    const float2 t = mul2(a, both(1.44269504088896341f));
    float2 r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(t.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(t.y));
    return r;
}

// A net's constants of both axes, for its pins' gradients
struct PairTerms {
    float2 ibp, ibm;    // 1/b+, 1/b-
    float2 nwp, nwm;    // -(WA+ - x_max), -(WA- - x_min)
    __device__ __forceinline__ PairTerms(float2 bp, float2 bm, float2 cp, float2 cm) {
        ibp = make_float2(rcp(bp.x), rcp(bp.y));
        ibm = make_float2(rcp(bm.x), rcp(bm.y));
        nwp = neg2(mul2(cp, ibp));
        nwm = neg2(mul2(cm, ibm));
    }
    // a+/b+ (1 + (x - WA+)/g) - a-/b- (1 - (x - WA-)/g) of sp = x - WA+, sm = x - WA-
    __device__ __forceinline__ float2 grad(float2 ep, float2 em, float2 sp, float2 sm, float2 ig, float2 nig) const {
        const float2 tp = fma2(sp, ig, both(1.f)), tm = fma2(sm, nig, both(1.f));
        return fma2(mul2(ep, ibp), tp, neg2(mul2(mul2(em, ibm), tm)));
    }
};

// one pin's gradient into its node's accumulators; `raw` is the pin_node entry
__device__ __forceinline__ void add_grad(ull *gq, ull *gqx, ull *gqy, int raw, float gx, float gy) {
    const int n = raw & kPinNode;
    if (__builtin_expect(raw >= 0, 1)) {  // nodes of more than kPackMaxPins pins are rare
        atomicAdd(gq + n, pack_q(grad_q32(gx), grad_q32(gy)));
    } else {
        atomicAdd(gqx + n, grad_q(gx));
        atomicAdd(gqy + n, grad_q(gy));
    }
}

// Sums of 8 values at once over an aligned group of G lanes (transposed
// butterfly): halving exchanges at offsets G/2, G/4, G/8 leave lane-in-group
// l with a partial of quantity (l / (G/8)) & 7, the remaining offsets finish
// it, and 8 broadcasts hand every lane of the group every total -- 3 + log2(G/8)
// + 8 shuffles instead of 8 log2(G).  Fixed order, so the same on every run.
// `mask`: the group's lanes; `base`: its first lane.
template <int G>
__device__ __forceinline__ void group_sum8(float v[8], int l, unsigned mask, int base) {
    static_assert(G >= 8 && G <= 32, "group of 8..32 lanes");
    const bool a = l & (G / 2), b = l & (G / 4), c = l & (G / 8);
    float u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float send = a ? v[k] : v[k + 4];
        u[k] = (a ? v[k + 4] : v[k]) + __shfl_xor_sync(mask, send, G / 2);
    }
    float t[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float send = b ? u[k] : u[k + 2];
        t[k] = (b ? u[k + 2] : u[k]) + __shfl_xor_sync(mask, send, G / 4);
    }
    float sum = (c ? t[1] : t[0]) + __shfl_xor_sync(mask, c ? t[0] : t[1], G / 8);
#pragma unroll
    for (int o = G / 16; o > 0; o >>= 1) sum += __shfl_xor_sync(mask, sum, o);
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = __shfl_sync(mask, sum, base + q * (G / 8));
}

// Maxima of 4 values at once over an aligned group of G lanes, the same scheme.
template <int G>
__device__ __forceinline__ void group_max4(float v[4], int l, unsigned mask, int base) {
    const bool a = l & (G / 2), b = l & (G / 4);
    float u[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float send = a ? v[k] : v[k + 2];
        u[k] = fmaxf(a ? v[k + 2] : v[k], __shfl_xor_sync(mask, send, G / 2));
    }
    float m = fmaxf(b ? u[1] : u[0], __shfl_xor_sync(mask, b ? u[0] : u[1], G / 4));
#pragma unroll
    for (int o = G / 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(mask, m, o));
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __shfl_sync(mask, m, base + q * (G / 4));
}

// One net of degree d <= G P by an aligned group of G lanes, P pins per lane
// in registers (pin j on lane j mod G): one load pass, each exponential once.
template <int G, int P>
__device__ __forceinline__ void net_group(const WaArgs &a, int s, int d, int l, unsigned mask, int base,
                                          const float2 *xy, float inv_g, float &hpf, float &waf) {
    bool v[P];
    int nd[P];
    float2 c[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int j = l + p * G;
        v[p] = j < d;
        // a slot past the net's end repeats its last pin: the extrema are
        // unchanged and no load waits on a branch (its terms are zeroed below)
        nd[p] = __ldg(a.pin_node + s + min(j, d - 1));  // raw entry (heavy flag)
        c[p] = __ldg(xy + (nd[p] & kPinNode));
    }
    float m4[4] = {-3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f};  // max x, max y, -min x, -min y
#pragma unroll
    for (int p = 0; p < P; ++p) {
        m4[0] = fmaxf(m4[0], c[p].x);
        m4[1] = fmaxf(m4[1], c[p].y);
        m4[2] = fmaxf(m4[2], -c[p].x);
        m4[3] = fmaxf(m4[3], -c[p].y);
    }
    group_max4<G>(m4, l, mask, base);
    const float mx[2] = {m4[0], m4[1]}, mn[2] = {-m4[2], -m4[3]};
    // the shifted coordinates are formed again for the gradients (two
    // instructions a pin, against registers that hold four blocks an SM)
    const float2 ig = both(inv_g), nig = both(-inv_g);
    const float2 nmx = make_float2(-mx[0], -mx[1]), nmn = make_float2(-mn[0], -mn[1]);
    float2 ep[P], em[P], bp = both(0.f), bm = both(0.f), cp = both(0.f), cm = both(0.f);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const float2 dp = add2(c[p], nmx), dm = add2(c[p], nmn);
        ep[p] = exp2_pair(mul2(dp, ig));
        em[p] = exp2_pair(mul2(dm, nig));
        if (!v[p]) ep[p] = em[p] = both(0.f);
        bp = add2(bp, ep[p]);
        bm = add2(bm, em[p]);
        cp = fma2(ep[p], dp, cp);
        cm = fma2(em[p], dm, cm);
    }
    float s8[8] = {bp.x, bm.x, cp.x, cm.x, bp.y, bm.y, cp.y, cm.y};
    group_sum8<G>(s8, l, mask, base);
    const PairTerms t(make_float2(s8[0], s8[4]), make_float2(s8[1], s8[5]), make_float2(s8[2], s8[6]),
                      make_float2(s8[3], s8[7]));
    if (l == 0) {
        hpf += (mx[0] - mn[0]) + (mx[1] - mn[1]);
        float wa_net = 0.f;
        wa_net += (mx[0] - mn[0]) - t.nwp.x + t.nwm.x;
        wa_net += (mx[1] - mn[1]) - t.nwp.y + t.nwm.y;
        waf += wa_net;
    }
    const float2 ncp = make_float2(-s8[2], -s8[6]), ncm = make_float2(-s8[3], -s8[7]);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (!v[p] || (nd[p] & kPinNode) >= a.n_grad) continue;
        // x - WA+- fused with the quotient (by hand: left to the compiler it
        // changed the last bit of some gradients with the code around it)
        const float2 g = t.grad(ep[p], em[p], fma2(ncp, t.ibp, add2(c[p], nmx)), fma2(ncm, t.ibm, add2(c[p], nmn)), ig,
                                nig);
        add_grad(a.gq, a.gqx, a.gqy, nd[p], g.x, g.y);
    }
}

// Nets of sub-bucket [lo, hi) by groups of G lanes; the launch's blocks
// [b0, b0 + nb) serve this sub-bucket, this one is block `bid`.
template <int G, int P>
__device__ __forceinline__ void net_groups(const WaArgs &a, int bid, int lo, int hi, int b0, int nb,
                                           const float2 *xy, float inv_g, float &hpf, float &waf) {
    constexpr int per_block = kThreads / G;
    const int lane = threadIdx.x & 31, l = lane & (G - 1), base = lane - l;
    const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << base);
    const int group = (bid - b0) * per_block + (int)threadIdx.x / G, n_groups = nb * per_block;
    for (int e = lo + group; e < hi; e += n_groups) {
        const int s = __ldg(a.net_ptr + e), d = __ldg(a.net_ptr + e + 1) - s;
        net_group<G, P>(a, s, d, l, mask, base, xy, inv_g, hpf, waf);
    }
}

// One net with d <= D pins held in registers by one thread.
template <int D>
__device__ __forceinline__ void net_thread(const int *__restrict__ pins, int d, const float2 *__restrict__ xy,
                                           float inv_g, ull *gq, ull *gqx, ull *gqy, int n_grad, float &hp_acc,
                                           float &wa_acc) {
    int node[D];
    float2 c[D];
    float xmx = -3.0e38f, xmn = 3.0e38f, ymx = -3.0e38f, ymn = 3.0e38f;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        if (j < d) {
            node[j] = __ldg(pins + j);  // raw entry (heavy flag)
            c[j] = __ldg(xy + (node[j] & kPinNode));
            xmx = fmaxf(xmx, c[j].x);
            xmn = fminf(xmn, c[j].x);
            ymx = fmaxf(ymx, c[j].y);
            ymn = fminf(ymn, c[j].y);
        }
    }
    const float2 ig = both(inv_g), nig = both(-inv_g);
    const float2 nmx = make_float2(-xmx, -ymx), nmn = make_float2(-xmn, -ymn);
    float2 ep[D], em[D], bp = both(0.f), bm = both(0.f), cp = both(0.f), cm = both(0.f);
#pragma unroll
    for (int j = 0; j < D; ++j) {
        if (j < d) {
            const float2 dp = add2(c[j], nmx), dm = add2(c[j], nmn);
            ep[j] = exp2_pair(mul2(dp, ig));
            em[j] = exp2_pair(mul2(dm, nig));
            bp = add2(bp, ep[j]);
            bm = add2(bm, em[j]);
            cp = fma2(ep[j], dp, cp);
            cm = fma2(em[j], dm, cm);
        }
    }
    const PairTerms t(bp, bm, cp, cm);
    float wa_net = 0.f;
    wa_net += (xmx - xmn) - t.nwp.x + t.nwm.x;
    wa_net += (ymx - ymn) - t.nwp.y + t.nwm.y;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        if (j < d && (node[j] & kPinNode) < n_grad) {
            const float2 g =
                t.grad(ep[j], em[j], add2(add2(c[j], nmx), t.nwp), add2(add2(c[j], nmn), t.nwm), ig, nig);
            add_grad(gq, gqx, gqy, node[j], g.x, g.y);
        }
    }
    hp_acc += (xmx - xmn) + (ymx - ymn);
    wa_acc += wa_net;
}

// One 2-pin net (pins a, b) in closed form.  With d = |x_a - x_b|, e =
// exp(-d/g) and r = 1/(1 + e), the terms above reduce to b+ = b- = 1 + e and
//   dWA/dx_max = (1 - e) r + 2 d e r^2 / g = -dWA/dx_min,
//   WA = d (1 - e) r,  HPWL = d
// (the same quantities; one exponential per axis instead of four).
__device__ __forceinline__ void net_pair(const WaArgs &a, int s, const float2 *__restrict__ xy, float inv_g,
                                         float &hp_acc, float &wa_acc) {
    const int na = __ldg(a.pin_node + s), nb = __ldg(a.pin_node + s + 1);  // raw entries (heavy flag)
    const float2 pa = __ldg(xy + (na & kPinNode)), pb = __ldg(xy + (nb & kPinNode));
    const float dd[2] = {pa.x - pb.x, pa.y - pb.y};
    float g[2];
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
        const float d = fabsf(dd[ax]);
        const float e = __expf(-d * inv_g);
        const float r = rcp(1.f + e);
        const float gmax = r * (1.f - e) + 2.f * d * e * r * r * inv_g;
        g[ax] = dd[ax] >= 0.f ? gmax : -gmax;  // pin a is the larger coordinate, or they coincide (g = 0)
        hp_acc += d;
        wa_acc += d * (1.f - e) * r;
    }
    if ((na & kPinNode) < a.n_grad) add_grad(a.gq, a.gqx, a.gqy, na, g[0], g[1]);
    if ((nb & kPinNode) < a.n_grad) add_grad(a.gq, a.gqx, a.gqy, nb, -g[0], -g[1]);
}

}  // namespace

// Bucket B (degree <= D) of the thread-per-net nets: registers sized for D.
template <int D, int B>
__device__ __forceinline__ void wa_small_body(const WaArgs &a, VBlock vb) {
    __shared__ double red[32];
    const float gamma = a.gamma > 0.f ? a.gamma : a.sc->f_gamma;
    const float inv_g = 1.f / gamma;
    const float2 *xy = a.xy;  // every node's position, interleaved
    // per-thread partials in FP32 (a thread owns a few nets), FP64 from the
    // block sum on: the FP64 pipe of this part is narrow
    float hpf = 0.f, waf = 0.f;
    const int lo = a.bucket_lo[B], hi = a.bucket_lo[B + 1];
    // every net of the 2-pin bucket has degree 2: its pins sit at a computed
    // offset, one dependent load fewer per net
    const int s0 = D == 2 && lo < hi ? __ldg(a.net_ptr + lo) : 0;
    for (int e = lo + vb.id * blockDim.x + threadIdx.x; e < hi; e += vb.n * blockDim.x) {
        if (D == 2) {
            net_pair(a, s0 + 2 * (e - lo), xy, inv_g, hpf, waf);
        } else {
            const int s = __ldg(a.net_ptr + e);
            net_thread<D>(a.pin_node + s, __ldg(a.net_ptr + e + 1) - s, xy, inv_g, a.gq, a.gqx, a.gqy, a.n_grad,
                          hpf, waf);
        }
    }
    // per-block partials in FP32 (folded with compensation by the last block
    // of the warp-per-net launch)
    const float hp = block_sum_ff(hpf, reinterpret_cast<float *>(red));
    const float wa = block_sum_ff(waf, reinterpret_cast<float *>(red));
    int off = 0;
#pragma unroll
    for (int b = 0; b < B; ++b) off += a.bucket_blocks[b];
    if (threadIdx.x == 0) {
        float *pf = reinterpret_cast<float *>(a.partials);
        pf[2 * (off + vb.id)] = hp;
        pf[2 * (off + vb.id) + 1] = wa;
    }
}

// The launches of several do not read one another's results: each is a
// programmatic dependent that starts in the slots that the last blocks of the
// one before leave free, and waits for it only at its end, so that the
// end of the last is the end of all (2M cells: the stage 100 -> 85 us).
template <int D, int B>
__global__ void __launch_bounds__(kThreads) wa_small_kernel(WaArgs a) {
    grid_release();
    wa_small_body<D, B>(a, grid_block());
    grid_wait();
}

// General path of one net of any degree by a warp: three passes over the pins
// (extrema; sums; gradients), pins lane, lane + 32, ...
__device__ __forceinline__ void net_warp_loop(const WaArgs &a, int s, int d, const float2 *xy, float inv_g,
                                              float &hpf, float &waf) {
    const int lane = threadIdx.x & 31;
    float m4[4] = {-3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f};  // max x, max y, -min x, -min y
    for (int j = lane; j < d; j += 32) {
        const int n = __ldg(a.pin_node + s + j) & kPinNode;
        const float2 q = __ldg(xy + n);
        const float x = q.x, y = q.y;
        m4[0] = fmaxf(m4[0], x);
        m4[1] = fmaxf(m4[1], y);
        m4[2] = fmaxf(m4[2], -x);
        m4[3] = fmaxf(m4[3], -y);
    }
    group_max4<32>(m4, lane, 0xffffffffu, 0);
    const float xmx = m4[0], ymx = m4[1], xmn = -m4[2], ymn = -m4[3];
    float s8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // bp bm cp cm for x then y
    for (int j = lane; j < d; j += 32) {
        const int n = __ldg(a.pin_node + s + j) & kPinNode;
        const float2 q = __ldg(xy + n);
        const float c2[2] = {q.x, q.y};
#pragma unroll
        for (int ax = 0; ax < 2; ++ax) {
            const float dp = c2[ax] - (ax ? ymx : xmx), dm = c2[ax] - (ax ? ymn : xmn);
            const float ep = __expf(dp * inv_g), em = __expf(-dm * inv_g);
            s8[4 * ax + 0] += ep;
            s8[4 * ax + 1] += em;
            s8[4 * ax + 2] += ep * dp;
            s8[4 * ax + 3] += em * dm;
        }
    }
    group_sum8<32>(s8, lane, 0xffffffffu, 0);
    AxisTerms t[2];
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
        t[ax].inv_bp = rcp(s8[4 * ax + 0]);
        t[ax].inv_bm = rcp(s8[4 * ax + 1]);
        t[ax].wp = s8[4 * ax + 2] * t[ax].inv_bp;
        t[ax].wm = s8[4 * ax + 3] * t[ax].inv_bm;
    }
    for (int j = lane; j < d; j += 32) {
        const int raw = __ldg(a.pin_node + s + j), n = raw & kPinNode;
        if (n >= a.n_grad) continue;
        const float2 q = __ldg(xy + n);
        const float c2[2] = {q.x, q.y};
        float g[2];
#pragma unroll
        for (int ax = 0; ax < 2; ++ax) {
            const float dp = c2[ax] - (ax ? ymx : xmx), dm = c2[ax] - (ax ? ymn : xmn);
            const float ep = __expf(dp * inv_g), em = __expf(-dm * inv_g);
            g[ax] = ep * t[ax].inv_bp * (1.f + (dp - t[ax].wp) * inv_g) -
                    em * t[ax].inv_bm * (1.f - (dm - t[ax].wm) * inv_g);
        }
        add_grad(a.gq, a.gqx, a.gqy, raw, g[0], g[1]);
    }
    if (lane == 0) {
        hpf += (xmx - xmn) + (ymx - ymn);
        waf += ((xmx - xmn) + t[0].wp - t[0].wm) + ((ymx - ymn) + t[1].wp - t[1].wm);
    }
}

// Nets of degree > 8 (buckets 3..6): blocks [0, b3) take degrees 9..16 with
// 8 lanes per net (two pins per lane, four nets per warp), then 17..32 with 16
// lanes (two pins per lane), 33..64 with 16 lanes (four pins per lane), and
// above 64 with a warp looping over the pins -- the lane group fits the net,
// so few lanes idle, and each group reduction serves two or four pins per lane
// (one pin per lane on 16 and 32 lanes took 9% longer for the stage).
__device__ __forceinline__ void wa_large_body(const WaArgs &a, VBlock vb) {
    __shared__ double red[32];
    const float gamma = a.gamma > 0.f ? a.gamma : a.sc->f_gamma;
    const float inv_g = 1.f / gamma;
    const float2 *xy = a.xy;  // every node's position, interleaved
    // per-thread partials in FP32 (a thread owns a few nets), FP64 from the
    // block sum on: the FP64 pipe of this part is narrow
    float hpf = 0.f, waf = 0.f;
    int b0 = 0;
    const int bid = vb.id;
    if (bid < b0 + a.bucket_blocks[3]) {
        net_groups<8, 2>(a, bid, a.bucket_lo[3], a.bucket_lo[4], b0, a.bucket_blocks[3], xy, inv_g, hpf, waf);
    } else if (bid < (b0 += a.bucket_blocks[3]) + a.bucket_blocks[4]) {
        net_groups<16, 2>(a, bid, a.bucket_lo[4], a.bucket_lo[5], b0, a.bucket_blocks[4], xy, inv_g, hpf, waf);
    } else if (bid < (b0 += a.bucket_blocks[4]) + a.bucket_blocks[5]) {
        net_groups<16, 4>(a, bid, a.bucket_lo[5], a.bucket_lo[6], b0, a.bucket_blocks[5], xy, inv_g, hpf, waf);
    } else {
        b0 += a.bucket_blocks[5];
        const int warp = ((bid - b0) * kThreads + (int)threadIdx.x) >> 5, nwarps = (a.bucket_blocks[6] * kThreads) >> 5;
        for (int e = a.bucket_lo[6] + warp; e < a.bucket_lo[7]; e += nwarps) {
            const int s = __ldg(a.net_ptr + e), d = __ldg(a.net_ptr + e + 1) - s;
            net_warp_loop(a, s, d, xy, inv_g, hpf, waf);
        }
    }
    const float hp = block_sum_ff(hpf, reinterpret_cast<float *>(red));
    const float wa = block_sum_ff(waf, reinterpret_cast<float *>(red));
    float *pf = reinterpret_cast<float *>(a.partials);
    if (threadIdx.x == 0) {
        pf[2 * (a.small_blocks + vb.id)] = hp;
        pf[2 * (a.small_blocks + vb.id) + 1] = wa;
    }
}

// HPWL and WA of partials [0, nb) of all four bucket launches (one block).
__device__ __forceinline__ void wa_fold(const WaArgs &a, int nb) {
    __shared__ double red[32];
    const float *pf = reinterpret_cast<const float *>(a.partials);
    const double h = block_sum_f(kahan_strided(pf, threadIdx.x, nb, blockDim.x, 2), red);
    const double w = block_sum_f(kahan_strided(pf + 1, threadIdx.x, nb, blockDim.x, 2), red);
    if (threadIdx.x == 0) {
        if (a.out) {
            a.out[0] = h;
            a.out[1] = w;
        }
        DevScalars *sc = a.sc;
        if (a.mode == WA_INIT) {
            sc->hpwl = h;
            sc->hpwl_prev = h;
            sc->wa = w;
        } else if (a.mode == WA_LOOP) {
            sc->t_hpwl = h;  // becomes the reported HPWL if the trial is accepted
            sc->t_wa = w;
        }
        *a.counter = 0u;
    }
}

// The last of the four launches: it folds the partials of all of them (the
// three before it have ended behind grid_wait).
__global__ void __launch_bounds__(kThreads, 4) wa_large_kernel(WaArgs a) {
    wa_large_body(a, grid_block());
    grid_wait();
    if (arrive_last(a.counter, gridDim.x)) wa_fold(a, a.small_blocks + (int)gridDim.x);
}

// The four launches in one, by block range: where all their blocks are
// resident at once.  At its largest bucket's registers it holds fewer blocks an
// SM, and past one wave that costs more than three launches (an iteration
// with the four / with the one: 576 cells 27.1 / 25.1 us, 5k 31.6 / 27.3, 60k
// 36.0 / 35.4; 200k, 1582 blocks, 72.2 / 75.2; 2M 210 / 254).
__global__ void __launch_bounds__(kThreads, 3) wa_all_kernel(WaArgs a) {
    int b = (int)blockIdx.x;
    if (b < a.bucket_blocks[0]) {
        wa_small_body<2, 0>(a, VBlock{b, a.bucket_blocks[0]});
    } else if ((b -= a.bucket_blocks[0]) < a.bucket_blocks[1]) {
        wa_small_body<4, 1>(a, VBlock{b, a.bucket_blocks[1]});
    } else if ((b -= a.bucket_blocks[1]) < a.bucket_blocks[2]) {
        wa_small_body<8, 2>(a, VBlock{b, a.bucket_blocks[2]});
    } else {
        wa_large_body(a, VBlock{b - a.bucket_blocks[2], (int)gridDim.x - a.small_blocks});
    }
    if (arrive_last(a.counter, gridDim.x)) wa_fold(a, (int)gridDim.x);
}

int wa_plan(WaArgs &a) {
    const int per = a.block_nets > kThreads ? a.block_nets : kThreads;
    auto grid = [per](int items) {
        int b = (items + per - 1) / per;
        return b < 1 ? 1 : (b > kWaMaxBlocks ? kWaMaxBlocks : b);
    };
    for (int b = 0; b < 3; ++b) a.bucket_blocks[b] = grid(a.bucket_lo[b + 1] - a.bucket_lo[b]);
    // large-net sub-buckets: lanes per net 16, 32, 16, 32; <= kWaMaxBlocks in all
    const int lanes[4] = {8, 16, 16, 32};
    int large = 0;
    for (int b = 3; b < kWaBuckets; ++b) {
        a.bucket_blocks[b] = std::min(grid((a.bucket_lo[b + 1] - a.bucket_lo[b]) * lanes[b - 3]), kWaMaxBlocks / 4);
        large += a.bucket_blocks[b];
    }
    a.small_blocks = a.bucket_blocks[0] + a.bucket_blocks[1] + a.bucket_blocks[2];
    a.all_blocks = a.small_blocks + large;
    return a.all_blocks;
}

// Positions (px, py) of all nodes -> the interleaved copy the WA kernels read.
__global__ void interleave_kernel(int n, const float *__restrict__ px, const float *__restrict__ py,
                                  float2 *__restrict__ xy) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        xy[i] = make_float2(px[i], py[i]);
}

void launch_interleave(int n, const float *px, const float *py, float2 *xy, cudaStream_t st) {
    if (n <= 0) return;
    int blocks = (n + kThreads - 1) / kThreads;
    if (blocks > 2048) blocks = 2048;
    interleave_kernel<<<blocks, kThreads, 0, st>>>(n, px, py, xy);
}

// Up to here the density chain is the longer branch of a trial: its stream goes
// first (ap_create) and the larger nets' launch, which would fill what the
// chain needs, waits for the three before it.  Beyond, the branches have equal
// priority and all four launches follow one another without a gap.  (A trial,
// the first form / the second / four ordinary launches going first, started at
// the centre and spread: 100k cells 31.8, 30.6 / 33.0, 32.3 / 33.5, 32.0 us;
// 350k 86.6, 54.9 / 88.0, 60.1 / 92.4, 56.7; 500k 91.6, 64.9 / 89.6, 71.0 /
// 94.4, 67.5; 700k 127.8, 118.9 / 119.8, 114.7 / 123.5, 119.4; 2M 245.7, 201.8 /
// 191.5, 188.6 / 194.6, 192.4.)
bool wa_longer(int n_nets) { return n_nets > 600000; }

void launch_wirelength(const WaArgs &a0, cudaStream_t st) {
    WaArgs a = a0;
    if (a.mode != WA_LOOP) launch_interleave(a.n_nodes, a.px, a.py, a.xy, st);
    const int all = wa_plan(a), large = all - a.small_blocks;
    static int wave = 0;
    if (wave <= 0) wave = wave_of((const void *)wa_all_kernel, kThreads, 456);
    if (all <= wave) {
        wa_all_kernel<<<all, kThreads, 0, st>>>(a);
        return;
    }
    wa_small_kernel<2, 0><<<a.bucket_blocks[0], kThreads, 0, st>>>(a);
    launch_dependent(wa_small_kernel<4, 1>, a.bucket_blocks[1], kThreads, 0, st, a);
    launch_dependent(wa_small_kernel<8, 2>, a.bucket_blocks[2], kThreads, 0, st, a);
    if (wa_longer(a.n_nets))
        launch_dependent(wa_large_kernel, large, kThreads, 0, st, a);
    else
        wa_large_kernel<<<large, kThreads, 0, st>>>(a);
}

// The batched form: the four bucket launches of every instance as records of
// one persistent launch (WaArgs::bucket), so that the buckets with few blocks
// fill the GPU together; an instance's sums fold in the last of all its blocks.
// (As four launches one after the other, the 3-4- and 5-8-pin nets on a third
// and a tenth of the resident blocks: 186 us for 32 instances, 126 in one.)
__global__ void __launch_bounds__(kThreads, 3) persist_wa_kernel(PersistQueue q, const WaArgs *recs) {
    persist_loop(q, recs, [](const WaArgs &a, VBlock vb, int) {
        if (a.bucket == 0) wa_small_body<2, 0>(a, vb);
        else if (a.bucket == 1) wa_small_body<4, 1>(a, vb);
        else if (a.bucket == 2) wa_small_body<8, 2>(a, vb);
        else wa_large_body(a, vb);
        if (arrive_last(a.counter, a.all_blocks)) wa_fold(a, a.all_blocks);
    });
}

int persist_wa_wave() {
    static int wave = 0;
    if (!wave) wave = wave_of((const void *)persist_wa_kernel, kThreads, 456);
    return wave;
}

void launch_persist_wa(const PersistQueue &q, int items, const WaArgs *recs, cudaStream_t st) {
    persist_wa_kernel<<<persist_blocks(persist_wa_wave(), items), kThreads, 0, st>>>(q, recs);
}

}  // namespace ap
