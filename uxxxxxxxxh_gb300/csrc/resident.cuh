// Resident runs: a whole rank-2 program (T sweeps) in one cooperative launch,
// the grid held in shared memory from the first sweep to the last.
//
// A 2D grid of up to a few million cells is bound by latency when each sweep
// is its own launch: a row is little work, so a CTA spends it waiting for
// loads and barriers, and FP64 runs add a range scan with a host round trip
// and four conversion launches.  152 SMs hold 33 MB of shared memory, though:
// a domain that fits is cut into one box per CTA (one CTA per SM), loaded
// once, swept T times in place, and written once (step T to a, step T - 1 to
// b).  Between steps the CTAs exchange only the cells within R of their
// boxes' edges -- 500 of 14000 cells a box at 1448^2, radius 1.  (3D boxes
// were built too and measured: their surfaces are a third of their cells, and
// from 64^3 on the streaming sweeps are faster, 5.7 against 10 us a sweep for
// an FP32 3d1r star at 128^3.)
//
//  * Exchange.  A published cell is its value and the step number in one
//    8-byte word (float pairs: two words), written by its owner during the
//    step and polled by its readers until the number matches: no fence, no
//    flag, no grid barrier; one L2 round trip per step.  Two buffers
//    alternate by the step's parity: a CTA publishes step s + 2 only after it
//    has read its readers' step s + 1, which they computed after reading its
//    step s.  The step numbers are cleared before the first step, behind the
//    launch's only grid-wide barrier.
//  * In place.  A step's results go to the slots G + R rows below (odd steps,
//    groups of rows ascending) or above (even steps, descending) the rows that
//    they were computed from, so the CTA needs bz + 3R + G + 1 rows and a block
//    barrier every G rows instead of a second copy.  G is as large as shared
//    memory allows (the whole box for small ones).
//  * A thread computes two rows of a column at a time (packed float-pair
//    sums, the column queue in registers) and walks L rows.
//  * FP64 grids under UHS_ARITH_AUTO: the kernel scans its cells' exponents
//    itself, the barrier folds them over the grid, and every CTA derives the
//    pairs' power-of-two scale (pair_range); when the range needs native FP64
//    it returns with both grids untouched and says so in *verdict.
//  * Per point the sums are the streaming kernel's: the same terms, order and
//    roundings, so results are bit-identical to it.  A program whose sweeps
//    would run in place (fewer than 8, or fewer than 4 from 2^21 points on)
//    rounds to FP64 between steps (round64), as they do.
//
// Bound: instruction issue (float pairs) and latency in the walk, then the
// exchange's round trip (about 1 us of the step).
//
// All waits are bounded (kResidentWaitCycles): one that runs out sets the
// timeout flag, and every CTA returns.
// Other streams' work delays a run but uses up none of its waits: a cooperative
// launch starts when all of its CTAs can be placed (measured: beside a kernel that
// held two SMs for 3 s, a run that needs every SM started at its end).
#pragma once
#include <type_traits>

#include "df32.cuh"
#include "resident.h"

namespace uhs {

constexpr long long kResidentWaitCycles = 1ll << 31;

template <int SHAPE, int R>
struct ResShape {
    static_assert(is_rank2_shape(SHAPE), "resident runs are rank 2");
    static constexpr bool star = SHAPE == kStar2, sep = SHAPE == kSep2;
    static constexpr int D = 2 * R + 1;
    static constexpr int NT = sep ? 2 * D : star ? 4 * R + 1 : D * D;
};

template <int NT>
struct ResArgs {
    ResCall c;
    float2 chl[NT];
    float cl_sum[3];
    float cab[NT];
};

// ---- published cells: {value, step} words, each written and read whole ----
__device__ __forceinline__ uint64_t pub_word(float v, unsigned step) {
    return static_cast<uint64_t>(step) << 32 | __float_as_uint(v);
}
__device__ __forceinline__ void pub_store(uint4 *p, float2 v, unsigned step, unsigned when) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n}" ::"l"(
                     p),
                 "l"(pub_word(v.x, step)), "l"(pub_word(v.y, step)), "r"(when)
                 : "memory");
}
__device__ __forceinline__ bool pub_load(const uint4 *p, float2 &v, unsigned step) {
    uint64_t a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = make_float2(__uint_as_float(static_cast<unsigned>(a)), __uint_as_float(static_cast<unsigned>(b)));
    return static_cast<unsigned>(a >> 32) == step && static_cast<unsigned>(b >> 32) == step;
}
__device__ __forceinline__ void pub_store(uint2 *p, float v, unsigned step, unsigned when) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p st.relaxed.gpu.global.b64 [%0], %1;\n}" ::"l"(p),
                 "l"(pub_word(v, step)), "r"(when)
                 : "memory");
}
__device__ __forceinline__ bool pub_load(const uint2 *p, float &v, unsigned step) {
    uint64_t a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    v = __uint_as_float(static_cast<unsigned>(a));
    return static_cast<unsigned>(a >> 32) == step;
}

// i / d for i < 2^16, d < 2^16 by a multiply (m = ceil(2^32 / d); d = 1 by itself)
struct FastDiv {
    unsigned m;
    int d;
    __device__ __forceinline__ explicit FastDiv(int d_) : m(d_ > 1 ? 0xffffffffu / d_ + 1u : 0u), d(d_) {}
    __device__ __forceinline__ int div(int i) const { return d > 1 ? static_cast<int>(__umulhi(i, m)) : i; }
};

// Two rows' points of one column, in the streaming kernel's order.
// c: the upper point's own cell; q[R + dz]: its column.
template <int SHAPE, int R, class Args>
__device__ __forceinline__ void res_pair(const Args &a, const float2 *c, const float2 *q, int W, float2 &o0,
                                         float2 &o1) {
    using SI = ResShape<SHAPE, R>;
    const float2 *const c1 = c + W;
    u64 h, l;
    if constexpr (SI::star) {
        constexpr int SC = 4 * R, SX = 2 * R;  // slots of the centre and the first x neighbour
        float2 x0[2 * R], x1[2 * R];           // -d, +d
#pragma unroll
        for (int d = 1; d <= R; ++d) {
            x0[2 * d - 2] = c[-d];
            x0[2 * d - 1] = c[d];
            x1[2 * d - 2] = c1[-d];
            x1[2 * d - 1] = c1[d];
        }
        float b0 = anchor_add(0.0f, a.cab[SC], q[R]), b1 = anchor_add(0.0f, a.cab[SC], q[R + 1]);
#pragma unroll
        for (int d = 1; d <= R; ++d) {
            b0 = anchor_add(b0, a.cab[2 * d - 2], q[R - d]);
            b0 = anchor_add(b0, a.cab[2 * d - 1], q[R + d]);
            b1 = anchor_add(b1, a.cab[2 * d - 2], q[R + 1 - d]);
            b1 = anchor_add(b1, a.cab[2 * d - 1], q[R + 1 + d]);
        }
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) {
            b0 = anchor_add(b0, a.cab[SX + k], x0[k]);
            b1 = anchor_add(b1, a.cab[SX + k], x1[k]);
        }
        dfa2 s;
        dfa2_first(s, pk2(b0, b1), a.chl[SC].x, a.chl[SC].y, q[R], q[R + 1]);
#pragma unroll
        for (int d = 1; d <= R; ++d) {
            dfa2_add(s, a.chl[2 * d - 2].x, a.chl[2 * d - 2].y, q[R - d], q[R + 1 - d]);
            dfa2_add(s, a.chl[2 * d - 1].x, a.chl[2 * d - 1].y, q[R + d], q[R + 1 + d]);
        }
#pragma unroll
        for (int k = 0; k < 2 * R; ++k) dfa2_add(s, a.chl[SX + k].x, a.chl[SX + k].y, x0[k], x1[k]);
        dfa2_renorm(dfa2_end(s), h, l);
    } else if constexpr (SI::sep) {
        // q holds x-filtered rows; the row pass
        float b0 = 0.0f, b1 = 0.0f;
#pragma unroll
        for (int k = 0; k < SI::D; ++k) {
            b0 = anchor_add(b0, a.cab[k], q[k]);
            b1 = anchor_add(b1, a.cab[k], q[k + 1]);
        }
        dfa2 s;
        dfa2_first(s, pk2(b0, b1), a.chl[0].x, a.chl[0].y, q[0], q[1]);
#pragma unroll
        for (int k = 1; k < SI::D; ++k) dfa2_add(s, a.chl[k].x, a.chl[k].y, q[k], q[k + 1]);
        dfa2_renorm(dfa2_end(s), h, l);
    } else {
        df2 s;
#pragma unroll
        for (int dz = -R; dz <= R; ++dz)
#pragma unroll
            for (int dx = -R; dx <= R; ++dx) {
                const int k = (dz + R) * SI::D + dx + R, off = dz * W + dx;
                if (k == 0) df2_mul_s(s, a.chl[k].x, a.chl[k].y, c[off], c1[off]);
                else df2_fma_s(s, a.chl[k].x, a.chl[k].y, c[off], c1[off]);
            }
        renorm2(s, h, l);
    }
    upk2(h, o0.x, o1.x);
    upk2(l, o0.y, o1.y);
}

template <int SHAPE, int R, class Args>
__device__ __forceinline__ float res_point(const Args &a, const float *c, const float *q, int W) {
    using SI = ResShape<SHAPE, R>;
    float s;
    if constexpr (SI::star) {
        s = fmaf(a.cl_sum[0], q[R], a.chl[4 * R].x * q[R]);
#pragma unroll
        for (int d = 1; d <= R; ++d) {
            s = fmaf(a.chl[2 * d - 2].x, q[R - d], s);
            s = fmaf(a.chl[2 * d - 1].x, q[R + d], s);
        }
#pragma unroll
        for (int d = 1; d <= R; ++d) {
            s = fmaf(a.chl[2 * R + 2 * d - 2].x, c[-d], s);
            s = fmaf(a.chl[2 * R + 2 * d - 1].x, c[d], s);
        }
    } else if constexpr (SI::sep) {
        s = a.chl[0].x * q[0];
#pragma unroll
        for (int k = 1; k < SI::D; ++k) s = fmaf(a.chl[k].x, q[k], s);
        s = fmaf(a.cl_sum[0], q[R], s);
    } else {
        s = 0.0f;
#pragma unroll
        for (int dz = -R; dz <= R; ++dz)
#pragma unroll
            for (int dx = -R; dx <= R; ++dx) {
                const int k = (dz + R) * SI::D + dx + R;
                const float v = c[dz * W + dx];
                s = k == 0 ? a.chl[k].x * v : fmaf(a.chl[k].x, v, s);
                if (dz == 0 && dx == 0) s = fmaf(a.cl_sum[0], v, s);
            }
    }
    return s;
}

// x pass of a separable box at cell c
template <int R, class Args>
__device__ __forceinline__ float2 res_xpass(const Args &a, const float2 *c) {
    constexpr int D = 2 * R + 1;
    float b = 0.0f;
#pragma unroll
    for (int k = 0; k < D; ++k) b = anchor_add(b, a.cab[D + k], c[k - R]);
    dfa s;
    dfa_first(s, b, a.chl[D].x, a.chl[D].y, c[-R]);
#pragma unroll
    for (int k = 1; k < D; ++k) dfa_add(s, a.chl[D + k].x, a.chl[D + k].y, c[k - R]);
    return dfa_renorm(dfa_end(s));
}
template <int R, class Args>
__device__ __forceinline__ float res_xpass(const Args &a, const float *c) {
    constexpr int D = 2 * R + 1;
    float s = a.chl[D].x * c[-R];
#pragma unroll
    for (int k = 1; k < D; ++k) s = fmaf(a.chl[D + k].x, c[k - R], s);
    return fmaf(a.cl_sum[1], c[0], s);
}

template <int SHAPE, int R, int ST>
__global__ void __launch_bounds__(resident_threads(ST == kStF64), 1)
    k_resident(const __grid_constant__ ResArgs<ResShape<SHAPE, R>::NT> args) {
    using SI = ResShape<SHAPE, R>;
    constexpr bool F64 = ST == kStF64;
    constexpr bool QUEUE = SI::star || SI::sep;
    constexpr int CORNER = SI::star ? 0 : R;  // box shapes read the halo's corners too
    constexpr int NT = resident_threads(F64);
    using TS = std::conditional_t<F64, double, float>;
    using TC = std::conditional_t<F64, float2, float>;
    using PUB = std::conditional_t<F64, uint4, uint2>;
    const ResCall &a = args.c;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TC *const cell0 = reinterpret_cast<TC *>(smem_raw) + R;  // slot 0's column 0
    unsigned *const halo = reinterpret_cast<unsigned *>(smem_raw + a.halo_off);
    __shared__ unsigned s_hi, s_lo;
    const int tid = threadIdx.x;

    // this CTA's box of the domain
    const int cx = blockIdx.x % a.px, cz = blockIdx.x / a.px;
    const int x0 = cx * a.nx / a.px, z0 = cz * a.nz / a.pz;
    const int bx = (cx + 1) * a.nx / a.px - x0, bz = (cz + 1) * a.nz / a.pz - z0;
    const int W = bx + 2 * R;
    const int shift = a.G + R;  // rows between a step's source and its results
    PUB *const pub = static_cast<PUB *>(a.pub);
    const int64_t pub_stride = static_cast<int64_t>(a.nz) * a.nx;
    // cells left of the first or from the second number on are published
    const int sx0 = x0 > 0 ? R : 0, sx1 = x0 + bx < a.nx ? bx - R : bx;
    const int sz0 = z0 > 0 ? R : 0, sz1 = z0 + bz < a.nz ? bz - R : bz;
    auto grid_at = [&](int par, int z, int x) -> TS * {  // box coordinates (may lie in the halo)
        return par == 0 ? static_cast<TS *>(a.a) + (a.lb0 + z0 + z) * a.as0 + (a.lb2 + x0 + x)
                        : static_cast<TS *>(a.b) + (a.lb0 + z0 + z) * a.bs0 + (a.lb2 + x0 + x);
    };
    auto pub_index = [&](int z, int x) { return static_cast<int64_t>(z0 + z) * a.nx + (x0 + x); };
    auto in_domain = [&](int z, int x) {
        return static_cast<unsigned>(z0 + z) < static_cast<unsigned>(a.nz) &&
               static_cast<unsigned>(x0 + x) < static_cast<unsigned>(a.nx);
    };
    // the halo cells' places in the box with its halo (below 2^16 cells), the
    // top bit set inside the domain: the rows above and below, then the columns
    const int hw = bx + 2 * CORNER, n_rows = 2 * R * hw, n_halo = n_rows + 2 * R * bz;
    const FastDiv dhw(hw), dbx(bx), dw(W);
    for (int i = tid; i < n_halo; i += NT) {
        int z, x;
        if (i < n_rows) {
            const int r = dhw.div(i);
            x = i - r * hw - CORNER;
            z = r < R ? r - R : bz + r - R;
        } else {
            const int k = (i - n_rows) % (2 * R);
            z = (i - n_rows) / (2 * R);
            x = k < R ? k - R : bx + k - R;
        }
        halo[i] = (in_domain(z, x) ? 0x80000000u : 0u) | static_cast<unsigned>((z + R) * W + x + R);
    }
    auto halo_cell = [&](unsigned w, int &z, int &x) {
        const int o = static_cast<int>(w & 0xffffu), r = dw.div(o);
        z = r - R;
        x = o - r * W - R;
    };
    __syncthreads();

    // ---- clear the step numbers of the cells this CTA publishes; scan exponents
    unsigned hi = 0u, lo = 0u;  // largest exponent field; largest 0x800 - exponent of a nonzero value
    auto scan = [&](double v) {
        const unsigned h = static_cast<unsigned>(__double2hiint(v)), e = (h >> 20) & 0x7ffu;
        hi = max(hi, e);
        if ((h << 1) | static_cast<unsigned>(__double2loint(v))) lo = max(lo, 0x800u - e);
    };
    const int n_own = bz * bx;
    for (int i = tid; i < n_own; i += NT) {
        const int z = dbx.div(i), x = i - z * bx;
        if (x < sx0 || x >= sx1 || z < sz0 || z >= sz1) {
            pub_store(pub + pub_index(z, x), TC{}, 0u, 1u);
            pub_store(pub + pub_stride + pub_index(z, x), TC{}, 0u, 1u);
        }
        if constexpr (F64) scan(*grid_at(0, z, x));
    }
    if constexpr (F64) {
        for (int i = tid; i < n_halo; i += NT) {
            int z, x;
            halo_cell(halo[i], z, x);
            scan(*grid_at(0, z, x));
            if (!(halo[i] >> 31)) scan(*grid_at(1, z, x));
        }
        for (int o = 16; o > 0; o >>= 1) {
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        }
        if (tid == 0) s_hi = s_lo = 0u;
        __syncthreads();
        if ((tid & 31) == 0) {
            atomicMax(&s_hi, hi);
            atomicMax(&s_lo, lo);
        }
    }
    // ---- the launch's only grid-wide barrier (ctl: arrivals, leavers, hi, lo; zero between runs)
    bool ok = true;
    __syncthreads();
    if (tid == 0) {
        if constexpr (F64) {
            atomicMax(a.ctl + 2, s_hi);
            atomicMax(a.ctl + 3, s_lo);
        }
        __threadfence();
        atomicAdd(a.ctl, 1u);
        const long long t0 = clock64();
        while (*reinterpret_cast<volatile unsigned *>(a.ctl) < gridDim.x) {
            if (clock64() - t0 > kResidentWaitCycles) {
                ok = false;
                break;
            }
        }
        __threadfence();
        if constexpr (F64) {
            s_hi = *reinterpret_cast<volatile unsigned *>(a.ctl + 2);
            s_lo = *reinterpret_cast<volatile unsigned *>(a.ctl + 3);
        }
        // the last CTA to have read them resets the words for the stream's next run
        __threadfence();
        if (atomicAdd(a.ctl + 1, 1u) == gridDim.x - 1) {
            a.ctl[0] = a.ctl[1] = a.ctl[2] = a.ctl[3] = 0u;
        }
        if (!ok) atomicOr(a.err, kDevErrTimeout);
    }
    if (__syncthreads_or(!ok)) return;
    int bias = 896;
    if constexpr (F64) {
        const PairRange pr = pair_range(static_cast<int>(s_hi), s_lo ? static_cast<int>(0x800u - s_lo) : -1, a.growth);
        if (blockIdx.x == 0 && tid == 0) *a.verdict = pr.ok ? 1 : 2;
        if (!pr.ok) return;
        bias = pair_bias(pr.shift);
    }
    unsigned range_err = 0u;
    auto to_tc = [&](TS v) -> TC {
        if constexpr (F64) return split_f64(v, range_err, bias);
        else return v;
    };
    // ---- load the box and its halo from a; the source of step 1 sits `shift` rows up
    {
        TC *const src = cell0 + (shift + R) * W;
        for (int i = tid; i < n_own; i += NT) {
            const int z = dbx.div(i), x = i - z * bx;
            src[z * W + x] = to_tc(*grid_at(0, z, x));
        }
        for (int i = tid; i < n_halo; i += NT) {
            int z, x;
            halo_cell(halo[i], z, x);
            src[z * W + x] = to_tc(*grid_at(0, z, x));
        }
    }
    __syncthreads();

    // FP32: two iterations of the walk make the 4-row queue of radius 1 whole
    constexpr int UNROLL = !F64 && QUEUE && R == 1 ? 2 : 1;
    const int L = a.L, n_groups = (bz + a.G - 1) / a.G;
#pragma unroll 1
    for (int s = 1; s <= a.T; ++s) {
        const bool down = s & 1;  // results `shift` rows below their source
        const TC *const src = cell0 + (down ? shift + R : R) * W;
        TC *const dst = cell0 + (down ? R : shift + R) * W;
        const bool out = s + 1 >= a.T;  // steps T - 1 and T go to the grids
        const bool join = out || (F64 && a.round64);
        const int par = s & 1;
        PUB *const pubs = pub + par * pub_stride;
#pragma unroll 1
        for (int gi = 0; gi < n_groups; ++gi) {
            if (gi > 0) __syncthreads();
            // rows [gz, gz + gn): ascending groups when results move down
            const int gz = (down ? gi : n_groups - 1 - gi) * a.G, gn = min(a.G, bz - gz);
            const int items = bx * ((gn + L - 1) / L);
#pragma unroll 1
            for (int i = tid; i < items; i += NT) {
                const int run = dbx.div(i), x = i - run * bx;
                const int za = gz + run * L, n = min(L, gz + gn - za);
                const TC *c = src + za * W + x;
                TC *d = dst + za * W + x;
                TC q[QUEUE ? 2 * R + 2 : 1];
                if constexpr (QUEUE) {
#pragma unroll
                    for (int k = 0; k < 2 * R; ++k) {
                        if constexpr (SI::sep) q[k + 2] = res_xpass<R>(args, c + (k - R) * W);
                        else q[k + 2] = c[(k - R) * W];
                    }
                }
                // the walk's rows that are published, one bit each
                unsigned pm = x < sx0 || x >= sx1 ? ~0u : 0u;
                if (za < sz0) pm |= (1u << (sz0 - za)) - 1u;
                if (za + n > sz1) pm |= za >= sz1 ? ~0u : ~0u << (sz1 - za);
                pm &= n < 32 ? (1u << n) - 1u : ~0u;
                if (s == a.T) pm = 0u;
                // (an odd last pair's second row lies past the box or in a halo
                // slot of the result, which is loaded afterwards)
#pragma unroll UNROLL
                for (int j = 0; j < n; j += 2) {
                    if constexpr (QUEUE) {
#pragma unroll
                        for (int k = 0; k < 2 * R; ++k) q[k] = q[k + 2];
                        if constexpr (SI::sep) {
                            q[2 * R] = res_xpass<R>(args, c + R * W);
                            q[2 * R + 1] = res_xpass<R>(args, c + (R + 1) * W);
                        } else {
                            q[2 * R] = c[R * W];
                            q[2 * R + 1] = c[(R + 1) * W];
                        }
                    }
                    TC o0, o1;
                    if constexpr (F64) {
                        res_pair<SHAPE, R>(args, c, q, W, o0, o1);
                    } else {
                        o0 = res_point<SHAPE, R>(args, c, q, W);
                        o1 = res_point<SHAPE, R>(args, c + W, q + (QUEUE ? 1 : 0), W);
                    }
                    if (join) {
                        const bool two = j + 1 < n;
                        TS v0, v1;
                        if constexpr (F64) {
                            if (!two) o1 = make_float2(0.0f, 0.0f);
                            range_err |= (__float_as_uint(o0.x) & 0x7f800000u) == 0x7f800000u;
                            range_err |= (__float_as_uint(o1.x) & 0x7f800000u) == 0x7f800000u;
                            v0 = join_f64(o0.x, o0.y, bias);
                            v1 = join_f64(o1.x, o1.y, bias);
                            if (a.round64) {
                                o0 = split_f64(v0, range_err, bias);
                                o1 = split_f64(v1, range_err, bias);
                            }
                        } else {
                            v0 = o0;
                            v1 = o1;
                        }
                        if (out) {
                            TS *const go = grid_at(par, za + j, x);
                            go[0] = v0;
                            if (two) go[par == 0 ? a.as0 : a.bs0] = v1;
                        }
                    }
                    d[0] = o0;
                    d[W] = o1;
                    if (pm & 3u) {
                        PUB *const pk = pubs + pub_index(za + j, x);
                        pub_store(pk, o0, s, pm & 1u);
                        pub_store(pk + a.nx, o1, s, pm & 2u);
                    }
                    pm >>= 2;
                    c += 2 * W;
                    d += 2 * W;
                }
            }
        }
        if (s == a.T) break;
        // ---- the next step's halo: published cells inside the domain, the
        // grid's own halo outside.  The halo slots of the result hold nothing
        // any thread still reads once every group is done.
        __syncthreads();
        bool late = false;
        const long long t0 = clock64();
#pragma unroll 1
        for (int i0 = tid; i0 < n_halo; i0 += 4 * NT) {
            const PUB *pp[4];
            TC *sp[4];
            unsigned pend = 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * NT;
                pp[k] = nullptr;
                sp[k] = nullptr;
                if (i < n_halo) {
                    const unsigned w = halo[i];
                    int z, x;
                    halo_cell(w, z, x);
                    sp[k] = dst + z * W + x;
                    if (w >> 31) {
                        pp[k] = pubs + pub_index(z, x);
                        pend |= 1u << k;
                    } else {
                        *sp[k] = to_tc(*grid_at(par, z, x));
                    }
                }
            }
            while (pend) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (pend >> k & 1u) {
                        TC v;
                        if (pub_load(pp[k], v, s)) {
                            *sp[k] = v;
                            pend &= ~(1u << k);
                        }
                    }
                }
                if (pend && clock64() - t0 > kResidentWaitCycles) {
                    late = true;
                    break;
                }
            }
            if (late) break;
        }
        if (__syncthreads_or(late)) {
            if (tid == 0) {
                atomicOr(a.err, kDevErrTimeout);
                if (atomicCAS(a.err + 2, 0u, 1u) == 0u) {  // first timeout: which block, which step
                    a.err[3] = blockIdx.x;
                    a.err[4] = 0u;
                    a.err[5] = static_cast<unsigned>(s);
                    a.err[6] = a.err[7] = 0u;
                }
            }
            return;
        }
    }
    if constexpr (F64) {
        if (range_err) atomicOr(a.err, kDevErrRange);
    }
}

}  // namespace uhs
