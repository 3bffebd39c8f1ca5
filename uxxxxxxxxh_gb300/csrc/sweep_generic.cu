// Generic sweep: any linear stencil expression (up to UHS_MAX_TERMS terms,
// |offset| <= UHS_MAX_RADIUS), evaluated term by term in the order the .dsl
// expression writes them.
//
// This is the kernel shape UHStencil's GPU lowering emits
// (examples/2d5pt_star/2d5pt_gpu.mlir:10-102; its hand-written twin
// examples/3d27pt_box/3d27pt.cu:20-129): a shared-memory input tile with the
// halo around it.  What differs is the schedule:
//   * each CTA streams a chunk of planes along the slowest axis and keeps the
//     2*rz+1 planes a point needs in a ring of shared-memory slots, so every
//     input plane is fetched from global memory once per CTA instead of once
//     per neighbouring plane;
//   * planes arrive by cp.async one plane ahead of the compute, so the fetch
//     of plane z+rz+1 overlaps the sums for plane z;
//   * a thread computes VY points, TY rows apart, so the term's coefficient
//     and its place in the ring are read once for all of them (a table of
//     places per plane, written by the first threads while the plane before
//     is summed), and VY independent sums hide the FP64 and load latency;
//   * results go straight from registers to global memory (no output tile).
// With UHS_ARITH_EXACT every product and sum is rounded separately in
// expression order, which makes the result bit-identical to the serial CPU
// loops (UH-SW/*/stencil_*_driver.serial.c mpe_verify).
//
// Bound: FP64 programs by the FP64 pipe (a DFMA, or DMUL and DADD, per term:
// 90-93 % of the measured DFMA rate); FP32 programs by instruction issue (79 %
// of the slots).  us per sweep with one point per thread and coefficients
// converted at each use -> now, 7-term one-sided program at 256^3: FP32 224 ->
// 64, FP64 265 -> 248, EXACT 445 -> 445 (FP64 takes several rows only where they
// pay, generic_vy); 64^3 FP32 20 -> 11, FP64 21 -> 14;
// 5-term 2D at 4096^2: FP32 209 -> 58 (8 points a thread; 90 at 4), FP64 211 ->
// 169.
#include "uhs_kernels.h"

#include <algorithm>
#include <cstring>

namespace uhs {
namespace {

template <class T, int MAXT>
struct GenericArgs {
    const T *in;
    T *out;
    int64_t in_s0, in_s1, out_s0, out_s1;
    int64_t n0, n1, n2;
    int64_t lb0, lb1, lb2, ub0, ub1, ub2;
    int rz, ry, rx;
    int W, H, NS;
    int zchunk;
    int nterms;
    int place[MAXT];  // dy * W + dx, and dz in the next array
    signed char dz[MAXT];
    T coef[MAXT];
};

template <class T>
__device__ __forceinline__ void cp_async_elem(T *smem, const T *gmem, bool valid) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    const int n = valid ? static_cast<int>(sizeof(T)) : 0;
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::); }

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

// blockDim = (TX, TY); VY output points per thread per plane.
template <class T, int MAXT, bool EXACT, int VY>
__global__ void __launch_bounds__(256) k_generic(const __grid_constant__ GenericArgs<T, MAXT> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *const ring = reinterpret_cast<T *>(smem_raw);
    __shared__ int s_place[2][MAXT];

    const int TX = blockDim.x, TY = blockDim.y;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx, threads = TX * TY;
    const int64_t x0 = a.lb2 + static_cast<int64_t>(blockIdx.x) * TX;
    const int64_t y0 = a.lb1 + static_cast<int64_t>(blockIdx.y) * (TY * VY);
    const int64_t zs = a.lb0 + static_cast<int64_t>(blockIdx.z) * a.zchunk;
    const int64_t ze = min(zs + static_cast<int64_t>(a.zchunk), a.ub0);
    const int plane_elems = a.W * a.H;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the sweep before has completed

    // Ring slots count from the chunk's first plane, zs - rz in slot 0.
    // Planes outside the grid (a program that reaches only upwards in z from
    // a domain starting at 0) are zero-filled.  A thread copies its column of
    // the tile's first TX, TY rows apart, and the 2 rx columns after them go
    // to all threads in turn.
    const int64_t gy0 = y0 - a.ry, gx0 = x0 - a.rx;
    const bool col_ok = gx0 + tx >= 0 && gx0 + tx < a.n2;
    const int tail = 2 * a.rx, tail_rows = tail ? threads / tail : 1;
    const int tr = tail ? tid / tail : 0, tc = TX + (tail ? tid % tail : 0);
    const bool tail_ok = tail && tr < tail_rows && gx0 + tc < a.n2;
    const T *const main0 = a.in + (gy0 + ty) * a.in_s1 + gx0 + tx, *const tail0 = a.in + (gy0 + tr) * a.in_s1 + gx0 + tc;
    auto load_plane = [&](int64_t p, int slot) {
        T *const dst = ring + slot * plane_elems;
        const bool zin = p >= 0 && p < a.n0;
        const int64_t lo = zin ? -gy0 : a.H, hi = zin ? a.n1 - gy0 : 0;  // tile rows inside the grid
        const T *g = main0 + p * a.in_s0;
        for (int r = ty; r < a.H; r += TY, g += TY * a.in_s1) {
            const bool ok = col_ok && r >= lo && r < hi;
            cp_async_elem(dst + r * a.W + tx, ok ? g : a.in, ok);
        }
        if (tail && tr < tail_rows) {
            g = tail0 + p * a.in_s0;
            for (int r = tr; r < a.H; r += tail_rows, g += tail_rows * a.in_s1) {
                const bool ok = tail_ok && r >= lo && r < hi;
                cp_async_elem(dst + r * a.W + tc, ok ? g : a.in, ok);
            }
        }
    };
    // places of every term's cell relative to a point's own, centre plane in slot `cur`
    auto fill_places = [&](int *to, int cur) {
        for (int k = tid; k < a.nterms; k += threads) {
            int s = cur + a.dz[k];
            s += s < 0 ? a.NS : 0;
            s -= s >= a.NS ? a.NS : 0;
            to[k] = s * plane_elems + a.place[k];
        }
    };

    // Prologue: planes zs-rz .. zs+rz, then one plane of look-ahead.
    const int64_t last_needed = ze - 1 + a.rz;
    for (int d = 0; d <= 2 * a.rz; ++d) {
        load_plane(zs - a.rz + d, d);
        cp_async_commit();
    }
    if (zs + a.rz + 1 <= last_needed) load_plane(zs + a.rz + 1, 2 * a.rz + 1);
    cp_async_commit();
    int cur = a.rz, next = 0;  // slots of plane z and of the next plane to load (z + rz + 2)
    fill_places(s_place[0], cur);

    const int64_t y = y0 + ty, x = x0 + tx;
    const T *const c0 = ring + (ty + a.ry) * a.W + (tx + a.rx);
    const int vstep = TY * a.W;
    T *optr = a.out + zs * a.out_s0 + y * a.out_s1 + x;
    int buf = 0;
    for (int64_t z = zs; z < ze; ++z) {
        cp_async_wait_1();
        __syncthreads();
        const int *const place = s_place[buf];
        T acc[VY];
        {
            const T *const p = c0 + place[0];
            const T c = a.coef[0];
#pragma unroll
            for (int v = 0; v < VY; ++v) acc[v] = EXACT ? mul_rn(c, p[v * vstep]) : c * p[v * vstep];
        }
#pragma unroll 4
        for (int k = 1; k < a.nterms; ++k) {
            const T *const p = c0 + place[k];
            const T c = a.coef[k];
#pragma unroll
            for (int v = 0; v < VY; ++v) {
                if constexpr (EXACT) acc[v] = add_rn(acc[v], mul_rn(c, p[v * vstep]));
                else acc[v] = fma(c, p[v * vstep], acc[v]);
            }
        }
        if (x < a.ub2) {
#pragma unroll
            for (int v = 0; v < VY; ++v)
                if (y + v * TY < a.ub1) optr[v * TY * a.out_s1] = acc[v];
        }
        optr += a.out_s0;
        cur = cur + 1 == a.NS ? 0 : cur + 1;
        buf ^= 1;
        fill_places(s_place[buf], cur);
        __syncthreads();
        if (z + a.rz + 2 <= last_needed) load_plane(z + a.rz + 2, next);
        cp_async_commit();
        next = next + 1 == a.NS ? 0 : next + 1;
    }
}

// Points per thread (up to 4, in 2D 8): as many rows as the domain has for them, while the ring
// leaves two CTAs an SM and the tiles, in chunks of 8 planes, still make two
// CTAs for each SM.  FP64 programs gain less from more rows (a row costs an FP64
// pipe term for each of its own, and a thread the time of one or two terms) than
// the last tile's idle rows and, in 2D, an uneven last CTA an SM cost.  So of the
// rows that rule allows they take those with the shortest estimate: 2D of the
// busiest SM, 3D (whose chunks even the SMs out) of all rows, idle ones too.  us a
// run, one row a thread / the most rows / these: 2D 49 points 217 x 2528 T = 8 518
// / 776 / 518, 25 points EXACT 659 x 479 335 / 424 / 335, 5 points 4096^2 T = 2 460
// / 372 / 372; 3D 125 points 152 x 37 x 213 T = 8 3080 / 3370 / 3080, 19 points 116 x
// 77 x 257 915 / 1165 / 914, 7 points EXACT 182 x 156 x 128 978 / 817 / 820.
int generic_vy(const SweepSpec &sp, int TX, int TY, int eb, bool exact) {
    const int64_t nz = sp.ub[0] - sp.lb[0], ny = sp.ub[1] - sp.lb[1], nx = sp.ub[2] - sp.lb[2], sms = device_sm_count();
    const auto tiles_y = [&](int vy) { return (ny + TY * vy - 1) / (TY * vy); };
    int best = 1;
    double shortest = 0.0;
    for (int vy = sp.rank == 2 ? 8 : 4; vy >= 1; vy /= 2) {
        const size_t smem = static_cast<size_t>(2 * sp.rz + 2) * (TX + 2 * sp.rx) * (TY * vy + 2 * sp.ry) * eb;
        const int64_t ctas = (nx + TX - 1) / TX * tiles_y(vy) * ((nz + 7) / 8);
        if (vy > 1 && (smem > 100 * 1024 || ctas < 2 * sms)) continue;
        if (eb == 4) return vy;
        const double terms = sp.nterms;
        const double est = sp.rank == 3 ? static_cast<double>(tiles_y(vy)) * (vy + 2.0 / terms)
                                        : static_cast<double>((ctas + sms - 1) / sms) * (vy + (exact ? 0.75 : 1.5) / terms);
        if (shortest == 0.0 || est < shortest) {
            shortest = est;
            best = vy;
        }
    }
    return best;
}

template <class T, int MAXT, bool EXACT, int VY>
cudaError_t launch_v(const SweepSpec &sp, const LaunchCfg &cfg, const GridView &in, const GridView &out,
                     cudaStream_t st) {
    GenericArgs<T, MAXT> a;
    std::memset(&a, 0, sizeof a);
    a.in = static_cast<const T *>(in.data);
    a.out = static_cast<T *>(out.data);
    a.in_s0 = in.s[0];
    a.in_s1 = in.s[1];
    a.out_s0 = out.s[0];
    a.out_s1 = out.s[1];
    a.n0 = in.n[0];
    a.n1 = in.n[1];
    a.n2 = in.n[2];
    a.lb0 = sp.lb[0];
    a.lb1 = sp.lb[1];
    a.lb2 = sp.lb[2];
    a.ub0 = sp.ub[0];
    a.ub1 = sp.ub[1];
    a.ub2 = sp.ub[2];
    a.rz = sp.rz;
    a.ry = sp.ry;
    a.rx = sp.rx;
    const int TX = cfg.tile_x > 0 ? cfg.tile_x : 32;
    const int TY = cfg.tile_y > 0 ? cfg.tile_y : 8;
    a.W = TX + 2 * sp.rx;
    a.H = TY * VY + 2 * sp.ry;
    a.NS = 2 * sp.rz + 2;
    a.nterms = sp.nterms;
    for (int k = 0; k < sp.nterms; ++k) {
        a.dz[k] = static_cast<signed char>(sp.dz[k]);
        a.place[k] = sp.dy[k] * a.W + sp.dx[k];
        a.coef[k] = static_cast<T>(sp.coef[k]);
    }
    const int64_t nz = sp.ub[0] - sp.lb[0], ny = sp.ub[1] - sp.lb[1], nx = sp.ub[2] - sp.lb[2];
    const int64_t tiles = ((nx + TX - 1) / TX) * ((ny + TY * VY - 1) / (TY * VY));
    int zchunk = cfg.tile_z;
    if (zchunk <= 0) {
        // Enough CTAs to fill the SMs several times over, chunks long enough
        // that the 2*rz warm-up planes stay a small fraction.
        const int64_t want = static_cast<int64_t>(device_sm_count()) * 16;
        const int64_t want_chunks = std::max<int64_t>(1, (want + tiles - 1) / tiles);
        // (grids too small for that: chunks down to 2 planes)
        const int64_t least = std::max(8, 4 * sp.rz), few = device_sm_count() * 4;
        zchunk = (int)std::max<int64_t>(tiles * ((nz + least - 1) / least) < few ? 2 : least,
                                        (nz + want_chunks - 1) / want_chunks);
    }
    if (sizeof(T) == 8 && VY > 1 && cfg.tile_z <= 0 && sp.rank == 3) {
        // FP64 chunks that even the SMs out: several rows a thread make few CTAs an
        // SM, and the busiest SM ends the sweep.  Up to twice the planes, where that
        // leaves four CTAs an SM (below, they wait for latency and not for one
        // another).  us a run, one row a thread / these rows in the usual chunks / in
        // these: 7 points EXACT 160 x 247 x 195 T = 16 3822 / 4083 / 3856, 13 points 342 x
        // 335 x 152 T = 8 3944 / 4068 / 3840.
        const int64_t sms = device_sm_count();
        const auto busiest = [&](int64_t zc) { return (tiles * ((nz + zc - 1) / zc) + sms - 1) / sms * (zc + 1); };
        const int64_t z0 = zchunk;
        int64_t best = busiest(z0) * 19 / 20;
        for (int64_t z = z0 + 1; z <= 2 * z0 && tiles * ((nz + z - 1) / z) >= 4 * sms; ++z)
            if (busiest(z) < best) {
                best = busiest(z);
                zchunk = static_cast<int>(z);
            }
    }
    a.zchunk = (int)std::min<int64_t>(zchunk, nz);
    const size_t smem = (size_t)a.NS * a.W * a.H * sizeof(T);
    auto kern = k_generic<T, MAXT, EXACT, VY>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3((unsigned)((nx + TX - 1) / TX), (unsigned)((ny + TY * VY - 1) / (TY * VY)),
                      (unsigned)((nz + a.zchunk - 1) / a.zchunk));
    lc.blockDim = dim3(TX, TY);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at{};  // programmatic dependent launch (stream_launch.cuh)
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, kern, a);
    if (e == cudaSuccess) count_launch();
    return e;
}

template <class T, int MAXT, bool EXACT>
cudaError_t launch_t(const SweepSpec &sp, const LaunchCfg &cfg, const GridView &in, const GridView &out,
                     cudaStream_t st) {
    for (int i = 0; i < 3; ++i)
        if (sp.ub[i] <= sp.lb[i]) return cudaSuccess;
    const int TX = cfg.tile_x > 0 ? cfg.tile_x : 32, TY = cfg.tile_y > 0 ? cfg.tile_y : 8;
    switch (generic_vy(sp, TX, TY, sizeof(T), EXACT)) {
        case 8: return launch_v<T, MAXT, EXACT, 8>(sp, cfg, in, out, st);
        case 4: return launch_v<T, MAXT, EXACT, 4>(sp, cfg, in, out, st);
        case 2: return launch_v<T, MAXT, EXACT, 2>(sp, cfg, in, out, st);
        default: return launch_v<T, MAXT, EXACT, 1>(sp, cfg, in, out, st);
    }
}

}  // namespace

cudaError_t launch_generic(const SweepSpec &sp, const LaunchCfg &cfg, const GridView &in, const GridView &out,
                           cudaStream_t st) {
    const bool exact = cfg.arith == UHS_ARITH_EXACT;
    const int tx = cfg.tile_x > 0 ? cfg.tile_x : 32, ty = cfg.tile_y > 0 ? cfg.tile_y : 8;
    if (tx * ty > 256 || tx <= 0 || ty <= 0) return cudaErrorInvalidValue;
    if (sp.dtype == UHS_F64) {
        if (sp.nterms <= 64)
            return exact ? launch_t<double, 64, true>(sp, cfg, in, out, st)
                         : launch_t<double, 64, false>(sp, cfg, in, out, st);
        return exact ? launch_t<double, UHS_MAX_TERMS, true>(sp, cfg, in, out, st)
                     : launch_t<double, UHS_MAX_TERMS, false>(sp, cfg, in, out, st);
    }
    if (sp.dtype == UHS_F32) {
        if (sp.nterms <= 64)
            return exact ? launch_t<float, 64, true>(sp, cfg, in, out, st)
                         : launch_t<float, 64, false>(sp, cfg, in, out, st);
        return exact ? launch_t<float, UHS_MAX_TERMS, true>(sp, cfg, in, out, st)
                     : launch_t<float, UHS_MAX_TERMS, false>(sp, cfg, in, out, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace uhs
