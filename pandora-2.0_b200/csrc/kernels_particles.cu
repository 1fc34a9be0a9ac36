// kernels_particles.cu -- Lagrangian particle advance on sm_100a.
//
// A group of threads per particle: tensor-product Lagrange interpolation of order ORD
// of the physical velocity of the current stage (the reference evaluates the
// same polynomial by Neville's scheme, p_InterpInterpolate3D / FindMolecule /
// Neville3D, src/pp_interp.f90:313-560), the tracer or Stokes-drag RK3 update
// (p_RK3SolveParticle, src/pp_rk3.f90:57-165, drag 927-946) and the periodic
// wrap (p_MPICorrectPosition, src/pp_mpi.f90:1011-1057; x3 uses '>' where x1
// and x2 use '>=').  The reference fetches a halo of NHALO = order/2 planes by
// DMGlobalToLocal (src/pp_interp.f90:115-264); on one GPU the stencil indices
// wrap modulo N.  Physical velocity layout: [z][y][x][4], the three components of a point
// side by side (and a pad), so that a stencil point is one vector load.
//
// Particles are kept sorted by spatial bin (z slowest), re-sorted once per step,
// so that a wave of threads reads a compact set of velocity rows that stays in
// L2 instead of gathering at random from a field larger than L2.
#include <cuda_runtime.h>
#include <algorithm>
#include <type_traits>
#include "pandora_internal.cuh"
#include "bfrot.cuh"

namespace pd {

// Lagrange basis weight m at x over the ORD nodes: prod_{n != m} (x - x_n) / (x_m - x_n),
// formed as one quotient of the two products (one FP64 division per weight).
template <int ORD>
__device__ __forceinline__ double lagrange_weight(double x, const double* nodes, int m) {
    double xm = nodes[0];
#pragma unroll
    for (int n = 1; n < ORD; n++)
        if (n == m) xm = nodes[n];   // m may be a run-time value: select, do not index
    double num = 1.0, den = 1.0;
#pragma unroll
    for (int n = 0; n < ORD; n++)
        if (n != m) { num *= x - nodes[n]; den *= xm - nodes[n]; }
    return num / den;
}

// G threads per particle (G = the power of two at or above ORD): thread `sub` of a
// group gathers the stencil column x = i0 + sub (threads sub >= ORD add nothing),
// so one warp load touches 32/G particles' rows of consecutive values instead of
// 32 scattered rows; the group sums its partial results with shuffles.
// The kernel is bound by the L1 lookups of its gathers and by the trips to memory of each
// group's chain (position, stencil, RK3 state).  Against one component per field (48 loads of 8
// bytes a thread at order 4, 84 sectors a particle; the state read at the end by one thread in
// four; every thread dividing for all three directions): 16 loads of 32 bytes, 64 sectors; the
// state asked for first and updated by one thread per component.  0.320 -> 0.230 ms per stage for
// 2^20 tracers in 256^3 (FP32-mixed 0.300 -> 0.213), 0.246 -> 0.156 for 2^18 in 512^3 (0.188 ->
// 0.124).
template <int ORD> constexpr int part_group() { return ORD <= 1 ? 1 : (ORD <= 2 ? 2 : (ORD <= 4 ? 4 : 8)); }
// CTAs of 256 threads per SM asked of the register allocator: 80 registers hold a plane of the
// order-4 FP64 stencil in flight, 64 two planes of the FP32 one.  2^20 tracers in 256^3: FP64
// 0.230 ms with 3 (0.286 with 4), FP32-mixed 0.213 with 4 (0.225 with 3).
template <int ORD, class T> constexpr int part_ctas() { return ORD <= 4 && sizeof(T) == 4 ? 4 : 3; }

// Stencil index q wrapped into [0, n): one period away at most for a position inside the
// domain, so the division is off the common path.
__device__ __forceinline__ int wrap_index(int q, int n) {
    if ((unsigned)q >= (unsigned)n) {
        q %= n;
        if (q < 0) q += n;
    }
    return q;
}

// Start of the stencil along one direction, from the same rounded arithmetic as
// p_InterpFindMolecule (src/pp_interp.f90:313-560).
template <int ORD> __device__ __forceinline__ int stencil_start(double x, double d) {
    constexpr int nh = ORD / 2;
    double halo = __dmul_rn((double)nh, d);
    double xd;
    if ((ORD & 1) == 0) {
        halo = __dsub_rn(halo, __dmul_rn(0.5, d));
        xd = __dadd_rn(__dadd_rn(__dadd_rn(x, halo), d), __dmul_rn(0.5, d));
    } else {
        xd = __dadd_rn(__dadd_rn(x, halo), __dmul_rn(0.5, d));
    }
    return (int)__ddiv_rn(xd, d) - nh - nh;
}

// The velocity of all three components at one grid point: one 32-byte (FP64) or 16-byte
// (FP32) load of the interleaved field.
__device__ __forceinline__ void load_point(const double* p, double* v) {
    asm("{\n .reg .f64 pad;\n ld.global.nc.v4.f64 {%0, %1, %2, pad}, [%3];\n}" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]) : "l"(p));
}
__device__ __forceinline__ void load_point(const float* p, double* v) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = (double)q.x; v[1] = (double)q.y; v[2] = (double)q.z;
}
__device__ __forceinline__ double pick(int c, double a, double b, double d) { return c == 0 ? a : (c == 1 ? b : d); }
__device__ __forceinline__ double* pick(int c, double* const* p) { return c == 0 ? p[0] : (c == 1 ? p[1] : p[2]); }

// T: precision of the stored physical velocity (the particle state and its
// arithmetic are FP64 in both forms).
template <int ORD, class T, int CAP>
__global__ void __launch_bounds__(256, part_ctas<ORD, T>()) k_particles(const __grid_constant__ MemberSet<T, CAP> ms, int stage) {
    constexpr int G = part_group<ORD>();
    // Components a thread advances: with four or more threads per particle, thread c < 3 of
    // the group holds and updates component c; with one or two, the first thread all three.
    constexpr int NC = G >= 4 ? 1 : 3;
    const Member<T>& mm = ms.m[CAP == 1 ? 0 : blockIdx.y];
    if (!mm.active) return;
    if constexpr (CAP > 1) {   // a batch slot between members
        if (mm.F.clock->status & PD_ST_IDLE) return;
    }                             // uniform over the CTA
    const Particles& P = mm.P;
    const Geo& g = mm.g;
    const T* __restrict__ phys = mm.F.phys;
    Clock* ck = mm.F.clock;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = t / G;
    const int sub = (int)(t % G);
    const int tstep = ck->tstep;
    if (tstep < mm.pp.release) return;                  // uniform over the member
    if (G == 1 && n >= P.np) return;
    // With G > 1 every lane of a warp reaches the shuffles: lanes past the last
    // particle (whole groups at the tail) gather for the last particle and store nothing.
    const bool valid = n < P.np;
    const long long nn = valid ? n : P.np - 1;
    const int base = (threadIdx.x & 31) & ~(G - 1);     // the group's first lane
    double xp[3];
#pragma unroll
    for (int c = 0; c < 3; c++) xp[c] = P.xp[c][nn];
    // the RK3 state, asked for ahead of the gather; a tracer's velocity is the fluid's and its
    // velocity register idle, so neither is read
    const double dpv = P.dp[nn];
    double up[NC], ur[NC], pr[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) {
        const int c = G >= 4 ? (sub < 3 ? sub : 2) : q;
        ur[q] = pick(c, P.uprk)[nn];
        up[q] = pr[q] = 0.0;
        if (dpv > 0.0) { up[q] = pick(c, P.up)[nn]; pr[q] = pick(c, P.prk)[nn]; }
    }
    // the stencil's start: with four or more threads per particle each of the first three
    // forms one direction's (one FP64 division instead of three) and the group exchanges them
    int i0[3];
    if constexpr (G >= 4) {
        const int mine = stencil_start<ORD>(pick(sub, xp[0], xp[1], xp[2]), pick(sub, g.dx, g.dy, g.dz));
#pragma unroll
        for (int c = 0; c < 3; c++) i0[c] = __shfl_sync(0xffffffffu, mine, base + c);
    } else {
        i0[0] = stencil_start<ORD>(xp[0], g.dx);
        i0[1] = stencil_start<ORD>(xp[1], g.dy);
        i0[2] = stencil_start<ORD>(xp[2], g.dz);
    }
    // weights of x (this thread's column), y and z: each thread of the group forms the
    // weight of its own offset in every direction; those of y and z the group exchanges
    double wx[G == 1 ? ORD : 1], wy[ORD], wz[G == 1 ? ORD : 1];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double d = c == 0 ? g.dx : (c == 1 ? g.dy : g.dz);
        double nodes[ORD];
#pragma unroll
        for (int m = 0; m < ORD; m++) nodes[m] = __dmul_rn((double)(i0[c] + m), d);
        if constexpr (G == 1) {
            double* w = c == 0 ? wx : (c == 1 ? wy : wz);
#pragma unroll
            for (int m = 0; m < ORD; m++) w[m] = lagrange_weight<ORD>(xp[c], nodes, m);
        } else {
            const double mine = lagrange_weight<ORD>(xp[c], nodes, sub < ORD ? sub : ORD - 1);
            if (c == 0) wx[0] = sub < ORD ? mine : 0.0;
            else if (c == 2) wz[0] = mine;   // exchanged plane by plane below
            else {
#pragma unroll
                for (int m = 0; m < ORD; m++) wy[m] = __shfl_sync(0xffffffffu, mine, base + m);
            }
        }
    }
    // gather: a point's three components are one load of 4 T (32 bytes in FP64)
    double uf[3] = {0.0, 0.0, 0.0};
    int yo[ORD];
#pragma unroll
    for (int m = 0; m < ORD; m++) yo[m] = wrap_index(i0[1] + m, g.ny) * g.nx;
    if constexpr (G == 1) {
        int xo[ORD];
#pragma unroll
        for (int m = 0; m < ORD; m++) xo[m] = wrap_index(i0[0] + m, g.nx);
#pragma unroll
        for (int zi = 0; zi < ORD; zi++) {
            const T* pl = phys + 4 * ((long long)wrap_index(i0[2] + zi, g.nz) * g.ny * g.nx);
            double ay[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int yi = 0; yi < ORD; yi++) {
                double ax[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int xi = 0; xi < ORD; xi++) {
                    double v[3];
                    load_point(pl + 4 * (long long)(yo[yi] + xo[xi]), v);
#pragma unroll
                    for (int c = 0; c < 3; c++) ax[c] += wx[xi] * v[c];
                }
#pragma unroll
                for (int c = 0; c < 3; c++) ay[c] += wy[yi] * ax[c];
            }
#pragma unroll
            for (int c = 0; c < 3; c++) uf[c] += wz[zi] * ay[c];
        }
    } else {
        // column x = i0 + sub (lanes past the stencil: its last column, weight 0); the x
        // weight is applied before the group sum
        const int xs = wrap_index(i0[0] + (sub < ORD ? sub : ORD - 1), g.nx);
#pragma unroll(ORD > 4 ? 1 : (sizeof(T) == 8 ? ORD : 2))
        for (int zi = 0; zi < ORD; zi++) {
            const T* pl = phys + 4 * ((long long)wrap_index(i0[2] + zi, g.nz) * g.ny * g.nx + xs);
            const double w = __shfl_sync(0xffffffffu, wz[0], base + zi);
            double v[ORD][3];
#pragma unroll
            for (int yi = 0; yi < ORD; yi++) load_point(pl + 4 * (long long)yo[yi], v[yi]);
            double ay[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int yi = 0; yi < ORD; yi++)
#pragma unroll
                for (int c = 0; c < 3; c++) ay[c] += wy[yi] * v[yi][c];
#pragma unroll
            for (int c = 0; c < 3; c++) uf[c] += w * ay[c];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double v = wx[0] * uf[c];
#pragma unroll
            for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            uf[c] = v;
        }
        if (NC == 3 && (sub != 0 || !valid)) return;   // NC == 1: the group exchanges components below
    }
    const double dt = ck->dt;
    double beta, gamma;
    if (stage == 1) { beta = 0.0; gamma = 1.0 / 3.0; }
    else if (stage == 2) { beta = -(5.0 / 9.0); gamma = 15.0 / 16.0; }
    else { beta = -(153.0 / 128.0); gamma = 8.0 / 15.0; }
    const bool release = tstep == mm.pp.release && stage == 1;
    // BF-rot shear transforms to the laboratory frame and back; the R forms
    // (p_RK3SolveParticleR, src/pp_rk3.f90:307-403, dispatched at src/pp_control.f90:
    // 568-571) interpolate laboratory components and advance the moving position with
    // them directly, the isotropic arithmetic
    const bool bfrot = g.shear && !g.rrot;
    double xw[3] = {xp[0], xp[1], xp[2]};   // frame in which the RK3 update runs
    BF bf;
    if (bfrot) {
        // p_RK3SolveParticleBF (src/pp_rk3.f90:169-303): velocity and position to
        // the laboratory frame (p_RK3Mov2Lab, src/pp_rk3.f90:989-1014), RK3 there,
        // back with p_RK3Lab2Mov (1016-1042) at the same B.
        bf = make_bf(g, ck);
        double xl[3] = {0.0, 0.0, 0.0}, ul[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
                if (bex(a, b)) { xl[a] += bf.bi[a][b] * xp[b]; ul[a] += bf.bi[a][b] * uf[b]; }
#pragma unroll
        for (int c = 0; c < 3; c++) { xw[c] = xl[c]; uf[c] = ul[c]; }
    }
    // the components of this thread
    double xc[NC], uc[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) {
        xc[q] = NC == 3 ? xw[q] : pick(sub, xw[0], xw[1], xw[2]);
        uc[q] = NC == 3 ? uf[q] : pick(sub, uf[0], uf[1], uf[2]);
        // p_ControlInitPartVelocity(BF) at the release step (src/pp_control.f90:378-516)
        if (release) { up[q] = uc[q]; pr[q] = 0.0; ur[q] = 0.0; }
    }
    // shear: minus the homogeneous source amat up (p_RK3ComputeHomogeneousSourceTerm,
    // src/pp_rk3.f90:1080-1102); amat has the single entry (1,3).  Exchanged ahead of the drag
    // branch, which parts a warp that holds tracers and heavy particles.
    double hs0 = 0.0;
    if (bfrot) {       // uniform over the CTA
        double up3 = up[NC - 1];
        if constexpr (NC == 1) up3 = __shfl_sync(0xffffffffu, up[0], base + 2);
        hs0 = g.shear_s * up3;
    }
    if (dpv > 0.0) {   // uniform over the group
        const double tau = ((dpv * dpv) / (18.0 * mm.pp.f_nu)) * (mm.pp.p_rho / mm.pp.f_rho);
#pragma unroll
        for (int q = 0; q < NC; q++) {
            const bool first = NC == 3 ? q == 0 : sub == 0;
            const double acc = ((uc[q] - up[q]) / tau) - (first ? hs0 : 0.0);
            pr[q] = (beta * pr[q]) + acc;
            up[q] = up[q] + (gamma * dt * pr[q]);
        }
    } else {
#pragma unroll
        for (int q = 0; q < NC; q++) up[q] = uc[q];
    }
#pragma unroll
    for (int q = 0; q < NC; q++) {
        ur[q] = (beta * ur[q]) + up[q];
        xc[q] = xc[q] + (gamma * dt * ur[q]);
    }
    if (bfrot) {   // back to the moving frame: bmat has the diagonal and (1,3)
        double x3 = xc[NC - 1];
        if constexpr (NC == 1) x3 = __shfl_sync(0xffffffffu, xc[0], base + 2);
#pragma unroll
        for (int q = 0; q < NC; q++) {
            const bool first = NC == 3 ? q == 0 : sub == 0;
            double v = 0.0;
            v += (NC == 3 ? bf.bm[q][q] : pick(sub, bf.bm[0][0], bf.bm[1][1], bf.bm[2][2])) * xc[q];
            if (first) v += bf.bm[0][2] * x3;
            xc[q] = v;
        }
    }
    if (NC == 1 && (sub >= 3 || !valid)) return;
#pragma unroll
    for (int q = 0; q < NC; q++) {
        const int c = NC == 3 ? q : sub;
        const double d = pick(c, g.dx, g.dy, g.dz), l = pick(c, g.lx, g.ly, g.lz);
        const double lo = -0.5 * d, hi = lo + l;
        double x = xc[q];
        if (x < lo) x = x + l;
        if (c < 2 ? x >= hi : x > hi) x = x - l;
        // lost: outside the domain after the wrap (components 2 and 3)
        const double mn = -(0.5 * d), mx = (double)(c == 1 ? g.ny : g.nz) * d - (0.5 * d);
        if (c > 0 && !(x >= mn && x < mx)) atomicOr(&ck->status, PD_ST_LOST);
        pick(c, P.xp)[n] = x;
        pick(c, P.up)[n] = up[q];
        pick(c, P.uprk)[n] = ur[q];
        if (dpv > 0.0 || release) pick(c, P.prk)[n] = pr[q];
    }
}

// P_INIT_RANDOM (src/pp_control.f90:663-707): three draws per particle, in order.
__global__ void k_init_particles(Particles P, Geo g, uint64_t key, double dia) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= P.np) return;
    const double L[3] = {g.lx, g.ly, g.lz}, D[3] = {g.dx, g.dy, g.dz};
    for (int c = 0; c < 3; c++) {
        const double rn = uniform(key, (uint64_t)(3 * n + c));
        P.xp[c][n] = __dsub_rn(__dmul_rn(rn, L[c]), __dmul_rn(D[c], 0.5));
        P.up[c][n] = 0.0; P.uprk[c][n] = 0.0; P.prk[c][n] = 0.0;
    }
    P.dp[n] = dia;
    P.pid[n] = n;
}

// ---------------------------------------------------------------------------
// Spatial sort: counting sort by bin (z slowest, then y, then x).  Bins are
// whole blocks of cells; positions lie in [-d/2, L-d/2) after the wrap, so
// x + d/2 is in [0, L).  Order inside a bin follows atomics; every particle's
// update is independent of the order, and pid keeps the caller's numbering.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int bin_of(double x, double d, int cells, int nb) {
    int b = (int)floor((x + 0.5 * d) / (d * cells));
    return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}

__global__ void k_part_key(Particles P, Geo g, PartSort s) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= P.np) return;
    const int bx = bin_of(P.xp[0][n], g.dx, s.bin_cells[0], s.nb[0]);
    const int by = bin_of(P.xp[1][n], g.dy, s.bin_cells[1], s.nb[1]);
    const int bz = bin_of(P.xp[2][n], g.dz, s.bin_cells[2], s.nb[2]);
    const unsigned k = ((unsigned)bz * s.nb[1] + by) * s.nb[0] + bx;
    s.key[n] = k;
    atomicAdd(&s.count[k], 1u);
}

// exclusive scan of count[0..n) in place: per-block scan of 1024 entries ...
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* warp_tot, unsigned& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned t = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;   // inclusive prefix of warp totals
    }
    __syncthreads();
    total = warp_tot[(blockDim.x >> 5) - 1];
    const unsigned base = wid ? warp_tot[wid - 1] : 0u;
    return base + x - v;
}

__global__ void __launch_bounds__(1024) k_scan_blocks(unsigned* a, unsigned* sums, long long n) {
    __shared__ unsigned wt[32];
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    const unsigned v = i < n ? a[i] : 0u;
    unsigned total;
    const unsigned ex = block_exclusive_scan(v, wt, total);
    if (i < n) a[i] = ex;
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// ... one block scans the block totals (at most 1024 of them) ...
__global__ void __launch_bounds__(1024) k_scan_sums(unsigned* sums, int nblocks) {
    __shared__ unsigned wt[32];
    const unsigned v = threadIdx.x < (unsigned)nblocks ? sums[threadIdx.x] : 0u;
    unsigned total;
    const unsigned ex = block_exclusive_scan(v, wt, total);
    if (threadIdx.x < (unsigned)nblocks) sums[threadIdx.x] = ex;
}

// ... and the block offsets are added back.
__global__ void __launch_bounds__(1024) k_scan_add(unsigned* a, const unsigned* sums, long long n) {
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    if (i < n) a[i] += sums[blockIdx.x];
}

__global__ void k_part_scatter(Particles src, PartSort s) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= src.np) return;
    const long long d = atomicAdd(&s.count[s.key[n]], 1u);
    const Particles& t = s.tmp;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        t.xp[c][d] = src.xp[c][n]; t.up[c][d] = src.up[c][n];
        t.uprk[c][d] = src.uprk[c][n]; t.prk[c][d] = src.prk[c][n];
    }
    t.dp[d] = src.dp[n];
    t.pid[d] = src.pid[n];
}

template <class T>
cudaError_t launch_particles(const Geo& g, const Member<T>* M, int B, long long np, int order, int stage,
                             cudaStream_t st) {
    if (np == 0) return cudaSuccess;
    switch (order) {
#define PD_ORD(O)                                                                                  \
    case O:                                                                                        \
        return for_member_sets(M, B, [&](const auto& ms, int nm) {                                 \
            constexpr int CAP = std::decay_t<decltype(ms)>::cap;                                   \
            k_particles<O, T, CAP><<<dim3((unsigned)((np * part_group<O>() + 255) / 256), nm), 256, 0, st>>>(ms, stage); \
        });
        PD_ORD(1) PD_ORD(2) PD_ORD(3) PD_ORD(4) PD_ORD(5) PD_ORD(6)
#undef PD_ORD
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_init_particles(const Geo& g, const Particles& p, uint64_t key, double dia, cudaStream_t st) {
    if (p.np == 0) return cudaSuccess;
    const long long nb = (p.np + 255) / 256;
    k_init_particles<<<(unsigned)nb, 256, 0, st>>>(p, g, key, dia);
    return cudaGetLastError();
}

// Sorts P by bin into s.tmp, then copies back into P's storage (so that the
// pointers captured in the step's CUDA graph stay valid).
cudaError_t launch_particle_sort(const Geo& g, const Particles& P, const PartSort& s, cudaStream_t st,
                                 int* nlaunch) {
    if (P.np == 0) return cudaSuccess;
    const long long nbins = (long long)s.nb[0] * s.nb[1] * s.nb[2];
    const int nblk = (int)((nbins + 1023) / 1024);
    if (nblk > 1024) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(s.count, 0, sizeof(unsigned) * nbins, st);
    if (e) return e;
    const unsigned pb = (unsigned)((P.np + 255) / 256);
    k_part_key<<<pb, 256, 0, st>>>(P, g, s);
    k_scan_blocks<<<nblk, 1024, 0, st>>>(s.count, s.block_sums, nbins);
    k_scan_sums<<<1, 1024, 0, st>>>(s.block_sums, nblk);
    k_scan_add<<<nblk, 1024, 0, st>>>(s.count, s.block_sums, nbins);
    k_part_scatter<<<pb, 256, 0, st>>>(P, s);
    if ((e = cudaGetLastError())) return e;
    // the 13 double arrays and pid are contiguous in both buffers (14 * np words)
    e = cudaMemcpyAsync(P.xp[0], s.tmp.xp[0], sizeof(double) * 14 * (size_t)P.np, cudaMemcpyDeviceToDevice, st);
    if (nlaunch) *nlaunch += 5;
    return e;
}

// p_StatsPrimary (src/pp_stats.f90:119-200): the sums over particles of up_i up_j and of
// the kinetic energy (1/2)(pi/6 dp^3 P_RHO)|up|^2; the caller divides by P_NP_GLOBAL.
__global__ void __launch_bounds__(256) k_part_stats(Particles p, long long np, double rho_p, double* acc) {
    double s[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double c = 3.14159265358979323846264338327950288 / 6.0;
    for (long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x; n < np; n += (long long)gridDim.x * blockDim.x) {
        const double u1 = p.up[0][n], u2 = p.up[1][n], u3 = p.up[2][n], d = p.dp[n];
        s[0] += u1 * u1; s[1] += u2 * u2; s[2] += u3 * u3;
        s[3] += u1 * u2; s[4] += u1 * u3; s[5] += u2 * u3;
        s[6] += 0.5 * ((c * (d * d * d)) * rho_p) * ((u1 * u1) + (u2 * u2) + (u3 * u3));
    }
    __shared__ double red[8][7];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 7; a++) {
        double x = s[a];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[w][a] = x;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double x = 0.0;
        for (int v = 0; v < (int)(blockDim.x >> 5); v++) x += red[v][threadIdx.x];
        atomicAdd(acc + threadIdx.x, x);
    }
}

cudaError_t launch_particle_stats(const Particles& p, long long np, double rho_p, double* acc, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(acc, 0, sizeof(double) * 7, st);
    if (e || np <= 0) return e;
    unsigned nb = (unsigned)std::min<long long>((np + 255) / 256, 1024);
    k_part_stats<<<nb, 256, 0, st>>>(p, np, rho_p, acc);
    return cudaGetLastError();
}

template cudaError_t launch_particles<double>(const Geo&, const Member<double>*, int, long long, int, int,
                                             cudaStream_t);
template cudaError_t launch_particles<float>(const Geo&, const Member<float>*, int, long long, int, int,
                                            cudaStream_t);

}  // namespace pd
