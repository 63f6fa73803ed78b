// stage.cu -- one RK stage of the coupled atmosphere-wildfire model on sm_100a.
//
// A stage evaluates k_s = Phi(X_s) (reference src/cu/pde.cu:910-917: RHS,
// Smagorinsky SGS terms, boundary/IBM rules) and folds the RK combination into
// the same pass (reference solver.cu:14-93, utils.cu:14-21), so no k-buffer is
// ever stored:
//   k_utau        : per column, wall friction velocity from the k = 0 plane (first
//                   stage; k_stage_edge leaves it for the following ones);
//   k_stage_march : per tile of cells, plane by plane along x in shared memory, the
//                   SGS inputs of the tile and its frame, then advection +
//                   diffusion + forces + reaction + SGS divergence and the acc /
//                   X_{s+1} updates of every cell the boundary rules do not
//                   overwrite;
//   k_stage_edge  : the fuel, the boundary/IBM values of k_s (cut node, top) and
//                   their RK updates.
// The right-hand side of cells on the walls (k = 0, k = Nz-1) and below the
// cut node is never used by the reference (boundary_conditions overwrites it,
// pde.cu:58-97), so the fused pass evaluates interior stencils only.
// Arithmetic follows the reference expression by expression; divisions by
// grid constants are folded into precomputed weights (ZCoef, KRow).
#include <cuda.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "stage_common.cuh"

namespace wf {

namespace {

// The kernels of a stage start while the one before them still runs (programmatic
// dependent launch) and read or write nothing that it touches before after_previous(),
// which waits for all of it: launch latency, the weights and the index loads are off
// the chain of a step.  k_stage_march lets the next kernel start in the last iteration of
// its walk (from its first one on, waiting blocks took the place of other contexts':
// 33 x 33 x 16 FP64 63 us a step with three contexts in turn against 49; 52 without
// early starts), the two small kernels at once.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// ---------------------------------------------------------------------------
// wall friction velocity of every column from its k = 0 plane
// (pde.cu:767-772: tau_w = sqrt((mu uz)^2 + (mu vz)^2), u_tau = sqrt(tau_w/rho))
template <class R> __device__ __forceinline__ R utau_of(const StageArgs<R> &a, const R (&u)[3], const R (&v)[3], R T)
{
    const int Nz = a.g.Nz;
    const R w0 = (R)a.g.zc[ZF0 * Nz], w1 = (R)a.g.zc[ZF1 * Nz], w2 = (R)a.g.zc[ZF2 * Nz];
    const R uz = w0 * u[0] + w1 * u[1] + w2 * u[2];
    const R vz = w0 * v[0] + w1 * v[1] + w2 * v[2];
    const R rho = fdiv(a.pr.Trho, T);
    R mu = a.pr.mu;
    if (a.ph.sutherland_viscosity == 1)
        mu = R(1.716e-5) * rpow(T / R(273.15), R(1.5)) * (R(273.15) + R(110.4)) / (T + R(110.4));
    const R a1 = mu * uz, a2 = mu * vz;
    return rsqrt_(fdiv(rsqrt_(a1 * a1 + a2 * a2), rho));
}

template <class R>
__global__ void __launch_bounds__(128) k_utau(const StageArgs<R> a)
{
    const Geom &g = a.g;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    start_next();
    if (col >= g.Nx * g.Ny) return;
    const int Nz = g.Nz, N = g.N;
    const R *X = a.X + (size_t)col * Nz;
    const R u[3] = {X[0], X[1], X[2]}, v[3] = {X[N], X[N + 1], X[N + 2]};
    a.utau[col] = utau_of(a, u, v, X[3 * (size_t)N]);
}

// ---------------------------------------------------------------------------
// The fused stage pass.  A block owns a tile of TJ rows (j) x TK planes (k) of
// cells and walks it along x, one x-plane per iteration; an interior thread owns
// VW cells in k (FP32: 2, every operation on packed pairs; FP64: 1) of one row.
// In iteration c it
//   A. forms from the state planes c-2 .. c+2 in shared memory the SGS inputs of
//      plane c (strain S', raw mu_sgs, the divergence source), the upwind
//      advection, the Laplacians and the source terms;
//   B. completes plane c-1: the SGS divergence from the SGS inputs of planes
//      c-2, c-1 and c, and the RK update.
// The fuel and the boundary cells (cut node, top) are k_stage_edge's; what
// part B writes there is lost, and it leaves the k-values they need in a.bc.
// In iteration c plane c + 3 is fetched, and waited for at its end: it is read from
// iteration c + 1 on, so a load has one iteration to arrive in.  It comes by TMA, one
// box per plane (one per row where the tile's halo wraps around in y; in x the wrap is
// the choice of a coordinate);
// grids whose columns are no multiple of 16 bytes are copied by cp.async instead.
// One barrier per plane.  FR further threads own the one-cell frame around the
// tile, whose SGS inputs part B of the tile's edge reads.
constexpr int kColRing = 8;   // x-planes of column tables kept (power of two)
// Planes of a tile at most: the two row lengths compiled.  Rows of 24 leave shared memory for more rows
// per tile where a column divides into so few planes (step, us, three contexts in turn, against rows of
// 32 alone: 33 x 33 x 16 FP64 50 / 57, 100 x 100 x 24 FP64 175 / 199, 201 x 150 x 45 FP32 with all source
// terms 366 / 408, 160 x 128 x 48 FP32 316 / 322).
constexpr int kTileK = 32, kTileK2 = 24;

// value of a thread's VW cells
struct F2 {
    float2 v;
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return {__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return {__ffma2_rn(b.v, make_float2(-1.0f, -1.0f), a.v)}; }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return {__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
template <class R> struct Vec;
template <> struct Vec<float> {
    using V = F2;
    static constexpr int W = 2;
};
template <> struct Vec<double> {
    using V = double;
    static constexpr int W = 1;
};
template <class V> __device__ __forceinline__ V splat(float a) { return {make_float2(a, a)}; }
template <class V> __device__ __forceinline__ V splat(double a) { return a; }
__device__ __forceinline__ float el(const F2 &a, int e) { return e ? a.v.y : a.v.x; }
__device__ __forceinline__ double el(double a, int) { return a; }
__device__ __forceinline__ void set_el(F2 &a, int e, float x) { (e ? a.v.y : a.v.x) = x; }
__device__ __forceinline__ void set_el(double &a, int, double x) { a = x; }
__device__ __forceinline__ F2 vpos(F2 a) { return {make_float2(fmaxf(a.v.x, 0.0f), fmaxf(a.v.y, 0.0f))}; }
__device__ __forceinline__ F2 vneg(F2 a) { return {make_float2(fminf(a.v.x, 0.0f), fminf(a.v.y, 0.0f))}; }
__device__ __forceinline__ double vpos(double a) { return rmax(a, 0.0); }
__device__ __forceinline__ double vneg(double a) { return rmin(a, 0.0); }
__device__ __forceinline__ F2 vsqrt(F2 a) { return {make_float2(rsqrt_(a.v.x), rsqrt_(a.v.y))}; }
__device__ __forceinline__ double vsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ F2 vdiv(F2 a, F2 b) { return {make_float2(fdiv(a.v.x, b.v.x), fdiv(a.v.y, b.v.y))}; }
__device__ __forceinline__ double vdiv(double a, double b) { return a / b; }

// per-k weights in shared memory, each a row over the tile's planes: upwind from
// below (k-2, k-1, k) and from above (k, k+1, k+2), negated, the part of w each carries
// (from below: max(w,0) WP + w WW, from above the rest of w), centred first
// derivative, Smagorinsky length squared, centred second derivative (k-1, k+1),
// height, spacing.  Weights apply to differences from the value at k.
enum ZRow { ZB = 0, ZF = 3, ZWP = 6, ZWW, ZD1, ZL, ZD2, ZZ = ZD2 + 2, ZDZ, ZROW };
// SGS inputs in shared memory
enum GRow { G_MU, G_Q, G_S11, G_S12, G_S13, G_S22, G_S23, G_S33, GROW };

// Shared memory of a block, in bytes from its start.  A row of the state holds
// its four fields one after the other (the layout of a TMA box), KH planes of
// halo on either side; consecutive cells are consecutive words, so every access
// of a warp is free of bank conflicts.
template <class R, int KW> struct StageSmem {
    static constexpr uint32_t E = sizeof(R);
    static constexpr int KH = 16 / E;                              // halo planes: a 16-byte boundary
    static constexpr int PX = KW + 2 * KH, PG = KW + 4, RS = 6, RG = 3;
    static constexpr uint32_t FX = PX * E;                         // one field of a row
    static constexpr uint32_t ROW_S = 4 * FX;                      // a multiple of 128 bytes, as a box's start must be
    static constexpr uint32_t FG = PG * E, ROW_G = GROW * FG;
    static constexpr uint32_t FZ = PG * E;
    uint32_t planeS, planeG;
    uint32_t g0;            // start of the SGS ring
    uint32_t zr;            // [ZROW][PG]
    uint32_t wall;          // bottom and top: weights of the value beyond the wall (3) and of the second derivative (4)
    uint32_t corr;          // V [2][2][TJ + 2]: second z derivative of T on the bottom and top wall; then a zero
    uint32_t cidx;          // [kColRing][TJ + 2] int2: fuel top, cut node
    uint32_t ctopo, cut_;   // [kColRing][TJ + 2] terrain height, wall friction velocity
    uint32_t bnd;           // [2][TJ][2] highest terrain and least friction / A of the five columns around a cell
    uint32_t zero;          // [2][TJ] int: which of them have no friction (bits: centre, x+, x-, y+, y-)
    uint32_t bar;           // [RS] mbarriers of the state planes
    uint32_t end;
    __host__ __device__ explicit StageSmem(int tj)
    {
        planeS = (uint32_t)(tj + 4) * ROW_S;
        planeG = (uint32_t)(tj + 2) * ROW_G;
        g0 = RS * planeS;
        bar = g0 + RG * planeG;
        zr = bar + RS * 8;
        wall = zr + ZROW * FZ;
        corr = wall + 16 * E;
        cidx = corr + (8 * (tj + 2) + 2) * E;
        ctopo = cidx + kColRing * (tj + 2) * 8;
        cut_ = ctopo + kColRing * (tj + 2) * E;
        bnd = cut_ + kColRing * (tj + 2) * E;
        zero = bnd + 4 * tj * E;
        end = zero + 2 * tj * 4;
    }
    __device__ static uint32_t s(int jj, int kk) { return (uint32_t)(jj + 2) * ROW_S + (uint32_t)(kk + KH) * E; }
    __device__ static uint32_t g(int jj, int kk) { return (uint32_t)(jj + 1) * ROW_G + (uint32_t)(kk + 2) * E; }
    __device__ static uint32_t z(int kk) { return (uint32_t)(kk + 2) * E; }
};
extern __shared__ __align__(128) unsigned char stage_smem[];
template <class T> __device__ __forceinline__ T &sh(uint32_t o) { return *reinterpret_cast<T *>(stage_smem + o); }

template <int B>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(stage_smem) + dst;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(B), "r"(valid ? B : 0)
                 : "memory");
}

// Bounded wait on an mbarrier phase (false when the limit ran out).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit)
{
    for (int it = 0; it < limit; it++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// SGS inputs of a thread's cells
template <class V> struct Sgs { V mu, g7, S11, S12, S13, S22, S23, S33; };
template <class SM, class V> __device__ __forceinline__ void put_sgs(uint32_t o, const Sgs<V> &q)
{
    sh<V>(o + G_MU * SM::FG) = q.mu;
    sh<V>(o + G_Q * SM::FG) = q.g7;
    sh<V>(o + G_S11 * SM::FG) = q.S11;
    sh<V>(o + G_S12 * SM::FG) = q.S12;
    sh<V>(o + G_S13 * SM::FG) = q.S13;
    sh<V>(o + G_S22 * SM::FG) = q.S22;
    sh<V>(o + G_S23 * SM::FG) = q.S23;
    sh<V>(o + G_S33 * SM::FG) = q.S33;
}

// the z neighbours of the value at byte offset o (own value c): one plane below
// and above, and two (FP32: the pair of cells k, k+1 takes k-2 .. k+3 from three
// aligned pairs)
template <class R, class V> struct ZNb { V m2, m1, p1, p2; };
template <class R> __device__ __forceinline__ ZNb<R, typename Vec<R>::V> z_nb(uint32_t o, typename Vec<R>::V c)
{
    ZNb<R, typename Vec<R>::V> n;
    if constexpr (sizeof(R) == 4) {
        n.m2 = sh<F2>(o - 8);
        n.p2 = sh<F2>(o + 8);
        n.m1.v = make_float2(n.m2.v.y, c.v.x);
        n.p1.v = make_float2(c.v.y, n.p2.v.x);
    } else {
        n.m2 = sh<double>(o - 16);
        n.m1 = sh<double>(o - 8);
        n.p1 = sh<double>(o + 8);
        n.p2 = sh<double>(o + 16);
    }
    return n;
}
// difference of the planes above and below
template <class R> __device__ __forceinline__ typename Vec<R>::V z_diff(uint32_t o, typename Vec<R>::V c)
{
    if constexpr (sizeof(R) == 4) {
        const F2 p = {make_float2(c.v.y, sh<float>(o + 8))}, m = {make_float2(sh<float>(o - 4), c.v.x)};
        return p - m;
    } else {
        return sh<double>(o + 8) - sh<double>(o - 8);
    }
}

// Constants of the model as values of a thread's cells: a 64-bit constant is one
// load, where a scalar would take two moves to fill a pair.
template <class R> struct StageVec {
    using V = typename Vec<R>::V;
    V hx, hy, lx, ly, c12, c4, kT, inv_Trho_cp, H_C_cp, mu_Trho, Trho, two_inv_Trho, inv_Trho_Pr, g_Tinf, T_inf, third, m_third, half, p4, m_hx,
        m_hy, ar, cA, cK;
};

// Source terms of T and the divergence source g7 = nu T_RHS / T of the SGS model
// (pde.cu:640-760): conduction and radiation over rho c_p, reaction, and unless
// LEAN the Sutherland laws and the convective exchange.  1 / rho is
// T / (T_inf rho_inf); x^(3/2) and x^(1/4) are taken by square roots.
template <class R, class V, bool LEAN>
__device__ __forceinline__ void sources(const StageArgs<R> &a, const StageVec<R> &q, V Tx, V Ty, V Tz, V lapT, V T, V Y, V K_T, int gk,
                                        int nzy, V dz, V &src, V &nu, V &g7)
{
    const V T2 = T * T, gg = vfma(Tz, Tz, vfma(Ty, Ty, Tx * Tx));
    V mu_Trho = q.mu_Trho, kT = q.kT, dk = splat<V>(R(0)), ex = dk, ext = dk;
    if constexpr (!LEAN) {
        const PhysR<R> &p = a.pr;
        auto c = [](double x) { return splat<V>((R)x); };
        if (a.ph.sutherland_viscosity == 1 || a.ph.sutherland_conductivity == 1) {
            const V x = T * c(1.0 / 273.15), sx = vsqrt(x), x15 = x * sx;
            if (a.ph.sutherland_viscosity == 1)
                mu_Trho = vdiv(x15 * c(1.716e-5 * (273.15 + 110.4)), (T + c(110.4)) * splat<V>(p.Trho));
            if (a.ph.sutherland_conductivity == 1) {
                const V d = vdiv(c(0.0241 * (273.15 + 194)), T + c(194));
                kT = d * x15;
                dk = d * vfma(c(1.5), sx, vdiv(c(-1.0) * x15, T + c(194)));
            }
        }
        if (p.alpha_s * p.sigma_s != R(0)) {
            // the gas is at T where the cell holds no fuel, the solid where it does; the other
            // of the two, and both above the fuel zone, at T_inf
            V dT, Tg;
#pragma unroll
            for (int e = 0; e < Vec<R>::W; e++) {
                const bool solid = el(Y, e) > R(0);
                set_el(Tg, e, solid ? p.T_inf : el(T, e));
                set_el(dT, e, gk + e > nzy ? R(0) : solid ? p.T_inf - el(T, e) : el(T, e) - p.T_inf);
            }
            V ad;
#pragma unroll
            for (int e = 0; e < Vec<R>::W; e++) set_el(ad, e, rfabs(el(dT, e)));
            const V h = splat<V>(p.h_c) * dz * vsqrt(vsqrt(vdiv(ad, dz)));
            ex = h * splat<V>(-p.alpha_s * p.sigma_s) * dT;
            ext = Tg * q.inv_Trho_cp;
        }
    }
    const V cond = vfma(q.c4, T2 * T, kT);
    const V flux = LEAN ? q.c12 * T2 * gg : vfma(q.c12 * T2, gg, dk);
    src = vfma(cond, lapT, flux) * (T * q.inv_Trho_cp);
    src = vfma(q.H_C_cp * Y, K_T, src);
    if constexpr (!LEAN) src = vfma(ex, ext, src);
    nu = mu_Trho * T;
    g7 = mu_Trho * src;
}

// differences of one field across a cell, over two spacings
template <class V> struct Grad { V x, y, z; };

// Squared Van Driest factors (turbulence.cu:255-454) of points at heights zh in a
// column of terrain height topo and friction velocity ut, with q = -1 / (A nu) of
// the cells they are taken for.
template <class R, class V> __device__ __forceinline__ V vd_factor2(V zh, R topo, R ut, V q)
{
    V f = vpos(zh - splat<V>(topo)) * splat<V>(ut) * q;
#pragma unroll
    for (int e = 0; e < Vec<R>::W; e++) set_el(f, e, van_driest(el(f, e)));
    return f * f;
}
__device__ __forceinline__ F2 vshfl(F2 a, int l)
{
    return {make_float2(__shfl_sync(0xffffffffu, a.v.x, l), __shfl_sync(0xffffffffu, a.v.y, l))};
}
__device__ __forceinline__ double vshfl(double a, int l) { return __shfl_sync(0xffffffffu, a, l); }

// SGS inputs from the differences (pde.cu:632-765): traceless strain S_ii = d_i u_i
// - div / 3, mu_sgs = rho l2 |S|.  Every sum of products is an explicit fused
// multiply-add, here and wherever the frame and the tile evaluate the same value:
// left to the compiler, the two came out differently in the last bit.
template <class R, class V> __device__ __forceinline__ Sgs<V> strain(const StageVec<R> &c, const Grad<V> (&d)[4], V hz, V T, V l2, V g7)
{
    Sgs<V> q;
    const V ux = d[0].x * c.hx, vy = d[1].y * c.hy, wz = d[2].z * hz;
    const V s12 = vfma(d[0].y, c.hy, d[1].x * c.hx), s13 = vfma(d[0].z, hz, d[2].x * c.hx), s23 = vfma(d[2].y, c.hy, d[1].z * hz);
    const V sq = vfma(wz, wz, vfma(vy, vy, ux * ux));
    const V mod2 = vfma(s23, s23, vfma(s12, s12, vfma(s13, s13, sq + sq)));
    const V div = vfma(d[2].z, hz, vfma(d[1].y, c.hy, ux));
    q.S11 = vfma(div, c.m_third, ux);
    q.S22 = vfma(div, c.m_third, vy);
    q.S33 = vfma(div, c.m_third, wz);
    q.S12 = c.half * s12;
    q.S13 = c.half * s13;
    q.S23 = c.half * s23;
    q.mu = vdiv(c.Trho * l2, T) * vsqrt(mod2);
    q.g7 = g7;
    return q;
}

template <class R, int NT, int FR, int NB, int KW, bool LEAN, bool VEC>
__global__ void __launch_bounds__(NT + FR, NB)
    k_stage_march(const StageArgs<R> a, const StageVec<R> cv, const StageGrid sg, const __grid_constant__ CUtensorMap m_tile,
                  const __grid_constant__ CUtensorMap m_row)
{
    using SM = StageSmem<R, KW>;
    using V = typename Vec<R>::V;
    constexpr int VW = Vec<R>::W;
    constexpr uint32_t E = sizeof(R);
    const Geom &g = a.g;
    const PhysR<R> &p = a.pr;
    const int Nx = g.Nx, Ny = g.Ny, Nz = g.Nz;
    const int tj = sg.tj, tk = sg.tk;
    const SM sm(tj);
    int bid = blockIdx.x;
    const int k0 = (bid % sg.ntk) * tk;
    bid /= sg.ntk;
    const int j0 = (bid % sg.ntj) * tj, ib = (bid / sg.ntj) * sg.L;
    const int ie = min(ib + sg.L, Nx);
    const int tid = threadIdx.x;
    const bool tma = sg.tma;
    // offsets within one field are below 4 GiB (wf_create's limit on the grid), so
    // addresses are a uniform base per field and a 32-bit byte offset
    const uint32_t plane = (uint32_t)Ny * (uint32_t)Nz * E;
    const size_t FB = (size_t)g.N * E;
    const int CW = tj + 2;
    auto at = [&](const R *base, int f, uint32_t o) -> const R & {
        return *reinterpret_cast<const R *>(reinterpret_cast<const char *>(base) + f * FB + o);
    };
    auto c_ = [](R x) { return splat<V>(x); };
    const bool rd = stage_reads_acc(a.method, a.stage), kp = stage_keeps_acc(a.method, a.stage), kstore = a.method == 3;

    // z weights of the tile's planes and the walls' one-sided weights
    for (int c = tid; c < SM::PG * ZROW; c += NT + FR) {
        const int e = c / SM::PG, kk = c - e * SM::PG, gk = k0 - 2 + kk;
        R v = R(0);
        if (gk >= 0 && gk < Nz) {
            const R *r = a.krow + (size_t)gk * KROW;
            const bool wall = gk == 0 || gk == Nz - 1;
            if (e < ZF) v = (gk >= 2) ? -r[RKM + e] : R(0);
            else if (e < ZWP) v = (gk <= Nz - 3) ? -r[RKP + 2 + e - ZF] : R(0);
            else if (e == ZWP) v = (gk == 1 || gk == Nz - 2) ? R(0) : R(1);
            else if (e == ZWW) v = gk == Nz - 2 ? R(1) : R(0);
            else if (e == ZD1) v = wall ? a.krow[(gk == 0 ? 1 : Nz - 2) * KROW + RD1] : r[RD1];
            else if (e == ZL) v = a.coef ? r[RDD2] : r[RDEL2];
            else if (e < ZZ) v = r[RD2 + 2 * (e - ZD2)];
            else v = e == ZZ ? r[RZ] : r[RDZ];
        }
        if (e == ZDZ && v == R(0)) v = R(1);   // outside the grid: a divisor
        sh<R>(sm.zr + c * E) = v;
    }
    // The one-sided first derivative on a wall (pde.cu:363-576) as the centred one
    // with a value beyond the wall, f1 - D / w (w the centred weight): weights of
    // that value; and the one-sided second derivative of T
    if (tid < 14) {
        const double *zc = g.zc;
        const int q = tid % 7, top = Nz - 1;
        const bool bot = tid < 7;
        const double w = bot ? zc[ZC * Nz + 1] : zc[ZC * Nz + top - 1];
        double v;
        if (q < 3) {
            v = bot ? -zc[(ZF0 + q) * Nz] / w : zc[(ZB2 - q) * Nz + top] / w;
            if (q == 1) v += 1.0;
        } else {
            v = bot ? zc[(ZFF0 + q - 3) * Nz] : zc[(ZBB3 - (q - 3)) * Nz + top];
        }
        sh<R>(sm.wall + tid * E) = (R)v;
    }
    if (tid < VW) sh<R>(sm.corr + (4 * CW * VW + tid) * E) = R(0);

    auto block_sync = [&]() { asm volatile("bar.sync 0, %0;" ::"n"(NT + FR) : "memory"); };
    auto up = [](int r, int d, int n) { return r + d >= n ? r + d - n : r + d; };   // ring slot d planes on
    auto col_slot = [&](int c) { return (uint32_t)((c & (kColRing - 1)) * CW); };
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(stage_smem);

    // ---- state planes into the ring ----
    if (tma && tid == 0) {
        for (int r = 0; r < SM::RS; r++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbase + sm.bar + r * 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tma) block_sync();
    after_previous();   // the weights and the barriers above need nothing of it
    // by TMA, issued by one lane of the block's last warp: a box of the tile's rows,
    // or one per row where the tile's halo wraps around in y
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // uniform in a warp
    const bool issuer = warp == (NT + FR) / 32 - 1 && (tid & 31) == 0;
    const bool wraps = j0 < 2 || j0 + tj + 1 > Ny - 2;
    auto fetch_box = [&](int c, int slot) {
        if (!issuer) return;
        const uint32_t bar = sbase + sm.bar + slot * 8, dst = sbase + slot * sm.planeS;
        const int ci = wrap_p(c, Nx - 1);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(tj + 4) * SM::ROW_S) : "memory");
        const uint64_t map = reinterpret_cast<uint64_t>(wraps ? &m_row : &m_tile);
        const int n = wraps ? tj + 4 : 1;
#pragma unroll 1
        for (int r = 0; r < n; r++)
            asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                         "[%0], [%1, {%2, %3, %4, %5}], [%6];"
                         :
                         : "r"(dst + r * SM::ROW_S), "l"(map), "r"(k0 - SM::KH), "r"(0), "r"(wrap_p(j0 - 2 + r, Ny - 1)), "r"(ci), "r"(bar)
                         : "memory");
    };
    // the RK operands of x-plane c of the tile into L2: frame threads, a row of one
    // field each
    auto prefetch_rk = [&](int c) {
        for (int q = tid - NT; q < 8 * tj; q += FR) {
            const int f = q & 3, row = q >> 3;
            const bool acc = q & 4;
            if (j0 + row < Ny && (acc ? rd : !kstore))
                asm volatile("prefetch.global.L2 [%0];" ::"l"(
                    &at(acc ? a.acc : a.yn, f, (uint32_t)c * plane + ((uint32_t)(j0 + row) * (uint32_t)Nz + k0) * E)));
        }
    };
    // column tables of x-plane c, row jj: loaded, and put into the ring
    struct Col {
        double topo;
        R ut;
        int2 ix;
    };
    auto get_col = [&](int c, int jj) {
        Col q = {0.0, R(0), make_int2(0, 0)};
        if (j0 + jj <= Ny) {
            const int col = wrap_p(c, Nx - 1) * Ny + wrap_p(j0 + jj, Ny - 1);
            q.topo = g.topo[col];
            q.ut = a.utau[col];
            q.ix = make_int2(g.nzy[col], g.cut[col]);
        }
        return q;
    };
    auto put_col = [&](int c, int jj, const Col &q) {
        const uint32_t o = col_slot(c) + jj + 1;
        sh<R>(sm.ctopo + o * E) = (R)q.topo;
        sh<R>(sm.cut_ + o * E) = q.ut;
        sh<int2>(sm.cidx + o * 8) = q.ix;
    };

    // ---- this thread's cells: of the tile (tid < NT), or of the frame ----
    const bool frame = warp >= NT / 32;
    const int h = tid - NT;   // frame thread
    int jj, kk;
    bool in;
    if (!frame) {
        const int w = tk / VW;
        jj = tid / w;
        kk = (tid - jj * w) * VW;
        in = jj < tj;
    } else {
        // rows above and below the tile, then the planes above and below it (FP32:
        // the pair that holds the plane)
        const int w = tk / VW;
        in = h < 2 * w + 2 * tj;
        if (h < 2 * w) {
            jj = h < w ? -1 : tj;
            kk = (h < w ? h : h - w) * VW;
        } else {
            const int e = h - 2 * w;
            jj = e < tj ? e : e - tj;
            kk = e < tj ? -VW : tk;
        }
    }
    if (!in) jj = kk = 0;
    const int gj = j0 + jj, gk = k0 + kk;
    const bool comp = in && gj <= Ny && gk < Nz && gk + VW > 0;   // SGS inputs wanted
    const bool fuelz = comp && gk < g.NzY;                        // may hold fuel
    const uint32_t so = SM::s(jj, kk), go = sm.g0 + SM::g(jj, kk), zo = sm.zr + SM::z(kk);
    const uint32_t off = comp ? ((uint32_t)wrap_p(gj, Ny - 1) * (uint32_t)Nz + (uint32_t)max(gk, 0)) * E : 0;
    // second z derivative of T of a wall cell (others: the zero)
    const int side = gk <= 0 ? 0 : gk + VW >= Nz ? 1 : 2;
    const uint32_t co = sm.corr + (side == 2 || !comp ? 4 * CW : side * CW + jj + 1) * (VW * E), cstep = side == 2 || !comp ? 0 : 2 * CW * VW * E;
    // fuel fraction and learned coefficient of the stage input at x-plane c
    auto fuel_at = [&](int c) -> V {
        V Y = c_(R(0));
        if (fuelz) {
            const int nzy = sh<int2>(sm.cidx + (col_slot(c) + jj + 1) * 8).x;
            const uint32_t o = (uint32_t)(wrap_p(c, Nx - 1) * Ny + wrap_p(gj, Ny - 1)) * (uint32_t)g.NzY;
#pragma unroll
            for (int e = 0; e < VW; e++)
                if (gk + e >= 0 && gk + e < nzy) set_el(Y, e, at(a.X, 4, (o + gk + e) * E));
        }
        return Y;
    };
    auto coef_at = [&](int c) -> V {
        V q = c_(R(1));
        if (a.coef && comp) {
#pragma unroll
            for (int e = 0; e < VW; e++)
                if (gk + e >= 0 && gk + e < Nz)
                    set_el(q, e, a.coef[((size_t)wrap_p(c, Nx - 1) * Ny + wrap_p(gj, Ny - 1)) * Nz + gk + e]);
        }
        return q;
    };
    auto arrhenius_v = [&](V T) {
        V K = c_(R(0));
        if (fuelz)
#pragma unroll
            for (int e = 0; e < VW; e++) set_el(K, e, arrhenius(p, el(T, e)));
        return K;
    };

    // by cp.async: every thread its own cells, and of the frame the rows two away (the
    // planes two away are in its pairs) or a corner; zeros outside the grid
    int j2 = jj;
    if (frame && in) j2 = jj < 0 ? -2 : jj == tj ? tj + 1 : jj == 0 ? -1 : jj == tj - 1 ? tj : jj;
    auto copy_cells = [&](int c, int slot, int row) {
        const int gr = j0 + row;
        const uint32_t ci = (uint32_t)wrap_p(c, Nx - 1) * plane + ((uint32_t)wrap_p(gr, Ny - 1) * (uint32_t)Nz + gk) * E;
        // FP64: a frame thread of the planes next to the tile also takes those two away
        const int e0 = VW == 1 && frame && kk < 0 ? -1 : 0, e1 = VW == 1 && frame && kk == tk ? 2 : VW;
#pragma unroll
        for (int e = -1; e < 2; e++) {
            if (e < e0 || e >= e1) continue;
            const bool ok = gk + e >= 0 && gk + e < Nz && gr <= Ny + 1;
            const uint32_t d = slot * sm.planeS + SM::s(row, kk + e);
#pragma unroll
            for (int f = 0; f < 4; f++) cp_async<E>(d + f * SM::FX, &at(a.X, f, ok ? ci + e * E : 0), ok);
        }
    };
    auto fetch_copy = [&](int c, int slot) {
        if (in) {
            copy_cells(c, slot, jj);
            if (j2 != jj) copy_cells(c, slot, j2);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // polls of the waits after the first plane's: FP32 takes the constant, FP64 the argument, each for the
    // fewer spills
    const int wait = E == 4 ? kPlaneWaitLimit : a.plane_wait;
    // Parities of the slots' next arrivals; when a plane did not arrive in time, kLost and its slot (+ 8 in
    // the walk) in the second byte: flagged, no further fetches and waits.  In one register: a word
    // more spilled 48 bytes in the FP32 form with rows of 24, a limit from the arguments 16 (3 to 4% of an
    // ensemble's step).
    constexpr uint32_t kLost = 0x80000000u;
    uint32_t phases = 0;
    auto fetch = [&](int c, int slot) {
        if (!tma) fetch_copy(c, slot);
        else if (!(phases & kLost)) fetch_box(c, slot);
    };
    auto arrived = [&](int slot, int walk, int limit) {
        if (tma && !(phases & kLost)) {
            if (mbar_wait(sbase + sm.bar + slot * 8, (phases >> slot) & 1, limit)) {
                phases ^= 1u << slot;
            } else {
                phases |= kLost | (uint32_t)(slot + walk) << 8;
                if (a.kerr) *(volatile int *)a.kerr = 1;
            }
        }
    };
    // the thread that fetches gives the planes still due a bounded chance to land before the block gives up
    // its shared memory: of the first four those not waited for, in the walk the one
    auto settle = [&]() {
        const int lost = (phases >> 8) & 15;
        if ((phases & kLost) && issuer)
            for (int r = lost & 7; r <= (lost < 8 ? 3 : lost & 7); r++)
                mbar_wait(sbase + sm.bar + r * 8, (phases >> r) & 1, kPlaneWaitLimit);
    };
    for (int c = ib - 2; c <= ib + 1; c++) fetch(c, c - (ib - 2));

    if (frame && h < CW) {
        Col q[3];
#pragma unroll
        for (int n = 0; n < 3; n++) q[n] = get_col(ib - 2 + n, h - 1);
#pragma unroll
        for (int n = 0; n < 3; n++) put_col(ib - 2 + n, h - 1, q[n]);
    }
    if (!tma) asm volatile("cp.async.wait_group 0;" ::: "memory");
    arrived(0, 0, a.plane_wait);
    for (int r = 1; r < 4; r++) arrived(r, 0, wait);
    block_sync();
    V Y = fuel_at(ib - 1), coef = coef_at(ib - 1);

    // values beyond the walls and second derivatives of T on them, of plane c in the
    // ring slot at byte offset b: frame threads, a row each
    const bool has_bot = k0 == 0, has_top = k0 + tk >= Nz;
    auto walls = [&](int c, uint32_t b) {
        for (int q = h; q < 2 * CW; q += FR) {
            const bool lo = q < CW;
            if (!(lo ? has_bot : has_top)) continue;
            const int row = lo ? q : q - CW, kw = lo ? 0 : Nz - 1 - k0, st = lo ? (int)E : -(int)E;
            const uint32_t o = b + SM::s(row - 1, kw), w = sm.wall + (lo ? 0 : 7 * E);
            auto W = [&](int n) { return sh<const R>(w + n * E); };
#pragma unroll
            for (int f = 0; f < 4; f++) {
                const uint32_t of = o + f * SM::FX;
                const R f0 = sh<const R>(of);   // the weights' sum is one
                sh<R>(of - st) = f0 + (W(1) * (sh<const R>(of + st) - f0) + W(2) * (sh<const R>(of + 2 * st) - f0));
            }
            const uint32_t oT = o + 3 * SM::FX, d = sm.corr + (((c & 1) * 2 + (lo ? 0 : 1)) * CW + row) * (VW * E);
            const int e = VW == 2 && !lo ? (Nz - 1) & 1 : 0;   // the wall cell's place among its thread's cells
            if (VW == 2) sh<R>(d + (1 - e) * E) = R(0);
            const R T0 = sh<const R>(oT);   // the weights' sum is zero
            sh<R>(d + e * E) = W(4) * (sh<const R>(oT + st) - T0) + W(5) * (sh<const R>(oT + 2 * st) - T0) + W(6) * (sh<const R>(oT + 3 * st) - T0);
        }
    };
    // The bytes that walls() writes belong to a TMA box: ordered before the copy that refills the slot (the
    // barriers between order the threads, not the two ways of writing).  Plane q is written in iteration q - 1
    // and its slot refilled from iteration q + 3 on, so one fence in four iterations is enough, at an
    // iteration's end: right after the writes it waited for the loads in flight (256 x 256 x 128 FP64 3.35 ms
    // a step; at every iteration's end 3.28)
    auto fence_walls = [&](int c) {
        if (tma && (has_bot || has_top) && h < 2 * CW && (c & 3) == 3) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    if (frame) {
        walls(ib - 1, sm.planeS);
        fence_walls(3);   // written before the first iteration: three are left
    }
    block_sync();

    // byte offsets of this thread's cells in the ring slots of planes c-2 .. c+2 and
    // of the SGS planes c, c-1, c-2, moved on by one slot per iteration
    const uint32_t endS = SM::RS * sm.planeS + so, endG = SM::RG * sm.planeG + go;
    uint32_t am2 = endS - sm.planeS, am1 = so, a0 = so + sm.planeS, ap1 = a0 + sm.planeS, ap2 = ap1 + sm.planeS;
    uint32_t g0 = go, g1 = endG - sm.planeG, g2 = g1 - sm.planeG;
    int rn = 4;   // ring slot of plane c + 3
    auto next_plane = [&](int c) {
        // the plane fetched in this iteration (c + 3) is used from the next one on
        if (!tma) asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (c + 3 <= ie + 1) arrived(rn, 8, wait);
        rn = rn == SM::RS - 1 ? 0 : rn + 1;
        am2 = am1;
        am1 = a0;
        a0 = ap1;
        ap1 = ap2;
        ap2 += sm.planeS;
        if (ap2 == endS) ap2 = so;
        const uint32_t t = g2;
        g2 = g1;
        g1 = g0;
        g0 = t;
        block_sync();
    };

    if (frame) {
#pragma unroll 1
        for (int c = ib - 1; c <= ie; c++) {
            if (c + 3 <= ie + 1) fetch(c + 3, rn);
            if (c + 1 < ie) prefetch_rk(c + 1);
            if (c == ie) start_next();
            V Yn = c_(R(0)), coefn = c_(R(1));
            Col col = {};
            if (c < ie) {
                Yn = fuel_at(c + 1);
                coefn = coef_at(c + 1);
                if (h < CW) col = get_col(c + 2, h - 1);
                if (has_bot || has_top) walls(c + 1, ap1 - so);
            }
            if (c >= ib && h < tj) {
                // Van Driest bound of the columns around (c, h): see part B
                const uint32_t oc = col_slot(c) + h + 1, o5[5] = {oc, col_slot(c + 1) + h + 1, col_slot(c - 1) + h + 1, oc + 1, oc - 1};
                R hmax = R(-1e30), umin = R(1e30);
                int zero = 0;
#pragma unroll
                for (int q = 0; q < 5; q++) {
                    const R ut = sh<R>(sm.cut_ + o5[q] * E);
                    if (ut == R(0)) {
                        zero |= 1 << q;
                    } else {
                        hmax = rmax(hmax, sh<R>(sm.ctopo + o5[q] * E));
                        umin = rmin(umin, ut);
                    }
                }
                const uint32_t o = (c & 1) * tj + h;
                sh<R>(sm.bnd + 2 * o * E) = hmax;
                sh<R>(sm.bnd + (2 * o + 1) * E) = rmax(umin, R(0)) * p.inv_avd;
                sh<int>(sm.zero + o * 4) = zero;
            }
            if (comp) {
                const uint32_t s = a0, sp = ap1, sm1 = am1;
                const V hz = sh<V>(zo + ZD1 * SM::FZ);
                Grad<V> d[4];
                V lapT;
#pragma unroll
                for (int f = 0; f < 4; f++) {
                    const uint32_t o = f * SM::FX;
                    const V f0 = sh<V>(s + o);
                    const auto zn = z_nb<R>(s + o, f0);
                    const V xm = f0 - sh<V>(sm1 + o), xp = sh<V>(sp + o) - f0, ym = f0 - sh<V>(s + o - SM::ROW_S), yp = sh<V>(s + o + SM::ROW_S) - f0;
                    const V zm = zn.m1 - f0, zp = zn.p1 - f0;
                    d[f].x = xp + xm;
                    d[f].y = yp + ym;
                    d[f].z = zp - zm;
                    if (f == 3)
                        lapT = vfma(sh<V>(zo + (ZD2 + 1) * SM::FZ), zp, vfma(sh<V>(zo + ZD2 * SM::FZ), zm, vfma(cv.ly, yp - ym, cv.lx * (xp - xm)))) +
                               sh<V>(co + (c & 1) * cstep);
                }
                const V T = sh<V>(s + 3 * SM::FX), K_T = arrhenius_v(T);
                const int nzy = LEAN ? 0 : sh<int2>(sm.cidx + (col_slot(c) + jj + 1) * 8).x;
                V src, nu, g7;
                const V Tx = d[3].x * cv.hx, Ty = d[3].y * cv.hy, Tz = d[3].z * hz;
                sources<R, V, LEAN>(a, cv, Tx, Ty, Tz, lapT, T, Y, K_T, gk, nzy, LEAN ? T : sh<V>(zo + ZDZ * SM::FZ), src, nu, g7);
                V l2 = sh<V>(zo + ZL * SM::FZ);
                if (a.coef) l2 = l2 * coef;
                put_sgs<SM, V>(g0, strain<R, V>(cv, d, hz, T, l2, g7));
            }
            if (h < CW && c < ie) put_col(c + 2, h - 1, col);
            Y = Yn;
            coef = coefn;
            fence_walls(c);
            next_plane(c);
        }
        settle();
    } else {
        // ---- the tile ----
        const bool act = in && gj < Ny && gk < Nz;                  // holds cells of the grid
        const bool low = act && gk <= a.kcmax + 2, top3 = act && gk + VW > Nz - 3;
        const uint32_t own = act ? ((uint32_t)gj * (uint32_t)Nz + (uint32_t)gk) * E : 0;
        // carried from part A of plane c-1 to its part B: right-hand side without the
        // SGS terms, gradient and Laplacian of T
        V kA[4], gT[4];
#pragma unroll
        for (int f = 0; f < 4; f++) kA[f] = gT[f] = c_(R(0));

#pragma unroll 1
        for (int c = ib - 1; c <= ie; c++) {
            if (!tma && c + 3 <= ie + 1) fetch(c + 3, rn);
            V Yn = c_(R(0)), coefn = c_(R(1));
            if (c < ie) {
                Yn = fuel_at(c + 1);
                coefn = coef_at(c + 1);
            }
            // ---- A. plane c ----
            const uint32_t s = a0, sp = ap1, sp2 = ap2, sm1 = am1, sm2 = am2;
            const V hz = sh<V>(zo + ZD1 * SM::FZ);
            const V u = sh<V>(s), v = sh<V>(s + SM::FX), w = sh<V>(s + 2 * SM::FX), T = sh<V>(s + 3 * SM::FX);
            // Upwind advection (pde.cu:341-437) on differences from the cell's value, which leaves no
            // rounding of the value itself: u+ (3f - 4f_{i-1} + f_{i-2})/(2dx) = u+ (4(f - f_{i-1}) -
            // (f - f_{i-2}))/(2dx), likewise u-; in z the backward form (weights ZB) carries w+ and the
            // forward form (ZF) w-, except next to the walls, where one form carries both.
            const bool rhs = c >= ib && c < ie;   // else only the SGS inputs are wanted
            // adv holds minus the advection.
            const V ax = vpos(u) * cv.m_hx, bx = vneg(u) * cv.m_hx, ay = vpos(v) * cv.m_hy, by = vneg(v) * cv.m_hy;
            const V wb = vfma(sh<V>(zo + ZWW * SM::FZ), w, sh<V>(zo + ZWP * SM::FZ) * vpos(w)), wf = w - wb;
            const V Czm2 = wb * sh<V>(zo + ZB * SM::FZ), Czm = wb * sh<V>(zo + (ZB + 1) * SM::FZ);
            const V Czp = wf * sh<V>(zo + (ZF + 1) * SM::FZ), Czp2 = wf * sh<V>(zo + (ZF + 2) * SM::FZ);
            const V Lzm = sh<V>(zo + ZD2 * SM::FZ), Lzp = sh<V>(zo + (ZD2 + 1) * SM::FZ);
            Grad<V> d[4];
            V lap[4], adv[4];
#pragma unroll
            for (int f = 0; f < 4; f++) {
                const uint32_t o = f * SM::FX;
                const V f0 = f == 0 ? u : f == 1 ? v : f == 2 ? w : T;
                const auto zn = z_nb<R>(s + o, f0);
                const V xm = f0 - sh<V>(sm1 + o), xp = sh<V>(sp + o) - f0, ym = f0 - sh<V>(s + o - SM::ROW_S), yp = sh<V>(s + o + SM::ROW_S) - f0;
                const V zm = zn.m1 - f0, zp = zn.p1 - f0;
                if (rhs) {
                    V r = ax * vfma(cv.p4, xm, sh<V>(sm2 + o) - f0);
                    r = vfma(bx, vfma(cv.p4, xp, f0 - sh<V>(sp2 + o)), r);
                    r = vfma(ay, vfma(cv.p4, ym, sh<V>(s + o - 2 * SM::ROW_S) - f0), r);
                    r = vfma(by, vfma(cv.p4, yp, f0 - sh<V>(s + o + 2 * SM::ROW_S)), r);
                    r = vfma(Czm, zm, r);
                    r = vfma(Czm2, zn.m2 - f0, r);
                    r = vfma(Czp, zp, r);
                    adv[f] = vfma(Czp2, zn.p2 - f0, r);
                }
                if (rhs || f == 3) lap[f] = vfma(Lzp, zp, vfma(Lzm, zm, vfma(cv.ly, yp - ym, cv.lx * (xp - xm))));
                d[f].x = xp + xm;
                d[f].y = yp + ym;
                d[f].z = zp - zm;
            }
            const uint32_t oq = (uint32_t)(c - 1) * plane + own;
            const bool upd = act && c > ib;
            // RK operands of plane c-1, early (what is written to the cut node and the top plane is
            // lost: k_stage_edge has their values)
            V yv[4], av[4];
#pragma unroll
            for (int f = 0; f < 4; f++) {
                yv[f] = av[f] = c_(R(0));
                if constexpr (VEC) {
                    if (upd && !kstore) yv[f] = *reinterpret_cast<const V *>(&at(a.yn, f, oq));
                    if (upd && rd) av[f] = *reinterpret_cast<const V *>(&at(a.acc, f, oq));
                } else {
#pragma unroll
                    for (int e = 0; e < VW; e++)
                        if (upd && gk + e < Nz) {
                            if (!kstore) set_el(yv[f], e, at(a.yn, f, oq + e * E));
                            if (rd) set_el(av[f], e, at(a.acc, f, oq + e * E));
                        }
                }
            }
            lap[3] = lap[3] + sh<V>(co + (c & 1) * cstep);
            const V K_T = arrhenius_v(T);
            const int nzy = LEAN ? 0 : sh<int2>(sm.cidx + (col_slot(c) + jj + 1) * 8).x;
            V src, nu, g7;
            const V Tx = d[3].x * cv.hx, Ty = d[3].y * cv.hy, Tz = d[3].z * hz;
            sources<R, V, LEAN>(a, cv, Tx, Ty, Tz, lap[3], T, Y, K_T, gk, nzy, LEAN ? T : sh<V>(zo + ZDZ * SM::FZ), src, nu, g7);
            V l2 = sh<V>(zo + ZL * SM::FZ);
            if (a.coef) l2 = l2 * coef;
            const Sgs<V> q0 = strain<R, V>(cv, d, hz, T, l2, g7);
            if (comp) put_sgs<SM, V>(g0, q0);

            // ---- B. plane c-1 ----
            if (c > ib) {
                int kc = -3;
                if (low) kc = sh<int2>(sm.cidx + (col_slot(c - 1) + jj + 1) * 8).y;
                const V Tq = sh<V>(sm1 + 3 * SM::FX), nuq = cv.mu_Trho * Tq;
                auto G1 = [&](int f) { return sh<V>(g1 + f * SM::FG); };
                auto G2 = [&](int f) { return sh<V>(g2 + f * SM::FG); };
                auto Gyp = [&](int f) { return sh<V>(g1 + f * SM::FG + SM::ROW_G); };
                auto Gym = [&](int f) { return sh<V>(g1 + f * SM::FG - SM::ROW_G); };
                V mu_c = G1(G_MU), mu_xp = q0.mu, mu_xm = G2(G_MU), mu_yp = Gyp(G_MU), mu_ym = Gym(G_MU), mu_kp, mu_km;
                if constexpr (VW == 2) {
                    mu_km.v = make_float2(sh<float>(g1 - 4), mu_c.v.x);
                    mu_kp.v = make_float2(mu_c.v.y, sh<float>(g1 + 8));
                } else {
                    mu_km = sh<V>(g1 - 8);
                    mu_kp = sh<V>(g1 + 8);
                }
                // Van Driest damping (turbulence.cu:255-454): the factor of a point is
                // 1 - exp(-z_ibm u_tau / (A nu)) with its column's distance and friction and this
                // cell's nu.  Where the least z_ibm u_tau / A of the columns with friction
                // exceeds the cut-off times nu, their factors are exactly 1; a column without
                // friction (u_tau = 0, as over the hills) has the factor 1 - exp(-0) = 0.
                const uint32_t ob = ((c - 1) & 1) * tj + jj;
                const R hb = sh<R>(sm.bnd + 2 * ob * E), ub = sh<R>(sm.bnd + (2 * ob + 1) * E);
                const R zlow = rmax(sh<R>(zo + ZZ * SM::FZ - E) - hb, R(0)) * ub, cutoff = VanDriestCut<R>::v * R(1.001);
                bool far = zlow > cutoff * el(nuq, 0);
                if (VW == 2) far = far && zlow > cutoff * el(nuq, 1);
                far = far || !act;
                const int zero = sh<int>(sm.zero + ob * 4);
                if (far && zero) {
                    const V z0 = c_(R(0)), z1 = c_(R(1));
                    const V fc = (zero & 1) ? z0 : z1;
                    mu_c = mu_c * fc;
                    mu_kp = mu_kp * fc;
                    mu_km = mu_km * fc;
                    mu_xp = mu_xp * ((zero & 2) ? z0 : z1);
                    mu_xm = mu_xm * ((zero & 4) ? z0 : z1);
                    mu_yp = mu_yp * ((zero & 8) ? z0 : z1);
                    mu_ym = mu_ym * ((zero & 16) ? z0 : z1);
                }
                // the others, few lanes of a warp, with the whole warp: four of them at a
                // time, a lane for one of the seven points of one of them
                unsigned near = __ballot_sync(0xffffffffu, !far);
                while (near) {
                    const int lane = tid & 31, pt = lane % 7;
                    unsigned m = near;
                    int src = 0, rank = -1;   // the cell this lane works for, this lane's own place among the four
#pragma unroll
                    for (int n = 0; n < 4; n++) {
                        const int l = __ffs(m) - 1;
                        if (n == lane / 7 && l >= 0) src = l;
                        if (n == 0 || l >= 0) rank = l == lane ? n : rank;
                        m &= m - 1;
                    }
                    near = m;
                    const V q = vdiv(c_(-p.inv_avd), vshfl(nuq, src));
                    const int jr = __shfl_sync(0xffffffffu, jj, src), kr = __shfl_sync(0xffffffffu, kk, src);
                    const uint32_t o = (col_slot(pt == 1 ? c : pt == 2 ? c - 2 : c - 1) + jr + (pt == 3 ? 2 : pt == 4 ? 0 : 1)) * E;
                    const uint32_t oz = sm.zr + ZZ * SM::FZ + SM::z(kr + (pt == 5 ? 1 : pt == 6 ? -1 : 0));
                    V zh;
#pragma unroll
                    for (int e = 0; e < VW; e++) set_el(zh, e, sh<R>(oz + e * E));
                    const V f = vd_factor2<R, V>(zh, sh<R>(sm.ctopo + o), sh<R>(sm.cut_ + o), q);
                    const int from = (rank < 0 ? 0 : rank) * 7;
                    auto damp = [&](V &mu, int n) {
                        const V x = vshfl(f, from + n);
                        if (rank >= 0) mu = mu * x;
                    };
                    damp(mu_c, 0);
                    damp(mu_xp, 1);
                    damp(mu_xm, 2);
                    damp(mu_yp, 3);
                    damp(mu_ym, 4);
                    damp(mu_kp, 5);
                    damp(mu_km, 6);
                }
                const V mu_x = (mu_xp - mu_xm) * cv.hx, mu_y = (mu_yp - mu_ym) * cv.hy, mu_z = (mu_kp - mu_km) * hz;
                const V S11 = G1(G_S11), S12 = G1(G_S12), S13 = G1(G_S13), S22 = G1(G_S22), S23 = G1(G_S23), S33 = G1(G_S33);
                auto zd = [&](int f, V own_v) { return z_diff<R>(g1 + f * SM::FG, own_v); };
                const V two_inv_rho = cv.two_inv_Trho * Tq;
                V k[4];
                V dS = vfma(zd(G_S13, S13), hz, vfma(Gyp(G_S12) - Gym(G_S12), cv.hy, (q0.S11 - G2(G_S11)) * cv.hx));
                V t = vfma(mu_c, dS, vfma(mu_z, S13, vfma(mu_y, S12, mu_x * S11)));
                k[0] = vfma(two_inv_rho, t, vfma((q0.g7 - G2(G_Q)) * cv.hx, cv.third, kA[0]));
                dS = vfma(zd(G_S23, S23), hz, vfma(Gyp(G_S22) - Gym(G_S22), cv.hy, (q0.S12 - G2(G_S12)) * cv.hx));
                t = vfma(mu_c, dS, vfma(mu_z, S23, vfma(mu_y, S22, mu_x * S12)));
                k[1] = vfma(two_inv_rho, t, vfma((Gyp(G_Q) - Gym(G_Q)) * cv.hy, cv.third, kA[1]));
                dS = vfma(zd(G_S33, S33), hz, vfma(Gyp(G_S23) - Gym(G_S23), cv.hy, (q0.S13 - G2(G_S13)) * cv.hx));
                t = vfma(mu_c, dS, vfma(mu_z, S33, vfma(mu_y, S23, mu_x * S13)));
                k[2] = vfma(two_inv_rho, t, vfma(zd(G_Q, G1(G_Q)) * hz, cv.third, kA[2]));
                t = vfma(mu_c, gT[3], vfma(mu_z, gT[2], vfma(mu_y, gT[1], mu_x * gT[0])));
                k[3] = vfma(cv.inv_Trho_Pr * Tq, t, kA[3]);
                if (low || top3) {
                    // k-values the boundary rules extrapolate from
                    R *bg = a.bc + (size_t)((c - 1) * Ny + gj) * kBcSlots;
#pragma unroll
                    for (int e = 0; e < VW; e++) {
                        const int q = gk + e;
                        if (q == kc + 1 || q == kc + 2) bg[q - kc - 1] = el(k[3], e);
                        if (q < kc) {   // below the cut node (pde.cu:88-97)
#pragma unroll
                            for (int f = 0; f < 4; f++) set_el(k[f], e, p.dead[f]);
                        }
                        if (q == Nz - 2 || q == Nz - 3) {
#pragma unroll
                            for (int f = 0; f < 4; f++) bg[(q == Nz - 2 ? 2 : 6) + f] = el(k[f], e);
                        }
                    }
                }
#pragma unroll
                for (int f = 0; f < 4; f++) {
                    const V out = vfma(cv.ar, vfma(cv.cA, av[f], k[f]), yv[f]);
                    const V acc = vfma(cv.cK, k[f], av[f]);
                    if constexpr (VEC) {
                        if (act) *reinterpret_cast<V *>(&const_cast<R &>(at(a.Xout, f, oq))) = out;
                        if (act && kp) *reinterpret_cast<V *>(&const_cast<R &>(at(a.acc, f, oq))) = acc;
                    } else {
#pragma unroll
                        for (int e = 0; e < VW; e++)
                            if (act && gk + e < Nz) {
                                const_cast<R &>(at(a.Xout, f, oq + e * E)) = el(out, e);
                                if (kp) const_cast<R &>(at(a.acc, f, oq + e * E)) = el(acc, e);
                            }
                    }
                }
            }
            // right-hand side of plane c without the SGS terms; buoyancy
            // g (rho - rho_inf) / rho with rho = T_inf rho_inf / T
            if (!rhs) {
#pragma unroll
                for (int f = 0; f < 4; f++) adv[f] = lap[f] = c_(R(0));   // not used
            }
            kA[0] = vfma(nu, lap[0], adv[0]);
            kA[1] = vfma(nu, lap[1], adv[1]);
            kA[2] = vfma(cv.g_Tinf, cv.T_inf - T, vfma(nu, lap[2], adv[2]));
            if (a.ph.temperature_convection == 0) adv[3] = c_(R(-1)) * vfma(w, Tz, vfma(v, Ty, u * Tx));
            kA[3] = src + adv[3];
            if constexpr (!LEAN) {
                const V drag = c_(-p.cd) * Y * vsqrt(vfma(w, w, vfma(v, v, u * u)));   // Y is 0 above the fuel
                kA[0] = vfma(drag, u, kA[0]);
                kA[1] = vfma(drag, v, kA[1]);
                kA[2] = vfma(drag, w, kA[2]);
            }
            gT[0] = Tx;
            gT[1] = Ty;
            gT[2] = Tz;
            gT[3] = lap[3];
            Y = Yn;
            coef = coefn;
            next_plane(c);
        }
    }
}

// ---------------------------------------------------------------------------
// What the fused pass leaves of a stage (pde.cu:14-99, 713-720), eight threads per
// column: the top plane (threads 0-3, a field each), the cut node (4-7) and the
// fuel (all).  The k-values they extrapolate from, and their accumulators, are in
// a.bc.  These cells are few, each a chain of dependent loads: as a kernel of their
// own all chains run at once, where at the end of each block of the fused pass they
// cost 75 of its 436 us (256 x 256 x 128 with hills, FP32).  Fuel entries above a
// column's fuel top never change and are not read, so only the stage that makes
// the new state copies them.  The thread of the cut node's T also takes the next
// stage's wall friction velocity, which saves that stage its k_utau.
// The last planes in x and y repeat the first ones, but for the fuel: the fused
// pass takes the first planes' for both, and what a seam cell's own fuel changes in
// its drag, reaction and convective exchange is added here (inside the fused
// pass the second evaluation spilled 32 to 96 bytes and cost 5% of the FP32 step; here
// 1 us of a 56 us step of 33 x 33 x 16 in FP64, nothing on the larger grids).
template <class R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 12 : 8) k_stage_edge(const StageArgs<R> a, int all_fuel)
{
    const Geom &g = a.g;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = t >> 3, p = t & 7, f = p & 3;
    if (col >= g.Nx * g.Ny) return;
    const size_t N = (size_t)g.N, cb = (size_t)col * g.Nz;
    const int i = col / g.Ny, wc = wrap_p(i, g.Nx - 1) * g.Ny + wrap_p(col - i * g.Ny, g.Ny - 1);
    const bool seam = wc != col;
    const int kc = __ldg(g.cut + wc), nzy = __ldg(g.nzy + wc), nf = all_fuel ? g.NzY : nzy;
    start_next();
    after_previous();
    const bool rd = stage_reads_acc(a.method, a.stage), kp = stage_keeps_acc(a.method, a.stage);
    const R an = (R)a.a_next;
    R *bc = a.bc + (size_t)col * kBcSlots;
    const R *w = a.krow + (size_t)kc * KROW;
    // the top plane and the cut node: no slip, T extrapolated (loads before stores, which may alias them)
    const bool top = p < 4, cutT = p == 7;
    const size_t o = f * N + cb + (top ? g.Nz - 1 : kc);
    const R y = a.yn[o];
    R *bacc = bc + (top ? 11 + f : 10);
    // whether plane q of a seam column holds other fuel than its copy, and what that adds to the
    // k-value of field f there
    auto fuel_jumps = [&](int q) {
        return seam && q < nzy && a.X[4 * N + (size_t)col * g.NzY + q] != a.X[4 * N + (size_t)wc * g.NzY + q];
    };
    auto own_fuel = [&](int q, int f) {
        const PhysR<R> &r = a.pr;
        const R Y = a.X[4 * N + (size_t)col * g.NzY + q], Yw = a.X[4 * N + (size_t)wc * g.NzY + q];
        const R *X = a.X + (size_t)wc * g.Nz + q;
        if (f < 3) {
            const R u = X[0], v = X[N], w = X[2 * N];
            return -r.cd * (Y - Yw) * rsqrt_(u * u + v * v + w * w) * X[f * N];
        }
        const R T = X[3 * N], K = r.H_C_cp * (Y - Yw) * arrhenius(r, T);
        if (r.alpha_s * r.sigma_s == R(0) || (Y > R(0)) == (Yw > R(0))) return K;
        // the exchange of a cell with fuel less that of one without (sources)
        const R dz = a.krow[(size_t)q * KROW + RDZ], dT = T - r.T_inf;
        const R h = r.h_c * dz * rsqrt_(rsqrt_(fdiv(rfabs(dT), dz))) * r.alpha_s * r.sigma_s * dT * r.inv_Trho_cp * (r.T_inf + T);
        return Y > R(0) ? K + h : K - h;
    };
    // added to what is there already: the update is linear in the k-value
    auto add = [&](size_t at, R *accv, R d) {
        R dacc = R(0);
        a.Xout[at] += rk_update(a.method, a.stage, d, R(0), dacc, an);
        if (kp) *accv += dacc;
    };
    const int q1 = top ? g.Nz - 2 : kc + 1, q2 = top ? g.Nz - 3 : kc + 2;   // the cells extrapolated from
    const bool jumps1 = (top || cutT) && fuel_jumps(q1), jumps2 = (top || cutT) && fuel_jumps(q2);
    R kv = R(0), acc = R(0), T0 = R(1), u[3] = {R(0), R(0), R(0)}, v[3] = {R(0), R(0), R(0)};
    const bool utau = cutT && a.make_utau && !seam;   // of the first planes only, which stand for the last
    if (utau) {
        // for the wall friction velocity: u and v of the cut node keep y_n, the others the
        // fused pass has written
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const R *src = q == kc ? a.yn : a.Xout;
            u[q] = src[cb + q];
            v[q] = src[N + cb + q];
        }
        if (kc > 0) T0 = a.Xout[3 * N + cb];
    }
    if (top || cutT) {
        kv = top ? a.pr.top_w1 * bc[2 + f] - a.pr.top_w2 * bc[6 + f] : w[RCUT1] * bc[0] - w[RCUT2] * bc[1];
        if (rd) acc = *bacc;
    }
    const R out = rk_update(a.method, a.stage, kv, y, acc, an);
    a.Xout[o] = out;
    if ((top || cutT) && kp) *bacc = acc;
#pragma unroll 1
    for (int n = jumps1 ? 0 : 1; n < (jumps2 ? 2 : 1); n++) {
        const R wt = top ? (n ? -a.pr.top_w2 : a.pr.top_w1) : n ? -w[RCUT2] : w[RCUT1];
        add(o, bacc, wt * own_fuel(n ? q2 : q1, f));
    }
    if (utau) a.utau[col] = utau_of(a, u, v, kc == 0 ? out : T0);
    for (int k = p; k < nf; k += 8) {
        // rate -Y_f K(T) Y below the fuel top
        const size_t oY = 4 * N + (size_t)col * g.NzY + k;
        auto rate = [&](int q) {
            return q < nzy ? -a.pr.Y_f * arrhenius(a.pr, a.X[3 * N + (size_t)wc * g.Nz + q]) * a.X[oY + q - k] : R(0);
        };
        const R yY = a.yn[oY];
        const bool jumps = k > kc && k < g.Nz - 1 && fuel_jumps(k);
        R aY = (rd && k < nzy) ? a.acc[oY] : R(0), r = R(0);
        if (k < nzy) r = k == kc ? w[RCUT1] * rate(kc + 1) - w[RCUT2] * rate(kc + 2) : k < kc ? a.pr.dead[4] : rate(k);
        a.Xout[oY] = rk_update(a.method, a.stage, r, yY, aY, an);
        if (kp && k < nzy) a.acc[oY] = aY;
#pragma unroll 1
        for (int q = 0; jumps && q < 4; q++) add(q * N + cb + k, a.acc + q * N + cb + k, own_fuel(k, q));
    }
}

// Block forms of the fused pass, by the names wf_set_stage_tile takes (the last
// number is the threads of a block): interior and frame threads, blocks per
// multiprocessor.
template <int NT_, int FR_, int NB_> struct StageForm { static constexpr int NT = NT_, FR = FR_, NB = NB_; };
template <class R> struct StageForms;
template <> struct StageForms<float> {
    static constexpr int count = 3;
    static constexpr int ti[3] = {8, 8, 8}, tj[3] = {16, 16, 8}, name[3] = {512, 384, 256};
};
template <> struct StageForms<double> {
    static constexpr int count = 2;
    static constexpr int ti[2] = {8, 8}, tj[2] = {8, 8}, name[2] = {512, 256};
};
// f(form) for the form with index idx
template <class R, class F> cudaError_t with_form(int idx, F f)
{
    if constexpr (sizeof(R) == 4) {
        switch (idx) {
        case 0: return f(StageForm<416, 96, 1>());
        case 1: return f(StageForm<288, 96, 1>());
        case 2: return f(StageForm<192, 64, 2>());
        default: return cudaErrorInvalidValue;
        }
    } else {
        switch (idx) {
        case 0: return f(StageForm<416, 96, 1>());
        case 1: return f(StageForm<160, 96, 2>());
        default: return cudaErrorInvalidValue;
        }
    }
}

}  // namespace

// Planes of a z-tile: nearly equal tiles of at most 32 planes, multiples of 16
// bytes, the last with at least 4, so that the top plane and the two below it
// share a tile, and a wall plane and the three next to it a tile or its halo.
int stage_tile_k(int Nz)
{
    for (int n = (Nz + 31) / 32;; n++) {
        const int tk = ((Nz + n - 1) / n + 3) / 4 * 4;
        if ((Nz - 1) % tk >= 3) return tk;
    }
}

namespace {

// Shared memory of a block with tj rows.
template <class R> size_t stage_bytes(int tk, int tj) { return tk > kTileK2 ? StageSmem<R, kTileK>(tj).end : StageSmem<R, kTileK2>(tj).end; }

// Tiling of a grid for blocks of form F on sms multiprocessors: rows per tile and
// x-planes per block of least cost.  A block takes L + 3 iterations (the two
// planes around its own, and the first loads); an iteration of a partly filled tile is
// shorter, but by far less than its share of the threads (latency).  Where the blocks
// fill the machine, passes of short blocks balance better than one of long ones
// (those next to the terrain or the top do more), hence the quarter pass.  Where they
// do not, the cost is two fifths the time of a block and three fifths the share of the
// machine it takes: the first is what a call alone waits for, the second what
// other contexts and ensemble members lose.  The weights are those of least loss over
// 8 FP64 and 6 FP32 grids of 17 x 17 x 12 to 128 x 128 x 64, 30 tilings each, timed
// alone and by three contexts in turn.  Per step, alone / in turn (us), the tilings
// these weights choose against those of weights that favour small tiles (0.4 + 0.6 of
// the fill, half and half): 33 x 33 x 16 FP64 135 / 53 (132 / 58), 48 x 40 x 20 FP64 with
// all source terms 165 / 78 (164 / 92), 64 x 64 x 32 FP32 146 / 67 (139 / 78).
template <class R, class F> StageGrid plan_form(int Nx, int Ny, int Nz, int sms)
{
    constexpr int VW = Vec<R>::W;
    StageGrid s;
    s.tma = false;
    s.tk = stage_tile_k(Nz);
    s.ntk = (Nz + s.tk - 1) / s.tk;
    int jmax = F::NT / (s.tk / VW);
    if (jmax > F::FR / 2 - s.tk / VW) jmax = F::FR / 2 - s.tk / VW;
    while (jmax > 1 && stage_bytes<R>(s.tk, jmax) > (size_t)(227 / F::NB - (F::NB > 1 ? 1 : 0)) * 1024) jmax--;
    double best = 0.0;
    s.L = 0;
    for (int n = (Ny + jmax - 1) / jmax; n <= Ny; n++) {
        const int tj = (Ny + n - 1) / n;
        if ((Ny + tj - 1) / tj != n) continue;
        const double iter = 0.6 + 0.4 * (double)(tj * (s.tk / VW)) / F::NT;
        for (int m = 1; m <= Nx; m++) {
            const int L = (Nx + m - 1) / m;
            if ((Nx + L - 1) / L != m) continue;
            const long long blocks = (long long)s.ntk * n * m, slots = (long long)F::NB * sms;
            const double waves = (double)((blocks + slots - 1) / slots);
            const double cost = (blocks < slots ? 0.5 + 0.75 * (double)blocks / slots : waves + 0.25) * (L + 3) * iter;
            if (s.L == 0 || cost < best) {
                best = cost;
                s.L = L;
                s.tj = tj;
                s.ntj = n;
                s.nti = m;
            }
        }
        if (tj <= 4) break;
    }
    return s;
}

}  // namespace

int g_stage_sms = 0;   // multiprocessors of the device, read at set-up

template <class R> cudaError_t stage_set_attributes()
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (!e) e = cudaDeviceGetAttribute(&g_stage_sms, cudaDevAttrMultiProcessorCount, dev);
    for (int q = 0; !e && q < StageForms<R>::count; q++)
        e = with_form<R>(q, [](auto f) {
            using F = decltype(f);
            const int most = 227 * 1024;
            const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
            cudaError_t e = cudaSuccess;
            auto set = [&](auto kw) {
                constexpr int KW = decltype(kw)::value;
                if (!e) e = cudaFuncSetAttribute(k_stage_march<R, F::NT, F::FR, F::NB, KW, true, true>, attr, most);
                if (!e) e = cudaFuncSetAttribute(k_stage_march<R, F::NT, F::FR, F::NB, KW, false, true>, attr, most);
                if constexpr (Vec<R>::W > 1) {
                    if (!e) e = cudaFuncSetAttribute(k_stage_march<R, F::NT, F::FR, F::NB, KW, true, false>, attr, most);
                    if (!e) e = cudaFuncSetAttribute(k_stage_march<R, F::NT, F::FR, F::NB, KW, false, false>, attr, most);
                }
            };
            set(std::integral_constant<int, kTileK>());
            set(std::integral_constant<int, kTileK2>());
            return e;
        });
    return e;
}
template cudaError_t stage_set_attributes<double>();
template cudaError_t stage_set_attributes<float>();

static F2 host_splat(float x)
{
    F2 v;
    v.v = make_float2(x, x);
    return v;
}
static double host_splat(double x) { return x; }
template <class R> static StageVec<R> stage_vec(const StageArgs<R> &a)
{
    const PhysR<R> &p = a.pr;
    const bool kstore = a.method == 3, last = stage_reads_acc(a.method, a.stage) && !stage_keeps_acc(a.method, a.stage);
    auto s = [](R x) { return host_splat(x); };
    StageVec<R> q;
    q.hx = s(p.inv2dx); q.hy = s(p.inv2dy); q.lx = s(p.invdx2); q.ly = s(p.invdy2);
    q.c12 = s(p.c12); q.c4 = s(p.c4); q.kT = s(p.kT); q.inv_Trho_cp = s(p.inv_Trho_cp); q.H_C_cp = s(p.H_C_cp);
    q.mu_Trho = s(p.mu_Trho); q.Trho = s(p.Trho); q.two_inv_Trho = s(p.two_inv_Trho); q.inv_Trho_Pr = s(p.inv_Trho_Pr);
    q.g_Tinf = s(p.g_Tinf); q.T_inf = s(p.T_inf);
    q.third = s(R(1.0 / 3.0)); q.m_third = s(R(-1.0 / 3.0)); q.half = s(R(0.5)); q.p4 = s(R(4));
    q.m_hx = s(-p.inv2dx); q.m_hy = s(-p.inv2dy);
    // RK update out = ar (k + cA acc) + y_n, acc' = acc + cK k (rk_update)
    q.ar = s(kstore ? R(1) : (R)a.a_next);
    q.cA = s(last ? R(1) : R(0));
    q.cK = s(a.method == 2 && a.stage > 1 && a.stage < 4 ? R(2) : R(1));
    return q;
}

template <class R> cudaError_t launch_stage(const StageArgs<R> &a, cudaStream_t s, cudaEvent_t *ev)
{
    const int ncol = a.g.Nx * a.g.Ny;
    if (a.coef) {
        cudaError_t e = launch_closure_coef_tc<R>(a.X, a.g, a.ph.dx, a.ph.dy, a.theta, a.coef, a.closure_err, s,
                                                  a.closure_wait);
        if (e) return e;
    }
    if (!a.have_utau) k_utau<R><<<(ncol + 127) / 128, 128, 0, s>>>(a);
    if (ev) cudaEventRecord(ev[0], s);
    const bool lean = a.ph.sutherland_viscosity != 1 && a.ph.sutherland_conductivity != 1 && a.ph.alpha_s * a.ph.sigma_s == 0.0;
    const StageVec<R> cv = stage_vec(a);
    cudaError_t e = with_form<R>(a.tile, [&](auto f) {
        using F = decltype(f);
        StageGrid sg = a.grid;
        CUtensorMap m[2];   // X by tiles and by rows
        memset(m, 0, sizeof(m));
        sg.tma = a.tmap[0] && a.tmap[1];
        for (int q = 0; q < 2 && sg.tma; q++) memcpy(&m[q], a.tmap[q], sizeof(m[q]));
        const int blocks = sg.ntk * sg.ntj * sg.nti, threads = F::NT + F::FR;
        const size_t smem = stage_bytes<R>(sg.tk, sg.tj);
        auto go = [&](auto kw, auto lean_, auto vec_) {
            return launch_early(k_stage_march<R, F::NT, F::FR, F::NB, decltype(kw)::value, decltype(lean_)::value, decltype(vec_)::value>,
                                blocks, threads, smem, s, a, cv, sg, m[0], m[1]);
        };
        auto go_kw = [&](auto kw) {
            if (Vec<R>::W == 1 || a.g.Nz % Vec<R>::W == 0) {   // a thread's cells are one aligned access
                return lean ? go(kw, std::true_type(), std::true_type()) : go(kw, std::false_type(), std::true_type());
            } else if constexpr (Vec<R>::W > 1) {
                return lean ? go(kw, std::true_type(), std::false_type()) : go(kw, std::false_type(), std::false_type());
            }
            return cudaErrorInvalidValue;
        };
        return sg.tk > kTileK2 ? go_kw(std::integral_constant<int, kTileK>()) : go_kw(std::integral_constant<int, kTileK2>());
    });
    if (e) return e;
    if (ev) cudaEventRecord(ev[1], s);
    const bool last = a.method == 3 || !stage_keeps_acc(a.method, a.stage);
    if ((e = launch_early(k_stage_edge<R>, (unsigned)((8 * (size_t)ncol + 127) / 128), 128, 0, s, a, (int)last))) return e;
    if (ev) cudaEventRecord(ev[2], s);
    return cudaGetLastError();
}

StageGrid stage_plan(int precision, int form, int Nx, int Ny, int Nz)
{
    StageGrid sg;
    const int sms = g_stage_sms;
    if (precision == 0) with_form<double>(form, [&](auto f) { sg = plan_form<double, decltype(f)>(Nx, Ny, Nz, sms); return cudaSuccess; });
    else with_form<float>(form, [&](auto f) { sg = plan_form<float, decltype(f)>(Nx, Ny, Nz, sms); return cudaSuccess; });
    return sg;
}

bool stage_tensor_map(void *out, const void *X, int precision, int Nx, int Ny, int Nz, int rows, void *encode_fn)
{
    const size_t E = precision == 0 ? 8 : 4;
    if (!encode_fn || Nz * E % 16 != 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0) return false;
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    const cuuint64_t dims[4] = {(cuuint64_t)Nz, 4, (cuuint64_t)Ny, (cuuint64_t)Nx};
    const cuuint64_t strides[3] = {(cuuint64_t)Nx * Ny * Nz * E, Nz * E, (cuuint64_t)Ny * Nz * E};
    const bool wide = stage_tile_k(Nz) > kTileK2;
    const int px = precision == 0 ? (wide ? StageSmem<double, kTileK>::PX : StageSmem<double, kTileK2>::PX)
                                  : (wide ? StageSmem<float, kTileK>::PX : StageSmem<float, kTileK2>::PX);
    const cuuint32_t box[4] = {(cuuint32_t)px, 4, (cuuint32_t)rows, 1}, estr[4] = {1, 1, 1, 1};
    const CUresult r = reinterpret_cast<Encode>(encode_fn)(
        reinterpret_cast<CUtensorMap *>(out), precision == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
        const_cast<void *>(X), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Measured at 512 x 512 x 128 FP32 (ms per launch): 1.19 / 1.25 / 1.11.  FP64, whole
// steps alone / by three contexts in turn (us), first form against second: 256 x 256 x 128
// 0.69 / 0.86 ms per launch, 64 x 64 x 32 201 / 99 against 178 / 112, 64 x 48 x 50 211 / 135
// against 235 / 157, 100 x 20 x 30 (60,000 cells) equal, 33 x 33 x 16 139 / 54 against 135 / 53,
// 24 x 24 x 24 129 / 48 against 116 / 46 (a block of 512 threads holds a whole
// multiprocessor, however few of them a small grid uses).
int stage_default_form(int precision, long long cells) { return precision == 0 ? (cells < 100000 ? 1 : 0) : 2; }
int stage_tile_count(int precision) { return precision == 0 ? StageForms<double>::count : StageForms<float>::count; }
void stage_tile_shape(int precision, int idx, int *ti, int *tj, int *nt)
{
    if (precision == 0) {
        *ti = StageForms<double>::ti[idx];
        *tj = StageForms<double>::tj[idx];
        if (nt) *nt = StageForms<double>::name[idx];
    } else {
        *ti = StageForms<float>::ti[idx];
        *tj = StageForms<float>::tj[idx];
        if (nt) *nt = StageForms<float>::name[idx];
    }
}

template cudaError_t launch_stage<double>(const StageArgs<double> &, cudaStream_t, cudaEvent_t *);
template cudaError_t launch_stage<float>(const StageArgs<float> &, cudaStream_t, cudaEvent_t *);

}  // namespace wf
