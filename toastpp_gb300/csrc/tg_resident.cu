// tg_resident.cu -- the mixed path's solve as one kernel: each thread-block
// cluster runs a conjugate-gradient process on its own right-hand sides from
// the first residual to the last FP64 correction.
//
// Why.  As separate launches an iteration was one SpMM, 2 x (levels) launches
// of the triangular sweeps, five vector and reduction kernels, and every
// fourth one a host read; each of them took 2 to 10 us whatever its size, so
// solves were bound by launches and level latency (3.2k-node request: 92
// iterations of 70 us; 30k-node request: 290 us an iteration of which about
// 60 were memory time).  Right-hand sides never exchange data, so a cluster
// that owns a few columns needs only its own barrier (a fraction of a
// microsecond), the dot products meet in distributed shared memory, and the
// host is not asked until the solve has ended.
//
// Preconditioner.  A triangular sweep has one dependent step per level (22 in
// 3D with a colour ordering).  In its place stands a factorised sparse
// approximate inverse (Kolotilina and Yeremin 1993): G lower triangular on
// A's own pattern with G A G^T close to 1, row i of G from the small system
// A(S, S) y = e_last over the row's pattern S, scaled to unit diagonal of
// G A G^T.  Applying it is two sparse products without any dependence.  On
// these systems it takes 1.12 to 1.15 times the iterations of IC(0) in the
// colour ordering.  G works for the complex symmetric systems unchanged, with
// the bilinear product throughout.
//
// On-chip state.  A cluster of cs CTAs splits the rows (the mesh's Morton
// layout) into cs contiguous ranges.  Each CTA keeps its rows of p, r and
// t = G r in shared memory, with a copy of the rows of other CTAs that its
// matrix rows refer to (its halo); whoever computes such a row stores it into
// the halos too, through distributed shared memory.  So every gather of the
// three products is a shared-memory read; only matrix values (10 bytes an
// entry with 16-bit local columns) and x stream from L2, and where the matrices
// fit too they are copied in once.  With the vectors in global memory the same
// process was bound by the rate of L1 lookups: 50 us an iteration on the
// 12.5k-node disc with 64 columns, 35 with them on chip, and 22 against 11 on
// the 3.2k-node disc with 32.
//
// Measured, whole requests before and after: 217 nodes, 8 columns 2.88 -> 0.40
// ms; 3.2k nodes CW, 32 columns 8.41 -> 1.06 ms; data gradient on 12.5k nodes
// (two solves of 32 columns) 157 -> 8.6 ms, of which most was columns whose
// residuals the float-float product could not resolve (below).
//
// Precision.  Vectors, the matrices and G are FP32, as in the batched FP32
// processes; sums are compensated FP32 pairs (TwoSum, about 2^-46) of FP32
// products, where those add four rows in FP32 and then in FP64; the recursion's
// scalars and G's rows are formed in pairs.  The solution and its true residual
// are FP64: the product in float-float, a row in FP64 where that is too noisy for
// it, and for CG requests and tolerances below 1e-13 always in FP64.
//
// Thread mapping: a thread per row, with the cluster's LV columns as one word
// of 4 to 16 bytes.  (Sharing a row between lanes, for more columns a cluster,
// was never faster.)
#include "tg_cluster.cuh"
#include "tg_jac.cuh"

namespace tg {

constexpr double RES_GOAL = 0.02;  // of the backward error's bound, where a correction more is due

template <int LV, class V>
struct alignas(LV * sizeof(V)) VecN {
    V v[LV];
};

__device__ __forceinline__ int cl_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}

// all threads of the cluster (cs = 1: of the CTA); writes before it are seen
// by every thread after it
__device__ __forceinline__ void cl_sync(int cs)
{
    if (cs == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
}

// the shared::cluster address of this CTA's shared variable p in CTA `rank`
__device__ __forceinline__ unsigned cl_map(const void* p, int rank)
{
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_store(unsigned a, float2 v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void cl_store(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
template <int B>
__device__ __forceinline__ void cl_store_bytes(unsigned a, const void* v)
{
    const float* f = (const float*)v;
    if constexpr (B == 4) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(f[0]) : "memory");
    else if constexpr (B == 8) cl_store(a, make_float2(f[0], f[1]));
    else asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
}

// a compensated FP32 sum (TwoSum): about 2^-46 relative, without FP64 adds
struct FSum {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float x)
    {
        const float s = __fadd_rn(h, x), b = __fsub_rn(s, h);
        l += __fadd_rn(__fsub_rn(h, __fsub_rn(s, b)), __fsub_rn(x, b));
        h = s;
    }
    // x^2 to about 2^-46
    __device__ __forceinline__ void add_square(double x)
    {
        const float2 f = ff_split(x);
        const float p = __fmul_rn(f.x, f.x);
        l += __fmaf_rn(2.f * f.x, f.y, __fmaf_rn(f.x, f.x, -p));
        add(p);
    }
    __device__ __forceinline__ void add(const FSum& o)
    {
        l += o.l;
        add(o.h);
    }
};

// The recursion's scalars (r.z, alpha, beta): unevaluated sums h + l of two
// floats, about 2^-45 relative.  In FP64, as the batched methods keep them, the
// divisions of one thread stood in every iteration's chain (1.8 us of it: 217
// nodes 0.39 -> 0.47 ms a request); the vectors take alpha and beta as FP32
// either way.
struct Sc {
    float h = 0.f, l = 0.f;
};
struct Scc {
    Sc x, y;
};
template <class V> struct ScOf { using T = Sc; };
template <> struct ScOf<cf> { using T = Scc; };

__device__ __forceinline__ Sc sc_norm(float h, float l)  // |l| <= |h|
{
    const float s = __fadd_rn(h, l);
    return Sc{s, __fsub_rn(l, __fsub_rn(s, h))};
}
__device__ __forceinline__ Sc sc_add(Sc a, Sc b)
{
    const float s = __fadd_rn(a.h, b.h), t = __fsub_rn(s, a.h);
    return sc_norm(s, __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, t)), __fsub_rn(b.h, t)) + (a.l + b.l));
}
__device__ __forceinline__ Sc sc_neg(Sc a) { return Sc{-a.h, -a.l}; }
__device__ __forceinline__ Sc sc_mul(Sc a, Sc b)
{
    const float p = __fmul_rn(a.h, b.h);
    return sc_norm(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p))));
}
// a / b, with f = 1 / b.h: a quotient, and its remainder's
__device__ __forceinline__ Sc sc_div(Sc a, Sc b, float f)
{
    const float q = __fmul_rn(a.h, f);
    return sc_norm(q, __fmaf_rn(-q, b.l, __fmaf_rn(-q, b.h, a.h) + a.l) * f);
}
__device__ __forceinline__ Sc sc_div(Sc a, Sc b) { return sc_div(a, b, 1.f / b.h); }
__device__ __forceinline__ Sc sc_scale(Sc a, float f) { return Sc{a.h * f, a.l * f}; }  // f: a power of two
__device__ __forceinline__ Scc sc_scale(Scc a, float f) { return Scc{sc_scale(a.x, f), sc_scale(a.y, f)}; }
// a conj(b) / |b|^2, with b scaled to between 1 and 2 first
__device__ __forceinline__ Scc sc_div(Scc a, Scc b)
{
    const float m = fmaxf(fabsf(b.x.h), fabsf(b.y.h));
    // 2^-e for m = 2^e (1 ..), e within +-126; zero, infinite and NaN m: 1
    const int e = (int)(__float_as_uint(m) >> 23);
    const float f = e > 0 && e < 254 ? __uint_as_float((unsigned)(254 - e) << 23) : 1.f;
    a = sc_scale(a, f);
    b = sc_scale(b, f);
    const Sc d = sc_add(sc_mul(b.x, b.x), sc_mul(b.y, b.y));
    const float g = 1.f / d.h;
    return Scc{sc_div(sc_add(sc_mul(a.x, b.x), sc_mul(a.y, b.y)), d, g),
               sc_div(sc_add(sc_mul(a.y, b.x), sc_neg(sc_mul(a.x, b.y))), d, g)};
}
__device__ __forceinline__ bool sc_zero(Sc a) { return a.h == 0.f; }
__device__ __forceinline__ bool sc_zero(Scc a) { return a.x.h == 0.f && a.y.h == 0.f; }
__device__ __forceinline__ bool sc_finite(Sc a) { return isfinite(a.h); }
__device__ __forceinline__ bool sc_finite(Scc a) { return isfinite(a.x.h) && isfinite(a.y.h); }
__device__ __forceinline__ float sc_cast(Sc a) { return a.h; }
__device__ __forceinline__ cf sc_cast(Scc a) { return cf{a.x.h, a.y.h}; }

// square root with non-negative real part
__device__ __forceinline__ double ssqrt(double a) { return sqrt(a); }
__device__ __forceinline__ cd ssqrt(cd z) { return csqrt_d(z); }
__device__ __forceinline__ bool sfinite(float a) { return isfinite(a); }
__device__ __forceinline__ bool sfinite(cf a) { return isfinite(a.x) && isfinite(a.y); }

// ---------------------------------------------------------------------------
// An entry of a row's matrix: a real value as Sc, a complex one as (re, im) of
// the high and of the low floats
struct alignas(16) Pc {
    f2x h, l;
};
template <class V> struct PairOf { using T = Sc; };
template <> struct PairOf<cf> { using T = Pc; };
__device__ __forceinline__ Scc p_sc(Pc a)
{
    const float2 h = f2_unpack(a.h), l = f2_unpack(a.l);
    return Scc{sc_norm(h.x, l.x), sc_norm(h.y, l.y)};
}
__device__ __forceinline__ Pc p_sc(Scc a) { return Pc{f2_pack(a.x.h, a.y.h), f2_pack(a.x.l, a.y.l)}; }
// entry e of the float-float matrix (re_hi, re_lo, im_hi, im_lo), times f
__device__ __forceinline__ void p_load(Sc& p, const void* A, int e, float f)
{
    const float2 v = ((const float2*)A)[e];
    p = Sc{v.x * f, v.y * f};
}
__device__ __forceinline__ void p_load(Pc& p, const void* A, int e, float f)
{
    const float4 v = ((const float4*)A)[e];
    p = Pc{f2_pack(v.x * f, v.z * f), f2_pack(v.y * f, v.w * f)};
}
__device__ __forceinline__ void p_set(Sc& p, float x) { p = Sc{x, 0.f}; }
__device__ __forceinline__ void p_set(Pc& p, float x) { p = Pc{f2_pack(x, 0.f), 0ull}; }
__device__ __forceinline__ double p_get(Sc a) { return (double)a.h + (double)a.l; }
__device__ __forceinline__ cd p_get(Pc a)
{
    const float2 h = f2_unpack(a.h), l = f2_unpack(a.l);
    return cd{(double)h.x + (double)l.x, (double)h.y + (double)l.y};
}
__device__ __forceinline__ float p_re(Sc a) { return a.h; }
__device__ __forceinline__ float p_re(Pc a) { return f2_unpack(a.h).x; }
__device__ __forceinline__ bool p_finite(Sc a) { return isfinite(a.h); }
__device__ __forceinline__ bool p_finite(Pc a) { const float2 h = f2_unpack(a.h); return isfinite(h.x) && isfinite(h.y); }
__device__ __forceinline__ Sc p_div(Sc a, Sc b) { return sc_div(a, b); }
__device__ __forceinline__ Pc p_div(Pc a, Pc b) { return p_sc(sc_div(p_sc(a), p_sc(b))); }
// c - a b
__device__ __forceinline__ Sc p_nms(Sc c, Sc a, Sc b) { return sc_add(c, sc_neg(sc_mul(a, b))); }
__device__ __forceinline__ Pc p_nms(Pc c, Pc a, Pc b)
{
    const float2 ah = f2_unpack(a.h), al = f2_unpack(a.l), bh = f2_unpack(b.h), bl = f2_unpack(b.l);
    ff2_mac(c.h, c.l, f2_bcast(-ah.x), f2_bcast(-al.x), b.h, b.l);
    ff2_mac(c.h, c.l, f2_pack(ah.y, -ah.y), f2_pack(al.y, -al.y), f2_pack(bh.y, bh.x), f2_pack(bl.y, bl.x));
    return c;
}
__device__ __forceinline__ Sc p_shfl(Sc a, int r)
{
    return Sc{__shfl_sync(0xffffffffu, a.h, r), __shfl_sync(0xffffffffu, a.l, r)};
}
__device__ __forceinline__ Pc p_shfl(Pc a, int r)
{
    return Pc{__shfl_sync(0xffffffffu, a.h, r), __shfl_sync(0xffffffffu, a.l, r)};
}

// 1 / sqrt(d), Re d > 0, for values that have been scaled to about 1: an FP32
// seed and two Newton steps in FP64
__device__ __forceinline__ double nr_rsqrt(double d)
{
    double x = 1.f / sqrtf((float)d);
    x = x * fma(-0.5 * d * x, x, 1.5);
    return x * fma(-0.5 * d * x, x, 1.5);
}
__device__ __forceinline__ cd nr_rsqrt(cd d)
{
    // sqrt d = (t, Im d / 2t) with t^2 = (|d| + Re d) / 2, its inverse the conjugate over |d|
    const float r = hypotf((float)d.x, (float)d.y), t = sqrtf(0.5f * (r + (float)d.x)), u = 1.f / r;
    cd x{t * u, -((float)d.y / (2.f * t)) * u};
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const cd y = vmul(d, vmul(x, x));
        x = vmul(x, cd{1.5 - 0.5 * y.x, -0.5 * y.y});
    }
    return x;
}

// G of the approximate inverse: GL lanes per row.  The row's pattern S (m
// entries, ascending, the row itself last) is in the slice layout; the lanes
// gather A(S, S) into shared memory, factor it L D L^T in place (lane = row),
// and back-substitute L^T y = e_m; the row is y / sqrt(d_m), from the
// float-float matrix (scaled by a power of four of its diagonal), and cast.  A row whose pivots are not positive, or whose entries are no FP32
// numbers, keeps its scaled diagonal alone.
// Values are pairs of floats: on disc and cylinder matrices the rows differ from
// an FP64 elimination's (which the IC(0) factor is formed by) by at most 4e-14,
// and after the cast in no entry.  FP64 instructions hold a warp's pipe for 16
// clocks, and a row's pivots are a chain: a warp per row in FP64 was 10 % of a
// request on 3D meshes of 2k to 4k nodes.
// Rows of at most 8 entries (2D) go four to a warp and rows of at most 16 two to
// a warp, each size in CTAs of its own.
// ---------------------------------------------------------------------------
template <class V64, class V, int GL, class P>
__device__ __forceinline__ void fsai_rows_of(P (*sm)[GL][GL + 1], int (*ss)[GL], int block, int n,
                                             const int* __restrict__ rowptr, const int* __restrict__ colidx,
                                             const int* __restrict__ diagpos, const void* __restrict__ A,
                                             const int* __restrict__ gptr, const int* __restrict__ gcol,
                                             const int* __restrict__ gcnt, V* __restrict__ gval)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, q = threadIdx.x / GL, gl = lane % GL, g0 = lane - gl;
    if (q >= fsai_rows(GL)) return;
    const int i = block * fsai_rows(GL) + q;
    P(*M)[GL + 1] = sm[q];
    int* S = ss[q];
    int m = i < n ? gcnt[i] : 0;
    if (m > GL || (GL > 8 && m <= GL / 2)) m = 0;  // other CTAs' row
    const int mm = (int)__reduce_max_sync(ALL, (unsigned)m);  // the warp's rows step together
    if (mm == 0) return;
    const int base = m ? gptr[i >> 5] + (i & 31) : 0;
    P dg;
    p_set(dg, 1.f);
    if (m) p_load(dg, A, diagpos[i], 1.f);
    bool ok = m && p_finite(dg) && p_re(dg) > 0.f;  // the same value in a row's lanes, here and below
    const int ex = ok ? ilogbf(p_re(dg)) >> 1 : 0;
    const float sc = ldexpf(1.f, -2 * ex);
    if (gl < m) S[gl] = gcol[base + 32 * gl];
    for (int a = 0; a < m; a++)
        if (gl < m) p_set(M[a][gl], 0.f);
    __syncwarp();
    // each lane its row of A, four entries in flight
    if (gl < m) {
        const int ra = S[gl], p1 = rowptr[ra + 1];
        for (int p = rowptr[ra]; p < p1; p += 4) {
            int c[4];
            P v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                c[u] = p + u < p1 ? colidx[p + u] : ra + 1;
                p_load(v[u], A, min(p + u, p1 - 1), sc);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                int at = -1;
                for (int b = 0; b < mm; b++)
                    if (b <= gl && S[b] == c[u]) at = b;
                if (at >= 0) M[gl][at] = v[u];
            }
        }
    }
    __syncwarp();
    for (int j = 0; j < mm; j++) {
        const P d = M[j < m ? j : 0][j < m ? j : 0];
        ok &= j >= m || (p_finite(d) && p_re(d) > 0.f);
        const bool on = ok && gl > j && gl < m;
        P l = d;
        if (on) {
            l = p_div(M[gl][j], d);
            for (int c = j + 1; c <= gl; c += 4) {
                P v[4], w[4];
#pragma unroll
                for (int u = 0; u < 4; u++) { v[u] = M[gl][min(c + u, gl)]; w[u] = M[min(c + u, gl)][j]; }
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = p_nms(v[u], l, w[u]);
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (c + u <= gl) M[gl][c + u] = v[u];
            }
        }
        __syncwarp();
        if (on) M[gl][j] = l;
        __syncwarp();
    }
    // lane j of the row holds y_j
    P t;
    p_set(t, gl == m - 1 ? 1.f : 0.f);
    for (int r = mm - 1; r > 0; r--) {
        const P tr = p_shfl(t, g0 + r);
        if (ok && r < m && gl < r) t = p_nms(t, M[r][gl], tr);
    }
    V y = vzero<V>();
    if (ok) y = vcast<V, V64>(vscale(vmul(p_get(t), nr_rsqrt(p_get(M[m - 1][m - 1]))), ldexp(1.0, -ex)));
    constexpr unsigned ROW = GL == 32 ? ALL : (1u << (GL & 31)) - 1u;
    ok &= ((__ballot_sync(ALL, gl >= m || sfinite(y)) >> g0) & ROW) == ROW;
    if (m == 0) return;
    if (!ok) y = gl == m - 1 ? vcast<V, V64>(vrecip(ssqrt(p_get(dg)))) : vzero<V>();
    if (gl < m) gval[base + 32 * gl] = y;
    // padding entries of the slice
    const int wd = (gptr[(i >> 5) + 1] - gptr[i >> 5]) >> 5;
    for (int e = m + gl; e < wd; e += GL) gval[base + 32 * e] = vzero<V>();
}

template <class V64, class V>
__global__ void __launch_bounds__(FSAI_NT) fsai_kernel(int n, int n32, int n16, const int* __restrict__ rowptr,
                                                      const int* __restrict__ colidx, const int* __restrict__ diagpos,
                                                      const void* __restrict__ A, const int* __restrict__ gptr,
                                                      const int* __restrict__ gcol, const int* __restrict__ gcnt,
                                                      V* __restrict__ gval)
{
    using P = typename PairOf<V>::T;
    __shared__ union Sm {
        P m8[fsai_rows(8)][8][9], m16[fsai_rows(16)][16][17], m32[fsai_rows(32)][32][33];
        __device__ Sm() {}
    } sm;
    __shared__ int ss[FSAI_NT];
    const int b = blockIdx.x;
    if (b < n32)
        fsai_rows_of<V64, V, 32, P>(sm.m32, (int(*)[32])ss, b, n, rowptr, colidx, diagpos, A, gptr, gcol, gcnt, gval);
    else if (b < n32 + n16)
        fsai_rows_of<V64, V, 16, P>(sm.m16, (int(*)[16])ss, b - n32, n, rowptr, colidx, diagpos, A, gptr, gcol, gcnt, gval);
    else
        fsai_rows_of<V64, V, 8, P>(sm.m8, (int(*)[8])ss, b - n32 - n16, n, rowptr, colidx, diagpos, A, gptr, gcol, gcnt, gval);
}

// ---------------------------------------------------------------------------
// The resident solve.
// ---------------------------------------------------------------------------
// per-column state of the process, in every CTA's shared memory; alpha and beta
// as the vectors' updates take them
template <class V>
struct ResCols {
    V alpha[CL_MAXCG], beta[CL_MAXCG];
    typename ScOf<V>::T zr[CL_MAXCG];
    float bn[CL_MAXCG], err[CL_MAXCG], fs[CL_MAXCG], thr[CL_MAXCG], trig[CL_MAXCG];
    double bnorm[CL_MAXCG], oerr[CL_MAXCG], scale[CL_MAXCG], berr[CL_MAXCG];
    int outer[CL_MAXCG], on[CL_MAXCG], rel[CL_MAXCG], its[CL_MAXCG], st[CL_MAXCG], ost[CL_MAXCG], nupd[CL_MAXCG], met[CL_MAXCG];
    int fail[CL_MAXCG];  // the column ended short of its bounds for another reason than the iteration limit
};

template <class V64, class V, int LV>
__global__ void __launch_bounds__(CL_NT, 1) resident_cg_kernel(ResArgs<V64, V> a)
{
    constexpr bool CPLX = vt<V>::cplx;
    const int NT = blockDim.x, NW = NT >> 5;
    using VN = VecN<LV, V>;
    constexpr int U = 8;   // entries of a matrix row in flight
    constexpr int RX = 2;  // rows in flight of the x update
    __shared__ ResCols<V> S;
    __shared__ __align__(16) float2 s_w[CL_NT / 32][CL_MAXCG * CL_NV];
    __shared__ float2 s_red[2][CL_MAXCS][CL_MAXCG * CL_NV];
    __shared__ double s_nrm[CL_MAXCS][CL_MAXCG * 2];
    extern __shared__ __align__(16) unsigned char cl_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int CG = LV;
    const int cs = a.cs, rank = cs > 1 ? cl_rank() : 0;
    const int grp = blockIdx.x / cs, cg0 = grp * CG;       // this cluster's first column
    const int nc = min(CG, a.k - cg0);                     // columns of the cluster
    const int n = a.n, k = a.k, ns = (n + 31) >> 5;
    const int R0 = (int)((long long)ns * rank / cs) * 32, R1 = min(n, (int)((long long)ns * (rank + 1) / cs) * 32);
    const int rb = R0 + tid, rs = NT;                      // a thread per row
    // gather buffers of p, r and t (q in between), and z of the own rows
    V* bp = reinterpret_cast<V*>(cl_sm);
    V* br = bp + (size_t)a.slots * CG;
    V* bt = br + (size_t)a.slots * CG;
    V* bz = bt + (size_t)a.slots * CG;
    V* x = a.x + (size_t)grp * n * CG;
    // the slice pointers of this CTA's rows, and the matrices where they fit, go
    // to shared memory behind the vectors
    Sell<V> M[3] = {a.A, a.G, a.T};
    {
        const int s0 = R0 >> 5, s1 = (R1 + 31) >> 5;
        V* vp = reinterpret_cast<V*>(cl_sm + a.mofs_val);
        unsigned short* cp = reinterpret_cast<unsigned short*>(cl_sm + a.mofs_col);
        int* pp = reinterpret_cast<int*>(cl_sm + a.mofs_ptr);
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const int b = M[m].ptr[s0], len = M[m].ptr[s1] - b;
            for (int o = tid; o <= s1 - s0; o += NT) pp[o] = M[m].ptr[s0 + o];
            if (a.msm) {
                for (int o = tid; o < len; o += NT) { vp[o] = M[m].val[b + o]; cp[o] = M[m].col[b + o]; }
                M[m].val = vp - b;
                M[m].col = cp - b;
                vp += len;
                cp += len;
            }
            M[m].ptr = pp - s0;
            pp += s1 - s0 + 1;
        }
    }
    int rbuf = 0;
    auto at = [&](V* v, int i) -> VN& { return *reinterpret_cast<VN*>(v + (i - R0) * CG); };
    auto gx = [&](int i) -> VN& { return *reinterpret_cast<VN*>(x + (size_t)i * CG); };
    // this CTA's rows of a gather buffer into the other CTAs' halos, then the
    // cluster's barrier
    uint2* const push = reinterpret_cast<uint2*>(cl_sm + a.mofs_push);
    const int npush = cs > 1 ? a.pofs[rank + 1] - a.pofs[rank] : 0;
    auto share = [&](V* v) {
        if (cs > 1) {
            __syncthreads();
            for (int t = tid; t < npush; t += NT) {
                const uint2 e = push[t];
                const VN y = *reinterpret_cast<const VN*>(v + e.x * CG);
                cl_store_bytes<sizeof(VN)>(cl_map(v + (e.y & 0xffffu) * CG, (int)(e.y >> 16)), &y);
            }
        }
        cl_sync(cs);
    };
    // Sums (mx: the last quantity is a maximum) of nv quantities per column
    // over the cluster, in a fixed order; red(c, i) reads the result.  All
    // writes before it are visible after it.
    auto reduce = [&](FSum (&v)[LV][CL_NV], int nv, bool mx) {
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int j = 0; j < LV; j++)
#pragma unroll
                for (int i = 0; i < CL_NV; i++)
                    if (i < nv) {
                        FSum t;
                        t.h = __shfl_xor_sync(0xffffffffu, v[j][i].h, o);
                        t.l = __shfl_xor_sync(0xffffffffu, v[j][i].l, o);
                        if (mx && i == nv - 1) v[j][i].h = fmaxf(v[j][i].h, t.h);
                        else v[j][i].add(t);
                    }
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < LV; j++)
#pragma unroll
                for (int i = 0; i < CL_NV; i++)
                    if (i < nv) s_w[warp][j * CL_NV + i] = make_float2(v[j][i].h, v[j][i].l);
        __syncthreads();
        for (int t = warp; t < CG * CL_NV; t += NW) {
            const int i = t % CL_NV;
            if (i >= nv) continue;
            FSum s;
            if (lane < NW) { const float2 w = s_w[lane][t]; s.h = w.x; s.l = w.y; }
            for (int o = 16; o; o >>= 1) {
                FSum u;
                u.h = __shfl_xor_sync(0xffffffffu, s.h, o);
                u.l = __shfl_xor_sync(0xffffffffu, s.l, o);
                if (mx && i == nv - 1) s.h = fmaxf(s.h, u.h);
                else s.add(u);
            }
            if (cs == 1) { if (lane == 0) s_red[rbuf][0][t] = make_float2(s.h, s.l); }
            else if (lane < cs) cl_store(cl_map(&s_red[rbuf][rank][t], lane), make_float2(s.h, s.l));
        }
        cl_sync(cs);
        rbuf ^= 1;
    };
    auto red = [&](int c, int i, bool mx) {
        FSum s;
        for (int d = 0; d < cs; d++) {
            const float2 t = s_red[rbuf ^ 1][d][c * CL_NV + i];
            if (mx) s.h = fmaxf(s.h, t.x);
            else { FSum u; u.h = t.x; u.l = t.y; s.add(u); }
        }
        return sc_norm(s.h, s.l);
    };
    // the (bilinear) product of quantities 0 and 1
    auto product = [&](int c) {
        if constexpr (CPLX) return Scc{red(c, 0, false), red(c, 1, false)};
        else return red(c, 0, false);
    };
    for (int t = tid; t < npush; t += NT) push[t] = a.push[a.pofs[rank] + t];
    // every CTA of the cluster runs before any stores into another's shared memory
    cl_sync(cs);
    // ---- start: r = b (zero guess) or the residual in R; norms in FP64
    {
        double v[LV][2];
#pragma unroll
        for (int j = 0; j < LV; j++) v[j][0] = v[j][1] = 0.0;
        for (int i = rb; i < R1; i += rs)
#pragma unroll
            for (int j = 0; j < LV; j++)
                if (j < nc) {
                    const size_t o = (size_t)i * k + cg0 + j;
                    v[j][0] += nrm2(a.B[o]);
                    if (!a.zero_guess) v[j][1] += nrm2(a.R[o]);
                }
        double* w = reinterpret_cast<double*>(s_w);  // [NW][2 CG]
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int j = 0; j < LV; j++)
#pragma unroll
                for (int i = 0; i < 2; i++) v[j][i] += __shfl_xor_sync(0xffffffffu, v[j][i], o);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < LV; j++)
#pragma unroll
                for (int i = 0; i < 2; i++) w[warp * 2 * CG + j * 2 + i] = v[j][i];
        __syncthreads();
        if (tid < 2 * CG) {
            double s = 0.0;
            for (int u = 0; u < NW; u++) s += w[u * 2 * CG + tid];
            if (cs == 1) s_nrm[0][tid] = s;
            else
                for (int d = 0; d < cs; d++) cl_store(cl_map(&s_nrm[rank][tid], d), s);
        }
        cl_sync(cs);
    }
    if (tid < CG) {
        const int c = tid;
        double b2 = 0.0, r2 = 0.0;
        for (int d = 0; d < cs; d++) { b2 += s_nrm[d][2 * c]; r2 += s_nrm[d][2 * c + 1]; }
        const double tol = c < nc ? a.co[cg0 + c].tol : 0.0, bn = sqrt(b2), er = a.zero_guess ? bn : sqrt(r2);
        int on = c < nc && bn > 0.0;
        S.berr[c] = 1.0;
        S.bnorm[c] = bn;
        S.oerr[c] = er;
        // with a componentwise bound only an exact initial guess stops here
        if (on && er <= tol * bn && (a.cwtol <= 0.0 || er == 0.0)) { on = 0; S.berr[c] = 0.0; }
        S.outer[c] = S.on[c] = on;
        S.scale[c] = pow2_floor(er);
        S.bn[c] = S.err[c] = (float)(er / S.scale[c]);
        S.rel[c] = S.its[c] = S.st[c] = S.ost[c] = S.nupd[c] = S.met[c] = S.fail[c] = 0;
        S.trig[c] = a.trig;
        S.alpha[c] = S.beta[c] = vzero<V>();
        S.zr[c] = typename ScOf<V>::T();
    }
    __syncthreads();
    for (int i = rb; i < R1; i += rs) {
        VN rv, zero;
#pragma unroll
        for (int j = 0; j < LV; j++) {
            zero.v[j] = rv.v[j] = vzero<V>();
            if (j < nc && S.outer[j]) {
                const size_t o = (size_t)i * k + cg0 + j;
                rv.v[j] = vcast<V, V64>(vscale(a.zero_guess ? a.B[o] : a.R[o], 1.0 / S.scale[j]));
            }
        }
        at(br, i) = rv;
        gx(i) = zero;
        at(bp, i) = zero;
    }
    share(br);
    // The process as a sequence of products, so that each piece of code stands
    // once (a turn is short enough for instruction fetches to count):
    //   1  t = G r
    //   2  z = G^T t, rho = r.z, then the scalars of the step that left r, the
    //      corrections when they are due, and p = z + beta p
    //   0  q = A p, alpha, then x += alpha p, r -= alpha q
    // mode: what r is, 0 the start, 1 an iteration's, 2 a corrected residual.
    int mode = 0, it = 0, ph = 1;
    bool run = true;
    FSum v[LV][CL_NV];
    for (;;) {
        const V* src = ph == 0 ? bp : ph == 1 ? br : bt;
        V* dst = ph == 2 ? bz : bt;
        const V* dw = ph == 0 ? bp : br;
        const Sell<V> Mx = ph == 0 ? M[0] : ph == 1 ? M[1] : M[2];
        if (run)
            for (int i = rb; i < R1; i += rs) {
                const int b = Mx.ptr[i >> 5], w = (Mx.ptr[(i >> 5) + 1] - b) >> 5;
                const unsigned short* col = Mx.col + b + (i & 31);
                const V* val = Mx.val + b + (i & 31);
                VN acc;
#pragma unroll
                for (int j = 0; j < LV; j++) acc.v[j] = vzero<V>();
#pragma unroll 1
                for (int e = 0; e < w; e += U) {
                    int c[U];
                    V av[U];
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (e + u < w) { c[u] = col[32 * (e + u)]; av[u] = val[32 * (e + u)]; }
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (e + u < w) {
                            const VN g = *reinterpret_cast<const VN*>(src + c[u] * CG);
#pragma unroll
                            for (int j = 0; j < LV; j++) acc.v[j] = vfma(acc.v[j], av[u], g.v[j]);
                        }
                }
                at(dst, i) = acc;
                if (ph != 1) {
                    const VN wv = *reinterpret_cast<const VN*>(dw + (i - R0) * CG);
#pragma unroll
                    for (int j = 0; j < LV; j++) {
                        const V t = vmul(wv.v[j], acc.v[j]);
                        v[j][0].add(re(t));
                        if (CPLX) v[j][1].add(im(t));
                    }
                }
            }
        if (ph == 1) {
            share(bt);
            ph = 2;
            continue;
        }
        reduce(v, 3, false);
        if (ph == 0) {
            if (tid < CG && S.on[tid]) {
                const auto pq = product(tid);
                const auto al = sc_div(S.zr[tid], pq);
                S.alpha[tid] = sc_cast(al);
                if (!sc_finite(al)) { S.on[tid] = 0; S.st[tid] = 2; }
                // a direction of negative curvature: the system is not positive
                // definite, and CG need not converge on it; the caller takes
                // the column elsewhere
                if constexpr (!CPLX)
                    if (pq.h < 0.f) { S.on[tid] = S.outer[tid] = 0; S.ost[tid] = S.fail[tid] = 1; }
            }
            __syncthreads();
            bool on[LV], any = false;
            V sc[LV];
#pragma unroll
            for (int j = 0; j < LV; j++) {
                on[j] = S.on[j]; any |= on[j]; sc[j] = S.alpha[j];
#pragma unroll
                for (int i = 0; i < CL_NV; i++) v[j][i] = FSum();
            }
            if (any)
                for (int i = rb; i < R1; i += RX * rs) {
                    VN xv[RX];
#pragma unroll
                    for (int u = 0; u < RX; u++)
                        if (i + u * rs < R1) xv[u] = gx(i + u * rs);
#pragma unroll
                    for (int u = 0; u < RX; u++) {
                        const int o = i + u * rs;
                        if (o >= R1) continue;
                        VN rv = at(br, o);
                        const VN pv = at(bp, o), qv = at(bt, o);
#pragma unroll
                        for (int j = 0; j < LV; j++)
                            if (on[j]) {
                                xv[u].v[j] = vfma(xv[u].v[j], sc[j], pv.v[j]);
                                rv.v[j] = vfms(rv.v[j], sc[j], qv.v[j]);
                                v[j][2].add(nrm2(rv.v[j]));
                            }
                        gx(o) = xv[u];
                        at(br, o) = rv;
                    }
                }
            share(br);
            mode = 1;
            run = any;
            ph = 1;
            continue;
        }
        if (tid < CG) {
            const int c = tid;
            const auto rz = product(c);
            bool go = S.on[c];
            if (mode == 1 && go) {
                S.err[c] = sqrtf(red(c, 2, false).h);
                S.its[c]++;
                go = false;
                if (S.err[c] <= S.trig[c] * S.bn[c]) { S.on[c] = 0; S.st[c] = 0; }
                else if (S.its[c] >= a.maxit) { S.on[c] = 0; S.st[c] = 1; }
                // a process that grows has lost its directions: it restarts
                else if (!(S.err[c] <= 100.f * S.bn[c])) { S.on[c] = 0; S.st[c] = 2; }
                else go = true;
            }
            if (mode == 2) go = S.rel[c] != 0;
            if (go) {
                const auto be = mode == 0 || S.rel[c] == 2 ? typename ScOf<V>::T() : sc_div(rz, S.zr[c]);
                S.beta[c] = sc_cast(be);
                S.zr[c] = rz;
                S.rel[c] = 0;
                if (sc_zero(rz) || !sc_finite(rz) || !sc_finite(be)) { S.on[c] = 0; S.st[c] = 2; }
            }
        }
        __syncthreads();
        if (mode == 1) {
        it++;
        int nact = 0, nwait = 0;
        for (int c = 0; c < CG; c++) { nact += S.outer[c]; nwait += S.outer[c] && !S.on[c]; }
        const bool limit = it >= a.maxit;
        if (nact == 0) break;
        // corrections: every fourth iteration, or when no column iterates
        if ((nwait && ((it & 3) == 0 || nwait == nact)) || limit) {
        __syncthreads();
        if (tid < CG) {
            const int c = tid;
            // 1: the trigger was reached, the process goes on; 2: it restarts
            S.rel[c] = S.outer[c] ? (S.on[c] ? (limit ? 1 : 0) : (S.st[c] == 0 ? 1 : 2)) : 0;
            // rows whose float-float residual may be off by more than a
            // thousandth of the residual to expect are formed in FP64 (float-float
            // carries about 2^-46 of |A||x|): the recursion's, or where it grew (or
            // is no number) and its correction is dropped, the last one
            const float ex = S.err[c] <= S.bn[c] ? S.err[c] : S.bn[c];
            S.thr[c] = (float)((double)ex * 1e-3 * 70368744177664.0);
        }
        __syncthreads();
        bool rel[LV], anyr = false;
#pragma unroll
        for (int j = 0; j < LV; j++) { rel[j] = S.rel[j]; anyr |= rel[j]; }
        if (anyr)
            for (int i = rb; i < R1; i += rs) {
                VN xv = gx(i);
#pragma unroll
                for (int j = 0; j < LV; j++)
                    if (rel[j]) {
                        const size_t o = (size_t)i * k + cg0 + j;
                        // (the correction of a process that grew is dropped)
                        const V64 s = S.err[j] <= S.bn[j] ? vadd(a.X[o], vscale(vcast<V64, V>(xv.v[j]), S.scale[j])) : a.X[o];
                        a.X[o] = s;
                        const float2 h = ff_split(re(s)), l = ff_split(im(s));
                        if constexpr (CPLX) ((float4*)a.Xff)[o] = make_float4(h.x, h.y, l.x, l.y);
                        else ((float2*)a.Xff)[o] = h;
                        xv.v[j] = vzero<V>();
                    }
                gx(i) = xv;
            }
        cl_sync(cs);
        // the true residual b - A x, its norm and the componentwise backward error
        {
            FSum w[LV][CL_NV];
            if (anyr)
                for (int i = rb; i < R1; i += rs) {
                    const int e0 = a.rowptr[i], e1 = a.rowptr[i + 1];
#pragma unroll
                    for (int j = 0; j < LV; j++) {
                        if (!rel[j]) continue;
                        const int c = cg0 + j;
                        float d = 0.f;
                        V64 ax;
                        f2x h = 0ull, l = 0ull;
                        // (every product in FP64: a CG request's; complex systems only
                        // for tolerances below 1e-13, and then both)
                        if (CPLX || !a.all64) {
#pragma unroll 2
                            for (int e = e0; e < e1; e++) {
                                const size_t o = (size_t)a.colidx[e] * k + c;
                                if constexpr (CPLX) {
                                    const float4 f = ((const float4*)a.Aff)[e], xf = ((const float4*)a.Xff)[o];
                                    ff2_mac(h, l, f2_bcast(f.x), f2_bcast(f.y), f2_pack(xf.x, xf.z),
                                            f2_pack(xf.y, xf.w));
                                    ff2_mac(h, l, f2_pack(-f.z, f.z), f2_pack(-f.w, f.w), f2_pack(xf.z, xf.x),
                                            f2_pack(xf.w, xf.y));
                                    d = fmaf(a.absA[e], fmaxf(fabsf(xf.x), fabsf(xf.z)), d);
                                } else {
                                    const float2 f = ((const float2*)a.Aff)[e], xf = ((const float2*)a.Xff)[o];
                                    ff2_mac(h, l, f2_bcast(f.x), f2_bcast(f.y), f2_bcast(xf.x), f2_bcast(xf.y));
                                    d = fmaf(a.absA[e], fabsf(xf.x), d);
                                }
                            }
                        } else {
                            for (int e = e0; e < e1; e++)
                                d = fmaf(a.absA[e], mag1f(a.X[(size_t)a.colidx[e] * k + c]), d);
                        }
                        const size_t o = (size_t)i * k + c;
                        const V64 b = a.B[o];
                        d += mag1f(b);
                        if (a.all64 || d > S.thr[j] * (float)S.scale[j]) {
                            ax = vzero<V64>();
                            for (int e = e0; e < e1; e++) ax = vfma(ax, a.A64[e], a.X[(size_t)a.colidx[e] * k + c]);
                        } else {
                            const float2 hh = f2_unpack(h), ll = f2_unpack(l);
                            if constexpr (CPLX) ax = V64{oz_to_double(hh.x, ll.x, 0), oz_to_double(hh.y, ll.y, 0)};
                            else ax = oz_to_double(hh.x, ll.x, 0);
                        }
                        const V64 rv = vsub(b, ax);
                        a.R[o] = rv;
                        const float m = mag1f(rv), qd = m == 0.f ? 0.f : (d > 0.f ? m / d : INFINITY);
                        // a NaN must not pass the test
                        w[j][1].h = qd <= w[j][1].h ? w[j][1].h : (qd == qd ? qd : INFINITY);
                        const V64 rs = vscale(rv, 1.0 / S.scale[j]);
                        w[j][0].add_square(re(rs));
                        if constexpr (CPLX) w[j][0].add_square(im(rs));
                    }
                }
            reduce(w, 2, true);
        }
        if (tid < CG && S.rel[tid]) {
            const int c = tid;
            const Sc r2 = red(c, 0, false);
            const double er = sqrt((double)r2.h + (double)r2.l) * S.scale[c], tol = a.co[cg0 + c].tol;
            S.oerr[c] = er;
            if (a.cwtol > 0.0) S.berr[c] = red(c, 1, true).h;
            // A column that meets its bounds without much to spare takes one
            // correction more, of no more than what is missing: the bound alone
            // left the data gradient, which sums small differences of the data,
            // up to 1.1e-9 from the exact one, a tenth of it 3e-10, a fiftieth
            // 1e-10, for 4 and 5 % of its time.  (Most columns have it from a
            // replacement of 1e-4.)
            const bool ok = er <= tol * S.bnorm[c] && (a.cwtol <= 0.0 || S.berr[c] <= a.cwtol);
            const bool spare = a.cwtol <= 0.0 || S.berr[c] <= RES_GOAL * a.cwtol;
            S.trig[c] = a.trig;
            if (ok && !spare)
                S.trig[c] = fmaxf(a.trig, 0.1f * (float)(RES_GOAL * a.cwtol / S.berr[c]));
            if (ok && (spare || limit || S.met[c]++ || S.nupd[c] + 1 >= a.max_upd)) {
                S.outer[c] = S.on[c] = S.rel[c] = 0;
                S.ost[c] = 0;
            } else if (limit || ++S.nupd[c] >= a.max_upd || !isfinite(er)) {
                S.outer[c] = S.on[c] = S.rel[c] = 0;
                S.ost[c] = 1;
                S.fail[c] = !limit || !isfinite(er);
            } else {
                // a true residual above the recursive one: the process no longer
                // follows the FP64 system and restarts from it.  (Off the rounding
                // floor the two agree to 1e-3; with the line at 8 a column at 7.4
                // kept its old directions and diverged on the 919-node disc.)
                if (er > 1.25 * S.err[c] * S.scale[c]) S.rel[c] = 2;
                const double old = S.scale[c];
                S.scale[c] = pow2_floor(er);
                const float f = (float)(old / S.scale[c]);
                S.fs[c] = f;
                S.bn[c] = (float)(er / S.scale[c]);
                S.zr[c] = sc_scale(S.zr[c], f * f);
                S.on[c] = 1;
                S.st[c] = 0;
            }
        }
        __syncthreads();
        if (limit) break;
        anyr = false;
#pragma unroll
        for (int j = 0; j < LV; j++) { rel[j] = S.rel[j]; anyr |= rel[j]; }
        int nrel = 0;
        for (int c = 0; c < CG; c++) nrel += S.rel[c] != 0;
        if (nrel) {
            // the columns go on from the true residual: r and p in the new scale
            if (anyr)
                for (int i = rb; i < R1; i += rs) {
                    VN rv = at(br, i), pv = at(bp, i);
#pragma unroll
                    for (int j = 0; j < LV; j++)
                        if (rel[j]) {
                            const int c = j;
                            rv.v[j] = vcast<V, V64>(vscale(a.R[(size_t)i * k + cg0 + c], 1.0 / S.scale[c]));
                            pv.v[j] = S.rel[c] == 2 ? vzero<V>() : vscale(pv.v[j], S.fs[c]);
                        }
                    at(br, i) = rv;
                    at(bp, i) = pv;
                }
            share(br);
            mode = 2;
            run = anyr;
            ph = 1;
#pragma unroll
            for (int j = 0; j < LV; j++)
#pragma unroll
                for (int i = 0; i < CL_NV; i++) v[j][i] = FSum();
            continue;
        }
        }
        }
        bool on[LV], any = false;
        V sc[LV];
#pragma unroll
        for (int j = 0; j < LV; j++) {
            on[j] = S.on[j]; any |= on[j]; sc[j] = S.beta[j];
#pragma unroll
            for (int i = 0; i < CL_NV; i++) v[j][i] = FSum();
        }
        if (any)
            for (int i = rb; i < R1; i += rs) {
                VN pv = at(bp, i);
                const VN zv = at(bz, i);
#pragma unroll
                for (int j = 0; j < LV; j++)
                    if (on[j]) pv.v[j] = vfma(zv.v[j], sc[j], pv.v[j]);
                at(bp, i) = pv;
            }
        share(bp);
        run = any;
        ph = 0;
    }
    // results; no CTA leaves while another may still write its shared memory
    __syncthreads();
    if (rank == 0 && tid < nc) {
        ColState& O = a.co[cg0 + tid];
        O.bnorm = S.bnorm[tid];
        O.err = S.oerr[tid];
        O.berr = S.berr[tid];
        O.its = (S.its[tid] + a.per - 1) / a.per;
        O.status = S.outer[tid] ? 1 : S.ost[tid];
        O.rel = S.fail[tid];
        O.active = 0;
    }
    cl_sync(cs);
}

// ---------------------------------------------------------------------------
// The IC(0) apply of the batched methods (FP64 path, natural ordering) as one
// launch.  A level per launch took 6 us, of which less than two were work: 190
// us an apply for 32 complex FP64 columns of the 12.5k-node disc (32 levels),
// 105 as clusters (560 -> 270 us on a 19.6k-node cylinder, 142 -> 57 for 8
// columns of a 1.3k-node disc).  y stays in shared memory with the halo rows of
// the CTA's matrix rows; at the end of a level its rows go to the other CTAs'
// halos and the cluster's barrier follows.  What the next level needs and no
// level writes (its rows, columns, factor entries, right-hand sides, pivots)
// loads before that barrier, so that after it a row is shared-memory reads and
// its sum.  (Loading it a whole level ahead, in a second register set, was
// slower: the barriers and each row's serial FP64 sum bound a level, not these
// loads; the FP64 pipe is a quarter busy.)  The rows of a level lie
// by their number of entries, so that a warp's rows end together.  Every row's
// sum runs in the same order as in the level kernels: the results are the same
// to the bit.
// ---------------------------------------------------------------------------
template <class V, int LV>
__global__ void __launch_bounds__(IC_NT) ic_cluster_kernel(IcClArgs<V> a)
{
    using VN = VecN<LV, V>;
    constexpr int WP = 8;  // entries of a row in flight
    extern __shared__ __align__(16) unsigned char cl_sm[];
    V* y = reinterpret_cast<V*>(cl_sm);  // [slots][LV]
    const int tid = threadIdx.x, cs = a.cs, rank = cs > 1 ? cl_rank() : 0;
    const int c0 = blockIdx.x / cs * LV, ns = (a.n + 31) >> 5, R0 = (int)((long long)ns * rank / cs) * 32;
    const size_t ld = a.k;
    bool on[LV], live = false;
#pragma unroll
    for (int j = 0; j < LV; j++) {
        on[j] = c0 + j < a.k && (!a.st || a.st[c0 + j].active == 1);
        live |= on[j];
    }
    if (!live) return;  // the same in every CTA of the cluster
    // the levels, their halo copies and the rows of both sweeps
    const int total = a.f.nlev + a.b.nlev;
    int4* lev = reinterpret_cast<int4*>(cl_sm + a.mofs);
    int2* pl = reinterpret_cast<int2*>(lev + total);
    unsigned short* rows = reinterpret_cast<unsigned short*>(pl + total);
    {
        const int4* lf = a.f.lev + rank * a.f.nlev;
        const int4* lb = a.b.lev + rank * a.b.nlev;
        const int f0 = lf[0].x, b0 = lb[0].x, own = lf[a.f.nlev - 1].x + lf[a.f.nlev - 1].y - f0;
        for (int t = tid; t < total; t += IC_NT) {
            const bool fwd = t < a.f.nlev;
            int4 L = fwd ? lf[t] : lb[t - a.f.nlev];
            L.x += fwd ? -f0 : own - b0;  // place in rows
            lev[t] = L;
            pl[t] = fwd ? a.f.pl[rank * a.f.nlev + t] : a.b.pl[rank * a.b.nlev + t - a.f.nlev];
        }
        for (int t = tid; t < own; t += IC_NT) { rows[t] = a.f.rows[f0 + t]; rows[own + t] = a.b.rows[b0 + t]; }
    }
    cl_sync(cs);        // every CTA runs before any stores into another's shared memory
    const V* in = a.in + (size_t)R0 * ld + c0;
    V* out = a.out + (size_t)R0 * ld + c0;
    const V* dinv = a.dinv + R0;
    int slot = 0, c[WP];
    V v[WP], di = vzero<V>();
    VN rhs;
    uint2 pe = make_uint2(0u, 0u);
    // row s of level L: its first entries, pivot and, forward, right-hand side
    auto fetch = [&](const IcSweepDev& w, const V* val, const int4& L, int s, bool fwd) {
        slot = rows[L.x + s];
#pragma unroll
        for (int u = 0; u < WP; u++)
            if (u < L.z) { c[u] = w.col[L.w + u * L.y + s]; v[u] = val[L.w + u * L.y + s]; }
        di = dinv[slot];
        if (fwd)
#pragma unroll
            for (int j = 0; j < LV; j++) rhs.v[j] = on[j] ? in[(size_t)slot * ld + j] : vzero<V>();
    };
    int4 L = lev[0];
    int2 P = pl[0];
    if (tid < L.y) fetch(a.f, a.vf, L, tid, true);
    if (tid < P.y) pe = a.f.push[P.x + tid];
    for (int l = 0; l < total; l++) {
        const bool fwd = l < a.f.nlev;
        const IcSweepDev& w = fwd ? a.f : a.b;
        const V* val = fwd ? a.vf : a.vb;
        for (int s = tid; s < L.y; s += IC_NT) {
            if (s != tid) fetch(w, val, L, s, fwd);
            VN acc = fwd ? rhs : *reinterpret_cast<const VN*>(y + slot * LV);
            for (int e = 0;;) {
#pragma unroll
                for (int u = 0; u < WP; u++)
                    if (e + u < L.z && c[u] != 0xffff) {
                        const VN g = *reinterpret_cast<const VN*>(y + c[u] * LV);
#pragma unroll
                        for (int j = 0; j < LV; j++) acc.v[j] = vfms(acc.v[j], v[u], g.v[j]);
                    }
                e += WP;
                if (e >= L.z) break;
#pragma unroll
                for (int u = 0; u < WP; u++)
                    if (e + u < L.z) { c[u] = w.col[L.w + (e + u) * L.y + s]; v[u] = val[L.w + (e + u) * L.y + s]; }
            }
#pragma unroll
            for (int j = 0; j < LV; j++) acc.v[j] = vmul(acc.v[j], di);
            *reinterpret_cast<VN*>(y + slot * LV) = acc;
            if (!fwd)
#pragma unroll
                for (int j = 0; j < LV; j++)
                    if (on[j]) out[(size_t)slot * ld + j] = acc.v[j];
        }
        if (l + 1 == total) break;
        if (cs > 1) {
            __syncthreads();
            for (int t = tid; t < P.y; t += IC_NT) {
                if (t != tid) pe = w.push[P.x + t];
                const VN x = *reinterpret_cast<const VN*>(y + pe.x * LV);
                cl_store_bytes<sizeof(VN)>(cl_map(y + (pe.y & 0xffffu) * LV, (int)(pe.y >> 16)), &x);
            }
        }
        const bool nf = l + 1 < a.f.nlev;
        const IcSweepDev& nw = nf ? a.f : a.b;
        L = lev[l + 1];
        P = pl[l + 1];
        if (tid < L.y) fetch(nw, nf ? a.vf : a.vb, L, tid, nf);
        if (tid < P.y) pe = nw.push[P.x + tid];
        cl_sync(cs);
    }
    cl_sync(cs);  // no CTA leaves while another may still write its shared memory
}

template <class V>
void (*ic_cluster_kernel_of(int lv))(IcClArgs<V>)
{
    if constexpr (sizeof(V) == 4)
        if (lv == 4) return ic_cluster_kernel<V, 4>;
    if constexpr (sizeof(V) <= 8)
        if (lv == 2) return ic_cluster_kernel<V, 2>;
    return ic_cluster_kernel<V, 1>;
}
template void (*ic_cluster_kernel_of<double>(int))(IcClArgs<double>);
template void (*ic_cluster_kernel_of<float>(int))(IcClArgs<float>);
template void (*ic_cluster_kernel_of<cd>(int))(IcClArgs<cd>);
template void (*ic_cluster_kernel_of<cf>(int))(IcClArgs<cf>);

template <class V64, class V32>
void (*resident_kernel(int lv))(ResArgs<V64, V32>)
{
    if constexpr (sizeof(V32) == 4)
        if (lv == 4) return resident_cg_kernel<V64, V32, 4>;
    return lv == 2 ? resident_cg_kernel<V64, V32, 2> : resident_cg_kernel<V64, V32, 1>;
}
template void (*resident_kernel<double, float>(int))(ResArgs<double, float>);
template void (*resident_kernel<cd, cf>(int))(ResArgs<cd, cf>);

template <class V64, class V>
void (*fsai_kernel_of())(int, int, int, const int*, const int*, const int*, const void*, const int*, const int*, const int*,
                         V*)
{
    return fsai_kernel<V64, V>;
}
template void (*fsai_kernel_of<double, float>())(int, int, int, const int*, const int*, const int*, const void*,
                                                 const int*, const int*, const int*, float*);
template void (*fsai_kernel_of<cd, cf>())(int, int, int, const int*, const int*, const int*, const void*, const int*,
                                          const int*, const int*, cf*);

}  // namespace tg
