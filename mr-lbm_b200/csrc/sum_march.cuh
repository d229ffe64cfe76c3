// sum_march.cuh -- the z-march of the D3Q27 sets without wall nodes, in sums
// instead of populations.
//
// On D3Q27 the weights are a product over the axes, w = w1(c_x) w1(c_y) w1(c_z)
// with w1 = (1, 4, 1) / 6, and the reconstructed population is a polynomial
// of order 2 in the c's times rho w.  So the streamed sums
//   M_abc(x) = sum_i c_ix^a c_iy^b c_iz^c f_i(x - c_i)
// factor into three passes of one-dimensional sums over c_y, c_z and c_x, and
// no population is ever formed: 18 values a node after the first pass, 18
// after the second, the 10 moments after the third.
//   y: the rows y - 1, y, y + 1 are read from the TMA stage (no row exchange);
//   z: in registers, a plane's c_z = +1 and 0 lines held until they are summed;
//   x: warp shuffles; the values that enter a 32-wide column from its two
//      sides come from one helper warp (lane = row and side) through a small
//      double-buffered edge buffer, the only exchange between warps.
// The sums carry the deviation from rho0 at rest (coefficient rho pics2 - rho0
// in place of rho pics2, whose sums are known): the second moments lose no
// digits to the 1/3 that the sums of whole populations cancel against.
//
// Measured (256^3 FP32, one step among others): 277 us against 322 for the 27
// populations (one row a lane, packed shared-memory row exchange); 252 thread
// instructions a node against 379; DRAM traffic 1.076 times the algorithmic
// bytes; 512^3 FP16 1,820 us against 2,117.  What bounds it: 5.0 TB/s of the
// 6.5 TB/s copy rate, with 13 warps an SM at 45 % issue.  Which domains run it:
// sums_domain.  R = 1 (one row a
// lane, 27 warps) took 313 us: 339 instructions, and the many columns in
// flight re-read their halos from DRAM (1.21 times).
//
// A thread holds R = 2 rows (R = 1 in batches): the z and x passes and the
// collision run on both at once as packed FP32 pairs (the two rows' values
// side by side from the first pass on, so packing costs no moves), the shared
// rows of the y pass are read once, and the addresses, waits and barriers of
// a step are paid once for two nodes.
#pragma once

namespace mrlbm {

constexpr int SUM_ROWS = 2;    // rows of a thread in the single-domain step
constexpr int SUM_CTAS = 3;    // its CTAs resident per SM
constexpr int SUM_EDGE = 8;    // floats of an edge slot and row (6 used)

// Shared memory: barriers, TMA ring, edge buffer [parity][side][row][SUM_EDGE]
template <typename T, int TYI, int NPM>
struct SumSmem {
    static constexpr int NR = TYI + 2;
    static constexpr size_t stage_max = ((size_t)NR * NPM * 2 * box_x<T>() * sizeof(T) + 127) / 128 * 128;
    static constexpr size_t edge_bytes = (size_t)2 * 2 * TYI * SUM_EDGE * sizeof(float);
    static constexpr size_t fixed = 128 + edge_bytes;
    static constexpr size_t budget = smem_share(SUM_CTAS);
    static constexpr int NS = fixed + NSTAGE_MAX * stage_max <= budget ? NSTAGE_MAX : NSTAGE_MAX - 1;
    static constexpr size_t bytes = fixed + NS * stage_max;
    static_assert(bytes <= budget, "shared memory over the CTA's share");
    static constexpr int CT = 0;
    uint64_t* bars;
    unsigned char* stages;
    float* edge;
    __device__ __forceinline__ explicit SumSmem(unsigned char* smem)
        : bars(reinterpret_cast<uint64_t*>(smem)), stages(smem + 128),
          edge(reinterpret_cast<float*>(smem + 128 + NS * stage_max))
    {
    }
    __device__ __forceinline__ float* sum_edge() const { return edge; }
};

// ------------------------------------------------ one row or two, the same ops

// two rows' values as one 64-bit register pair
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2_pack(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float row_of(float v, int) { return v; }
__device__ __forceinline__ float row_of(F2 v, int r)
{
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v.v));
    return r ? b : a;
}
__device__ __forceinline__ float p_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float p_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float p_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float p_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ F2 p_add(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 p_sub(F2 a, F2 b)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 p_mul(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 p_fma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// the value of both rows / of each
template <typename P>
__device__ __forceinline__ P p_all(float v);
template <>
__device__ __forceinline__ float p_all<float>(float v) { return v; }
template <>
__device__ __forceinline__ F2 p_all<F2>(float v) { return f2_pack(v, v); }
__device__ __forceinline__ void p_rows(float& p, const float (&v)[1]) { p = v[0]; }
__device__ __forceinline__ void p_rows(F2& p, const float (&v)[2]) { p = f2_pack(v[0], v[1]); }

// A node's words of a TMA stage, 16-bit ones in their storage scaling (the
// scales are folded into the products below); split storage adds the low
// words of 3u to the high ones.
template <typename T, int NM, int NML>
__device__ __forceinline__ void raw_moments(const T* sp, float* mc)
{
#pragma unroll
    for (int p = 0; p < (NM + 1) / 2; p++) {
        const T* q = sp + p * 2 * box_x<T>();
        const float2 v = MRLBM_SMEM_OK(q, 2 * (int)sizeof(T), BCK_STAGE) ? Stor2<T>::lds(q) : make_float2(0.f, 0.f);
        mc[2 * p] = v.x;
        if (2 * p + 1 < NM) mc[2 * p + 1] = v.y;
    }
    if constexpr (NML < NM) {
#pragma unroll
        for (int c = 0; c < 3; c++) mc[1 + c] = fmaf(mc[NML + c], 1.0f / F16_SCALE_LOW, mc[1 + c]);
    }
}

// u (stored scaling) in the unit of the second moments, plus b
template <typename T>
__device__ __forceinline__ float u_plus(float u, float b)
{
    if constexpr (scaled_storage<T>()) return fmaf(u, F16_SCALE_PI / F16_SCALE_U, b);
    else return u + b;
}
template <typename T>
__device__ __forceinline__ float u_minus(float u, float b)   // u - b
{
    if constexpr (scaled_storage<T>()) return fmaf(u, F16_SCALE_PI / F16_SCALE_U, -b);
    else return u - b;
}
template <typename T>
__device__ __forceinline__ float minus_u(float b, float u)   // b - u
{
    if constexpr (scaled_storage<T>()) return fmaf(u, -F16_SCALE_PI / F16_SCALE_U, b);
    else return b - u;
}

// rho in the unit that the products take (rho over the second moments'
// storage scale) and rho - rho0
template <typename T>
__device__ __forceinline__ float rho_unit(float m0, float rho0, float& dev)
{
    if constexpr (scaled_storage<T>()) {
        dev = m0 * (1.0f / F16_SCALE_RHO);
        return fmaf(m0, 1.0f / F16_SCALE_RHO, rho0) * (1.0f / F16_SCALE_PI);
    } else {
        dev = m0;
        return rho0 + m0;
    }
}

// The y pass: V[k][b], b = 0, 1, 2 the order in c_y, of the six coefficients
// k = (a, c), the orders in c_x and c_z: (0,0) (1,0) (0,1) (2,0) (1,1) (0,2),
// for R rows.  sp: the node's words in the stage row below the first; ROW:
// elements of a stage row.  Weights are 6 w1.  Each product that feeds a sum
// is fused by hand, so a node has the same bits for every R and in the helper.
struct YRow {       // a row's words as the pass needs them
    float rs, m0, tr, e, u[3], xx, xy, xz, yz, zz;
};
template <typename T, int NM, int NML>
__device__ __forceinline__ void y_row(const T* sp, float rho0, YRow& w)
{
    float m[NM];
    raw_moments<T, NM, NML>(sp, m);
    w.rs = rho_unit<T>(m[0], rho0, w.m0);
    w.tr = (m[4] + m[7]) + m[9];
    w.e = fmaf(w.tr, -1.0f / 3.0f, m[7]);
    w.u[0] = m[1]; w.u[1] = m[2]; w.u[2] = m[3];
    w.xx = m[4]; w.xy = m[5]; w.xz = m[6]; w.yz = m[8]; w.zz = m[9];
}
// c_y = +1 lines of the row below
template <typename T>
__device__ __forceinline__ void y_below(const YRow& w, float (&p)[6])
{
    p[0] = fmaf(w.rs, u_plus<T>(w.u[1], w.e), w.m0);
    p[1] = __fmul_rn(w.rs, u_plus<T>(w.u[0], w.xy));
    p[2] = __fmul_rn(w.rs, u_plus<T>(w.u[2], w.yz));
    p[3] = __fmul_rn(w.rs, w.xx);
    p[4] = __fmul_rn(w.rs, w.xz);
    p[5] = __fmul_rn(w.rs, w.zz);
}
// the sums, from the row below's lines p, the row itself (c_y = 0, weight 4)
// and the row above (c_y = -1)
template <typename T>
__device__ __forceinline__ void y_sums(const float (&p)[6], const YRow& o, const YRow& w, float (&V)[6][3])
{
    const float q0 = fmaf(w.rs, minus_u<T>(w.e, w.u[1]), w.m0);
    V[0][2] = p[0] + q0;
    V[0][1] = p[0] - q0;
    const float f[5] = {u_minus<T>(w.u[0], w.xy), u_minus<T>(w.u[2], w.yz), w.xx, w.xz, w.zz};
#pragma unroll
    for (int k = 1; k < 6; k++) {
        V[k][2] = fmaf(w.rs, f[k - 1], p[k]);
        V[k][1] = fmaf(-w.rs, f[k - 1], p[k]);
    }
    const float r4 = 4.0f * o.rs;
    const float ru = scaled_storage<T>() ? r4 * (F16_SCALE_PI / F16_SCALE_U) : r4;
    V[0][0] = fmaf(4.0f, o.m0, fmaf(r4, o.tr * (-1.0f / 3.0f), V[0][2]));
    V[1][0] = fmaf(ru, o.u[0], V[1][2]);
    V[2][0] = fmaf(ru, o.u[2], V[2][2]);
    V[3][0] = fmaf(r4, o.xx, V[3][2]);
    V[4][0] = fmaf(r4, o.xz, V[4][2]);
    V[5][0] = fmaf(r4, o.zz, V[5][2]);
}
template <typename T, int NM, int NML, int R, typename P>
__device__ __forceinline__ void y_pass(const T* sp, int row, float rho0, P (&V)[6][3])
{
    float v[R][6][3];
    YRow a, b;
    float p[6];
    y_row<T, NM, NML>(sp, rho0, a);
    y_below<T>(a, p);
    y_row<T, NM, NML>(sp + row, rho0, a);
#pragma unroll
    for (int r = 0; r < R; r++) {
        y_row<T, NM, NML>(sp + (r + 2) * row, rho0, b);
        y_sums<T>(p, a, b, v[r]);
        if (r + 1 < R) {
            y_below<T>(a, p);
            a = b;
        }
    }
#pragma unroll
    for (int k = 0; k < 6; k++)
#pragma unroll
        for (int o = 0; o < 3; o++) {
            float w[R];
#pragma unroll
            for (int r = 0; r < R; r++) w[r] = v[r][k][o];
            p_rows(V[k][o], w);
        }
}

// z lines of a plane: line l = a + 3 b; up: c_z = +1, dn: c_z = -1, and the
// c_z = 0 lines of a = 0, 1 (a = 2 has none of its own: it equals up)
template <typename P>
struct ZLines {
    P up[9], dn[9], md[6];
};
template <typename P>
__device__ __forceinline__ void z_lines(const P (&V)[6][3], ZLines<P>& L)
{
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const P h = p_add(V[0][b], V[5][b]);
        L.up[3 * b] = p_add(h, V[2][b]);
        L.dn[3 * b] = p_sub(h, V[2][b]);
        L.md[2 * b] = V[0][b];
        L.up[3 * b + 1] = p_add(V[1][b], V[4][b]);
        L.dn[3 * b + 1] = p_sub(V[1][b], V[4][b]);
        L.md[2 * b + 1] = V[1][b];
        L.up[3 * b + 2] = L.dn[3 * b + 2] = V[3][b];
    }
}

// The z pass: x lines of the output plane, U[i][a] of the six orders
// i = (b, c): (0,0) (1,0) (2,0) (0,1) (1,1) (0,2).  up0: the plane below's
// c_z = +1 lines, md / up1: the output plane's c_z = 0 lines, dn: the plane
// above's c_z = -1 lines.
template <typename P>
__device__ __forceinline__ void z_sum(const P (&up0)[9], const P (&up1)[9], const P (&md)[6], const P (&dn)[9],
                                      P (&U)[6][3])
{
    const P four = p_all<P>(4.0f);
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const P s = p_add(up0[3 * b + x], dn[3 * b + x]);
            U[b][x] = p_fma(four, x < 2 ? md[2 * b + x] : up1[3 * b + 2], s);         // c order 0
            if (b < 2) U[3 + b][x] = p_sub(up0[3 * b + x], dn[3 * b + x]);           // c order 1
            if (b < 1) U[5][x] = s;                                                    // c order 2
        }
}

// the values of an edge slot into q where on is set (no select per value)
__device__ __forceinline__ void edge_into(float (&q)[6], const float* e, bool on)
{
#ifdef MRLBM_BOUNDS_CHECK
    on = on && MRLBM_SMEM_OK(e, 24, BCK_EDGE);
#endif
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.s32 p, %7, 0;\n\t"
        "@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%6];\n\t"
        "@p ld.shared.v2.f32 {%4, %5}, [%6 + 16];\n\t}"
        : "+f"(q[0]), "+f"(q[1]), "+f"(q[2]), "+f"(q[3]), "+f"(q[4]), "+f"(q[5])
        : "r"((unsigned)__cvta_generic_to_shared(e)), "r"((int)on)
        : "memory");
}
__device__ __forceinline__ void edge_into(F2 (&q)[6], const float* e, bool on)
{
#ifdef MRLBM_BOUNDS_CHECK
    on = on && MRLBM_SMEM_OK(e, 48, BCK_EDGE);
#endif
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.s32 p, %7, 0;\n\t"
        "@p ld.shared.v2.b64 {%0, %1}, [%6];\n\t"
        "@p ld.shared.v2.b64 {%2, %3}, [%6 + 16];\n\t"
        "@p ld.shared.v2.b64 {%4, %5}, [%6 + 32];\n\t}"
        : "+l"(q[0].v), "+l"(q[1].v), "+l"(q[2].v), "+l"(q[3].v), "+l"(q[4].v), "+l"(q[5].v)
        : "r"((unsigned)__cvta_generic_to_shared(e)), "r"((int)on)
        : "memory");
}

__device__ __forceinline__ float from_left(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float from_right(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ F2 from_left(F2 v) { return f2_pack(from_left(row_of(v, 0)), from_left(row_of(v, 1))); }
__device__ __forceinline__ F2 from_right(F2 v) { return f2_pack(from_right(row_of(v, 0)), from_right(row_of(v, 1))); }
__device__ __forceinline__ float p_inv(float v) { return 1.0f / v; }
__device__ __forceinline__ F2 p_inv(F2 v) { return f2_pack(1.0f / row_of(v, 0), 1.0f / row_of(v, 1)); }

// The x pass and the collision: arriving x lines fl (from x - 1), fr (from
// x + 1), the node's own c_x = 0 lines U0; o: the stored moments 0 .. 9.
// The sums carry 6^3 = 216 times the moments.  Stored scaling: 3u = 3 j / rho,
// 9 Pi_ij = 9 P_ij / rho, 4.5 Pi_ii = (4.5 P_ii - 1.5 (rho - rho0)) / rho with
// P_ii the deviation from rho0 / 3; all from the quotient 1 / (72 rho) and its
// rounded multiples by 3 and 72, so a velocity meets the roundings of one
// quotient, which vary with the density, and the density deviation that of
// 1 / 216.  Drift of the sums over 20,000 steps of 32^3 boxes, here / with the
// 27 populations: mean density deviation 1.2e-5 / 1.6e-3 of itself (noise),
// 1.2e-4 / 1.1e-2 (waves), momentum 2.5e-5 / 1.4e-5 (shear), 4e-6 / 4.8e-5.
// The collision is collide_scaled's.
template <int FLAGS, typename P>
__device__ __forceinline__ void x_collide(const StepArgs& a, const P (&fl)[6], const P (&fr)[6], const P (&U0)[6],
                                          P (&o)[10])
{
    const P four = p_all<P>(4.0f);
    const P s0 = p_add(fl[0], fr[0]);
    const P M0 = p_fma(four, U0[0], s0);
    const P r = p_mul(M0, p_all<P>(1.0f / 216.0f));   // rho - rho0
    const P rho = p_add(p_all<P>(a.rho0), r);
    const P i3 = p_inv(p_mul(p_all<P>(72.0f), rho)), i9 = p_mul(p_all<P>(3.0f), i3);
    const P t = p_mul(p_all<P>(-0.5f), M0), c15 = p_all<P>(1.5f);
    P ux = p_mul(p_sub(fl[0], fr[0]), i3);
    P uy = p_mul(p_fma(four, U0[1], p_add(fl[1], fr[1])), i3);
    P uz = p_mul(p_fma(four, U0[3], p_add(fl[3], fr[3])), i3);
    P xx = p_mul(p_fma(c15, s0, t), i3);
    P yy = p_mul(p_fma(c15, p_fma(four, U0[2], p_add(fl[2], fr[2])), t), i3);
    P zz = p_mul(p_fma(c15, p_fma(four, U0[5], p_add(fl[5], fr[5])), t), i3);
    P xy = p_mul(p_sub(fl[1], fr[1]), i9);
    P xz = p_mul(p_sub(fl[3], fr[3]), i9);
    P yz = p_mul(p_fma(four, U0[4], p_add(fl[4], fr[4])), i9);
    const P t_om = p_all<P>(1.0f - a.omega0), om = p_all<P>(a.omega0), om_d2 = p_all<P>(0.5f * a.omega0);
    if constexpr ((FLAGS & F_FORCE) != 0) {
        const P ir = p_mul(p_all<P>(72.0f), i3), ir3 = p_mul(p_all<P>(3.0f), ir);
        ux = p_fma(ir3, p_all<P>(a.fx), ux);
        uy = p_fma(ir3, p_all<P>(a.fy), uy);
        uz = p_fma(ir3, p_all<P>(a.fz), uz);
    }
    const P ox = p_mul(om, ux), oy = p_mul(om, uy), hx = p_mul(om_d2, ux), hy = p_mul(om_d2, uy),
            hz = p_mul(om_d2, uz);
    xx = p_fma(t_om, xx, p_mul(hx, ux));
    yy = p_fma(t_om, yy, p_mul(hy, uy));
    zz = p_fma(t_om, zz, p_mul(hz, uz));
    xy = p_fma(t_om, xy, p_mul(ox, uy));
    xz = p_fma(t_om, xz, p_mul(ox, uz));
    yz = p_fma(t_om, yz, p_mul(oy, uz));
    if constexpr ((FLAGS & F_FORCE) != 0) {
        const float tt = 1.0f - 0.5f * a.omega0;
        const P ir = p_mul(p_all<P>(72.0f), i3), c3 = p_mul(p_all<P>(3.0f * tt), ir);
        const P Fx = p_mul(c3, p_all<P>(a.fx)), Fy = p_mul(c3, p_all<P>(a.fy)), Fz = p_mul(c3, p_all<P>(a.fz));
        xx = p_fma(Fx, ux, xx);
        yy = p_fma(Fy, uy, yy);
        zz = p_fma(Fz, uz, zz);
        xy = p_add(xy, p_fma(Fx, uy, p_mul(Fy, ux)));
        xz = p_add(xz, p_fma(Fx, uz, p_mul(Fz, ux)));
        yz = p_add(yz, p_fma(Fy, uz, p_mul(Fz, uy)));
    }
    o[0] = r; o[1] = ux; o[2] = uy; o[3] = uz;
    o[4] = xx; o[5] = xy; o[6] = xz; o[7] = yy; o[8] = yz; o[9] = zz;
}

// Pipeline of one column of TYI rows: warps 0 .. TYI/R - 1 hold R interior
// rows each, the next one the edge columns x = X0 - 1 (lanes 0 ..) and
// x = X0 + 32 (lanes 16 ..) of the same rows; further warps of the CTA only
// take the barriers.  Step j takes plane z0 - 1 + j from the ring through the
// y pass and, from j = 2 on, completes output plane z0 - 2 + j after the
// step's barrier.
template <typename T, int FLAGS, int TYI, int R, typename SM>
struct SumMarch : ZRing<T, TYI, npairs_of(FLAGS), SM, TYI / R> {
    using Ring = ZRing<T, TYI, npairs_of(FLAGS), SM, TYI / R>;
    using Ring::a;
    using Ring::advance;
    using Ring::cph;
    using Ring::cs;
    using Ring::nprod;
    using Ring::raise_timeout;
    using Ring::Ring;
    using Ring::ROW;
    using Ring::sm;
    using Ring::stage_base;
    using Ring::stage_off;
    using Ring::timed_out;
    using Ring::X0;
    using Ring::Y0;
    using Ring::z0;
    using P = std::conditional_t<R == 2, F2, float>;
    static constexpr int NM = nmoments_of(FLAGS);
    static constexpr int NML = nmoments_of(FLAGS & ~F_SPLITU);
    static_assert(TYI <= 16, "the helper warp holds both edge columns");
    static_assert(TYI % R == 0 && (R == 1 || R == 2), "rows of a thread");

    // edge slot of rows row .. row + R - 1 (R values of each of the six orders)
    __device__ __forceinline__ float* edge_slot(int par, int side, int row) const
    {
        return sm.sum_edge() + ((par * 2 + side) * TYI + row) * SUM_EDGE;
    }
#ifdef MRLBM_BOUNDS_CHECK
    __device__ void poison(int par) const
    {
        for (int i = threadIdx.x; i < 2 * TYI * SUM_EDGE; i += blockDim.x)
            edge_slot(par, 0, 0)[i] = __int_as_float(0x7fc00000);
    }
#endif
    // barrier of step j; false when a bounded wait timed out in the CTA
    __device__ __forceinline__ bool meet(int j, bool ok)
    {
        if (!ok) raise_timeout();
        __syncthreads();
        if (timed_out()) return false;
#ifdef MRLBM_BOUNDS_CHECK
        poison((j + 1) & 1);
        __syncthreads();
#endif
        advance(j);
        return true;
    }

    struct Node {
        int off;          // element offset of the first node's words in the row below it of a stage
        int x, y;         // first node
        unsigned at;      // byte offset of the first node's pair in a padded plane
        unsigned pitch;   // bytes of a padded row of pairs
        int lane, row;
        bool live[R], face[R];   // in the domain; on an x or y face of a periodic axis
    };

    __device__ __forceinline__ void store(const Node& nd, int zd, const P (&v)[10])
    {
        // the pair's plane: the same for the whole CTA; a node's place in it is a 32-bit offset
        const size_t zoff = (size_t)(zd + 1) * (size_t)a.plane * (2 * sizeof(T));
        const bool gz = (a.periodic & 4) && (zd == 0 || zd == a.nz - 1);
#pragma unroll
        for (int r = 0; r < R; r++) {
            float o[NM_MAX];
#pragma unroll
            for (int m = 0; m < 10; m++) o[m] = row_of(v[m], r);
            stored_words<T, NM, FLAGS>(a, o);
            if (!nd.live[r]) continue;
            const unsigned at = nd.at + r * nd.pitch;
            if (!MRLBM_GLOBAL_OK(zoff + at + 2 * sizeof(T) <= (size_t)a.field * 2 * sizeof(T), BCK_STORE, a.err)) continue;
#pragma unroll
            for (int p = 0; p < NM / 2; p++)
                Stor2<T>::st(reinterpret_cast<T*>(static_cast<char*>(a.out_p[p]) + zoff + at), o[2 * p], o[2 * p + 1]);
            if constexpr (NM % 2 != 0)
                Stor<T>::st(reinterpret_cast<T*>(static_cast<char*>(a.out_p[NM / 2]) + zoff + at), o[NM - 1]);
            if (nd.face[r] || gz) {
                const int y = nd.y + r;
                store_ghosts<T, NM>(a, (a.periodic & 1) && (nd.x == 0 || nd.x == a.nx - 1),
                                    (a.periodic & 2) && (y == 0 || y == a.ny - 1), gz, nd.x, y, zd, o);
            }
        }
    }

    // step j >= 2 of the interior; up0: c_z = +1 lines of plane j - 2
    // (replaced by plane j's), up1: those of plane j - 1
    template <int PAR>
    __device__ __forceinline__ bool step(const Node& nd, int j, P (&up0)[9], const P (&up1)[9], P (&md)[6])
    {
        const bool ok = mbar_wait(&sm.bars[cs], cph);
        P U[6][3];
        {
            P V[6][3];
            y_pass<T, NM, NML, R>(stage_base() + nd.off, ROW, a.rho0, V);
            ZLines<P> L;
            z_lines(V, L);
            z_sum(up0, up1, md, L.dn, U);
#pragma unroll
            for (int l = 0; l < 9; l++) up0[l] = L.up[l];
#pragma unroll
            for (int l = 0; l < 6; l++) md[l] = L.md[l];
        }
        P fl[6], fr[6], U0[6];   // arriving from x - 1, from x + 1; the own c_x = 0 lines
#pragma unroll
        for (int i = 0; i < 6; i++) {
            const P h = p_add(U[i][0], U[i][2]);
            fl[i] = from_left(p_add(h, U[i][1]));
            fr[i] = from_right(p_sub(h, U[i][1]));
            U0[i] = U[i][0];
        }
        if (!meet(j, ok)) return false;
        edge_into(fl, edge_slot(PAR, 0, nd.row), nd.lane == 0);
        edge_into(fr, edge_slot(PAR, 1, nd.row), nd.lane == TILE_X - 1);
        P o[10];
        x_collide<FLAGS>(a, fl, fr, U0, o);
        store(nd, z0 - 2 + j, o);
        return true;
    }

    // steps 0 and 1 only fill the z pipeline
    template <int RR, typename PP>
    __device__ __forceinline__ bool lead(int off, int j, PP (&up)[9], PP (&md)[6])
    {
        const bool ok = mbar_wait(&sm.bars[cs], cph);
        PP V[6][3];
        y_pass<T, NM, NML, RR>(stage_base() + off, ROW, a.rho0, V);
        ZLines<PP> L;
        z_lines(V, L);
#pragma unroll
        for (int l = 0; l < 9; l++) up[l] = L.up[l];
#pragma unroll
        for (int l = 0; l < 6; l++) md[l] = L.md[l];
        return meet(j, ok);
    }

    // each returns the step whose wait timed out, or -1
    __device__ __forceinline__ int interior_loop(int lane, int warp)
    {
        Node nd;
        nd.lane = lane;
        nd.row = R * warp;
        nd.x = X0 + lane;
        nd.y = Y0 + R * warp;
        nd.off = stage_off(R * warp, nd.x);
        nd.pitch = (unsigned)a.pitch * (unsigned)(2 * sizeof(T));
        nd.at = (unsigned)(nd.y + 1) * nd.pitch + (unsigned)(nd.x + XOFF) * (unsigned)(2 * sizeof(T));
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int y = nd.y + r;
            nd.live[r] = nd.x < a.nx && y < a.ny;
            nd.face[r] = ((a.periodic & 1) && (nd.x == 0 || nd.x == a.nx - 1)) ||
                         ((a.periodic & 2) && (y == 0 || y == a.ny - 1));
        }
        P upA[9], upB[9], md[6];
        if (!lead<R>(nd.off, 0, upA, md)) return 0;
        if (!lead<R>(nd.off, 1, upB, md)) return 1;
        for (int j = 2; j < nprod; j++) {
            if (!step<0>(nd, j, upA, upB, md)) return j;
            if (++j >= nprod) break;
            if (!step<1>(nd, j, upB, upA, md)) return j;
        }
        return -1;
    }

    __device__ __forceinline__ int helper_loop(int lane)
    {
        const int side = lane >> 4, row = (lane & 15) < TYI ? (lane & 15) : 0;
        const bool on = (lane & 15) < TYI;
        const int off = stage_off(row, side ? X0 + TILE_X : X0 - 1);
        const float sgn = side ? -1.0f : 1.0f;
        float up0[9], up1[9], md[6];
        if (!lead<1>(off, 0, up0, md)) return 0;
        if (!lead<1>(off, 1, up1, md)) return 1;
        for (int j = 2; j < nprod; j++) {
            const bool ok = mbar_wait(&sm.bars[cs], cph);
            float V[6][3], U[6][3];
            y_pass<T, NM, NML, 1>(stage_base() + off, ROW, a.rho0, V);
            ZLines<float> L;
            z_lines(V, L);
            z_sum(up0, up1, md, L.dn, U);
#pragma unroll
            for (int l = 0; l < 9; l++) { up0[l] = up1[l]; up1[l] = L.up[l]; }
#pragma unroll
            for (int l = 0; l < 6; l++) md[l] = L.md[l];
            float* e = edge_slot(j & 1, side, row - row % R) + row % R;
            if (on && MRLBM_SMEM_OK(e, 4 * (5 * R + 1), BCK_EDGE)) {
#pragma unroll
                for (int i = 0; i < 6; i++) e[i * R] = fmaf(sgn, U[i][1], __fadd_rn(U[i][0], U[i][2]));
            }
            if (!meet(j, ok)) return j;
        }
        return -1;
    }

    __device__ __forceinline__ int idle_loop()
    {
        for (int j = 0; j < nprod; j++)
            if (!meet(j, true)) return j;
        return -1;
    }
};

// One column of a sums-march domain; as zmarch_column.
template <typename T, int FLAGS, int TYI, int R, typename SM>
__device__ __forceinline__ bool sum_column(const StepArgs& a, const CUtensorMap* map, int X0, int Y0, int z0, int zend,
                                           const SM& sm, unsigned& g0)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SumMarch<T, FLAGS, TYI, R, SM> zm(a, map, sm, g0, X0, Y0, z0, zend);
#ifdef MRLBM_BOUNDS_CHECK
    if (threadIdx.x == 0) {
        g_bounds.stage_lo = smem_u32(sm.stages);
        g_bounds.stage_hi = smem_u32(sm.stages) + (unsigned)(SM::NS * SM::stage_max);
        g_bounds.ex_lo = g_bounds.ex_hi = 0;
        g_bounds.edge_lo = smem_u32(sm.sum_edge());
        g_bounds.edge_hi = g_bounds.edge_lo + (unsigned)(4 * TYI * SUM_EDGE * sizeof(float));
        g_bounds.err = a.err;
    }
    __syncthreads();
    zm.poison(0);
    zm.poison(1);
    __syncthreads();
#endif
    zm.fill();
    const int kfail = warp < TYI / R    ? zm.interior_loop(lane, warp)
                      : warp == TYI / R ? zm.helper_loop(lane)
                                        : zm.idle_loop();
    if (kfail >= 0) {
        zm.drain(kfail);
        __syncthreads();
        return false;
    }
    g0 += (unsigned)zm.nprod;
    // the last step read edge slots that the next column's helper writes
    __syncthreads();
    return true;
}

}  // namespace mrlbm
