// Line transforms of the Cartesian slices above 128 x 128 (slice_big.cu, slice_cluster.cu): 128 and 256 points on
// 16 values per thread, as reg_n2m / reg_m2n (slice_reg.cuh) with fewer instructions.
//   * The sums of the butterflies are packed f32x2 instructions (padd, psub).
//   * The twiddles W_N^(j a) come two to a load from a table in the order of use (tw[a / 2][j] =
//     {W^(j a), W^(j (a + 1))}): 15 complex products a line, where applying W^j, W^2j, W^4j, W^8j takes 32.
//   * The transform is always the forward one.  The inverse is the forward one between re and im exchanged
//     (swp): the passes exchange where a value is formed or stored anyway, and the slice between the inverse
//     column and row transforms lies in memory exchanged.
// At 1025 x 256 x 256 the three passes of an evaluation went from 855 to 699 us with these and the form of the
// column pass for real media: 4.58 GB at 6.6 TB/s, where the column pass was bound by instruction issue and
// latency at two blocks per multiprocessor before.
#pragma once
#include "common.cuh"
#include "dft_reg.cuh"

UPPE_DEV float2 swp(float2 a) { return make_float2(a.y, a.x); }

// 4-point DFT; TURN: the third input is to be multiplied by -i first
template <bool TURN = false>
UPPE_DEV void ldft4(float2& u0, float2& u1, float2& u2, float2& u3) {
    const float2 m2 = cmul_mi(u2);
    const float2 a0 = TURN ? cadd(u0, m2) : padd(u0, u2), a1 = TURN ? csub(u0, m2) : psub(u0, u2);
    const float2 a2 = padd(u1, u3), a3 = cmul_mi(psub(u1, u3));
    u0 = padd(a0, a2);
    u2 = psub(a0, a2);
    u1 = cadd(a1, a3);
    u3 = csub(a1, a3);
}

UPPE_DEV void ldft16(float2 (&v)[16]) {
#pragma unroll
    for (int n = 0; n < 4; ++n) ldft4(v[n], v[n + 4], v[n + 8], v[n + 12]);  // v[n + 4 k]: output k of row n
    v[5] = mul_w16<1, false>(v[5]);
    v[9] = mul_w16<2, false>(v[9]);
    v[13] = mul_w16<3, false>(v[13]);
    v[6] = mul_w16<2, false>(v[6]);
    v[14] = mul_w16<6, false>(v[14]);
    v[7] = mul_w16<3, false>(v[7]);
    v[11] = mul_w16<6, false>(v[11]);
    v[15] = mul_w16<9, false>(v[15]);
    ldft4(v[0], v[1], v[2], v[3]);
    ldft4(v[4], v[5], v[6], v[7]);
    ldft4<true>(v[8], v[9], v[10], v[11]);
    ldft4(v[12], v[13], v[14], v[15]);
    // v[4 k + m] = output k + 4 m: natural order
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int m = k + 1; m < 4; ++m) {
            const float2 x = v[4 * k + m];
            v[4 * k + m] = v[4 * m + k];
            v[4 * m + k] = x;
        }
}

template <int R>
UPPE_DEV void ldft_line(float2 (&u)[R]) {
    static_assert(R == 8 || R == 16, "lines of 128 or 256 points");
    if constexpr (R == 16) {
        ldft16(u);
    } else {
        float2 e[4] = {u[0], u[2], u[4], u[6]}, o[4] = {u[1], u[3], u[5], u[7]};
        ldft4(e[0], e[1], e[2], e[3]);
        ldft4(o[0], o[1], o[2], o[3]);
        const float2 t1 = mul_w16<2, false>(o[1]), t2 = cmul_mi(o[2]), t3 = mul_w16<6, false>(o[3]);
        u[0] = padd(e[0], o[0]);
        u[4] = psub(e[0], o[0]);
        u[1] = padd(e[1], t1);
        u[5] = psub(e[1], t1);
        u[2] = cadd(e[2], t2);
        u[6] = csub(e[2], t2);
        u[3] = padd(e[3], t3);
        u[7] = psub(e[3], t3);
    }
}

template <int R>
UPPE_DEV void line_twiddle(float2 (&v)[16], const float4* __restrict__ tw, int j) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float4 t = __ldg(&tw[i * R + j]);
        if (i) v[2 * i] = cmul(v[2 * i], make_float2(t.x, t.y));
        v[2 * i + 1] = cmul(v[2 * i + 1], make_float2(t.z, t.w));
    }
}

// natural -> mixed: v[m] = x[j + R m]  ->  w[s R + b] = X[j + R s + 16 b]
template <int R, class SY>
UPPE_DEV void line_n2m(float2 (&v)[16], float2 (&w)[16], float2* ex, int j, const float4* __restrict__ tw, const SY& sync) {
    ldft16(v);
    line_twiddle<R>(v, tw, j);
#pragma unroll
    for (int a = 0; a < 16; ++a) ex[j * 17 + a] = v[a];
    sync();
#pragma unroll
    for (int s = 0; s < 16 / R; ++s) {
        float2 u[R];
#pragma unroll
        for (int jj = 0; jj < R; ++jj) u[jj] = ex[jj * 17 + j + R * s];
        ldft_line<R>(u);
#pragma unroll
        for (int b = 0; b < R; ++b) w[s * R + b] = u[b];
    }
}

// mixed -> natural: w[s R + b] = X[j + R s + 16 b]  ->  v[m] = x[j + R m]
template <int R, class SY>
UPPE_DEV void line_m2n(float2 (&w)[16], float2 (&v)[16], float2* ex, int j, const float4* __restrict__ tw, const SY& sync) {
    sync();  // the line's last reads of this region are done
#pragma unroll
    for (int s = 0; s < 16 / R; ++s) {
        float2 u[R];
#pragma unroll
        for (int b = 0; b < R; ++b) u[b] = w[s * R + b];
        ldft_line<R>(u);
#pragma unroll
        for (int jj = 0; jj < R; ++jj) ex[jj * 17 + j + R * s] = u[jj];
    }
    sync();
#pragma unroll
    for (int a = 0; a < 16; ++a) v[a] = ex[j * 17 + a];
    line_twiddle<R>(v, tw, j);
    ldft16(v);
}

// the table of lines of 2^LN points within h->tw_line
template <int LN>
UPPE_DEV const float4* line_table(const float4* tw) {
    return tw + (LN == 8 ? 64 : 0);
}
