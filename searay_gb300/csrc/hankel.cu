// Cylindrical transverse transform: the radial Hankel transform of SeaRay's HankelTransformTool
// (modules/grid_tools.py:252-325; kernels fft.cl:363-385 RootVolumeMultiply/Divide, :443-477
// RadialTransform/InverseRadialTransform) as a batched complex x real GEMM per azimuthal mode,
// with the root-volume weights folded into the matrices:
//     forward  J_k = sum_r Mfwd[k][r] J_r,  Mfwd[k][r] = H[k][r] Lambda_r / Lambda_k  (k < Nk, else 0)
//     inverse  E_r = sum_k Minv[r][k] E_k,  Minv[r][k] = H[k][r] Lambda_k / Lambda_r
// The spectral-side operations are fused into the GEMM: the A-operand loader applies the propagator
// phase and i kz, the epilogue forms the ODE right-hand side and the RK4 stage update.
// The azimuthal FFT (FFT_axis2/IFFT_axis2, fft.cl:401-441) of grids with N2 > 1 runs as a separate
// DFT pass around the GEMM.
#include "common.cuh"
#include "hankel_tc.cuh"
#include "time_common.cuh"
#include "uppe_internal.h"

#define GBK 16  // reduction elements per shared tile

enum { A_PLAIN = 0, A_QPHASE_IKZ = 1, A_QPHASE = 2, A_SADJ = 3 };
enum { C_STORE = 0, C_FINISH1 = 1, C_SPEC = 2, C_QADJ = 3, C_FADJ = 4 };

struct GemmArgs {
    const float2* A;  // operand source ([w][r|k][m] layout, row length N1, N2 azimuthal nodes)
    const float* B;   // [N2][KP][LD], reduction-major: B[m][k][i], zero-padded (hankel_kmajor)
    int KP, LD;
    int which;        // 0 Mfwd, 1 Minv, 2 Mfwd^T, 3 Minv^T
    OpView op;
    float2* C0;       // store target / q_out / A_out
    float2* C1;       // E (finish) / qf
    const float2* qi;
    int N0, N1, N2, NI, NK;
    int spec_mode;
    float Cs, Ce;
    StepArgs z;
};

// One block: BM frequencies x BN output columns, threads of TM x TN; TX threads along the columns, a
// thread's columns in groups of four (TX groups apart).  The accumulators of two neighbouring columns
// share a packed f32x2 register, so a term costs two packed FMAs against the broadcast Re and Im of
// the field; each sum runs over k in ascending order.  B comes in by 16-byte asynchronous copies and the
// field (with its propagator factor, formed in registers) by way of the next tile's loads issued
// before this tile's products, both into the other half of a double buffer: one barrier per 16 k.  The
// products then go through shared memory, TY rows at a time, to a rolled loop along the columns: the
// epilogue's code exists once (unrolled over a thread's products it stalled on instruction fetch), its
// accesses are coalesced, and its operands are loaded four points ahead of the stores.
//
// At 2049 x 512 x 512 a product is 1.07e9 FMAs, 28 us at the 39e12/s of 152 multiprocessors.  Bound by the delivery of
// its operands from shared memory (L1 pipe 70 % busy, `mio_throttle` and `short_scoreboard` the top stalls, issue
// 46 to 52 % on 130 blocks).  Measured there, the propagator factor or the RK stage included: 67 and 70 us, against
// 127 and 120 us with 32 x 64 tiles of 2 x 4 and no copies ahead (512 threads of 2 x 8 against 256 of 4 x 8: 68 against
// 71 us; scalar FMAs in place of packed ones: the same).
template <int BM, int BN, int TM, int TN>
struct GemmShape {
    static constexpr int TX = BN / TN, TY = BM / TM, T = TX * TY, AE = BM * GBK / T, BE = GBK * BN / 4 / T;
    static_assert(TY == GBK && TX % 16 == 0 && TN % 4 == 0 && AE >= 1 && BE >= 1, "GEMM shape");
};

template <int AMODE, int CMODE, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) k_hankel_gemm(GemmArgs g) {
    using GS = GemmShape<BM, BN, TM, TN>;
    __shared__ float2 As[2][GBK][BM + 1];
    __shared__ __align__(16) float Bs[2][GBK][BN];
    const int tid = threadIdx.x;
    const int m = blockIdx.z;
    const int w0 = blockIdx.y * BM;
    const int i0 = blockIdx.x * BN;
    // a warp covers 16 column groups x 2 rows, so that its B reads are 256 bytes and two rows share them
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int WX = GS::TX / 16;
    const int tx = (lane & 15) + 16 * (warp % WX), ty = (lane >> 4) + 2 * (warp / WX);
    const PhaseArgs pa{g.z.zhi, g.z.zlo, g.z.plain};
    f2x accx[TM][TN / 2], accy[TM][TN / 2];
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) accx[r][j] = accy[r][j] = pk2(0.f, 0.f);
    const float* Bm = g.B + (size_t)m * g.KP * g.LD;

    const auto issue_B = [&](int k0, int half) {
#pragma unroll
        for (int s = 0; s < GS::BE; ++s) {
            const int e = tid + s * GS::T;
            const int kk = e / (BN / 4), c = 4 * (e % (BN / 4));
            if (i0 + c < g.LD)
                cp_async16_time(&Bs[half][kk][c], Bm + (size_t)(k0 + kk) * g.LD + i0 + c);
            else
                *reinterpret_cast<float4*>(&Bs[half][kk][c]) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // the field element e = (w, k) of a tile: loads first, the factor when it is stored
    float2 av[GS::AE], aK[GS::AE];
    float aki[GS::AE];
    const auto load_A = [&](int k0) {
#pragma unroll
        for (int s = 0; s < GS::AE; ++s) {
            const int e = tid + s * GS::T;
            const int w = w0 + e / GBK, k = k0 + e % GBK;
            av[s] = aK[s] = make_float2(0.f, 0.f);
            aki[s] = 0.f;
            if (w < g.N0 && k < g.NK) {
                const size_t idx = ((size_t)w * g.N1 + k) * g.N2 + m;
                av[s] = g.A[idx];
                if (AMODE != A_PLAIN) {
                    aK[s] = g.op.K[idx];
                    if (g.op.ki) aki[s] = g.op.ki[idx];
                }
            }
        }
    };
    const auto store_A = [&](int k0, int half) {
#pragma unroll
        for (int s = 0; s < GS::AE; ++s) {
            const int e = tid + s * GS::T;
            const int w = w0 + e / GBK, k = k0 + e % GBK;
            float2 v = av[s];
            if (AMODE != A_PLAIN && w < g.N0 && k < g.NK) {
                const float2 kgw = g.op.kg[w];
                OpPoint o;
                o.Khi = aK[s].x;
                o.Klo = aK[s].y;
                o.kzr = g.op.envelope ? kgw.x : (aK[s].x - kgw.x) + (aK[s].y - kgw.y);
                o.kzi = aki[s];
                if (AMODE == A_SADJ) {
                    // conj(D2) v, D2 = (i/2) exp(-i(kz+kg)z) / Re kz
                    const float2 f = cconj(propagator_factor(o, pa, -1.f));
                    v = cscale(cmul_mi(cmul(f, v)), 0.5f / o.kzr);
                } else {
                    v = cmul(propagator_factor(o, pa, 1.f), v);
                    if (AMODE == A_QPHASE_IKZ) v = op_field(g.op, o, v);
                }
            }
            As[half][e % GBK][e / GBK] = v;
        }
    };

    load_A(0);
    issue_B(0, 0);
    store_A(0, 0);
    int half = 0;
    for (int k0 = 0; k0 < g.NK; k0 += GBK, half ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();  // this tile has landed; the other half has been read
        const bool more = k0 + GBK < g.NK;
        if (more) {
            issue_B(k0 + GBK, half ^ 1);
            load_A(k0 + GBK);
        }
#pragma unroll
        for (int kk = 0; kk < GBK; ++kk) {
            f2x b[TN / 2];
#pragma unroll
            for (int q = 0; q < TN / 4; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(&Bs[half][kk][4 * (q * GS::TX + tx)]);
                b[2 * q] = pk2(v.x, v.y);
                b[2 * q + 1] = pk2(v.z, v.w);
            }
#pragma unroll
            for (int r = 0; r < TM; ++r) {
                const float2 a = As[half][kk][ty * TM + r];
                const f2x ax = pk2(a.x, a.x), ay = pk2(a.y, a.y);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) {
                    accx[r][j] = fma2(ax, b[j], accx[r][j]);
                    accy[r][j] = fma2(ay, b[j], accy[r][j]);
                }
            }
        }
        if (more) store_A(k0 + GBK, half ^ 1);
    }
    // ---- epilogue ----
    float2* stage = reinterpret_cast<float2*>(&Bs[0][0][0]);  // TY rows of BN products
    const bool need_a = CMODE == C_SPEC && (g.spec_mode == SPEC_STAGE1 || g.spec_mode == SPEC_STAGE23);
    const bool need_b = CMODE == C_SPEC && (g.spec_mode == SPEC_STAGE23 || g.spec_mode == SPEC_FINISH);
#pragma unroll 1
    for (int r = 0; r < TM; ++r) {
        __syncthreads();  // the last tile's products, or the previous rows, have been read
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            f2x vx = accx[0][j], vy = accy[0][j];
#pragma unroll
            for (int rr = 1; rr < TM; ++rr)
                if (r == rr) {
                    vx = accx[rr][j];
                    vy = accy[rr][j];
                }
            const float2 x = up2(vx), y = up2(vy);
            const int c = 4 * ((j / 2) * GS::TX + tx) + 2 * (j % 2);
            *reinterpret_cast<float4*>(&stage[ty * BN + c]) = make_float4(x.x, y.x, x.y, y.y);
        }
        __syncthreads();
        constexpr int NE = GS::TY * BN / GS::T, U = NE < 4 ? NE : 4;
#pragma unroll 1
        for (int e0 = 0; e0 < NE; e0 += U) {
            float2 v[U], K[U], qa[U], qb[U];
            float ki[U];
            size_t idx[U];
            bool in[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = tid + (e0 + u) * GS::T;
                const int c = e % BN, w = w0 + (e / BN) * TM + r, i = i0 + c;
                in[u] = w < g.N0 && i < g.NI;
                idx[u] = ((size_t)w * g.N1 + i) * g.N2 + m;
                v[u] = stage[(e / BN) * BN + c];
                K[u] = qa[u] = qb[u] = make_float2(0.f, 0.f);
                ki[u] = 0.f;
                if (CMODE != C_STORE && in[u]) {
                    K[u] = g.op.K[idx[u]];
                    if (g.op.ki) ki[u] = g.op.ki[idx[u]];
                    if (need_a) qa[u] = g.qi[idx[u]];
                    if (need_b) qb[u] = g.C1[idx[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!in[u]) continue;
                const int w = w0 + ((tid + (e0 + u) * GS::T) / BN) * TM + r;
                if constexpr (CMODE == C_STORE) {
                    g.C0[idx[u]] = v[u];
                    continue;
                }
                const float cond = (w < g.op.ncond) ? 0.f : 1.f;
                const float2 kgw = g.op.kg[w];
                OpPoint o;
                o.Khi = K[u].x;
                o.Klo = K[u].y;
                o.kzr = g.op.envelope ? kgw.x : (K[u].x - kgw.x) + (K[u].y - kgw.y);
                o.kzi = ki[u];
                if constexpr (CMODE == C_QADJ || CMODE == C_FADJ) {
                    float2 c = cmul(cconj(propagator_factor(o, pa, 1.f)), v[u]);
                    if (CMODE == C_QADJ) c = cmul(cconj(op_ikz(o)), c);
                    g.C0[idx[u]] = c;
                } else if constexpr (CMODE == C_FINISH1) {
                    if (g.C0) g.C0[idx[u]] = v[u];
                    g.C1[idx[u]] = op_field(g.op, o, v[u]);
                } else if constexpr (CMODE == C_SPEC) {
                    const float2 f = propagator_factor(o, pa, -1.f);
                    const float2 s = cscale(cmul_i(cmul_fixed(f, v[u])), 0.5f / o.kzr);
                    switch (g.spec_mode) {
                        case SPEC_STORE_K:
                            g.C0[idx[u]] = s;
                            break;
                        case SPEC_STAGE1:
                            g.C1[idx[u]] = caxpy(qa[u], s, g.Cs);
                            g.C0[idx[u]] = cscale(caxpy(qa[u], s, g.Ce), cond);
                            break;
                        case SPEC_STAGE23:
                            g.C1[idx[u]] = caxpy(qb[u], s, g.Cs);
                            g.C0[idx[u]] = cscale(caxpy(qa[u], s, g.Ce), cond);
                            break;
                        default:
                            g.C0[idx[u]] = cscale(caxpy(qb[u], s, g.Cs), cond);
                            break;
                    }
                }
            }
        }
    }
}

// Azimuthal DFT along the contiguous last axis (length N2): out[row][j] = scale * sum_m in[row][m] W^{jm},
// W = exp(-+2 pi i / N2) (numpy fft / ifft conventions, fft.cl:401-441).
__global__ void k_azimuth_dft(const float2* __restrict__ in, float2* __restrict__ out, size_t rows, int N2,
                              int logN2, bool inv, float scale, const float2* __restrict__ tw, int twLog) {
    const size_t n = rows * (size_t)N2;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i >> logN2;
        const int j = (int)(i & (N2 - 1));
        const float2* src = in + row * N2;
        float2 acc = make_float2(0.f, 0.f);
        for (int mm = 0; mm < N2; ++mm) {
            float2 w = __ldg(&tw[((j * mm) & (N2 - 1)) << (twLog - logN2)]);
            if (inv) w.y = -w.y;
            acc = cadd(acc, cmul(src[mm], w));
        }
        out[i] = cscale(acc, scale);
    }
}

// The forward azimuthal DFT of the mixed form, its outputs split straight into the operand tiles of the tensor-core
// transform that follows (tile order of k_hankel_tc_prep).  Eight neighbouring lanes take eight radial nodes
// of one azimuthal mode: their 2-byte stores fill 16-byte rows, their loads of one azimuthal node share sectors
// with those of the warp's other modes.
__global__ void k_azimuth_tiles(const float2* __restrict__ in, uint8_t* __restrict__ Atc, int N0, int N1, int N2,
                                int logN2, int nwt, int nkt, const float2* __restrict__ tw, int twLog) {
    const size_t rows = (size_t)N0 * N1, n = ((rows + 7) >> 3) << (3 + logN2);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(i >> 3) & (N2 - 1);
        const size_t row = ((i >> (3 + logN2)) << 3) + (i & 7);
        if (row >= rows) continue;
        const float2* src = in + row * N2;
        float2 acc = make_float2(0.f, 0.f);
        for (int mm = 0; mm < N2; ++mm)
            acc = cadd(acc, cmul(src[mm], __ldg(&tw[((j * mm) & (N2 - 1)) << (twLog - logN2)])));
        tc_store_split(Atc, nwt, nkt, j, (int)(row / N1), (int)(row % N1), acc);
    }
}

static cudaError_t launch_azimuth(UppeHandle* h, const float2* in, float2* out, bool inv) {
    const int logN2 = ilog2_exact(h->N2);
    const size_t rows = (size_t)h->N0 * h->N1;
    const size_t n = rows * h->N2;
    unsigned blocks = (unsigned)((n + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    h->launches++;
    k_azimuth_dft<<<blocks, 256, 0, h->stream>>>(in, out, rows, h->N2, logN2, inv, inv ? 1.f / h->N2 : 1.f, h->tw,
                                                  h->twLog);
    return cudaGetLastError();
}

cudaError_t launch_hankel_tc(UppeHandle* h, int amode, int cmode, const float2* A, int which, float2* C0,
                             float2* C1, int NI, int NK, StepArgs z);

static cudaError_t launch_azimuth_tiles(UppeHandle* h, const float2* in) {
    const int logN2 = ilog2_exact(h->N2);
    const size_t n = ((((size_t)h->N0 * h->N1 + 7) >> 3) << 3) * h->N2;
    unsigned blocks = (unsigned)((n + 255) / 256);
    if (blocks > 16u * h->num_sms) blocks = 16u * h->num_sms;
    h->launches++;
    h->atc_next = 0;
    k_azimuth_tiles<<<blocks, 256, 0, h->stream>>>(in, h->Atc, h->N0, h->N1, h->N2, logN2, (h->N0 + TC_W - 1) / TC_W,
                                                   (h->N1 + TC_K - 1) / TC_K, h->tw, h->twLog);
    return cudaGetLastError();
}

size_t hankel_kmajor_len(int N1, int N2) {
    const size_t KP = (size_t)(N1 + GBK - 1) / GBK * GBK, LD = (size_t)(N1 + 3) / 4 * 4;
    return (size_t)N2 * KP * LD;
}

// The matrix M[m][i][k] (rows of NK) as the FP32 GEMM reads it, out[m][k][i], zero-padded to KP x LD.
void hankel_kmajor(const float* M, int N1, int N2, int NK, float* out) {
    const size_t KP = (size_t)(N1 + GBK - 1) / GBK * GBK, LD = (size_t)(N1 + 3) / 4 * 4;
    for (size_t e = 0; e < (size_t)N2 * KP * LD; ++e) out[e] = 0.f;
    for (int m = 0; m < N2; ++m)
        for (int i = 0; i < N1; ++i)
            for (int k = 0; k < NK; ++k) out[((size_t)m * KP + k) * LD + i] = M[((size_t)m * N1 + i) * NK + k];
}

template <int AMODE, int CMODE, int BM, int BN, int TM, int TN>
static cudaError_t run_simt_shape(UppeHandle* h, const GemmArgs& g) {
    dim3 grid((g.NI + BN - 1) / BN, (g.N0 + BM - 1) / BM, g.N2);
    k_hankel_gemm<AMODE, CMODE, BM, BN, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, h->stream>>>(g);
    return cudaGetLastError();
}

// The plain FP32 GEMM.  Wide tiles reuse each field element (and its propagator factor) for more columns
// and need fewer shared loads per FMA, narrow ones make more blocks: the widest whose blocks still cover
// three quarters of the multiprocessors, and 16 x 64 below that.  Step times in us with tiles of 256 | 128 |
// 64 | 16 x 64 (the chosen one starred): 2049 x 512 609* | 693 | 705 | 821, 1025 x 512 574 | 381* | 406 |
// 493, 513 x 512 551 | 364 | 272* | 288, 257 x 256 316 | 214 | 168 | 132*, 257 x 64 145 | 108 | 92 | 78*.
template <int AMODE, int CMODE>
static cudaError_t run_simt(UppeHandle* h, GemmArgs& g) {
    if (!h->Bk[g.which]) return cudaErrorInvalidValue;
    g.B = h->Bk[g.which];
    g.KP = (h->N1 + GBK - 1) / GBK * GBK;
    g.LD = (h->N1 + 3) / 4 * 4;
    h->launches++;
    const auto blocks = [&](int bn) { return (long)((g.NI + bn - 1) / bn) * ((g.N0 + 31) / 32) * g.N2; };
    const long want = (long)h->num_sms * 3 / 4;
    if (g.NI > 128 && blocks(256) >= want) return run_simt_shape<AMODE, CMODE, 32, 256, 2, 8>(h, g);
    if (g.NI > 64 && blocks(128) >= want) return run_simt_shape<AMODE, CMODE, 32, 128, 2, 4>(h, g);
    if (blocks(64) >= want) return run_simt_shape<AMODE, CMODE, 32, 64, 2, 4>(h, g);
    return run_simt_shape<AMODE, CMODE, 16, 64, 1, 4>(h, g);
}

// Mixed-precision form: tensor-core GEMM (hankel_tc.cu); plain FP32 form: the FP32 SIMT GEMM above.
template <int AMODE, int CMODE>
static cudaError_t run_gemm(UppeHandle* h, GemmArgs& g) {
    if (h->cfg.precision == UPPE_PREC_MIXED)
        return launch_hankel_tc(h, AMODE, CMODE, g.A, g.which, g.C0, g.C1, g.NI, g.NK, g.z);
    return run_simt<AMODE, CMODE>(h, g);
}

static GemmArgs base_args(UppeHandle* h, StepArgs z) {
    GemmArgs g{};
    g.op = uppe_op_view(h);
    g.N0 = h->N0;
    g.N1 = h->N1;
    g.N2 = h->N2;
    g.z = z;
    return g;
}

// Inverse transform: E = T^-1(i kz exp(..) q) or, for finish, A = T^-1(exp(..) q) and E = i kz A.
cudaError_t launch_real_cyl(UppeHandle* h, int mode, const float2* src, float2* A_out, StepArgs z) {
    GemmArgs g = base_args(h, z);
    g.A = src;
    g.which = 1;
    g.NI = h->N1;
    g.NK = h->Nk;
    cudaError_t err;
    if (h->N2 == 1) {
        if (mode == REAL_E) {
            g.C0 = h->E;
            err = run_gemm<A_QPHASE_IKZ, C_STORE>(h, g);
        } else {
            g.C0 = A_out;
            g.C1 = h->E;
            err = run_gemm<A_QPHASE, C_FINISH1>(h, g);
        }
        return err;
    }
    g.C0 = h->scratch;
    if (mode == REAL_E) {
        err = run_gemm<A_QPHASE_IKZ, C_STORE>(h, g);
        if (err != cudaSuccess) return err;
        return launch_azimuth(h, h->scratch, h->E, true);
    }
    err = run_gemm<A_QPHASE, C_STORE>(h, g);
    if (err != cudaSuccess) return err;
    float2* A = A_out ? A_out : h->k1;  // k1 is free at finish time
    err = launch_azimuth(h, h->scratch, A, true);
    if (err != cudaSuccess) return err;
    return launch_ikz(h, A, h->E);
}

// Forward transform of J (or of the incoming field for SPEC_LOAD) and the spectral update: fused into the GEMM's
// epilogue in the SIMT form.  The tensor-core form stores its product over J (its pre-pass, or the azimuthal DFT, has
// read J by then) and a separate elementwise pass applies S and the RK stage: the update reads five arrays a point,
// which the GEMM's few blocks wait for and a pass over the whole grid streams (257 x 64 x 8 azimuthal: forward
// transform with the update 24 us in the epilogue, 17 us apart; a ten-step pass 1.98 -> 1.82 ms).
// z_next (stages whose estimate the next evaluation transforms at z_next): the tensor-core form's
// spectral update also writes that inverse transform's operand tiles (k_spec_point).
cudaError_t launch_spec_cyl(UppeHandle* h, int mode, const float2* src_real, float2* q_out, float2* qf_io,
                            const float2* qi, float Cs, float Ce, StepArgs z, const StepArgs* z_next) {
    GemmArgs g = base_args(h, z);
    g.which = 0;
    g.NI = h->N1;
    g.NK = h->N1;
    g.A = src_real;
    if (h->N2 > 1) {
        g.A = h->scratch;
        const bool tiles = h->cfg.precision == UPPE_PREC_MIXED && h->tc_next && h->Atc;
        cudaError_t err = tiles ? launch_azimuth_tiles(h, src_real) : launch_azimuth(h, src_real, h->scratch, false);
        if (err != cudaSuccess) return err;
        if (tiles) {
            h->atc_fwd = 1;
            h->atc_fwd_which = 0;
            h->atc_fwd_src = h->scratch;
        }
    }
    g.C0 = q_out;
    if (mode == SPEC_LOAD) return run_gemm<A_PLAIN, C_STORE>(h, g);
    if (h->cfg.precision == UPPE_PREC_MIXED) {
        g.C0 = h->J;
        cudaError_t err = run_gemm<A_PLAIN, C_STORE>(h, g);
        if (err != cudaSuccess) return err;
        return launch_spec_point(h, mode, h->J, q_out, qf_io, qi, Cs, Ce, z, z_next);
    }
    g.C1 = qf_io;
    g.qi = qi;
    g.Cs = Cs;
    g.Ce = Ce;
    g.spec_mode = mode;
    return run_simt<A_PLAIN, C_SPEC>(h, g);
}

// Adjoint transverse transforms on cylindrical grids (one azimuthal node) with the transposed folded
// matrices: ADJ_S / ADJ_LOAD apply Mfwd^T, ADJ_E / ADJ_FIN apply Minv^T; the tensor-core GEMM in the
// mixed-precision form, the FP32 SIMT GEMM in the plain form.
cudaError_t launch_adj_cyl(UppeHandle* h, int mode, const float2* in, float2* out, StepArgs z) {
    GemmArgs g = base_args(h, z);
    g.A = in;
    g.C0 = out;
    g.NI = h->N1;
    g.NK = h->N1;
    switch (mode) {
        case ADJ_S:
            g.which = 2;
            return run_gemm<A_SADJ, C_STORE>(h, g);
        case ADJ_LOAD:
            g.which = 2;
            return run_gemm<A_PLAIN, C_STORE>(h, g);
        case ADJ_E:
            g.which = 3;
            return run_gemm<A_PLAIN, C_QADJ>(h, g);
        default:
            g.which = 3;
            return run_gemm<A_PLAIN, C_FADJ>(h, g);
    }
}
