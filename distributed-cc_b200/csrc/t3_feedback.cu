// T3 -> r1 (r1r2_add_t3_tri_, distr_cc/rccsdt.py:262-296) in one pass over the canonical blocks.
//
// The reference contracts V = P3_422(t3) of a block with ERI slices E = <oo|vv>:
//   r1[i][a] += c1 sum_bc E[j,k][b,c] V[a,b,c],  r1[j][a] += c2 sum_bc E[i,k][b,c] V[b,a,c],
//   r1[k][a] += c3 sum_bc E[i,j][b,c] V[b,c,a].
// Moving the permutations of V onto E, output m (E_1 = E[j,k], E_2 = E[i,k], E_3 = E[i,j]) is
//   R_m[v] = sum_yz t[v,y,z] A_m[y,z] + sum_xz t[x,v,z] B_m[x,z] + sum_xy t[x,y,v] C_m[x,y]
// with A, B, C out of K1 = 4E - 2E^T, K2 = -2E + E^T, K3 = E - 2E^T:
//   A = K1(E1), K2(E2), K3(E3);  B = K2(E1), K1(E2), K2(E3);  C = K3(E1), K2(E2), K1(E3).
// So every element of t3 is read once and used nine times.
#include "dcc_common.cuh"

namespace dcc {

constexpr int R1_THREADS = 256, R1_WARPS = R1_THREADS / 32;
constexpr int R1_XC = 4;        // first indices x of a CTA
constexpr int R1_MAXNV = 128;   // z tiles of 32 in registers: at most four

// K[k][pair][y][z], k = 0, 1, 2 for K1, K2, K3 of every occupied pair
__global__ void k_r1_mix(const double *__restrict__ E, double *__restrict__ K, int64_t npair, int nv) {
    const int64_t nv2 = (int64_t)nv * nv, n = npair * nv2;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = e / nv2;
        const int yz = (int)(e - p * nv2), y = yz / nv, z = yz - y * nv;
        const double a = E[e], b = E[p * nv2 + (int64_t)z * nv + y];
        K[e] = 4.0 * a - 2.0 * b;
        K[n + e] = b - 2.0 * a;
        K[2 * n + e] = a - 2.0 * b;
    }
}

// CTA (q, x0): the sums of block q over x in [x0, x0 + 4), one warp per y, lanes along z (NZ tiles
// of 32).  A warp keeps B of its lanes' z in registers and A of its y for the four x; C comes
// broadcast from shared memory.  part[item][m][v] gets the CTA's share of R_m[v].  Bound by
// issue and load latency at eight warps an SM (229 registers; DRAM 32 %, FP64 pipe 23 % busy at nocc=6,
// nvir=90), so the loads run one y ahead of their use: nocc=10, nvir=90 (1.28 GB, A a quarter more from
// L2) 0.45 ms, 2.8 TB/s (0.61 without the loads ahead); the three batched GEMMs with three right-hand sides and the seventy launches around them took 1.9 ms.
template <int NZ>
__global__ void __launch_bounds__(R1_THREADS, 1)
    k_r1_t3(const double *__restrict__ t3, const double *__restrict__ K, const int32_t *__restrict__ ijk, int nocc,
            int nv, int nxc, double *__restrict__ part) {
    extern __shared__ double sm[];
    double *sC = sm;                      // [3][XC][nv]
    double *sY = sC + 3 * R1_XC * nv;     // [3][nv]
    double *sZ = sY + 3 * nv;             // [warp][3][nv]
    double *sX = sZ + R1_WARPS * 3 * nv;  // [warp][3][XC]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t q = blockIdx.x / nxc;
    const int x0 = (int)(blockIdx.x % nxc) * R1_XC, nx = min(R1_XC, nv - x0);
    const int i = ijk[3 * q], j = ijk[3 * q + 1], k = ijk[3 * q + 2];
    double *out = part + (int64_t)blockIdx.x * 3 * nv;
    if ((unsigned)i >= (unsigned)nocc || (unsigned)j >= (unsigned)nocc || (unsigned)k >= (unsigned)nocc) {
        for (int e = threadIdx.x; e < 3 * nv; e += R1_THREADS) out[e] = 0.0;  // not a block of this space
        return;
    }
    const int64_t nv2 = (int64_t)nv * nv, kn = (int64_t)nocc * nocc * nv2;
    const double *E1 = K + (int64_t)(j * nocc + k) * nv2, *E2 = K + (int64_t)(i * nocc + k) * nv2,
                 *E3 = K + (int64_t)(i * nocc + j) * nv2;
    const double *A[3] = {E1, E2 + kn, E3 + 2 * kn};
    const double *B[3] = {E1 + kn, E2, E3 + kn};
    const double *C[3] = {E1 + 2 * kn, E2 + kn, E3};
    for (int e = threadIdx.x; e < 3 * R1_XC * nv; e += R1_THREADS) {
        const int m = e / (R1_XC * nv), r = e - m * R1_XC * nv, x = r / nv, y = r - x * nv;
        const double *Cm = m == 0 ? C[0] : (m == 1 ? C[1] : C[2]);
        sC[e] = x < nx ? Cm[(int64_t)(x0 + x) * nv + y] : 0.0;
    }
    double b[3][R1_XC][NZ], accX[3][R1_XC], accZ[3][NZ];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
#pragma unroll
        for (int x = 0; x < R1_XC; ++x) {
            accX[m][x] = 0.0;
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int z = lane + 32 * u;
                b[m][x][u] = (x < nx && z < nv) ? B[m][(int64_t)(x0 + x) * nv + z] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < NZ; ++u) accZ[m][u] = 0.0;
    }
    __syncthreads();
    const double *tq = t3 + (q * nv + x0) * nv2;
    double tn[R1_XC][NZ];  // the next y's elements, in flight while this one's are used
    auto fetch = [&](int y) {
#pragma unroll
        for (int x = 0; x < R1_XC; ++x)
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int z = lane + 32 * u;
                tn[x][u] = (x < nx && z < nv && y < nv) ? __ldcs(tq + x * nv2 + (int64_t)y * nv + z) : 0.0;
            }
    };
    fetch(w);
    for (int y = w; y < nv; y += R1_WARPS) {
        double t[R1_XC][NZ], a[3][NZ], accY[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int x = 0; x < R1_XC; ++x)
#pragma unroll
            for (int u = 0; u < NZ; ++u) t[x][u] = tn[x][u];
        fetch(y + R1_WARPS);
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int z = lane + 32 * u;
                a[m][u] = z < nv ? __ldg(A[m] + (int64_t)y * nv + z) : 0.0;
            }
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int x = 0; x < R1_XC; ++x) {
                const double c = sC[(m * R1_XC + x) * nv + y];
#pragma unroll
                for (int u = 0; u < NZ; ++u) {
                    accX[m][x] = fma(t[x][u], a[m][u], accX[m][x]);
                    accY[m] = fma(t[x][u], b[m][x][u], accY[m]);
                    accZ[m][u] = fma(t[x][u], c, accZ[m][u]);
                }
            }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) accY[m] += __shfl_xor_sync(0xffffffffu, accY[m], o);
            if (lane == m) sY[m * nv + y] = accY[m];
        }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
#pragma unroll
        for (int u = 0; u < NZ; ++u)
            if (lane + 32 * u < nv) sZ[(w * 3 + m) * nv + lane + 32 * u] = accZ[m][u];
#pragma unroll
        for (int x = 0; x < R1_XC; ++x) {
            double v = accX[m][x];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) sX[(w * 3 + m) * R1_XC + x] = v;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * nv; e += R1_THREADS) {
        const int m = e / nv, v = e - m * nv;
        double s = sY[e];
        for (int g = 0; g < R1_WARPS; ++g) s += sZ[g * 3 * nv + e];
        if (v >= x0 && v < x0 + nx)
            for (int g = 0; g < R1_WARPS; ++g) s += sX[(g * 3 + m) * R1_XC + v - x0];
        out[e] = s;
    }
}

// r1[o][v] += the shares of every block that holds o, weighted by its case (c1, c2, c3) = (1, 1, 1)
// for i<j<k, (1, 0, 1/2) for i=j<k, (1/2, 1, 0) for i<j=k; a fixed order of summation.
constexpr int R1_SUM = 32;  // shares summed side by side
__global__ void __launch_bounds__(32 * R1_SUM) k_r1_sum(const double *__restrict__ part, const int32_t *__restrict__ ijk,
                                                        int64_t n, int nv, int nxc, double *__restrict__ r1) {
    __shared__ double red[R1_SUM][33];
    const int o = blockIdx.x, lane = threadIdx.x & 31, g = threadIdx.x >> 5, v = blockIdx.y * 32 + lane;
    double s = 0.0;
    for (int64_t q = 0; q < n; ++q) {
        const int i = ijk[3 * q], j = ijk[3 * q + 1], k = ijk[3 * q + 2];
        if ((i != o && j != o && k != o) || (i == j && j == k)) continue;
        const double c1 = i != o ? 0.0 : (i < j ? (j < k ? 1.0 : 0.5) : 1.0);
        const double c2 = j != o || i == j ? 0.0 : 1.0;
        const double c3 = k != o || j == k ? 0.0 : (i < j ? 1.0 : 0.5);
        if (v < nv)
            for (int c = g; c < nxc; c += R1_SUM) {
                const double *p = part + (q * nxc + c) * 3 * nv + v;
                if (c1 != 0.0) s += c1 * p[0];
                if (c2 != 0.0) s += c2 * p[nv];
                if (c3 != 0.0) s += c3 * p[2 * nv];
            }
    }
    red[g][lane] = s;
    __syncthreads();
    if (g == 0 && v < nv) {
        for (int u = 1; u < R1_SUM; ++u) s += red[u][lane];
        r1[(int64_t)o * nv + v] += s;
    }
}

// r2[y,z,b,c] += alpha sum_{x,a} f[x,a] X[x,y,z,a,b,c] (distr_cc/rccsdt.py:300-316) in FP64: a thread
// per (b, c) of one (y, z), so that every element of X is read once along rows.  Bound by that
// read: nocc=10, nvir=90 (an FP32 X, 2.9 GB) 0.52 ms, where a matrix-vector product and an
// addition per x took 0.75 ms and 2 nocc launches.
constexpr int FK_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(FK_THREADS) k_r2_fock(const T *__restrict__ X, const double *__restrict__ f,
                                                        double *__restrict__ r2, int no, int nv, double alpha) {
    extern __shared__ double sf[];
    for (int i = threadIdx.x; i < no * nv; i += FK_THREADS) sf[i] = f[i];
    __syncthreads();
    const int64_t nv2 = (int64_t)nv * nv, yz = blockIdx.y, sx = (int64_t)no * no * nv2 * nv;
    const int64_t bc = (int64_t)blockIdx.x * FK_THREADS + threadIdx.x;
    if (bc >= nv2) return;
    double s = 0.0;
    for (int x = 0; x < no; ++x) {
        const T *p = X + x * sx + yz * nv2 * nv + bc;
        const double *fx = sf + x * nv;
#pragma unroll 8
        for (int a = 0; a < nv; ++a) s = fma(fx[a], (double)__ldcs(p + a * nv2), s);
    }
    r2[yz * nv2 + bc] = fma(alpha, s, r2[yz * nv2 + bc]);
}

}  // namespace dcc

using namespace dcc;

extern "C" size_t dcc_t3_r1_workspace_bytes(int64_t nblocks, int64_t nocc, int64_t nvir) {
    const int64_t nxc = (nvir + R1_XC - 1) / R1_XC;
    return (size_t)(3 * nocc * nocc * nvir * nvir + nblocks * nxc * 3 * nvir) * sizeof(double);
}

extern "C" int dcc_t3_r1(const double *t3, const double *oovv, const int32_t *ijk, int64_t nblocks, int64_t nocc,
                         int64_t nvir, double *r1, void *workspace, size_t workspace_bytes, void *stream) {
    clear_error();
    DCC_REQUIRE(nblocks >= 0 && nocc >= 0 && nvir >= 0 && nocc < 32768, DCC_ERR_SHAPE, "bad size");
    if (nblocks == 0 || nocc == 0 || nvir == 0) return DCC_OK;
    DCC_REQUIRE(t3 && oovv && ijk && r1 && workspace, DCC_ERR_NULL, "NULL buffer");
    DCC_REQUIRE(nvir <= R1_MAXNV, DCC_ERR_UNSUPPORTED, "nvir above %d", R1_MAXNV);
    DCC_REQUIRE(workspace_bytes >= dcc_t3_r1_workspace_bytes(nblocks, nocc, nvir), DCC_ERR_WORKSPACE,
                "workspace too small");
    const int nv = (int)nvir, nxc = (nv + R1_XC - 1) / R1_XC;
    DCC_REQUIRE(nblocks * nxc < (1LL << 31), DCC_ERR_SHAPE, "too many blocks");
    cudaStream_t st = as_stream(stream);
    double *K = (double *)workspace, *part = K + 3 * nocc * nocc * nvir * nvir;
    const int64_t ne = nocc * nocc * nvir * nvir;
    const unsigned gm = ceil_div(ne, 256);
    k_r1_mix<<<gm < 148 * 16 ? gm : 148 * 16, 256, 0, st>>>(oovv, K, nocc * nocc, nv);
    int rc = launch_status("t3_r1 mix");
    if (rc) return rc;
    const size_t smem = (size_t)(3 * R1_XC * nv + 3 * nv + R1_WARPS * 3 * nv + R1_WARPS * 3 * R1_XC) * sizeof(double);
    auto launch = [&](auto kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
        kern<<<(unsigned)(nblocks * nxc), R1_THREADS, smem, st>>>(t3, K, ijk, (int)nocc, nv, nxc, part);
    };
    static_assert((3 * R1_XC + 3 + R1_WARPS * 3) * R1_MAXNV * 8 + R1_WARPS * 3 * R1_XC * 8 <= 64 * 1024, "shared memory");
    if (nv <= 32)
        launch(k_r1_t3<1>);
    else if (nv <= 64)
        launch(k_r1_t3<2>);
    else if (nv <= 96)
        launch(k_r1_t3<3>);
    else
        launch(k_r1_t3<4>);
    rc = launch_status("t3_r1");
    if (rc) return rc;
    k_r1_sum<<<dim3((unsigned)nocc, (unsigned)((nv + 31) / 32)), 32 * R1_SUM, 0, st>>>(part, ijk, nblocks, nv, nxc, r1);
    return launch_status("t3_r1 sum");
}

extern "C" int dcc_t3_r2_fock(const void *X, int x_f32, const double *fock_ov, double *r2, int64_t nocc, int64_t nvir,
                              double alpha, void *stream) {
    clear_error();
    DCC_REQUIRE(nocc >= 0 && nvir >= 0 && nocc < 256 && nvir < 32768, DCC_ERR_SHAPE, "bad size");
    if (nocc == 0 || nvir == 0) return DCC_OK;
    DCC_REQUIRE(X && fock_ov && r2, DCC_ERR_NULL, "NULL buffer");
    const size_t smem = (size_t)(nocc * nvir) * sizeof(double);
    DCC_REQUIRE(smem <= 48 * 1024, DCC_ERR_UNSUPPORTED, "nocc * nvir above 6144");
    const dim3 grid(ceil_div(nvir * nvir, FK_THREADS), (unsigned)(nocc * nocc));
    if (x_f32)
        k_r2_fock<float><<<grid, FK_THREADS, smem, as_stream(stream)>>>((const float *)X, fock_ov, r2, (int)nocc,
                                                                        (int)nvir, alpha);
    else
        k_r2_fock<double><<<grid, FK_THREADS, smem, as_stream(stream)>>>((const double *)X, fock_ov, r2, (int)nocc,
                                                                         (int)nvir, alpha);
    return launch_status("t3_r2_fock");
}
