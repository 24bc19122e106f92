// W_vvvv . t3 (distr_cc/rccsdt.py:421-427) over symmetric and antisymmetric index pairs.
//
// A W_vvvv with the pair symmetry W[x,y,d,e] = W[y,x,e,d] (<xy|de> = <yx|ed>) needs half the
// multiplications: with t+-[d<=e] = t[d,e] +- t[e,d] and W+-[x<=y][d<=e] = (W[x,y,d,e] +- W[x,y,e,d]) / 2
// (the diagonal d = e once, in the plus operands),
//   r+- = sum_{d<=e} W+- t+-,   r[x,y] = r+ + r-,   r[y,x] = r+ - r-.
// Each of the three strings becomes two split GEMMs of nvir(nvir+1)/2 columns and as long a
// contraction in place of one of nvir^2 and nvir^2.  Here: the operands t+-, W+- as K-major two-piece
// splits (sums and differences in FP64, then split), and the pass that adds the six FP32 results
// (the accumulation type of the products) into r3 in FP64.  nocc=10, nvir=90: the six GEMMs 8.2 ms in
// place of 17.4 (1.4 PFLOP/s of bf16 products either way), the three strings together 12.5 in
// place of 19.5; the relative error of the result about half (2.2e-5 against 4.4e-5 at nvir=112 on
// random data: the FP32 accumulation is half as long).
#include "dcc_common.cuh"
#include "split_util.cuh"

namespace dcc {

constexpr int PR_THREADS = 256;
constexpr int PR_MAXNV = 112;  // a plane of an odd pitch and two rows of pairs in shared memory

// The four piece arrays [row][Kp] of a plus / minus operand.
struct PairOut {
    void *ph, *pl, *mh, *ml;
    int64_t Kp;
};

// Eight consecutive pieces of a row (x: plus, y: minus values), written as 16-byte packs.
template <int KIND>
__device__ __forceinline__ void pair_store(const PairOut &o, int64_t at, const double (&x)[8], const double (&y)[8]) {
    if constexpr (KIND == 0) {
        uint32_t w[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            __nv_bfloat16 h[2], l[2];
            split_bf16(x[2 * j], h[0], l[0]);
            split_bf16(x[2 * j + 1], h[1], l[1]);
            w[0][j] = (uint32_t)__bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
            w[1][j] = (uint32_t)__bfloat16_as_ushort(l[0]) | ((uint32_t)__bfloat16_as_ushort(l[1]) << 16);
            split_bf16(y[2 * j], h[0], l[0]);
            split_bf16(y[2 * j + 1], h[1], l[1]);
            w[2][j] = (uint32_t)__bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
            w[3][j] = (uint32_t)__bfloat16_as_ushort(l[0]) | ((uint32_t)__bfloat16_as_ushort(l[1]) << 16);
        }
        void *p[4] = {o.ph, o.pl, o.mh, o.ml};
#pragma unroll
        for (int a = 0; a < 4; ++a)
            *(uint4 *)((__nv_bfloat16 *)p[a] + at) = make_uint4(w[a][0], w[a][1], w[a][2], w[a][3]);
    } else {
        float w[4][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            split_tf32(x[j], w[0][j], w[1][j]);
            split_tf32(y[j], w[2][j], w[3][j]);
        }
        void *p[4] = {o.ph, o.pl, o.mh, o.ml};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            ((float4 *)((float *)p[a] + at))[0] = make_float4(w[a][0], w[a][1], w[a][2], w[a][3]);
            ((float4 *)((float *)p[a] + at))[1] = make_float4(w[a][4], w[a][5], w[a][6], w[a][7]);
        }
    }
}

// Pair table entry: d << 8 | e, d <= e (lexicographic); 0xFFFF past the last pair.
__device__ __forceinline__ bool pair_of(uint16_t v, int &d, int &e) {
    d = v >> 8;
    e = v & 255;
    return v != 0xFFFFu;
}

// visit(d, e, src[d ds + e]) over a plane, rows over the warps, four rows' loads in flight a lane.
template <typename Visit>
__device__ __forceinline__ void plane_each(const double *__restrict__ src, int64_t ds, int nv, Visit visit) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int NW = PR_THREADS / 32, R = 4;
    for (int e0 = 0; e0 < nv; e0 += 64)
        for (int d0 = w; d0 < nv; d0 += NW * R) {
            double v[R][2];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int d = d0 + NW * r, e = e0 + 32 * u + lane;
                    v[r][u] = (d < nv && e < nv) ? __ldcs(src + d * ds + e) : 0.0;
                }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int d = d0 + NW * r, e = e0 + 32 * u + lane;
                    if (d < nv && e < nv) visit(d, e, v[r][u]);
                }
        }
}

// t+- of rows (q, f) whose plane (d, e) has e contiguous: t3[q][f fs + d ds + e].  One CTA per row:
// the plane is staged at an odd pitch (both orders read free of bank conflicts), then written as
// 16-byte packs.  Bound by the latency of a plane's loads at three CTAs an SM (its shared memory; DRAM
// 35 % busy at nocc=6, nvir=90): nocc=10, nvir=90 0.64 ms, 0.3 at 6.5 TB/s (8 bytes read, 4 written per
// element of t3).
template <int KIND>
__global__ void __launch_bounds__(PR_THREADS) k_pair_rows(const double *__restrict__ t3, const uint16_t *__restrict__ tab,
                                                          int nv, int64_t fs, int64_t ds, PairOut o) {
    extern __shared__ double S[];
    const int P = nv | 1;
    const int64_t row = blockIdx.x, q = row / nv;
    plane_each(t3 + q * nv * nv * nv + (row - q * nv) * fs, ds, nv, [&](int d, int e, double v) { S[d * P + e] = v; });
    __syncthreads();
    for (int64_t p = 8 * threadIdx.x; p < o.Kp; p += 8 * PR_THREADS) {
        double x[8], y[8];
        const uint4 t = __ldg((const uint4 *)(tab + p));
        const uint32_t tw[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int d, e;
            const bool ok = pair_of((uint16_t)(tw[j >> 1] >> (16 * (j & 1))), d, e);
            const double u = ok ? S[d * P + e] : 0.0, v = ok ? S[e * P + d] : 0.0;
            x[j] = d == e ? u : u + v;
            y[j] = d == e ? 0.0 : u - v;
        }
        pair_store<KIND>(o, row * o.Kp + p, x, y);
    }
}

// t+- of rows (q, c) of t3[q][d][e][c]: a warp takes 32 rows c and 16 pairs, so that both elements of
// every pair are read as runs along c and each row gets whole 32-byte sectors.
template <int KIND>
__global__ void __launch_bounds__(PR_THREADS) k_pair_cols(const double *__restrict__ t3, const uint16_t *__restrict__ tab,
                                                          int64_t nblk, int nv, PairOut o) {
    const int lane = threadIdx.x & 31;
    const int64_t npc = (o.Kp + 15) / 16, ncc = (nv + 31) / 32, total = nblk * ncc * npc;
    for (int64_t t = (int64_t)blockIdx.x * (PR_THREADS / 32) + (threadIdx.x >> 5); t < total;
         t += (int64_t)gridDim.x * (PR_THREADS / 32)) {
        const int64_t pc = t % npc, r = t / npc, q = r / ncc;
        const int c = (int)(r - q * ncc) * 32 + lane;
        const bool cv = c < nv;
        const double *src = t3 + q * nv * nv * nv + (cv ? c : 0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t p = pc * 16 + 8 * h;
            if (p >= o.Kp) break;  // Kp is a multiple of 8
            double x[8], y[8], u[8], v[8];
            int dd[8], ee[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {  // the table entry is the warp's
                const bool ok = pair_of(__ldg(tab + p + j), dd[j], ee[j]) && cv;
                u[j] = ok ? __ldg(src + ((int64_t)dd[j] * nv + ee[j]) * nv) : 0.0;
                v[j] = ok ? __ldg(src + ((int64_t)ee[j] * nv + dd[j]) * nv) : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                x[j] = dd[j] == ee[j] ? u[j] : u[j] + v[j];
                y[j] = dd[j] == ee[j] ? 0.0 : u[j] - v[j];
            }
            if (cv) pair_store<KIND>(o, (q * nv + c) * o.Kp + p, x, y);
        }
    }
}

// W+- of the pairs x <= y (one CTA each), with half of F_vv's three strings in each of the three
// contractions: W + (F[x,d] delta(y,e) + delta(x,d) F[y,e]) / 2.  sym[0], sym[1] (zeroed by the
// caller) get the bits of max |W[x,y,d,e] - W[y,x,e,d]| and max |W| (NaN above every number), by
// which the caller decides whether the pairs stand for W.
template <int KIND>
__global__ void __launch_bounds__(PR_THREADS) k_pair_w(const double *__restrict__ W, const double *__restrict__ F,
                                                       const uint16_t *__restrict__ tab, int nv, PairOut o,
                                                       unsigned long long *sym) {
    extern __shared__ double S[];
    __shared__ unsigned long long red[2][PR_THREADS / 32];
    const int P = nv | 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x, y;
    pair_of(tab[blockIdx.x], x, y);
    unsigned long long dev = 0, big = 0;
    auto bits = [](double v) { return (unsigned long long)__double_as_longlong(fabs(v)); };
    plane_each(W + ((int64_t)x * nv + y) * nv * nv, nv, nv, [&](int d, int e, double v) {
        S[d * P + e] = v;
        const unsigned long long b = bits(v);
        big = b > big ? b : big;
    });
    __syncthreads();
    plane_each(W + ((int64_t)y * nv + x) * nv * nv, nv, nv, [&](int d, int e, double v) {
        const unsigned long long a = bits(v - S[e * P + d]);
        dev = a > dev ? a : dev;
    });
    for (int k = 16; k > 0; k >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, dev, k), b = __shfl_xor_sync(0xffffffffu, big, k);
        dev = a > dev ? a : dev;
        big = b > big ? b : big;
    }
    if (lane == 0) {
        red[0][w] = dev;
        red[1][w] = big;
    }
    __syncthreads();  // every element compared before F goes in
    if (threadIdx.x == 0) {
        for (int k = 1; k < PR_THREADS / 32; ++k) {
            dev = red[0][k] > dev ? red[0][k] : dev;
            big = red[1][k] > big ? red[1][k] : big;
        }
        atomicMax(sym, dev);
        atomicMax(sym + 1, big);
    }
    if (F) {
        for (int d = threadIdx.x; d < nv; d += PR_THREADS) S[d * P + y] += 0.5 * F[(int64_t)x * nv + d];
        __syncthreads();
        for (int e = threadIdx.x; e < nv; e += PR_THREADS) S[x * P + e] += 0.5 * F[(int64_t)y * nv + e];
        __syncthreads();
    }
    for (int64_t p = 8 * threadIdx.x; p < o.Kp; p += 8 * PR_THREADS) {
        double u[8], v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int d, e;
            const bool ok = pair_of(__ldg(tab + p + j), d, e);
            const double a = ok ? S[d * P + e] : 0.0, b = ok ? S[e * P + d] : 0.0;
            u[j] = d == e ? a : 0.5 * (a + b);
            v[j] = d == e ? 0.0 : 0.5 * (a - b);
        }
        pair_store<KIND>(o, (int64_t)blockIdx.x * o.Kp + p, u, v);
    }
}

// r3[q][a][b][c] += E1[a,b] + E2[a,c] + E3[b,c] with E[x,y] = C+ + C- (x < y), C+ - C- (x > y), C+ (x = y)
// of the unordered pair: C1 as [q][pair][c], C2 as [q][pair][b], C3 as [q][a][pair], so that all but
// the transposition of C2 (through shared memory) is read along rows, and a block's 90 or so CTAs
// share its 9 MB of results in L2 (with q innermost, [pair][q][c], every 360-byte run was its own
// DRAM page: 4.0 ms).  One CTA per plane (q, a), two rows' loads in flight a lane.  Bound by
// the latency of its loads at two CTAs an SM (registers and the transposed plane; DRAM 26 % busy at
// nocc=6, nvir=90): nocc=10, nvir=90 (4.5 GB) 2.16 ms.
struct PairC {
    const float *p[3], *m[3];
};
__global__ void __launch_bounds__(PR_THREADS, 2) k_pair_add(PairC C, double *__restrict__ r3, int nv, int np,
                                                            double alpha) {
    extern __shared__ double T2[];  // [c][b], then C3's two rows
    constexpr int NW = PR_THREADS / 32, R = 2, NZ = (PR_MAXNV + 31) / 32;
    const int P = nv | 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *Tp = (float *)(T2 + nv * P), *Tm = Tp + np;
    const int64_t row = blockIdx.x, q = row / nv;
    const int a = (int)(row - q * nv);
    auto pr = [&](int x, int y) {
        const int lo = x < y ? x : y, hi = x < y ? y : x;
        return lo * nv - lo * (lo - 1) / 2 + hi - lo;
    };
    auto val = [&](float p, float m, int x, int y) {
        return x == y ? (double)p : (x < y ? (double)p + (double)m : (double)p - (double)m);
    };
    // (x, lane + 32 u) of rows x0, x0 + NW, ... of the pairs (a, x) of one string
    float vp[R][NZ], vm[R][NZ];
    auto fetch = [&](int s, int x0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int x = x0 + NW * r;
            const int64_t at = (q * np + pr(a, x < nv ? x : 0)) * nv;
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int i = lane + 32 * u;
                const bool ok = x < nv && i < nv;
                vp[r][u] = ok ? __ldg(C.p[s] + at + i) : 0.f;
                vm[r][u] = ok ? __ldg(C.m[s] + at + i) : 0.f;
            }
        }
    };
    for (int i = threadIdx.x; i < np; i += PR_THREADS) {
        Tp[i] = __ldcs(C.p[2] + row * np + i);
        Tm[i] = __ldcs(C.m[2] + row * np + i);
    }
    for (int c0 = w; c0 < nv; c0 += NW * R) {
        fetch(1, c0);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int c = c0 + NW * r, b = lane + 32 * u;
                if (c < nv && b < nv) T2[c * P + b] = val(vp[r][u], vm[r][u], a, c);
            }
    }
    __syncthreads();
    for (int b0 = w; b0 < nv; b0 += NW * R) {
        double old[R][NZ];
        fetch(0, b0);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int b = b0 + NW * r, c = lane + 32 * u;
                old[r][u] = (b < nv && c < nv) ? r3[(row * nv + b) * nv + c] : 0.0;
            }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < NZ; ++u) {
                const int b = b0 + NW * r, c = lane + 32 * u;
                if (b >= nv || c >= nv) continue;
                const int i = pr(b, c);
                const double e = val(vp[r][u], vm[r][u], a, b) + T2[c * P + b] + val(Tp[i], Tm[i], b, c);
                r3[(row * nv + b) * nv + c] = fma(alpha, e, old[r][u]);
            }
    }
}

// The small matrices of the residual's OO contractions in one launch (some fifteen element-wise
// launches otherwise, most of the host time of a small molecule's residual):
//   G2[i,a,l,d] = -(W_ovov[l,a,i,d] + W_ovvo[l,a,d,i]) / 2,   Wh = W_ovvo / 2,
//   A[(i,j)][(l,m)] = (W_oooo[l,m,i,j] - F_oo[l,i] delta(m,j)) / 2,
// and the bits of max |W_oooo[l,m,i,j] - W_oooo[m,l,j,i]| / 2 and max |W_oooo| in sym[0..1] (zeroed
// by the caller), by which the caller decides whether A stands for W_oooo.
__global__ void __launch_bounds__(256) k_oo_small(const double *__restrict__ Wov, const double *__restrict__ Wvo,
                                                  const double *__restrict__ Woo, const double *__restrict__ F, int no,
                                                  int nv, double *__restrict__ G2, double *__restrict__ Wh,
                                                  double *__restrict__ A, unsigned long long *sym) {
    const int64_t n1 = (int64_t)no * no * nv * nv, n2 = (int64_t)no * no * no * no;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = first; e < n1; e += step) {
        Wh[e] = 0.5 * Wvo[e];
        const int d = (int)(e % nv), l = (int)((e / nv) % no), a = (int)((e / ((int64_t)nv * no)) % nv),
                  i = (int)(e / ((int64_t)nv * no * nv));
        const int64_t la = (int64_t)l * nv + a;
        G2[e] = -0.5 * (Wov[(la * no + i) * nv + d] + Wvo[(la * nv + d) * no + i]);
    }
    unsigned long long dev = 0, big = 0;
    for (int64_t e = first; e < n2; e += step) {
        const int m = (int)(e % no), l = (int)((e / no) % no), j = (int)((e / ((int64_t)no * no)) % no),
                  i = (int)(e / ((int64_t)no * no * no));
        const double w = Woo[(((int64_t)l * no + m) * no + i) * no + j], wt = Woo[(((int64_t)m * no + l) * no + j) * no + i];
        A[e] = 0.5 * w - (m == j ? 0.5 * F[l * no + i] : 0.0);
        const unsigned long long x = (unsigned long long)__double_as_longlong(fabs(0.5 * (w - wt))),
                                 y = (unsigned long long)__double_as_longlong(fabs(w));
        dev = x > dev ? x : dev;
        big = y > big ? y : big;
    }
    for (int k = 16; k > 0; k >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, dev, k), y = __shfl_xor_sync(0xffffffffu, big, k);
        dev = x > dev ? x : dev;
        big = y > big ? y : big;
    }
    if ((threadIdx.x & 31) == 0 && big != 0) {  // a warp without elements adds nothing
        atomicMax(sym, dev);
        atomicMax(sym + 1, big);
    }
}

template <typename K>
static void pair_smem(K kern, size_t bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace dcc

using namespace dcc;

static int pair_check(int64_t nblocks, int64_t nvir, int64_t Kp, int kind, const uint16_t *pairs) {
    DCC_REQUIRE(kind == 0 || kind == 1, DCC_ERR_UNSUPPORTED, "kind must be 0 (bf16x3) or 1 (tf32x3)");
    DCC_REQUIRE(nblocks >= 0 && nvir >= 1 && nblocks * nvir < (1ll << 31), DCC_ERR_SHAPE, "bad size");
    DCC_REQUIRE(nvir <= PR_MAXNV, DCC_ERR_UNSUPPORTED, "nvir above %d", PR_MAXNV);
    DCC_REQUIRE(Kp >= nvir * (nvir + 1) / 2 && Kp % 8 == 0, DCC_ERR_SHAPE, "Kp below the pairs or not a multiple of 8");
    DCC_REQUIRE(pairs && ((uintptr_t)pairs & 15) == 0, DCC_ERR_NULL, "NULL or misaligned pair table");
    return DCC_OK;
}

static int pair_out(void *const *pieces, int64_t Kp, PairOut &o) {
    DCC_REQUIRE(pieces, DCC_ERR_NULL, "NULL pieces");
    for (int i = 0; i < 4; i++)
        DCC_REQUIRE(pieces[i] && ((uintptr_t)pieces[i] & 15) == 0, DCC_ERR_NULL, "NULL or misaligned piece array");
    o = PairOut{pieces[0], pieces[1], pieces[2], pieces[3], Kp};
    return DCC_OK;
}

extern "C" int dcc_t3_pair_split(const double *t3, int string, const uint16_t *pairs, int64_t nblocks, int64_t nvir,
                                 int64_t Kp, void *const *pieces, int kind, void *stream) {
    clear_error();
    int rc = pair_check(nblocks, nvir, Kp, kind, pairs);
    if (rc) return rc;
    DCC_REQUIRE(string >= 0 && string <= 2, DCC_ERR_SHAPE, "string must be 0, 1 or 2");
    if (nblocks == 0) return DCC_OK;
    DCC_REQUIRE(t3, DCC_ERR_NULL, "NULL t3");
    PairOut o;
    if ((rc = pair_out(pieces, Kp, o))) return rc;
    cudaStream_t st = as_stream(stream);
    const int nv = (int)nvir;
    if (string == 0) {
        const int64_t warps = nblocks * ((nv + 31) / 32) * ((Kp + 15) / 16), ctas = (warps + 7) / 8;
        const unsigned grid = (unsigned)(ctas < 148 * 16 ? ctas : 148 * 16);
        if (kind == 0)
            k_pair_cols<0><<<grid, PR_THREADS, 0, st>>>(t3, pairs, nblocks, nv, o);
        else
            k_pair_cols<1><<<grid, PR_THREADS, 0, st>>>(t3, pairs, nblocks, nv, o);
        return launch_status("t3_pair_split");
    }
    const size_t smem = (size_t)nv * (nv | 1) * sizeof(double);
    const int64_t fs = string == 1 ? nvir : nvir * nvir, ds = string == 1 ? nvir * nvir : nvir;
    const unsigned grid = (unsigned)(nblocks * nvir);
    if (kind == 0) {
        pair_smem(k_pair_rows<0>, smem);
        k_pair_rows<0><<<grid, PR_THREADS, smem, st>>>(t3, pairs, nv, fs, ds, o);
    } else {
        pair_smem(k_pair_rows<1>, smem);
        k_pair_rows<1><<<grid, PR_THREADS, smem, st>>>(t3, pairs, nv, fs, ds, o);
    }
    return launch_status("t3_pair_split");
}

extern "C" int dcc_wvvvv_pair_split(const double *W, const double *F, const uint16_t *pairs, int64_t nvir, int64_t Kp,
                                    void *const *pieces, int kind, uint64_t *sym, void *stream) {
    clear_error();
    int rc = pair_check(1, nvir, Kp, kind, pairs);
    if (rc) return rc;
    DCC_REQUIRE(W && sym, DCC_ERR_NULL, "NULL buffer");
    PairOut o;
    if ((rc = pair_out(pieces, Kp, o))) return rc;
    cudaStream_t st = as_stream(stream);
    const int nv = (int)nvir;
    const size_t smem = (size_t)nv * (nv | 1) * sizeof(double);
    const unsigned grid = (unsigned)(nvir * (nvir + 1) / 2);
    unsigned long long *s = (unsigned long long *)sym;
    if (kind == 0) {
        pair_smem(k_pair_w<0>, smem);
        k_pair_w<0><<<grid, PR_THREADS, smem, st>>>(W, F, pairs, nv, o, s);
    } else {
        pair_smem(k_pair_w<1>, smem);
        k_pair_w<1><<<grid, PR_THREADS, smem, st>>>(W, F, pairs, nv, o, s);
    }
    return launch_status("wvvvv_pair_split");
}

extern "C" int dcc_t3_pair_add(const float *const *plus, const float *const *minus, double *r3, int64_t nblocks,
                               int64_t nvir, double alpha, void *stream) {
    clear_error();
    DCC_REQUIRE(nblocks >= 0 && nvir >= 1 && nvir <= PR_MAXNV && nblocks * nvir < (1ll << 31), DCC_ERR_SHAPE, "bad size");
    if (nblocks == 0) return DCC_OK;
    DCC_REQUIRE(plus && minus && r3, DCC_ERR_NULL, "NULL buffer");
    PairC C;
    for (int i = 0; i < 3; i++) {
        DCC_REQUIRE(plus[i] && minus[i], DCC_ERR_NULL, "NULL result");
        C.p[i] = plus[i];
        C.m[i] = minus[i];
    }
    const int nv = (int)nvir, np = nv * (nv + 1) / 2;
    const size_t smem = (size_t)nv * (nv | 1) * sizeof(double) + 2 * (size_t)np * sizeof(float);
    pair_smem(k_pair_add, smem);
    k_pair_add<<<(unsigned)(nblocks * nvir), PR_THREADS, smem, as_stream(stream)>>>(C, r3, nv, np, alpha);
    return launch_status("t3_pair_add");
}

extern "C" int dcc_t3_oo_operands(const double *W_ovov, const double *W_ovvo, const double *W_oooo, const double *F_oo,
                                  int64_t nocc, int64_t nvir, double *G2, double *Wvo_half, double *A, uint64_t *sym,
                                  void *stream) {
    clear_error();
    DCC_REQUIRE(nocc >= 0 && nvir >= 0 && nocc < 4096 && nvir < 4096, DCC_ERR_SHAPE, "bad size");
    if (nocc == 0 || nvir == 0) return DCC_OK;
    DCC_REQUIRE(W_ovov && W_ovvo && W_oooo && F_oo && G2 && Wvo_half && A && sym, DCC_ERR_NULL, "NULL buffer");
    const int64_t n1 = nocc * nocc * nvir * nvir, n2 = nocc * nocc * nocc * nocc, n = n1 > n2 ? n1 : n2;
    const unsigned grid = ceil_div(n, 256);
    k_oo_small<<<grid < 148 * 8 ? grid : 148 * 8, 256, 0, as_stream(stream)>>>(
        W_ovov, W_ovvo, W_oooo, F_oo, (int)nocc, (int)nvir, G2, Wvo_half, A, (unsigned long long *)sym);
    return launch_status("t3_oo_operands");
}
