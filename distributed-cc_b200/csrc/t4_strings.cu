// The per-block strings of compute_r4_tri (distr_cc/rccsdtq.py:862-1055) in ONE
// persistent launch over the stored T4 blocks, FP64 on the tensor cores.
//
// The reference walks its stored blocks (i<=j<=k<=l) and, for each, adds about a
// hundred strings  r4[q][a,b,c,d] += alpha W[..] . T[..]  whose operands are
// slices of full tensors at the block's occupied indices.  Every such string is a
// small GEMM over the block's virtual indices: the output letters that sit in W
// are its rows, those in T its columns, the summed letters (one or two of e, f,
// m, n) its contraction.  Here one CTA owns the output rows a in [a0, a0+na) of
// one stored block in shared memory and runs every string of a descriptor table
// over it; the block is written once at the end.
//
// Consecutive strings with the same row and column letters (fields 20, 28, 29) form a
// run: a warp keeps its tile of the run's GEMM in registers (up to 16 8x8 accumulators of
// mma.m8n8k4.f64) through all of the run's strings and pairs and adds it into the shared
// accumulator once, so the whole table costs some thirty barriers and shared-memory
// updates instead of one per string and pair, and a string costs its operand loads and
// matrix instructions alone.  Operands are read in place through strides (they stay in
// L1/L2: at nvir ~ 11 the intermediates are a few MB); the plan orders columns and the
// contraction so that the lanes of a fragment load read neighbouring elements of T or W.
// A run whose GEMM has one row (the F_oo / W_oooo strings: no output letter in W) is a sum
// of scaled vectors and runs on the FP64 lanes.
//
// What bounds it: the latency of operand loads at sixteen warps an SM (16 GB from L2 at nocc=7,
// nvir=11, 17 % of its rate; DRAM 4 %); the contractions are short (7 to 121 summed values).  Measured (nocc=7, nvir=11, 161 blocks, B200): the kernel 3.5 ms, against
// 8.3 ms with FP64 lanes, one barrier and one shared-memory update per string and pair; at
// nocc=5, nvir=8 0.47 against 2.2 ms.
//
// The W_ovov / W_voov strings of the OO batch (distr_cc/rccsdtq.py:1062-1349) take a
// stored SOURCE block and an occupied m per term: they run in "pair mode", once for
// every (source, m) pair that the output block's sparse pair list holds for the
// string's group (the reference's masked prefactor slots, only the nonzero ones).
// The F_oo / W_oooo prefactor strings are plain strings over the unpacked T4 of every
// ordering.
//
// A descriptor is 32 int64 (DCC_T4S_DESC_LEN; layout in include/dcc_b200.h).  Every
// string is checked in the kernel before it runs: operand indices, non-negative
// strides, letters in exactly one operand, and the largest offset it can reach
// inside its operand's element count; a string that fails is skipped and sets bit
// 2 of *status, a block whose occupied indices fall outside [0, nocc) sets bit 1, a pair
// (or pair range) that fails the same checks is skipped and sets bit 4.
#include "dcc_common.cuh"
#include "dcc_b200.h"

namespace dcc {

constexpr int T4S_THREADS = 256;
constexpr int T4S_MAXOPS = 32;
constexpr int T4S_DESC = 32;
constexpr int64_t T4S_SMEM_MAX = 200 * 1024;

struct T4StrOps {
    const double *p[T4S_MAXOPS];
    int64_t n[T4S_MAXOPS];
    int nops;
};

__device__ __forceinline__ int t4s_ostride(int x, int nv) {  // accumulator stride of output letter x
    return x == 0 ? nv * nv * nv : (x == 1 ? nv * nv : (x == 2 ? nv : 1));
}

// One string of the table, decoded and checked for this CTA's block (shared memory).
struct T4Rec {
    const double *W, *T;  // operands at the block's occupied indices
    double alpha;
    int64_t wm, tq;          // pair mode: strides of m (W) and of the source block (T)
    int64_t wroom, troom;    // elements of W / T past the largest offset the string reaches
    int rws[4], cts[4];      // strides of the row / column letters by position
    int K0, wk0, tk0, K1, wk1, tk1;
    int mask, rord, cord;    // the run key
    int p0, p1, mode, ok;
};
constexpr int T4S_BATCH = 96;  // strings decoded at a time

struct T4Run {  // the GEMM of a run: extents and accumulator strides by position, its tile shape, its end
    int rext[4], cext[4], ros[4], cos[4];
    int R, C, shape, end;
};

// Decode and check descriptor d for block q, rows [a0, a0 + na); returns false when it must
// not run.
__device__ bool t4s_decode(const T4StrOps &ops, const int64_t *d, const int *occ, int q, int a0, int na, int nv,
                           const int32_t *pair_off, int ngroups, int npairs, T4Rec &o, int *status) {
    const int64_t wop = d[0], top = d[1], mask = d[20], K0 = d[21], wk0 = d[22], tk0 = d[23], K1 = d[24], wk1 = d[25],
                  tk1 = d[26], rord = d[28], cord = d[29], wm = d[30], mode = d[31];
    bool ok = wop >= 0 && wop < ops.nops && top >= 0 && top < ops.nops && mask >= 0 && mask < 16 && K0 >= 1 &&
              K1 >= 1 && wk0 >= 0 && tk0 >= 0 && wk1 >= 0 && tk1 >= 0 && d[10] >= 0 && d[11] >= 0 && rord >= 0 &&
              rord < 65536 && cord >= 0 && cord < 65536 && wm >= 0 && mode >= 0 && mode <= ngroups;
    int64_t wb = 0, tb = 0, wmax = 0, tmax = 0;
    int seen_r = 0, seen_c = 0, npos_r = 0, npos_c = 0;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int64_t ws = d[2 + x], ts = d[6 + x], wv = d[12 + x], tv = d[16 + x];
        const bool inw = (mask >> x) & 1;
        ok = ok && ws >= 0 && ts >= 0 && wv >= 0 && tv >= 0 && (inw ? tv == 0 : wv == 0);
        wb += ws * occ[x];
        tb += ts * occ[x];
        const int ex = x == 0 ? na : nv;
        wmax += wv * (ex - 1);
        tmax += tv * (ex - 1);
        const int xr = (int)((rord >> (4 * x)) & 15) - 1, xc = (int)((cord >> (4 * x)) & 15) - 1;
        if (xr >= 0) {
            npos_r++;
            seen_r |= 1 << (xr & 7);
            ok = ok && xr < 4;
        }
        if (xc >= 0) {
            npos_c++;
            seen_c |= 1 << (xc & 7);
            ok = ok && xc < 4;
        }
        o.rws[x] = (xr >= 0 && xr < 4) ? (int)d[12 + xr] : 0;
        o.cts[x] = (xc >= 0 && xc < 4) ? (int)d[16 + xc] : 0;
    }
    o.mask = (int)mask;
    o.rord = (int)rord;
    o.cord = (int)cord;
    o.mode = (int)mode;
    o.p0 = 0;
    o.p1 = 1;
    // the row order lists the letters of W once each, the column order those of T
    ok = ok && seen_r == (int)mask && seen_c == (int)(15 & ~mask) && npos_r == __popc(seen_r) &&
         npos_c == __popc(seen_c);
    if (ok) {
        wb += d[10] * q + d[12] * a0;
        tb += (mode == 0 ? d[11] * q : 0) + d[16] * a0;  // pair mode: field 11 strides the source block
        wmax += wb + wk0 * (K0 - 1) + wk1 * (K1 - 1);
        tmax += tb + tk0 * (K0 - 1) + tk1 * (K1 - 1);
        ok = wmax < ops.n[wop] && tmax < ops.n[top];
    }
    if (!ok) {
        atomicOr(status, 2);
        return false;
    }
    o.W = ops.p[wop] + wb;
    o.T = ops.p[top] + tb;
    o.alpha = __longlong_as_double((long long)d[27]);
    o.wroom = ops.n[wop] - wmax;
    o.troom = ops.n[top] - tmax;
    // operands hold fewer than 2^31 elements: a longer pair stride fails for every index but 0
    o.wm = wm < (1ll << 31) ? wm : (1ll << 31);
    o.tq = d[11] < (1ll << 31) ? d[11] : (1ll << 31);
    o.K0 = (int)K0;
    o.wk0 = (int)wk0;
    o.tk0 = (int)tk0;
    o.K1 = (int)K1;
    o.wk1 = (int)wk1;
    o.tk1 = (int)tk1;
    if (mode > 0) {  // once per (source block, m) pair of group mode-1 of this block
        const int32_t *po = pair_off + (int64_t)q * (ngroups + 1) + (mode - 1);
        o.p0 = po[0];
        o.p1 = po[1];
        if (o.p0 < 0 || o.p1 < o.p0 || o.p1 > npairs) {
            atomicOr(status, 4);
            return false;
        }
    }
    return true;
}

// Operand pointers of pair pr of string r (the string itself when it is not in pair mode);
// false when the pair fails its checks.
__device__ __forceinline__ bool t4s_pair(const T4Rec &r, int pr, const int32_t *__restrict__ pair_sm, int nocc,
                                         const double *&W, const double *&T, int *status) {
    W = r.W;
    T = r.T;
    if (r.mode == 0) return true;
    const int src = pair_sm[2 * (int64_t)pr], m = pair_sm[2 * (int64_t)pr + 1];
    if (src < 0 || m < 0 || m >= nocc || r.wm * m >= r.wroom || r.tq * src >= r.troom) {
        atomicOr(status, 4);
        return false;
    }
    W += r.wm * m;
    T += r.tq * src;
    return true;
}

// The digits of index x in the mixed radix ext, one byte per position (nvir <= 29).
__device__ __forceinline__ uint32_t t4s_digits(int x, const int *ext) {
    uint32_t pk = 0;
#pragma unroll
    for (int p = 3; p >= 0; --p) {
        const int y = x / ext[p];
        pk |= (uint32_t)(x - y * ext[p]) << (8 * p);
        x = y;
    }
    return pk;
}
__device__ __forceinline__ int t4s_dot(uint32_t pk, const int *st) {
    return (int)(pk & 255u) * st[0] + (int)((pk >> 8) & 255u) * st[1] + (int)((pk >> 16) & 255u) * st[2] +
           (int)(pk >> 24) * st[3];
}

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// One run on warp tiles of 8 RT rows x 8 CT columns; AHEAD: with the loads of a step issued during
// the products of the one before.  Fragments of m8n8k4: lane l holds
// A[row l/4][k l%4], B[k l%4][col l/4] and D[row l/4][cols 2(l%4), 2(l%4)+1].
template <bool AHEAD, int RT, int CT>
__device__ __forceinline__ void t4s_run(double *acc, const T4Rec *rec, int r0, int r1, const T4Run &g,
                                        const int32_t *__restrict__ pair_sm, int nocc, int warp, int lane, int *status) {
    const int nrt = (g.R + 8 * RT - 1) / (8 * RT), nct = (g.C + 8 * CT - 1) / (8 * CT);
    for (int tile = warp; tile < nrt * nct; tile += T4S_THREADS / 32) {
        const int rb = (tile / nct) * 8 * RT + (lane >> 2), cb = (tile % nct) * 8 * CT;
        uint32_t rpk[RT], cpk[CT];
#pragma unroll
        for (int u = 0; u < RT; ++u) rpk[u] = t4s_digits(rb + 8 * u < g.R ? rb + 8 * u : 0, g.rext);
#pragma unroll
        for (int v = 0; v < CT; ++v) {
            const int c = cb + 8 * v + (lane >> 2);
            cpk[v] = t4s_digits(c < g.C ? c : 0, g.cext);
        }
        double d[RT][CT][2];
#pragma unroll
        for (int u = 0; u < RT; ++u)
#pragma unroll
            for (int v = 0; v < CT; ++v) d[u][v][0] = d[u][v][1] = 0.0;
        for (int s = r0; s < r1; ++s) {
            const T4Rec &r = rec[s];
            if (!r.ok) continue;
            int wo[RT], to[CT];
#pragma unroll
            for (int u = 0; u < RT; ++u) wo[u] = t4s_dot(rpk[u], r.rws);
#pragma unroll
            for (int v = 0; v < CT; ++v) to[v] = t4s_dot(cpk[v], r.cts);
            const int K0 = r.K0, K1 = r.K1, wk0 = r.wk0, tk0 = r.tk0, wk1 = r.wk1, tk1 = r.tk1;
            const int64_t KK = (int64_t)K0 * K1;
            const double alpha = r.alpha;
            for (int pr = r.p0; pr < r.p1; ++pr) {
                const double *W, *T;
                if (!t4s_pair(r, pr, pair_sm, nocc, W, T, status)) continue;
                int k0 = lane & 3, k1 = 0;  // this lane's summed values of the step
                while (k0 >= K0) {
                    k0 -= K0;
                    k1++;
                }
                double a[RT], b[CT];
                auto fetch = [&]() {  // this lane's elements of the step; zeros past the last summed value
                    if (k1 < K1) {
                        const double *Wk = W + (k0 * wk0 + k1 * wk1), *Tk = T + (k0 * tk0 + k1 * tk1);
#pragma unroll
                        for (int u = 0; u < RT; ++u) a[u] = alpha * __ldg(Wk + wo[u]);
#pragma unroll
                        for (int v = 0; v < CT; ++v) b[v] = __ldg(Tk + to[v]);
                    } else {
#pragma unroll
                        for (int u = 0; u < RT; ++u) a[u] = 0.0;
#pragma unroll
                        for (int v = 0; v < CT; ++v) b[v] = 0.0;
                    }
                    k0 += 4;
                    while (k0 >= K0) {
                        k0 -= K0;
                        k1++;
                    }
                };
                if constexpr (AHEAD) {
                    fetch();
                    for (int64_t kb = 0; kb < KK; kb += 4) {
                        double x[RT], y[CT];
#pragma unroll
                        for (int u = 0; u < RT; ++u) x[u] = a[u];
#pragma unroll
                        for (int v = 0; v < CT; ++v) y[v] = b[v];
                        fetch();  // the next step's loads, in flight during this one's products
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < RT; ++u)
#pragma unroll
                            for (int v = 0; v < CT; ++v) dmma(d[u][v][0], d[u][v][1], x[u], y[v]);
                    }
                } else {
                    for (int64_t kb = 0; kb < KK; kb += 4) {
                        fetch();
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < RT; ++u)
#pragma unroll
                            for (int v = 0; v < CT; ++v) dmma(d[u][v][0], d[u][v][1], a[u], b[v]);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < CT; ++v)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = cb + 8 * v + 2 * (lane & 3) + j;
                if (c >= g.C) continue;
                const int oc = t4s_dot(t4s_digits(c, g.cext), g.cos);
#pragma unroll
                for (int u = 0; u < RT; ++u)
                    if (rb + 8 * u < g.R) acc[t4s_dot(rpk[u], g.ros) + oc] += d[u][v][j];
            }
    }
}

// A run whose GEMM has one row: acc[c] += sum of scalar x vector, columns on the lanes.
__device__ __forceinline__ void t4s_run_vector(double *acc, const T4Rec *rec, int r0, int r1, const T4Run &g,
                                               const int32_t *__restrict__ pair_sm, int nocc, int *status) {
    constexpr int V = 8;  // columns of a thread in flight
    for (int c0 = threadIdx.x; c0 < g.C; c0 += V * T4S_THREADS) {
        uint32_t cpk[V];
        double x[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int c = c0 + v * T4S_THREADS;
            cpk[v] = t4s_digits(c < g.C ? c : 0, g.cext);
            x[v] = 0.0;
        }
        for (int s = r0; s < r1; ++s) {
            const T4Rec &r = rec[s];
            if (!r.ok) continue;
            int to[V];
#pragma unroll
            for (int v = 0; v < V; ++v) to[v] = t4s_dot(cpk[v], r.cts);
            for (int pr = r.p0; pr < r.p1; ++pr) {
                const double *W, *T;
                if (!t4s_pair(r, pr, pair_sm, nocc, W, T, status)) continue;
                for (int k1 = 0; k1 < r.K1; ++k1)
                    for (int k0 = 0; k0 < r.K0; ++k0) {
                        const double w = r.alpha * __ldg(W + k0 * r.wk0 + k1 * r.wk1);
                        const double *Tk = T + (k0 * r.tk0 + k1 * r.tk1);
#pragma unroll
                        for (int v = 0; v < V; ++v) x[v] = fma(w, __ldg(Tk + to[v]), x[v]);
                    }
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int c = c0 + v * T4S_THREADS;
            if (c < g.C) acc[t4s_dot(cpk[v], g.cos)] += x[v];
        }
    }
}

// Issue cost of a run on RT x CT tiles: rounds of the CTA's warps times the matrix
// instructions and loads of a step.
__device__ __forceinline__ int t4s_cost(int R, int C, int RT, int CT) {
    const int n = ((R + 8 * RT - 1) / (8 * RT)) * ((C + 8 * CT - 1) / (8 * CT));
    return (n + T4S_THREADS / 32 - 1) / (T4S_THREADS / 32) * (2 * RT * CT + RT + CT);
}

// Tile shapes of a run (8 RT rows x 8 CT columns per warp); -1: one row, on the FP64 lanes.
template <bool AHEAD>
__device__ void t4s_plan(T4Run &g, int rord, int cord, int na, int nv) {
    g.R = g.C = 1;
    for (int p = 0; p < 4; ++p) {
        const int xr = ((rord >> (4 * p)) & 15) - 1, xc = ((cord >> (4 * p)) & 15) - 1;
        g.rext[p] = xr < 0 ? 1 : (xr == 0 ? na : nv);
        g.ros[p] = xr < 0 ? 0 : t4s_ostride(xr, nv);
        g.cext[p] = xc < 0 ? 1 : (xc == 0 ? na : nv);
        g.cos[p] = xc < 0 ? 0 : t4s_ostride(xc, nv);
        g.R *= g.rext[p];
        g.C *= g.cext[p];
    }
    g.shape = -1;
    if (g.R == 1) return;
    // at most 12 accumulators where a second set of operands is in flight
    const int rt[8] = {AHEAD ? 2 : 4, 4, 3, 2, AHEAD ? 4 : 8, 1, 8, 2},
              ct[8] = {AHEAD ? 6 : 4, 3, 4, AHEAD ? 4 : 8, 2, 8, 1, 2};
    int best = 0x7fffffff;
    for (int i = 0; i < 8; ++i) {  // the shape of least cost for these rows and columns
        const int c = t4s_cost(g.R, g.C, rt[i], ct[i]);
        if (c < best) {
            best = c;
            g.shape = i;
        }
    }
}

// AHEAD where all CTAs are resident at once: a warp's loads then have little company to hide
// behind, and issuing them a step ahead pays (nocc=4, nvir=12 0.80 -> 0.63 ms, nocc=6, nvir=9 1.08 ->
// 0.93; nocc=5, nvir=8 the same 0.47); with more rounds the SMs are busy and the smaller tiles
// cost more loads (nocc=7, nvir=11 3.56 -> 3.98).
template <bool AHEAD>
__global__ void __launch_bounds__(T4S_THREADS, 2)
    k_t4_strings(const __grid_constant__ T4StrOps ops, const int64_t *__restrict__ desc, int nstr,
                 const int32_t *__restrict__ quads, const int32_t *__restrict__ pair_off,
                 const int32_t *__restrict__ pair_sm, int ngroups, int npairs, int nocc, int nv, int na_step, int nsplit,
                 double beta, double *__restrict__ r4, int *status) {
    extern __shared__ double acc[];
    const int q = blockIdx.x / nsplit, part = blockIdx.x % nsplit;
    const int a0 = part * na_step;
    const int na = min(na_step, nv - a0);
    const int nv3 = nv * nv * nv;
    const int nacc = na * nv3;
    T4Rec *rec = reinterpret_cast<T4Rec *>(acc + (int64_t)na_step * nv3);
    T4Run *runs = reinterpret_cast<T4Run *>(rec + T4S_BATCH);  // runs[i]: the run that starts at rec[i]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < nacc; e += blockDim.x) acc[e] = 0.0;
    int occ[4];
    bool occ_ok = true;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        occ[x] = quads[4 * (int64_t)q + x];
        occ_ok = occ_ok && occ[x] >= 0 && occ[x] < nocc;
    }
    if (!occ_ok) {  // uniform over the CTA
        if (threadIdx.x == 0) atomicOr(status, 1);
        return;
    }
    for (int s0 = 0, nb; s0 < nstr; s0 += nb) {
        nb = min(T4S_BATCH, nstr - s0);
        __syncthreads();  // the previous batch's runs are done with rec
        if (threadIdx.x < nb) {
            T4Rec o = {};
            o.ok = t4s_decode(ops, desc + (int64_t)(s0 + threadIdx.x) * T4S_DESC, occ, q, a0, na, nv, pair_off, ngroups,
                              npairs, o, status);
            rec[threadIdx.x] = o;
        }
        __syncthreads();
        auto same = [&](int i, int j) {
            return rec[i].mask == rec[j].mask && rec[i].rord == rec[j].rord && rec[i].cord == rec[j].cord;
        };
        if (s0 + nb < nstr) {  // a run the batch cuts goes to the next batch whole (unless it fills this one)
            int e = nb - 1;
            while (e > 0 && same(e, e - 1)) e--;
            if (e > 0) nb = e;
        }
        if (threadIdx.x < nb && (threadIdx.x == 0 || !same(threadIdx.x, threadIdx.x - 1))) {
            const int i = threadIdx.x;
            int e = i;
            bool any = false;
            for (; e < nb && same(i, e); e++) any = any || rec[e].ok;
            if (any) t4s_plan<AHEAD>(runs[i], rec[i].rord, rec[i].cord, na, nv);
            runs[i].end = any ? e : -e;  // no string of the run passed its checks: skipped
        }
        __syncthreads();
        for (int r0 = 0, r1; r0 < nb; r0 = r1) {
            const T4Run &g = runs[r0];
            r1 = g.end;
            if (r1 < 0) {
                r1 = -r1;
                continue;
            }
#define T4S_CASE(ID, RT, CT)                                                             \
    case ID:                                                                             \
        t4s_run<AHEAD, RT, CT>(acc, rec, r0, r1, g, pair_sm, nocc, warp, lane, status);   \
        break;
            switch (g.shape) {
                T4S_CASE(0, (AHEAD ? 2 : 4), (AHEAD ? 6 : 4))
                T4S_CASE(1, 4, 3)
                T4S_CASE(2, 3, 4)
                T4S_CASE(3, 2, (AHEAD ? 4 : 8))
                T4S_CASE(4, (AHEAD ? 4 : 8), 2)
                T4S_CASE(5, 1, 8)
                T4S_CASE(6, 8, 1)
                T4S_CASE(7, 2, 2)
                default: t4s_run_vector(acc, rec, r0, r1, g, pair_sm, nocc, status);
            }
#undef T4S_CASE
            __syncthreads();  // the next run's tiles split the accumulator another way
        }
    }
    __syncthreads();
    double *out = r4 + (int64_t)q * nv * nv3 + (int64_t)a0 * nv3;
    if (beta == 0.0) {
        for (int e = threadIdx.x; e < nacc; e += blockDim.x) out[e] = acc[e];
    } else {
        for (int e = threadIdx.x; e < nacc; e += blockDim.x) out[e] = beta * out[e] + acc[e];
    }
}

// W_oooovv's T4 part over every ordering (distr_cc/rccsdtq.py:756-775),
//   out[j,k,l][m][a,b] = alpha sum_{i,f,e} E[m,i,e,f] Ts[i,j,k,l][f,a,b,e],
// read in place: a CTA owns one (j,k,l), its warps tiles of 8 m x 16 (a,b) on m8n8k4.f64, the
// contraction runs over (i, f) and the contiguous e.  The einsum through a transposed copy of Ts
// took 0.48 ms of copy and 0.1 of GEMM at nocc=7, nvir=11; this 0.09 ms (one read of Ts, 281 MB).
constexpr int WOO_THREADS = 256, WOO_CT = 2;
__global__ void __launch_bounds__(WOO_THREADS) k_t4_woo(const double *__restrict__ Ts, const double *__restrict__ E,
                                                        double *__restrict__ out, int no, int nv, double alpha) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nv2 = nv * nv;
    const int64_t v4 = (int64_t)nv2 * nv2, o3 = (int64_t)no * no * no, jkl = blockIdx.x;
    const double *T0 = Ts + jkl * v4;  // + i o3 v4
    const int nct = (nv2 + 8 * WOO_CT - 1) / (8 * WOO_CT), nmt = (no + 7) / 8;
    for (int t = warp; t < nct * nmt; t += WOO_THREADS / 32) {
        const int m = (t / nct) * 8 + (lane >> 2), cb = (t % nct) * 8 * WOO_CT;
        const bool mv = m < no;
        int to[WOO_CT];
#pragma unroll
        for (int v = 0; v < WOO_CT; ++v) {
            const int c = cb + 8 * v + (lane >> 2);  // (a, b)
            to[v] = (c < nv2 ? c : 0) * nv;
        }
        double d[WOO_CT][2] = {};
        for (int i = 0; i < no; ++i) {
            const double *Ti = T0 + i * o3 * v4, *Ei = E + ((int64_t)(mv ? m : 0) * no + i) * nv2;
            // (f, e) flattened, e fastest: T at f nv^3 + e, E at e nv + f
            int e = lane & 3, f = 0;
            while (e >= nv) {
                e -= nv;
                f++;
            }
            for (int kb = 0; kb < nv2; kb += 4) {
                double a = 0.0, b[WOO_CT] = {};
                if (f < nv) {
                    a = alpha * __ldg(Ei + e * nv + f);
                    const double *Tk = Ti + (int64_t)f * nv * nv2 + e;
#pragma unroll
                    for (int v = 0; v < WOO_CT; ++v) b[v] = __ldg(Tk + to[v]);
                }
                e += 4;
                while (e >= nv) {
                    e -= nv;
                    f++;
                }
                __syncwarp();
#pragma unroll
                for (int v = 0; v < WOO_CT; ++v) dmma(d[v][0], d[v][1], a, b[v]);
            }
        }
        if (mv) {
            double *o = out + (jkl * no + m) * nv2;
#pragma unroll
            for (int v = 0; v < WOO_CT; ++v)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int c = cb + 8 * v + 2 * (lane & 3) + j;
                    if (c < nv2) o[c] = d[v][j];
                }
        }
    }
}

}  // namespace dcc

using namespace dcc;

extern "C" int dcc_t4_strings_rows_per_cta(int64_t nq, int64_t nvir) {
    if (nq <= 0 || nvir <= 0) return -1;
    const int64_t row = nvir * nvir * nvir * (int64_t)sizeof(double);
    const int64_t na_max = T4S_SMEM_MAX / row;
    if (na_max < 1) return -1;
    // Rounds of resident CTAs (two per SM while their accumulators fit) times a CTA's time, which
    // grows as about 2.5 + na (measured at nocc=7, nvir=11, ms a round: na=1 0.95, 2 1.48, 3 1.70,
    // 4 1.77, 6 3.0; the best choices 3.6 ms there at na=4 against 5.1 at 3, 0.47 ms at nocc=5,
    // nvir=8 at na=2 against 0.86 at 1, 0.80 ms at nocc=4, nvir=12 at na=1 against 0.88 at 2).
    int64_t best_na = 1;
    double best = 1e300;
    for (int64_t na = 1; na <= nvir && na <= na_max; na++) {
        const int64_t smem = na * row + T4S_BATCH * (int64_t)(sizeof(T4Rec) + sizeof(T4Run)) + 1024;
        const int64_t slots = 148 * (2 * smem <= 228 * 1024 ? 2 : 1);
        const int64_t rounds = (nq * ((nvir + na - 1) / na) + slots - 1) / slots;
        const double cost = (double)rounds * (2.5 + (double)na);
        if (cost < best) {
            best = cost;
            best_na = na;
        }
    }
    return (int)best_na;
}

extern "C" int dcc_t4_strings(const double *const *ops, const int64_t *op_numel, int nops, const int64_t *desc,
                              int nstr, const int32_t *quads, int64_t nq, const int32_t *pair_off,
                              const int32_t *pair_sm, int ngroups, int64_t npairs, int64_t nocc, int64_t nvir,
                              double beta, double *r4, int *status, void *stream) {
    clear_error();
    DCC_REQUIRE(nops >= 1 && nops <= T4S_MAXOPS, DCC_ERR_SHAPE, "1 to 32 operands");
    DCC_REQUIRE(ngroups >= 0 && ngroups < 4096 && npairs >= 0 && npairs < (1LL << 30), DCC_ERR_SHAPE,
                "bad pair lists");
    DCC_REQUIRE(ngroups == 0 || (pair_off && pair_sm), DCC_ERR_NULL, "NULL pair lists");
    DCC_REQUIRE(nstr >= 0 && nq >= 0 && nocc >= 1 && nvir >= 1 && nq < (1LL << 24) && nvir < 1024, DCC_ERR_SHAPE,
                "bad size");
    if (nq == 0) return DCC_OK;
    DCC_REQUIRE(ops && op_numel && desc && quads && r4 && status, DCC_ERR_NULL, "NULL argument");
    T4StrOps o = {};
    for (int i = 0; i < nops; ++i) {
        DCC_REQUIRE(ops[i] && op_numel[i] >= 1, DCC_ERR_NULL, "NULL or empty operand");
        DCC_REQUIRE(op_numel[i] < (1LL << 31), DCC_ERR_SHAPE, "operands must hold fewer than 2^31 elements");
        o.p[i] = ops[i];
        o.n[i] = op_numel[i];
    }
    o.nops = nops;
    const int na = dcc_t4_strings_rows_per_cta(nq, nvir);
    DCC_REQUIRE(na >= 1, DCC_ERR_SHAPE, "nvir^3 doubles exceed the shared-memory accumulator");
    const int nsplit = (int)((nvir + na - 1) / na);
    const int64_t grid = nq * nsplit;
    DCC_REQUIRE(grid < (1LL << 31), DCC_ERR_SHAPE, "too many blocks");
    const size_t smem = (size_t)na * nvir * nvir * nvir * sizeof(double) + T4S_BATCH * (sizeof(T4Rec) + sizeof(T4Run));
    static_assert(T4S_SMEM_MAX + T4S_BATCH * (sizeof(T4Rec) + sizeof(T4Run)) <= 227 * 1024, "shared memory per CTA");
    const int64_t slots = 148 * (2 * ((int64_t)smem + 1024) <= 228 * 1024 ? 2 : 1);
    auto launch = [&](auto kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(T4S_SMEM_MAX + T4S_BATCH * (sizeof(T4Rec) + sizeof(T4Run))));
        kern<<<(unsigned)grid, T4S_THREADS, smem, as_stream(stream)>>>(o, desc, nstr, quads, pair_off, pair_sm, ngroups,
                                                                       (int)npairs, (int)nocc, (int)nvir, na, nsplit,
                                                                       beta, r4, status);
    };
    if (grid <= slots)
        launch(k_t4_strings<true>);
    else
        launch(k_t4_strings<false>);
    return launch_status("t4_strings");
}

extern "C" int dcc_t4_w_oooovv(const double *Ts, const double *E, double *out, int64_t nocc, int64_t nvir, double alpha,
                               void *stream) {
    clear_error();
    DCC_REQUIRE(nocc >= 0 && nvir >= 0 && nocc < 1024 && nvir < 1024, DCC_ERR_SHAPE, "bad size");
    if (nocc == 0 || nvir == 0) return DCC_OK;
    DCC_REQUIRE(Ts && E && out, DCC_ERR_NULL, "NULL buffer");
    k_t4_woo<<<(unsigned)(nocc * nocc * nocc), WOO_THREADS, 0, as_stream(stream)>>>(Ts, E, out, (int)nocc, (int)nvir,
                                                                                  alpha);
    return launch_status("t4_w_oooovv");
}
