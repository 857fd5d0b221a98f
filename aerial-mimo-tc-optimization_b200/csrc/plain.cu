// plain.cu -- the plain FP32 chain: the reference's scalar method (Gram,
// coef_apply, LLR) plus the FP32 Cholesky MMSE solve the reference lacks, stage
// by stage or as one kernel.  Every stage is bit-exact with the CPU restatement
// in the checker because each output element is accumulated in the same order
// with the same fused multiply-adds.
#include <algorithm>

#include "common.cuh"

namespace aeq {

// ---------------------------------------------------------------------------
// One kernel for the solve, the apply and the whole chain.  A block takes
// several subcarriers, a team of TEAM lanes each, with their H, then Y, and C in
// shared memory.
//
//   kCoef   G, H -> C, noiseInv          the FP32 Cholesky MMSE solve
//   kApply  C, Y -> Y_eq                 coef_apply_v1_scalar (src/aerial_coef_wmma.cu:71-104)
//   kChain  H, Y -> LLR (and Y_eq)       gram_scalar (src/aerial_bottleneck.cu:56-80, M = H^H),
//                                        all of the above and the demapper; G, C and
//                                        noiseInv never leave the SM
//
// Every value is accumulated in the serial specification's order with its
// fused multiply-adds; lanes only divide the values among themselves:
//   G       lane: row r, columns 2q, 2q + 1, antennas in order.
//   factor  right-looking, lane: row i: at step k = 0, 1, ... it takes
//           L_ik conj(L_jk) off its element j, the order of the left-looking sum.
//   C       lane: antennas tid, tid + TEAM, ... (two at a time, for two
//           independent chains); forward and backward substitution in registers.
//   mu      lane: one layer, antennas in order.
//   Y_eq    lane: one layer and up to TS symbols, antennas in order.
//
// What bounds it: instruction issue and the latency of each subcarrier's chain
// of phases.  A thread per output element, as the reference has it, reads two
// operands from L1 for each complex product; here a lane's operands serve two
// columns (G) or up to four symbols (Y_eq) from one 16-byte read each, rows are
// padded so that a warp's reads meet no bank conflicts, and the intermediates'
// 27.6 MB per 100 MHz slot of HBM traffic are gone.  The phases with fewer
// values than lanes (the factor, with its square roots and divisions, and mu)
// run for all subcarriers of a block in one warp: done by each subcarrier's own
// warp they were over a quarter of all instructions.  Y is copied where H was
// once H is spent (and asked into L2 at the start), which leaves room for 20
// subcarriers on an SM instead of 12.  4 slots of 132 PRB x 64 antennas x 8
// layers: 403 us as four scalar kernels per cell, 53 us with a warp for each
// subcarrier throughout, 48 us as here.
// ---------------------------------------------------------------------------
enum PlainMode : int { kCoef, kApply, kChain };

struct PlainCell {
    const cf* H;
    const cf* Y;
    const cf* G;        // kCoef: in
    cf* C;              // kCoef: out, kApply: in
    float* nInv;        // kCoef: out
    cf* O;              // kApply: out, kChain: optional out
    float* llr;
    float sigma2;
    int nSC, A, L, S, nPam;
    int vecH, vecY;     // 16-byte rows of H (L even, aligned); of Y and C (A even, aligned)
    unsigned block0;    // first block of this cell
    PamLut lut;
};
struct PlainParams {
    PlainCell cell[AERIAL_MAX_CELLS];
    int nCells;
    int teamValues;     // shared memory per team, in complex values (even)
};

// Lanes per subcarrier: 16 for up to 4 layers, a warp for 8, four warps for
// 16, whose C has enough antennas to occupy them.  A block's subcarriers have at
// most 32 rows between them (the factor's warp).
__host__ __device__ constexpr int plain_team(int LT) { return LT <= 4 ? 16 : LT == 8 ? 32 : 128; }
constexpr int kPlainThreads = 128;

// Row strides in complex values: even (16-byte rows) and 16 bytes past a
// multiple of the row, so that eight rows read at once differ in banks.
__host__ __device__ __forceinline__ int plain_hs(int L) { return ((L + 1) & ~1) + 2; }
__host__ __device__ __forceinline__ int plain_cs(int A) { return ((A + 1) & ~1) + 2; }

// Shared memory of a team, in complex values: H (kChain: then Y), C, Y (kApply),
// G and then the factor, and 3 L floats.
struct PlainSmem {
    int c, y, l, total;
};
__host__ __device__ __forceinline__ PlainSmem plain_smem(int mode, int A, int L, int S) {
    const int h = A * plain_hs(L), c = L * plain_cs(A), y = S * plain_cs(A);
    PlainSmem m;
    m.c = mode == kApply ? 0 : mode == kCoef ? h : (h > y ? h : y);
    m.y = mode == kApply ? c : 0;
    m.l = m.c + c + (mode == kApply ? y : 0);
    m.total = (m.l + (mode == kApply ? 0 : L * L + (3 * L + 1) / 2) + 1) & ~1;
    return m;
}

template <int TEAM>
__device__ __forceinline__ void team_sync() {
    if constexpr (TEAM > 32) __syncthreads();
    else __syncwarp();
}
__device__ __forceinline__ uint32_t sm_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(cf* d, const cf* s) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm_addr(d)), "l"(__cvta_generic_to_global(s))
                 : "memory");
}
__device__ __forceinline__ void cp8(cf* d, const cf* s) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sm_addr(d)), "l"(__cvta_generic_to_global(s))
                 : "memory");
}
__device__ __forceinline__ float4 ld4(const cf* p) { return *reinterpret_cast<const float4*>(p); }

// rows x cols values of src (contiguous) into rows of stride ds.  COLS: cols
// where known (a divisor of 2 TEAM), so that a lane's pieces lie a constant
// number of rows apart; else 0.
template <int TEAM, int COLS = 0>
__device__ __forceinline__ void stage_rows(cf* dst, int ds, const cf* src, int rows, int cols, int vec, int tid) {
    if (vec) {
        const int half = cols >> 1;
        if constexpr (COLS != 0) {
            constexpr int HALF = COLS / 2, STEP = TEAM / HALF;
            static_assert(TEAM % HALF == 0, "a lane keeps its piece of the row");
            dst += tid / HALF * ds + tid % HALF * 2;
            src += 2 * tid;
#pragma unroll 4
            for (int r = tid / HALF; r < rows; r += STEP, dst += STEP * ds, src += 2 * TEAM) cp16(dst, src);
        } else if (half >= TEAM) {
            for (int r = 0; r < rows; r++)
                for (int k = tid; k < half; k += TEAM) cp16(dst + r * ds + 2 * k, src + (long)r * cols + 2 * k);
        } else {
            for (int e = tid; e < rows * half; e += TEAM) {
                const int r = e / half, k = e - r * half;
                cp16(dst + r * ds + 2 * k, src + 2 * e);
            }
        }
    } else {
        for (int e = tid; e < rows * cols; e += TEAM) {
            const int r = e / cols;
            cp8(dst + r * ds + (e - r * cols), src + e);
        }
    }
}

// C columns of NA antennas a, a + TEAM: G x = conj(H[a][:]).
template <int LT, bool EX, int NA, int TEAM>
__device__ __forceinline__ void solve_antennas(const cf* sH, int hs, const cf* sL, const float* sInv, cf* sC, int cs,
                                               int L, int a) {
    cf w[NA][LT];
#pragma unroll
    for (int n = 0; n < NA; n++) {
        const cf* h = sH + (a + n * TEAM) * hs;
#pragma unroll
        for (int i = 0; i < LT; i += 2) {
            if (!EX && i >= L) break;
            const float4 v = ld4(h + i);
            w[n][i] = make_float2(v.x, -v.y);
            w[n][i + 1] = make_float2(v.z, -v.w);
        }
    }
#pragma unroll
    for (int i = 0; i < LT; i++) {
        if (!EX && i >= L) break;
#pragma unroll
        for (int k = 0; k < i; k++) {
            const cf lv = sL[i * L + k];
#pragma unroll
            for (int n = 0; n < NA; n++) {
                const cf y = w[n][k];
                cf& acc = w[n][i];
                acc.x = __fmaf_rn(-lv.x, y.x, acc.x);
                acc.x = __fmaf_rn(lv.y, y.y, acc.x);
                acc.y = __fmaf_rn(-lv.x, y.y, acc.y);
                acc.y = __fmaf_rn(-lv.y, y.x, acc.y);
            }
        }
        const float iv = sInv[i];
#pragma unroll
        for (int n = 0; n < NA; n++) w[n][i] = make_float2(__fmul_rn(w[n][i].x, iv), __fmul_rn(w[n][i].y, iv));
    }
#pragma unroll
    for (int i = LT - 1; i >= 0; i--) {
        if (!EX && i >= L) continue;
#pragma unroll
        for (int k = i + 1; k < LT; k++) {
            if (!EX && k >= L) break;
            const cf lv = sL[k * L + i];
#pragma unroll
            for (int n = 0; n < NA; n++) {
                const cf y = w[n][k];
                cf& acc = w[n][i];
                acc.x = __fmaf_rn(-lv.x, y.x, acc.x);
                acc.x = __fmaf_rn(-lv.y, y.y, acc.x);
                acc.y = __fmaf_rn(-lv.x, y.y, acc.y);
                acc.y = __fmaf_rn(lv.y, y.x, acc.y);
            }
        }
        const float iv = sInv[i];
#pragma unroll
        for (int n = 0; n < NA; n++) {
            w[n][i] = make_float2(__fmul_rn(w[n][i].x, iv), __fmul_rn(w[n][i].y, iv));
            sC[i * cs + a + n * TEAM] = w[n][i];
        }
    }
}

template <int N>
__device__ __forceinline__ void plain_llr_store(cf v, float noise, const PamLut& lut, float* dst) {
    float o[2 * N];
    pam_llr<N>(v.x, v.y, noise, lut, o);
    // rows of 8 N bytes from an 8-byte aligned array
#pragma unroll
    for (int j = 0; j < 2 * N; j += 2) *reinterpret_cast<float2*>(dst + j) = make_float2(o[j], o[j + 1]);
}

// Y_eq of layer l, symbols st, st + LPL, ... (TS of them; those past S are
// computed on row 0 and dropped).
template <int MODE, int TS, int LPL>
__device__ __forceinline__ void apply_symbols(const PlainCell& cl, const cf* sC, const cf* sY, int cs, float noise,
                                              long sc, int l, int st, bool out) {
    const int A = cl.A, S = cl.S, L = cl.L;
    const cf* c = sC + l * cs;
    const cf* y[TS];
    cf acc[TS];
#pragma unroll
    for (int t = 0; t < TS; t++) {
        const int s = st + t * LPL;
        y[t] = sY + (s < S ? s : 0) * cs;
        acc[t] = make_float2(0.f, 0.f);
    }
    int a = 0;
#pragma unroll 4
    for (; a + 1 < A; a += 2) {
        const float4 cv = ld4(c + a);
        float4 yv[TS];
#pragma unroll
        for (int t = 0; t < TS; t++) yv[t] = ld4(y[t] + a);
#pragma unroll
        for (int t = 0; t < TS; t++) acc[t] = cma(make_float2(cv.x, cv.y), make_float2(yv[t].x, yv[t].y), acc[t]);
#pragma unroll
        for (int t = 0; t < TS; t++) acc[t] = cma(make_float2(cv.z, cv.w), make_float2(yv[t].z, yv[t].w), acc[t]);
    }
    if (a < A) {
#pragma unroll
        for (int t = 0; t < TS; t++) acc[t] = cma(c[a], y[t][a], acc[t]);
    }
    const long row = (sc * L + l) * (long)S;
#pragma unroll
    for (int t = 0; t < TS; t++) {
        const int s = st + t * LPL;
        if (!out || s >= S) continue;
        if (MODE == kApply || cl.O) cl.O[row + s] = acc[t];
        if constexpr (MODE == kChain) {
            float* dst = cl.llr + (row + s) * 2 * cl.nPam;
            switch (cl.nPam) {
                case 1: plain_llr_store<1>(acc[t], noise, cl.lut, dst); break;
                case 2: plain_llr_store<2>(acc[t], noise, cl.lut, dst); break;
                case 3: plain_llr_store<3>(acc[t], noise, cl.lut, dst); break;
                default: plain_llr_store<4>(acc[t], noise, cl.lut, dst); break;
            }
        }
    }
}

// Cholesky factor of the block's subcarriers by one warp, lane (j, i) = row i of
// subcarrier j: G's lower triangle at sl (row stride L, next subcarrier ts
// later) is replaced by the factor's, 1 / its diagonal goes to sInv.
template <int LT, bool EX>
__device__ __forceinline__ void factor_rows(cf* sl, float* sInv, int L, int i) {
    cf r[LT];
#pragma unroll
    for (int c = 0; c < LT; c++) r[c] = (c <= i && i < L) ? sl[i * L + c] : make_float2(1.f, 0.f);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < LT; k++) {
        if (!EX && k >= L) break;
        float s = __shfl_sync(0xffffffffu, r[k].x, k, LT);
        if (!(s > 0.f)) s = 1e-30f;
        const float iv = __fdiv_rn(1.0f, __fsqrt_rn(s));
        if (i == k) sInv[k] = iv;
        const cf a = make_float2(__fmul_rn(r[k].x, iv), __fmul_rn(r[k].y, iv));
        if (i > k && i < L) sl[i * L + k] = a;
        __syncwarp();
#pragma unroll
        for (int c = k + 1; c < LT; c++) {
            if (!EX && c >= L) break;
            const cf b = sl[c * L + k];
            r[c].x = __fmaf_rn(-a.x, b.x, r[c].x);
            r[c].x = __fmaf_rn(-a.y, b.y, r[c].x);
            r[c].y = __fmaf_rn(-a.y, b.x, r[c].y);
            r[c].y = __fmaf_rn(a.x, b.y, r[c].y);
        }
    }
}

// EX: every cell has L == LT.  LT: layers rounded up to 2, 4, 8 or 16.
template <int MODE, int LT, bool EX>
__global__ void __launch_bounds__(kPlainThreads) plain_kernel(const __grid_constant__ PlainParams p) {
    constexpr int TEAM = plain_team(LT);
    constexpr int LPL = TEAM / LT;                     // lanes per layer of the apply phase
    extern __shared__ float4 plain_shared[];
    wait_previous();
    const int team = threadIdx.x / TEAM, tid = threadIdx.x % TEAM, teams = blockDim.x / TEAM;
    int ci = 0;
    while (ci + 1 < p.nCells && blockIdx.x >= p.cell[ci + 1].block0) ci++;
    const PlainCell& cl = p.cell[ci];
    const int A = cl.A, L = EX ? LT : cl.L, S = cl.S;
    const int hs = EX ? LT + 2 : plain_hs(L), cs = plain_cs(A);
    const long sc0 = (long)(blockIdx.x - cl.block0) * teams;
    const bool out = sc0 + team < cl.nSC;              // teams past the cell's end repeat its last subcarrier
    const long sc = out ? sc0 + team : cl.nSC - 1;
    const int ts = p.teamValues;
    const PlainSmem m = plain_smem(MODE, A, L, S);
    cf* sh = reinterpret_cast<cf*>(plain_shared);      // team 0's
    cf* sH = sh + team * ts;
    cf* sC = sH + m.c;
    cf* sY = sH + m.y;

    if constexpr (MODE == kApply) {
        stage_rows<TEAM>(sC, cs, cl.C + sc * A * L, L, A, cl.vecY, tid);
        stage_rows<TEAM>(sY, cs, cl.Y + sc * S * A, S, A, cl.vecY, tid);
    } else {
        stage_rows<TEAM, EX ? LT : 0>(sH, hs, cl.H + sc * A * L, A, L, cl.vecH, tid);
        if constexpr (MODE == kChain) {
            const char* y = reinterpret_cast<const char*>(cl.Y + sc * S * A);
            for (int e = 128 * tid; e < 8 * S * A; e += 128 * TEAM)
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(__cvta_generic_to_global(y + e)));
        } else {
            for (int e = tid; e < L * L; e += TEAM) sH[m.l + e] = cl.G[sc * L * L + e];
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");

    float noise = 0.f;
    if constexpr (MODE != kApply) {
        __syncthreads();
        if constexpr (MODE == kChain) {
            // the lower triangle of G: row pair R holds 2 (R + 1) column pairs,
            // after the R (R + 1) of the pairs above
            constexpr int PAIRS = LT / 2 * (LT / 2 + 1);
            for (int t = threadIdx.x; t < teams * PAIRS; t += blockDim.x) {
                const int j = t / PAIRS, v = t % PAIRS;
                int R = 0;
                while ((R + 1) * (R + 2) <= v) R++;
                const int u = v - R * (R + 1);
                const int r = 2 * R + (u > R ? 1 : 0), q = u > R ? u - R - 1 : u;
                if (!EX && r >= L) continue;
                const cf* hr = sh + j * ts + r;
                const cf* hc = sh + j * ts + 2 * q;
                cf g0 = make_float2(0.f, 0.f), g1 = g0;
#pragma unroll 8
                for (int k = 0; k < A; k++) {
                    const cf w = hr[k * hs];
                    const float4 c = ld4(hc + k * hs);
                    const cf n = make_float2(w.x, -w.y);
                    g0 = cma(n, make_float2(c.x, c.y), g0);
                    g1 = cma(n, make_float2(c.z, c.w), g1);
                }
                if (r == 2 * q) g0.x = __fadd_rn(g0.x, cl.sigma2);
                if (r == 2 * q + 1) g1.x = __fadd_rn(g1.x, cl.sigma2);
                cf* g = sh + j * ts + m.l + r * L + 2 * q;
                g[0] = g0;
                if (2 * q + 1 <= r) g[1] = g1;
            }
            __syncthreads();
        }
        // one warp, another one from block to block
        const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
        const bool mine = (int)(threadIdx.x >> 5) == (int)(blockIdx.x % (unsigned)warps);
        if (mine) {
            const int j = min(lane / LT, teams - 1);   // lanes past the last subcarrier repeat it
            cf* l = sh + j * ts + m.l;
            factor_rows<LT, EX>(l, reinterpret_cast<float*>(l + L * L), L, lane % LT);
        }
        __syncthreads();
        // ---- C: forward and backward substitution per antenna ----
        const cf* sL = sH + m.l;
        const float* sInv = reinterpret_cast<const float*>(sL + L * L);
        int a = tid;
        for (; a + TEAM < A; a += 2 * TEAM) solve_antennas<LT, EX, 2, TEAM>(sH, hs, sL, sInv, sC, cs, L, a);
        if (a < A) solve_antennas<LT, EX, 1, TEAM>(sH, hs, sL, sInv, sC, cs, L, a);
        __syncthreads();
        // ---- mu and the noise of the unbiased symbol ----
        if (mine) {
            const int j = lane / LT, l = lane % LT;
            if (j < teams && l < L) {
                float mu = 0.f;
                const cf* c = sh + j * ts + m.c + l * cs;
                const cf* h = sh + j * ts + l;
#pragma unroll 8
                for (int k = 0; k < A; k++) {
                    const cf cv = c[k], hv = h[k * hs];
                    mu = __fmaf_rn(cv.x, hv.x, mu);
                    mu = __fmaf_rn(-cv.y, hv.y, mu);
                }
                const float ni = __fdiv_rn(mu, __fsub_rn(1.0f, mu));
                float* f = reinterpret_cast<float*>(sh + j * ts + m.l + L * L) + L;
                f[l] = __fdiv_rn(1.0f, mu);
                f[L + l] = ni;
                if (MODE == kCoef && sc0 + j < cl.nSC) cl.nInv[(sc0 + j) * L + l] = ni;
            }
        }
        __syncthreads();
        if constexpr (MODE == kChain) {                // H is spent: Y takes its place
            stage_rows<TEAM>(sY, cs, cl.Y + sc * S * A, S, A, cl.vecY, tid);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        const float* sMuInv = sInv + L;
#pragma unroll
        for (int l = 0; l < LT; l++) {
            if (!EX && l >= L) break;
            const float im = sMuInv[l];
            for (int k = tid; k < A; k += TEAM) {
                const cf v = sC[l * cs + k];
                const cf w = make_float2(__fmul_rn(v.x, im), __fmul_rn(v.y, im));
                if constexpr (MODE == kChain) sC[l * cs + k] = w;
                else if (out) cl.C[(sc * L + l) * A + k] = w;
            }
        }
        if constexpr (MODE == kCoef) return;
        noise = sMuInv[L + min(tid / LPL, L - 1)];
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }

    // ---- Y_eq (and LLRs): lane (layer l, symbols st, st + LPL, ...) ----
    if constexpr (MODE != kCoef) {
        team_sync<TEAM>();
        const int l = tid / LPL, st = tid % LPL;
        if (l >= L) return;
        switch ((S + LPL - 1) / LPL) {
            case 1: apply_symbols<MODE, 1, LPL>(cl, sC, sY, cs, noise, sc, l, st, out); break;
            case 2: apply_symbols<MODE, 2, LPL>(cl, sC, sY, cs, noise, sc, l, st, out); break;
            case 3: apply_symbols<MODE, 3, LPL>(cl, sC, sY, cs, noise, sc, l, st, out); break;
            default: apply_symbols<MODE, 4, LPL>(cl, sC, sY, cs, noise, sc, l, st, out); break;
        }
    }
}

// ---------------------------------------------------------------------------
// Gram: G[sc][r][c] = sum_k cma(conj(H[k][r]), H[k][c]) (+ sigma2 if r == c):
// gram_scalar (src/aerial_bottleneck.cu:56-80) with M = H^H, the antenna sum of
// every element in order.
//
// A lane owns RT x CT elements, so its RT + CT operand reads serve RT CT
// complex products: shared-memory reads return 128 bytes a cycle however many
// lanes want the same value, and with one row and one column pair a lane
// (24 bytes for 8 FMAs) they, not the FMA pipe or HBM, set the time.  2 x 2
// (32 bytes for 16 FMAs; 4 x 4 for 16 layers) puts both near the HBM time of
// H; 4 x 2 leaves too few warps on an SM (20 KB of H per warp: 22 us).  A warp
// stages and multiplies its own 32 / lanes subcarriers; a spare row per
// subcarrier keeps those read together in different banks.  8 slots of 1,584
// subcarriers x 64 antennas x 8 layers (59 MB): 77 us one thread per element,
// 22 us one pair per lane, 19 us as here.
// ---------------------------------------------------------------------------
constexpr int kGramThreads = 32;
constexpr int kGramParts = 2;                  // a subcarrier's antennas arrive and are summed in two parts
// Where a subcarrier's part is at most this many pieces (two for each lane), the
// lanes walk the pieces of all the warp's subcarriers in one row: taken one
// subcarrier after another, 16 of them for 1 or 2 layers, a turn with most
// lanes idle cost as much as a full one.  60 subcarriers x 4 antennas x 1 layer
// 6.4 us in turns, 1.4 us in one row; x 64 x 2 5.6 and 3.6 us.
constexpr int kGramFlat = 64;
__host__ __device__ constexpr int gram_rt(int LT) { return LT == 2 ? 1 : LT == 16 ? 4 : 2; }
__host__ __device__ constexpr int gram_ct(int LT) { return LT == 16 ? 4 : 2; }
__host__ __device__ constexpr int gram_team(int LT) { return (LT / gram_rt(LT)) * (LT / gram_ct(LT)); }

struct GramParams {
    const cf* H;
    cf* G;
    float sigma2;
    int nSC, A, L, vecH, vecG;
    // for division of up to 2^16 by the part's antennas and by a row's pieces:
    // floor(2^32 / d) + 1, or 0 for 1
    unsigned rcpRows[kGramParts], rcpPieces;
};
__device__ __forceinline__ int div_rcp(int v, unsigned rcp) { return rcp ? (int)__umulhi((unsigned)v, rcp) : v; }
static unsigned rcp_of(int d) { return d > 1 ? (unsigned)(0x100000000ull / (unsigned)d) + 1u : 0u; }

template <int LT, bool EX>
__global__ void __launch_bounds__(kGramThreads) gram_kernel(const GramParams p) {
    constexpr int RT = gram_rt(LT), CT = gram_ct(LT), TEAM = gram_team(LT), PER = 32 / TEAM;
    extern __shared__ float4 gram_smem[];
    wait_previous();
    const int lane = threadIdx.x;                      // a block is one warp
    const int A = p.A, L = EX ? LT : p.L, hs = EX ? LT + 2 : plain_hs(L);
    const int ts = (A + 1) * hs;                       // values per subcarrier
    cf* sm = reinterpret_cast<cf*>(gram_smem);
    const long sc0 = (long)blockIdx.x * PER;
    const int n = (int)min((long)PER, (long)p.nSC - sc0);      // subcarriers of this warp
    const int part = (A + kGramParts - 1) / kGramParts;         // antennas of one copy group
    const int width = p.vecH ? 2 : 1, pieces = L / width;       // values a copy, copies a row
#pragma unroll
    for (int q = 0; q < kGramParts; q++) {
        const int a0 = q * part, rows = min(part, A - a0);
        if (part * pieces <= kGramFlat) {
            for (int e = lane; e < n * rows * pieces; e += 32) {
                const int row = div_rcp(e, p.rcpPieces), k = (e - row * pieces) * width;
                const int j = div_rcp(row, p.rcpRows[q]), a = a0 + row - j * rows;
                const cf* src = p.H + ((sc0 + j) * A + a) * L + k;
                cf* dst = sm + j * ts + a * hs + k;
                if (p.vecH) cp16(dst, src);
                else cp8(dst, src);
            }
        } else {
            for (int j = 0; j < n && rows > 0; j++)
                stage_rows<32, EX ? LT : 0>(sm + j * ts + a0 * hs, hs, p.H + ((sc0 + j) * A + a0) * L, rows, L, p.vecH,
                                            lane);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int j = lane / TEAM, t = lane % TEAM;
    const int r0 = t / (LT / CT) * RT, c0 = t % (LT / CT) * CT;
    const cf* hr = sm + j * ts + r0;
    const cf* hc = sm + j * ts + c0;
    cf acc[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int m = 0; m < CT; m++) acc[i][m] = make_float2(0.f, 0.f);
    auto antennas = [&](int k0, int k1) {
#pragma unroll 4
        for (int k = k0; k < k1; k++) {
            cf rv[RT], cv[CT];
            if constexpr (RT == 1) {
                rv[0] = hr[k * hs];
            } else {
#pragma unroll
                for (int i = 0; i < RT; i += 2) {
                    const float4 v = ld4(hr + k * hs + i);
                    rv[i] = make_float2(v.x, v.y);
                    rv[i + 1] = make_float2(v.z, v.w);
                }
            }
#pragma unroll
            for (int m = 0; m < CT; m += 2) {
                const float4 v = ld4(hc + k * hs + m);
                cv[m] = make_float2(v.x, v.y);
                cv[m + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int m = 0; m < CT; m++) acc[i][m] = cma(make_float2(rv[i].x, -rv[i].y), cv[m], acc[i][m]);
        }
    };
    static_assert(kGramParts == 2, "one wait per part");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncwarp();
    antennas(0, min(part, A));
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    antennas(part, A);
    if (j >= n || r0 >= L || c0 >= L) return;
    cf* g = p.G + ((sc0 + j) * L + r0) * L + c0;
#pragma unroll
    for (int i = 0; i < RT; i++) {
        const int r = r0 + i;
        if (!EX && r >= L) break;
#pragma unroll
        for (int m = 0; m < CT; m++)
            if (r == c0 + m) acc[i][m].x = __fadd_rn(acc[i][m].x, p.sigma2);
#pragma unroll
        for (int m = 0; m < CT; m += 2) {
            if (p.vecG) {                              // L even, G 16-byte aligned
                if (EX || c0 + m < L)
                    *reinterpret_cast<float4*>(g + i * L + m) =
                        make_float4(acc[i][m].x, acc[i][m].y, acc[i][m + 1].x, acc[i][m + 1].y);
            } else {
                if (c0 + m < L) g[i * L + m] = acc[i][m];
                if (c0 + m + 1 < L) g[i * L + m + 1] = acc[i][m + 1];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// LLR demapper (llr_v1_baseline / llr_v3 shape), a thread per symbol.  A launch
// of a block per SM or more is bound by its writes, 2 N values per symbol read:
// a thread takes four symbols, whose loads are under way together, and a row of
// LLRs goes out in one store as wide as it is (32 bytes of 256-QAM in FP32 fill a
// sector; as four 8-byte stores each of a warp's requests left every sector of
// 1 KB a quarter full).  FP32 rows without such a store, those of 64-QAM (24
// bytes) and those of 256-QAM in an output that is not aligned for it, cross
// through shared memory into contiguous stores.  14-symbol 256-QAM of 8 slots of
// 1,584 subcarriers x 8 layers, 57 MB: 21.5 us with a store per two LLRs, 10 us;
// 2 M symbols 8 bytes past the alignment 36 us with four stores a symbol, 13.8 us.
// Smaller launches are bound by one thread's chain, which four symbols and the
// crossing lengthen: a symbol a thread and direct stores (20,000 symbols of
// 64-QAM 2.3 us with four, 1.5 us).
// ---------------------------------------------------------------------------
constexpr int kLlrThreads = 256;
constexpr int kLlrSymbols = 4;                 // symbols a thread of a large launch loads before it demaps the first

// W: 4-byte words of LLRs per symbol.
template <int W>
__device__ __forceinline__ void store_words(uint32_t* dst, const uint32_t (&v)[W]) {
    if constexpr (W == 8)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(dst), "r"(v[0]), "r"(v[1]),
                     "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    else if constexpr (W == 4)
        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    else if constexpr (W == 2)
        *reinterpret_cast<uint2*>(dst) = make_uint2(v[0], v[1]);
    else
        *dst = v[0];
}

// LLRs of the symbols base .. base + 255 (count in all), a row of W words from
// each thread.  wide: out is aligned to the row's store, for rows of 6 words to 16
// bytes; otherwise stores of NARROW words (FP32 LLR rows are 8-byte aligned, FP16
// ones 4-byte).  CROSS: rows of 24 bytes or more that have no store of their own
// go by way of shared memory; shorter ones gain nothing there (2 M symbols of
// 64-QAM in FP16 9.0 us that way, 8.4 us in three direct stores).
template <int W, int NARROW, bool CROSS>
__device__ __forceinline__ void write_rows(uint32_t* out, long base, int count, const uint32_t (&v)[W], bool wide) {
    const long idx = base + threadIdx.x;
    if constexpr ((W & (W - 1)) == 0) {
        if (wide) {
            if (idx < count) store_words<W>(out + idx * W, v);
            return;
        }
    }
    if constexpr (CROSS && W >= 6) {
        static_assert(NARROW == 2 && W % 2 == 0, "FP32 rows");
        __shared__ __align__(16) uint32_t rows[kLlrThreads * W];
#pragma unroll
        for (int j = 0; j < W; j += 2)
            *reinterpret_cast<uint2*>(rows + threadIdx.x * W + j) = make_uint2(v[j], v[j + 1]);
        __syncthreads();
        uint32_t* dst = out + base * W;
        if (wide && base + kLlrThreads <= count) {
            for (int e = threadIdx.x; e < kLlrThreads * W / 4; e += kLlrThreads)
                reinterpret_cast<uint4*>(dst)[e] = reinterpret_cast<const uint4*>(rows)[e];
        } else {
            const int words = (int)min((long)kLlrThreads, count - base) * W;
            for (int e = 2 * threadIdx.x; e < words; e += 2 * kLlrThreads)
                *reinterpret_cast<uint2*>(dst + e) = *reinterpret_cast<const uint2*>(rows + e);
        }
        __syncthreads();
        return;
    }
    if (idx >= count) return;
#pragma unroll
    for (int j = 0; j < W; j += NARROW) {
        uint32_t part[NARROW];
#pragma unroll
        for (int i = 0; i < NARROW; i++) part[i] = v[j + i];
        store_words<NARROW>(out + idx * W + j, part);
    }
}

// U: symbols of a thread, 256 apart.
template <int N, int U>
__global__ void __launch_bounds__(kLlrThreads) llr_f16_kernel(const __half2* in, const float* ni, __half* out, int count,
                                                               bool wide, PamLut lut) {
    wait_previous();
    __half2 v[U];
    float nv[U];
    const long base = (long)blockIdx.x * kLlrThreads * U;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const long at = min(base + u * kLlrThreads + (long)threadIdx.x, (long)count - 1);
        v[u] = in[at];
        nv[u] = ni[at];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        float o[2 * N];
        pam_llr<N>(__low2float(v[u]), __high2float(v[u]), nv[u], lut, o);
        uint32_t w[N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            const __half2 h = __floats2half2_rn(o[2 * j], o[2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        write_rows<N, 1, (U > 1)>(reinterpret_cast<uint32_t*>(out), base + u * kLlrThreads, count, w, wide);
    }
}

// noiseInv index = symbol / symsPerNoise: the block's first quotient by one
// division, the rest from it (rcp = floor(2^32 / symsPerNoise) + 1, exact
// while symsPerNoise <= 1024; a larger count changes at most once in a block).
template <int N, int U>
__global__ void __launch_bounds__(kLlrThreads) llr_f32_kernel(const cf* in, const float* ni, float* out, int count,
                                                               int symsPerNoise, unsigned rcp, bool wide, PamLut lut) {
    wait_previous();
    cf v[U];
    float nv[U];
    const long base = (long)blockIdx.x * kLlrThreads * U;
    const int q0 = (int)(base / symsPerNoise);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const long at = min(base + u * kLlrThreads + (long)threadIdx.x, (long)count - 1);
        const unsigned r = (unsigned)(at - (long)q0 * symsPerNoise);
        const int q = q0 + (symsPerNoise == 1 ? (int)r
                            : symsPerNoise <= 1024 ? (int)__umulhi(r, rcp)
                                                   : (r >= (unsigned)symsPerNoise ? 1 : 0));
        v[u] = in[at];
        nv[u] = ni[q];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        float o[2 * N];
        pam_llr<N>(v[u].x, v[u].y, nv[u], lut, o);
        uint32_t w[2 * N];
#pragma unroll
        for (int j = 0; j < 2 * N; j++) w[j] = __float_as_uint(o[j]);
        write_rows<2 * N, 2, (U > 1)>(reinterpret_cast<uint32_t*>(out), base + u * kLlrThreads, count, w, wide);
    }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
static bool shape_ok(int nSC, int nSym, int L, int A) {
    return nSC >= 1 && nSC <= 12 * AERIAL_MAX_PRB && nSym >= 1 && nSym <= AERIAL_MAX_SYMS && L >= 1 && L <= AERIAL_MAX_LAYERS && A >= 1 &&
           A <= AERIAL_MAX_ANTS;
}

static int layers_tile(int L) { return L <= 2 ? 2 : L <= 4 ? 4 : L <= 8 ? 8 : 16; }

template <int MODE, int LT, bool EX>
static int launch_plain_t(PlainParams& p, cudaStream_t st) {
    constexpr int TEAM = plain_team(LT);
    int values = 0;
    for (int i = 0; i < p.nCells; i++)
        values = std::max(values, plain_smem(MODE, p.cell[i].A, p.cell[i].L, p.cell[i].S).total);
    // the subcarriers of a block that one warp reads together start LT values
    // apart in the banks
    if (LT < 16) values += (LT - values % 16 + 16) % 16;
    const int teamBytes = values * (int)sizeof(cf);
    // fewer teams (whole warps) where their rows do not fit: the largest team's
    // need (256 antennas, 16 layers, 16 symbols) is 72 KB
    constexpr int WARP_TEAMS = TEAM >= 32 ? 1 : 32 / TEAM;
    int teams = kPlainThreads / TEAM;
    while (teams > WARP_TEAMS && teams * teamBytes > kMaxSmemPerCta) teams -= WARP_TEAMS;
    if (teams * teamBytes > kMaxSmemPerCta) return AERIAL_ERR_UNSUPPORTED;
    const int s = allow_max_smem<plain_kernel<MODE, LT, EX>>();
    if (s) return s;
    unsigned blocks = 0;
    for (int i = 0; i < p.nCells; i++) {
        p.cell[i].block0 = blocks;
        blocks += (unsigned)((p.cell[i].nSC + teams - 1) / teams);
    }
    p.teamValues = values;
    return launch_after(plain_kernel<MODE, LT, EX>, blocks, teams * TEAM, (size_t)teams * teamBytes, st, p);
}

template <int MODE, int LT>
static int launch_plain_l(PlainParams& p, cudaStream_t st) {
    bool exact = true;
    for (int i = 0; i < p.nCells; i++) exact = exact && p.cell[i].L == LT;
    return exact ? launch_plain_t<MODE, LT, true>(p, st) : launch_plain_t<MODE, LT, false>(p, st);
}

// Cells whose layers round up to the same tile, in one launch.
template <int MODE>
static int launch_plain(PlainParams& p, cudaStream_t st) {
    switch (layers_tile(p.cell[0].L)) {
        case 2: return launch_plain_l<MODE, 2>(p, st);
        case 4: return launch_plain_l<MODE, 4>(p, st);
        case 8: return launch_plain_l<MODE, 8>(p, st);
        default: return launch_plain_l<MODE, 16>(p, st);
    }
}

static PlainCell plain_cell(const cf* H, const cf* Y, int nSC, int A, int L, int S) {
    PlainCell c{};
    c.H = H;
    c.Y = Y;
    c.nSC = nSC;
    c.A = A;
    c.L = L;
    c.S = S;
    c.vecH = (L % 2) == 0 && ((uintptr_t)H & 15) == 0;
    c.vecY = (A % 2) == 0 && ((uintptr_t)Y & 15) == 0;
    return c;
}

template <int LT, bool EX>
static int launch_gram_t(const GramParams& p, cudaStream_t st) {
    const int s = allow_max_smem<gram_kernel<LT, EX>>();
    if (s) return s;
    constexpr int PER = 32 / gram_team(LT);
    // 256 antennas x 16 layers need 131 KB, the most
    const size_t smem = (size_t)PER * (p.A + 1) * plain_hs(p.L) * sizeof(cf);
    const unsigned blocks = (unsigned)((p.nSC + PER - 1) / PER);
    return launch_after(gram_kernel<LT, EX>, blocks, kGramThreads, smem, st, p);
}

static int launch_gram(const cf* H, float sigma2, cf* G, int nSC, int A, int L, cudaStream_t st) {
    const bool even = (L % 2) == 0;
    GramParams p{H, G, sigma2, nSC, A, L, even && ((uintptr_t)H & 15) == 0, even && ((uintptr_t)G & 15) == 0, {}, 0};
    const int part = (A + kGramParts - 1) / kGramParts;
    for (int q = 0; q < kGramParts; q++) p.rcpRows[q] = rcp_of(std::min(part, A - q * part));
    p.rcpPieces = rcp_of(p.vecH ? L / 2 : L);
    switch (layers_tile(L)) {
        case 2: return L == 2 ? launch_gram_t<2, true>(p, st) : launch_gram_t<2, false>(p, st);
        case 4: return L == 4 ? launch_gram_t<4, true>(p, st) : launch_gram_t<4, false>(p, st);
        case 8: return L == 8 ? launch_gram_t<8, true>(p, st) : launch_gram_t<8, false>(p, st);
        default: return L == 16 ? launch_gram_t<16, true>(p, st) : launch_gram_t<16, false>(p, st);
    }
}

static int launch_mmse_coef(const cf* G, const cf* H, cf* C, float* nI, int nSC, int A, int L, cudaStream_t st) {
    PlainParams p;
    p.nCells = 1;
    p.cell[0] = plain_cell(H, nullptr, nSC, A, L, 1);
    p.cell[0].G = G;
    p.cell[0].C = C;
    p.cell[0].nInv = nI;
    return launch_plain<kCoef>(p, st);
}

static int launch_coef_apply(const cf* C, const cf* Y, cf* O, int nSC, int nSym, int L, int A, cudaStream_t st) {
    PlainParams p;
    p.nCells = 1;
    p.cell[0] = plain_cell(nullptr, Y, nSC, A, L, nSym);
    p.cell[0].C = const_cast<cf*>(C);
    p.cell[0].O = O;
    p.cell[0].vecY = p.cell[0].vecY && ((uintptr_t)C & 15) == 0;
    return launch_plain<kApply>(p, st);
}

// Whether rows of `words` 4-byte LLR words may be stored whole (write_rows).
static bool llr_wide(const void* out, int words) {
    const uintptr_t need = words == 6 ? 16 : 4 * (uintptr_t)words;
    return (uintptr_t)out % need == 0;
}

// Blocks of a demapper launch with U symbols a thread.
static unsigned llr_blocks(int N, int U) { return ((unsigned)N + kLlrThreads * U - 1) / (kLlrThreads * U); }
static bool llr_large(int N) { return llr_blocks(N, kLlrSymbols) >= (unsigned)sm_count(); }

template <int U>
static int launch_llr_f32(const cf* in, const float* ni, float* out, int N, int n, int spn, cudaStream_t st) {
    const PamLut lut = pam_lut(n);
    const unsigned g = llr_blocks(N, U);
    const unsigned rcp = spn > 1 ? (unsigned)(0x100000000ull / (unsigned)spn) + 1u : 0u;
    const bool w = llr_wide(out, 2 * n);
    switch (n) {
        case 1: return launch_after(llr_f32_kernel<1, U>, g, kLlrThreads, 0, st, in, ni, out, N, spn, rcp, w, lut);
        case 2: return launch_after(llr_f32_kernel<2, U>, g, kLlrThreads, 0, st, in, ni, out, N, spn, rcp, w, lut);
        case 3: return launch_after(llr_f32_kernel<3, U>, g, kLlrThreads, 0, st, in, ni, out, N, spn, rcp, w, lut);
        default: return launch_after(llr_f32_kernel<4, U>, g, kLlrThreads, 0, st, in, ni, out, N, spn, rcp, w, lut);
    }
}
static int launch_llr_f32(const cf* in, const float* ni, float* out, int N, int n, int spn, cudaStream_t st) {
    return llr_large(N) ? launch_llr_f32<kLlrSymbols>(in, ni, out, N, n, spn, st)
                        : launch_llr_f32<1>(in, ni, out, N, n, spn, st);
}

template <int U>
static int launch_llr_f16(const __half2* in, const float* ni, __half* out, int N, int n, cudaStream_t st) {
    const PamLut lut = pam_lut(n);
    const unsigned g = llr_blocks(N, U);
    const bool w = llr_wide(out, n);
    switch (n) {
        case 1: return launch_after(llr_f16_kernel<1, U>, g, kLlrThreads, 0, st, in, ni, out, N, w, lut);
        case 2: return launch_after(llr_f16_kernel<2, U>, g, kLlrThreads, 0, st, in, ni, out, N, w, lut);
        case 3: return launch_after(llr_f16_kernel<3, U>, g, kLlrThreads, 0, st, in, ni, out, N, w, lut);
        default: return launch_after(llr_f16_kernel<4, U>, g, kLlrThreads, 0, st, in, ni, out, N, w, lut);
    }
}

}  // namespace aeq

namespace aeq {

int static_scratch(char** out);

// Load the plain chain's kernels on the current device (aerial_prepare).
template <typename K>
static int prepare_one(K* k) {
    cudaFuncAttributes at;
    return rt_status(cudaFuncGetAttributes(&at, k));
}
template <int MODE, int LT>
static int prepare_plain_l() {
    int s = prepare_one(plain_kernel<MODE, LT, true>);
    if (!s) s = allow_max_smem<plain_kernel<MODE, LT, true>>();
    if (!s) s = prepare_one(plain_kernel<MODE, LT, false>);
    return s ? s : allow_max_smem<plain_kernel<MODE, LT, false>>();
}
template <int MODE>
static int prepare_plain_mode() {
    int s = prepare_plain_l<MODE, 2>();
    if (!s) s = prepare_plain_l<MODE, 4>();
    if (!s) s = prepare_plain_l<MODE, 8>();
    return s ? s : prepare_plain_l<MODE, 16>();
}
template <int LT>
static int prepare_gram() {
    int s = prepare_one(gram_kernel<LT, true>);
    if (!s) s = allow_max_smem<gram_kernel<LT, true>>();
    if (!s) s = prepare_one(gram_kernel<LT, false>);
    return s ? s : allow_max_smem<gram_kernel<LT, false>>();
}
template <int N>
static int prepare_llr() {
    int s = prepare_one(llr_f16_kernel<N, 1>);
    if (!s) s = prepare_one(llr_f16_kernel<N, kLlrSymbols>);
    if (!s) s = prepare_one(llr_f32_kernel<N, 1>);
    return s ? s : prepare_one(llr_f32_kernel<N, kLlrSymbols>);
}
int prepare_plain_kernels() {
    int s = prepare_gram<2>();
    if (!s) s = prepare_gram<4>();
    if (!s) s = prepare_gram<8>();
    if (!s) s = prepare_gram<16>();
    if (!s) s = prepare_plain_mode<kCoef>();
    if (!s) s = prepare_plain_mode<kApply>();
    if (!s) s = prepare_plain_mode<kChain>();
    if (!s) s = prepare_llr<1>();
    if (!s) s = prepare_llr<2>();
    if (!s) s = prepare_llr<3>();
    if (!s) s = prepare_llr<4>();
    return s;
}

}  // namespace aeq

using namespace aeq;

extern "C" int aerial_gram(const aerial_cf32* H, float sigma2, aerial_cf32* G, int nSC, int nAnt, int nLayers,
                           void* stream) {
    if (!H || !G || !shape_ok(nSC, 1, nLayers, nAnt)) return AERIAL_ERR_INVALID_ARG;
    return launch_gram((const cf*)H, sigma2, (cf*)G, nSC, nAnt, nLayers, to_stream(stream));
}

extern "C" int aerial_mmse_coef(const aerial_cf32* G, const aerial_cf32* H, aerial_cf32* C, float* noiseInv, int nSC,
                                int nAnt, int nLayers, void* stream) {
    if (!G || !H || !C || !noiseInv || !shape_ok(nSC, 1, nLayers, nAnt)) return AERIAL_ERR_INVALID_ARG;
    return launch_mmse_coef((const cf*)G, (const cf*)H, (cf*)C, noiseInv, nSC, nAnt, nLayers, to_stream(stream));
}

extern "C" int aerial_coef_apply(const aerial_cf32* C, const aerial_cf32* Y_rx, aerial_cf32* Y_eq, int nSC, int nSym,
                                 int nLayers, int nAnt, void* stream) {
    if (!C || !Y_rx || !Y_eq || !shape_ok(nSC, nSym, nLayers, nAnt)) return AERIAL_ERR_INVALID_ARG;
    return launch_coef_apply((const cf*)C, (const cf*)Y_rx, (cf*)Y_eq, nSC, nSym, nLayers, nAnt, to_stream(stream));
}

extern "C" int aerial_llr(const aerial_ch2* softEst, const float* noiseInv, uint16_t* llrOut, int N, int nPamBits,
                          void* stream) {
    if (!softEst || !noiseInv || !llrOut || N < 1 || nPamBits < 1 || nPamBits > 4) return AERIAL_ERR_INVALID_ARG;
    const auto run = llr_large(N) ? launch_llr_f16<kLlrSymbols> : launch_llr_f16<1>;
    return run((const __half2*)softEst, noiseInv, (__half*)llrOut, N, nPamBits, to_stream(stream));
}

extern "C" int aerial_llr_f32(const aerial_cf32* softEst, const float* noiseInv, float* llrOut, int N, int nPamBits,
                              int nSymPerNoise, void* stream) {
    if (!softEst || !noiseInv || !llrOut || N < 1 || nPamBits < 1 || nPamBits > 4 || nSymPerNoise < 1)
        return AERIAL_ERR_INVALID_ARG;
    return launch_llr_f32((const cf*)softEst, noiseInv, llrOut, N, nPamBits, nSymPerNoise, to_stream(stream));
}

// ---------------------------------------------------------------------------
// The plain chain over cells.  The chain's kernel keeps G, C and noiseInv on
// chip; the workspace (these and Y_eq of the largest cell) is part of the
// interface, checked, and used where a cell has to run stage by stage.
// ---------------------------------------------------------------------------
struct PlainWs {
    size_t C, nInv, yeq, total;        // offsets; G comes first
};
static PlainWs plain_ws_cell(const aerial_cell_desc& c) {
    size_t nSC = (size_t)c.nPRB * 12;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    PlainWs w;
    w.C = al(nSC * c.nLayers * c.nLayers * sizeof(cf));
    w.nInv = w.C + al(nSC * c.nLayers * c.nAnt * sizeof(cf));
    w.yeq = w.nInv + al(nSC * c.nLayers * sizeof(float));
    w.total = w.yeq + al(nSC * c.nLayers * c.nSym * sizeof(cf));
    return w;
}

extern "C" size_t aerial_pusch_eq_plain_workspace(const aerial_cell_desc* cells, int nCells) {
    size_t m = 0;
    for (int i = 0; cells && i < nCells; i++) {
        size_t w = plain_ws_cell(cells[i]).total;
        if (w > m) m = w;
    }
    return m;
}

// The checks of one cell, before anything is launched.
static int plain_cell_check(const aerial_cell_desc& c) {
    if (c.nPRB < 1 || c.nPRB > AERIAL_MAX_PRB) return AERIAL_ERR_INVALID_ARG;
    if (!c.H || !c.Y_rx || !c.llr || c.nPamBits < 1 || c.nPamBits > 4 ||
        !shape_ok(c.nPRB * 12, c.nSym, c.nLayers, c.nAnt))
        return AERIAL_ERR_INVALID_ARG;
    if (c.format != AERIAL_FMT_CF32) return AERIAL_ERR_UNSUPPORTED;   // the FP32 chain reads complex64 only
    return AERIAL_OK;
}

// A cell's buffers.  The specification runs the cells of a call in order, and
// each cell stage by stage, so a later cell may use what an earlier one wrote or
// write over what it is done with, and a cell's outputs may lie over inputs that
// its earlier stages have read.  The kernel runs all its subcarriers at once.
struct PlainBuffers {
    uintptr_t in[2], inEnd[2], out[2], outEnd[2];
};
static PlainBuffers plain_buffers(const aerial_cell_desc& c) {
    const size_t nSC = (size_t)c.nPRB * 12, res = nSC * c.nLayers * c.nSym;
    PlainBuffers b;
    b.in[0] = (uintptr_t)c.H;
    b.inEnd[0] = b.in[0] + nSC * c.nAnt * c.nLayers * sizeof(cf);
    b.in[1] = (uintptr_t)c.Y_rx;
    b.inEnd[1] = b.in[1] + nSC * c.nSym * c.nAnt * sizeof(cf);
    b.out[0] = (uintptr_t)c.llr;
    b.outEnd[0] = b.out[0] + res * 2 * c.nPamBits * sizeof(float);
    b.out[1] = (uintptr_t)c.Y_eq;
    b.outEnd[1] = c.Y_eq ? b.out[1] + res * sizeof(cf) : b.out[1];
    return b;
}
// Whether a buffer that `a` writes overlaps one that `b` reads, or (outs) writes.
static bool plain_touches(const PlainBuffers& a, const PlainBuffers& b, bool outs) {
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++)
            if ((a.out[i] < b.inEnd[j] && b.in[j] < a.outEnd[i]) ||
                (outs && a.out[i] < b.outEnd[j] && b.out[j] < a.outEnd[i]))
                return true;
    return false;
}

static int run_staged(const aerial_cell_desc& c, char* ws, cudaStream_t st) {
    const PlainWs w = plain_ws_cell(c);
    const int nSC = c.nPRB * 12;
    const cf* H = (const cf*)c.H;
    cf *G = (cf*)ws, *C = (cf*)(ws + w.C), *yeq = c.Y_eq ? (cf*)c.Y_eq : (cf*)(ws + w.yeq);
    float* nInv = (float*)(ws + w.nInv);
    int s = launch_gram(H, c.sigma2, G, nSC, c.nAnt, c.nLayers, st);
    if (!s) s = launch_mmse_coef(G, H, C, nInv, nSC, c.nAnt, c.nLayers, st);
    if (!s) s = launch_coef_apply(C, (const cf*)c.Y_rx, yeq, nSC, c.nSym, c.nLayers, c.nAnt, st);
    return s ? s : launch_llr_f32(yeq, nInv, c.llr, nSC * c.nLayers * c.nSym, c.nPamBits, c.nSym, st);
}

// Consecutive cells whose layers share a tile and whose buffers are independent
// go into one launch; a cell whose outputs overlap its own inputs runs stage by
// stage in the workspace.
static int run_plain(const aerial_cell_desc* cells, int nCells, char* ws, cudaStream_t st) {
    PlainBuffers held[AERIAL_MAX_CELLS];
    for (int i = 0; i < nCells;) {
        PlainParams p;
        p.nCells = 0;
        const int tile = layers_tile(cells[i].nLayers);
        long subcarriers = 0;                        // block indices stay in 31 bits
        bool staged = false;
        for (; i < nCells && p.nCells < AERIAL_MAX_CELLS && layers_tile(cells[i].nLayers) == tile; i++) {
            const aerial_cell_desc& c = cells[i];
            const int nSC = c.nPRB * 12;
            if (p.nCells && subcarriers + nSC > INT32_MAX / 2) break;
            const PlainBuffers b = plain_buffers(c);
            bool apart = !plain_touches(b, b, false);
            staged = !apart && !p.nCells;
            for (int j = 0; j < p.nCells && apart; j++)
                apart = !plain_touches(held[j], b, true) && !plain_touches(b, held[j], false);
            if (!apart) break;
            subcarriers += nSC;
            held[p.nCells] = b;
            PlainCell& d = p.cell[p.nCells++];
            d = plain_cell((const cf*)c.H, (const cf*)c.Y_rx, nSC, c.nAnt, c.nLayers, c.nSym);
            d.O = (cf*)c.Y_eq;
            d.llr = c.llr;
            d.sigma2 = c.sigma2;
            d.nPam = c.nPamBits;
            d.lut = pam_lut(c.nPamBits);
        }
        const int s = staged ? run_staged(cells[i++], ws, st) : launch_plain<kChain>(p, st);
        if (s) return s;
    }
    return AERIAL_OK;
}

extern "C" int aerial_pusch_eq_plain(const aerial_cell_desc* cells, int nCells, void* workspace, size_t wsBytes,
                                     void* stream) {
    if (!cells || nCells < 1 || !workspace) return AERIAL_ERR_INVALID_ARG;
    for (int i = 0; i < nCells; i++) {
        const int s = plain_cell_check(cells[i]);
        if (s != AERIAL_OK) return s;
        if (plain_ws_cell(cells[i]).total > wsBytes) return AERIAL_ERR_INVALID_ARG;
    }
    return run_plain(cells, nCells, static_cast<char*>(workspace), to_stream(stream));
}

// ---------------------------------------------------------------------------
// The plain chain for callers that must not allocate device memory.
//
// Some hosts cannot call cudaMalloc on the path that equalizes a slot: a
// real-time receiver loop where an allocation may block or synchronize the
// device and miss the slot deadline, or a plugin inside a framework that owns
// all device memory and hands out none.  The chain's intermediates (G, C,
// noiseInv) live in shared memory, so this entry point needs no device memory
// but for a cell that has to run stage by stage, which takes the library's static
// scratch; a batch whose largest cell's intermediates would exceed its
// AERIAL_STATIC_SCRATCH_BYTES is refused, as the interface states.
// ---------------------------------------------------------------------------
extern "C" int aerial_pusch_eq_plain_static(const aerial_cell_desc* cells, int nCells, void* stream) {
    if (!cells || nCells < 1) return AERIAL_ERR_INVALID_ARG;
    for (int i = 0; i < nCells; i++) {
        const int s = plain_cell_check(cells[i]);
        if (s != AERIAL_OK) return s;
    }
    if (aerial_pusch_eq_plain_workspace(cells, nCells) > (size_t)AERIAL_STATIC_SCRATCH_BYTES)
        return AERIAL_ERR_SCRATCH_LIMIT;
    char* ws = nullptr;
    for (int i = 0; i < nCells && !ws; i++) {
        const PlainBuffers b = plain_buffers(cells[i]);
        if (!plain_touches(b, b, false)) continue;
        const int s = static_scratch(&ws);
        if (s != AERIAL_OK) return s;
    }
    return run_plain(cells, nCells, ws, to_stream(stream));
}
