// coef_tc.cu -- coef_apply on the tensor cores: the semantics of
// coef_apply_v2_wmma (src/aerial_coef_wmma.cu:146-239), FP16 operands and
// FP32 accumulation, without its shared-memory staging.
//
// Y_eq[l][s] = sum_a C[l][a] Y[s][a] (no conjugate) as a real-embedded
// mma.sync m16n8k16: with B pairs (Re Y, Im Y), A row l carries
// (Re C, -Im C) -> Re out and A row l+8 carries (Im C, Re C) -> Im out.
// Thread (g, c) of k-step j owns antennas 8j+2c and 8j+2c+1, so its A operand
// is C[l][8j+2c .. +1] and its B operand Y[s][8j+2c .. +1]: one 16-byte load
// each, straight into registers, several k-steps' loads ahead of their MMAs.  One
// warp per subcarrier; L <= 16 (two m-tiles), nSym <= 16 (two n-tiles).
#include <algorithm>

#include "common.cuh"

namespace aeq {

__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

__device__ __forceinline__ void mma_f16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The pair p[a0], p[a0 + 1] of a row of A values; zeros for a row that does
// not exist (in = false) and past the row's end.  Ordinary and volatile loads
// (wait_previous): C and Y are what earlier kernels of the stream wrote.
template <bool VEC>
__device__ __forceinline__ float4 ld_pair(const float2* p, int a0, int A, bool in) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (VEC) {                         // A even, 16-byte rows
        if (in && a0 < A)
            asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                         : "l"(__cvta_generic_to_global(p + a0)));
    } else {
        if (in && a0 < A) { const float2 t = p[a0]; v.x = t.x; v.y = t.y; }
        if (in && a0 + 1 < A) { const float2 t = p[a0 + 1]; v.z = t.x; v.w = t.y; }
    }
    return v;
}

// k-steps whose loads are issued together.  The kernel is bound by the bytes
// it has in flight: one k-step's three 16-byte loads a lane before their MMAs
// left HBM at 4.2 TB/s.  8 slots of 1,584 subcarriers, 64 antennas, 8 layers,
// 14 symbols (154 MB): 37 us, 30 us with four k-steps at a time, 27 us with eight.
// Up to 8 antennas there is one k-step, and the registers of eight only take
// room from other warps (3,276 subcarriers x 8 antennas x 4 layers x 14 symbols
// 2.9 us with eight, 1.9 us with one).
constexpr int kTcSteps = 8;

// NMT, NNT: 8-layer and 8-symbol tiles; STEPS: k-steps loaded together.
template <int NMT, int NNT, bool VEC, int STEPS>
__global__ void __launch_bounds__(256) coef_apply_tc_kernel(const float2* C, const float2* Y, float2* O, int nSC, int nSym, int L, int A) {
    wait_previous();
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, c = lane & 3;
    const long w0 = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nw = ((long)gridDim.x * blockDim.x) >> 5;
    const int nK = (A + 7) >> 3;
    for (long sc = w0; sc < nSC; sc += nw) {
        float acc[NMT][NNT][4] = {};
        const float2* Cs = C + sc * (long)L * A;
        const float2* Ys = Y + sc * (long)nSym * A;
        for (int j0 = 0; j0 < nK; j0 += STEPS) {
            float4 cv[STEPS][NMT], yv[STEPS][NNT];
#pragma unroll
            for (int j = 0; j < STEPS; j++) {
                const int a0 = 8 * (j0 + j) + 2 * c;       // past A for steps past nK: zeros
#pragma unroll
                for (int mt = 0; mt < NMT; mt++)
                    cv[j][mt] = ld_pair<VEC>(Cs + (long)(8 * mt + g) * A, a0, A, 8 * mt + g < L);
#pragma unroll
                for (int nt = 0; nt < NNT; nt++)
                    yv[j][nt] = ld_pair<VEC>(Ys + (long)(8 * nt + g) * A, a0, A, 8 * nt + g < nSym);
            }
#pragma unroll
            for (int j = 0; j < STEPS; j++) {
                if (j0 + j >= nK) break;
                uint32_t b[NNT][2];
#pragma unroll
                for (int nt = 0; nt < NNT; nt++) {
                    b[nt][0] = h2u(__floats2half2_rn(yv[j][nt].x, yv[j][nt].y));
                    b[nt][1] = h2u(__floats2half2_rn(yv[j][nt].z, yv[j][nt].w));
                }
#pragma unroll
                for (int mt = 0; mt < NMT; mt++) {
                    const float4 v = cv[j][mt];
                    const uint32_t p0 = h2u(__floats2half2_rn(v.x, v.y)), p1 = h2u(__floats2half2_rn(v.z, v.w));
                    const uint32_t r0 = p0 ^ 0x80000000u, r1 = p1 ^ 0x80000000u;          // (Re, -Im)
                    const uint32_t i0 = __byte_perm(p0, 0, 0x1032), i1 = __byte_perm(p1, 0, 0x1032);  // (Im, Re)
#pragma unroll
                    for (int nt = 0; nt < NNT; nt++) mma_f16(acc[mt][nt], r0, i0, r1, i1, b[nt][0], b[nt][1]);
                }
            }
        }
#pragma unroll
        for (int mt = 0; mt < NMT; mt++)
#pragma unroll
            for (int nt = 0; nt < NNT; nt++) {
                const int l = 8 * mt + g, s = 8 * nt + 2 * c;
                if (l < L) {
                    float2* o = O + (sc * L + l) * (long)nSym;
                    if (s < nSym) o[s] = make_float2(acc[mt][nt][0], acc[mt][nt][2]);
                    if (s + 1 < nSym) o[s + 1] = make_float2(acc[mt][nt][1], acc[mt][nt][3]);
                }
            }
    }
}

template <int NMT, int NNT>
static int launch_tc(const float2* C, const float2* Y, float2* O, int nSC, int nSym, int L, int A, bool vec,
                      cudaStream_t st) {
    // a warp per subcarrier, at most eight blocks an SM: an SM holds one or two at a
    // time, and later ones start as others finish
    const unsigned blocks = (unsigned)std::min(((long)nSC + 7) / 8, (long)sm_count() * 8);
    auto kernel = A <= 8 ? (vec ? coef_apply_tc_kernel<NMT, NNT, true, 1> : coef_apply_tc_kernel<NMT, NNT, false, 1>)
                         : (vec ? coef_apply_tc_kernel<NMT, NNT, true, kTcSteps>
                                : coef_apply_tc_kernel<NMT, NNT, false, kTcSteps>);
    return launch_after(kernel, blocks, 256, 0, st, C, Y, O, nSC, nSym, L, A);
}

}  // namespace aeq

using namespace aeq;

extern "C" int aerial_coef_apply_tc(const aerial_cf32* C, const aerial_cf32* Y_rx, aerial_cf32* Y_eq, int nSC,
                                    int nSym, int nLayers, int nAnt, void* stream) {
    if (!C || !Y_rx || !Y_eq || nSC < 1 || nSym < 1 || nSym > AERIAL_MAX_SYMS || nLayers < 1 ||
        nLayers > AERIAL_MAX_LAYERS || nAnt < 1 || nAnt > AERIAL_MAX_ANTS)
        return AERIAL_ERR_INVALID_ARG;
    const bool vec = (nAnt % 2) == 0 && ((uintptr_t)C & 15) == 0 && ((uintptr_t)Y_rx & 15) == 0;
    auto run = nLayers > 8 ? (nSym > 8 ? launch_tc<2, 2> : launch_tc<2, 1>)
                           : (nSym > 8 ? launch_tc<1, 2> : launch_tc<1, 1>);
    return run((const float2*)C, (const float2*)Y_rx, (float2*)Y_eq, nSC, nSym, nLayers, nAnt, vec, to_stream(stream));
}
