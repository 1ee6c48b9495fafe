// lbm_kernels_inst.cuh -- instantiates the kernels of one storage type.
// Included by lbm_kernels_<type>.cu with LBM_S (element type), LBM_T (F-dump
// element type) and LBM_SFX (launcher suffix) defined.
#include <algorithm>

#include "lbm_kernels.cuh"
#include "lbm_launch.h"

namespace lbm {

#define LBM_CAT2(a, b) a##b
#define LBM_CAT(a, b) LBM_CAT2(a, b)

// One iteration (or reduction pass) with 16-byte vectors as two launches: the
// interior rows on s, the face rows on sf (s when null), so that the two can
// run side by side.  *nparts gets the number of reduction partial slots the
// two launches use.
template <int MODE>
static cudaError_t launch_rows_mode(const StepArgs &a0, unsigned block, cudaStream_t s, cudaStream_t sf,
                                    unsigned *nparts)
{
    constexpr int V = 16 / (int)sizeof(LBM_S);
    StepArgs a = a0;
    a.nvx = a0.dim / V;
    const size_t m = (size_t)(a.dim - 4);
    const unsigned gi = (unsigned)((m * m * (size_t)a.nvx + block - 1) / block);
    const unsigned gf = (unsigned)(((size_t)4 * (a.dim - 3) * (size_t)a.nvx + block - 1) / block);
    a.partial_base = 0u;
    if (gi > 0) pull_kernel<LBM_S, MODE, 16, ROWS_INTERIOR><<<gi, block, 0, s>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    a.partial_base = gi;
    pull_kernel<LBM_S, MODE, 16, ROWS_FACES><<<gf, block, 0, sf ? sf : s>>>(a);
    if (nparts) *nparts = gi + gf;
    return cudaGetLastError();
}

// One AA iteration (or reduction pass) of phase PHASE: interior rows, then
// face rows.
template <int VB, int PHASE>
static cudaError_t launch_aa_phase(int mode, const StepArgs &a0, unsigned block, cudaStream_t s, unsigned *nparts)
{
    constexpr int V = VB / (int)sizeof(LBM_S);
    StepArgs a = a0;
    a.nvx = a0.dim / V;
    const size_t m = (size_t)(a.dim - 4);
    const unsigned gi = (unsigned)((m * m * (size_t)a.nvx + block - 1) / block);
    const unsigned gf = (unsigned)(((size_t)4 * (a.dim - 3) * (size_t)a.nvx + block - 1) / block);
    for (int pass = 0; pass < 2; ++pass) {
        const unsigned grid = pass == 0 ? gi : gf;
        if (grid == 0) continue;
        a.partial_base = pass == 0 ? 0u : gi;
        if (pass == 0) {
            switch (mode) {
            case MODE_STEP: aa_kernel<LBM_S, MODE_STEP, VB, ROWS_INTERIOR, PHASE><<<grid, block, 0, s>>>(a); break;
            case MODE_STEP_MACRO:
                aa_kernel<LBM_S, MODE_STEP_MACRO, VB, ROWS_INTERIOR, PHASE><<<grid, block, 0, s>>>(a);
                break;
            case MODE_REDUCE: aa_kernel<LBM_S, MODE_REDUCE, VB, ROWS_INTERIOR, PHASE><<<grid, block, 0, s>>>(a); break;
            default: return cudaErrorInvalidValue;
            }
        } else {
            switch (mode) {
            case MODE_STEP: aa_kernel<LBM_S, MODE_STEP, VB, ROWS_FACES, PHASE><<<grid, block, 0, s>>>(a); break;
            case MODE_STEP_MACRO:
                aa_kernel<LBM_S, MODE_STEP_MACRO, VB, ROWS_FACES, PHASE><<<grid, block, 0, s>>>(a);
                break;
            case MODE_REDUCE: aa_kernel<LBM_S, MODE_REDUCE, VB, ROWS_FACES, PHASE><<<grid, block, 0, s>>>(a); break;
            default: return cudaErrorInvalidValue;
            }
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (nparts) *nparts = gi + gf;
    return cudaSuccess;
}

// AA variant: 8-byte vectors for FP32 (its fastest two-lattice width), 16-byte
// otherwise; a.aa_phase picks the A- or B-step.
cudaError_t LBM_CAT(launch_aa_, LBM_SFX)(int mode, const StepArgs &a, unsigned block, cudaStream_t s,
                                         unsigned *nparts)
{
    constexpr int VB = sizeof(LBM_S) == 4 ? 8 : 16;
    return a.aa_phase ? launch_aa_phase<VB, 1>(mode, a, block, s, nparts)
                      : launch_aa_phase<VB, 0>(mode, a, block, s, nparts);
}

cudaError_t LBM_CAT(launch_reduce_, LBM_SFX)(const StepArgs &a, unsigned block, cudaStream_t s, unsigned *nparts)
{
    return launch_rows_mode<MODE_REDUCE>(a, block, s, nullptr, nparts);
}

// (16-bit storage on large lattices, FP32 with 16-byte vectors; see step_shape
// in lbm_capi.cu)
cudaError_t LBM_CAT(launch_rows_, LBM_SFX)(int mode, const StepArgs &a, unsigned block, cudaStream_t s,
                                           cudaStream_t sf)
{
    if constexpr (sizeof(LBM_S) < 8) {
        switch (mode) {
        case MODE_STEP: return launch_rows_mode<MODE_STEP>(a, block, s, sf, nullptr);
        case MODE_STEP_MACRO: return launch_rows_mode<MODE_STEP_MACRO>(a, block, s, sf, nullptr);
        }
    }
    return cudaErrorInvalidValue;
}

// One iteration with VB-byte vectors in one launch, as a programmatic
// dependent of the launch before it on the stream.
template <int VB, int MODE>
static cudaError_t launch_step_mode(const StepArgs &a, unsigned block, cudaStream_t s)
{
    constexpr unsigned V = VB / (int)sizeof(LBM_S), VF = face_vec<LBM_S>();
    const unsigned dim = (unsigned)a.dim, m = dim - 4;
    const size_t ni = (size_t)m * m * (dim / V), nf = (size_t)4 * (dim - 3) * (dim / VF);
    if (ni >> 31) return cudaErrorInvalidValue;  // FastDiv's range
    StepRows r;
    r.face_blocks = (unsigned)((nf + block - 1) / block);
    r.div_face = FastDiv(dim / VF);
    r.div_row = FastDiv(dim / V);
    r.div_plane = FastDiv(m);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(r.face_blocks + (unsigned)((ni + block - 1) / block));
    lc.blockDim = dim3(block);
    lc.stream = s;
    lc.attrs = at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, step_kernel<LBM_S, MODE, VB>, a, r);
}

template <int VB> static cudaError_t launch_step_vb(int mode, const StepArgs &a, unsigned block, cudaStream_t s)
{
    switch (mode) {
    case MODE_STEP: return launch_step_mode<VB, MODE_STEP>(a, block, s);
    case MODE_STEP_MACRO: return launch_step_mode<VB, MODE_STEP_MACRO>(a, block, s);
    case MODE_STEP_ADJ:  // (16-bit storage: 8-byte vectors, launch_pull)
        if constexpr (sizeof(LBM_S) != 2 || VB < 16) return launch_step_mode<VB, MODE_STEP_ADJ>(a, block, s);
        return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t LBM_CAT(launch_step_, LBM_SFX)(int vb, int mode, const StepArgs &a, unsigned block, cudaStream_t s)
{
    switch (vb) {
    case 16:
        if constexpr (sizeof(LBM_S) != 4) return launch_step_vb<16>(mode, a, block, s);
        break;
    case 8: return launch_step_vb<8>(mode, a, block, s);
    case 4:
        if constexpr (sizeof(LBM_S) < 8) return launch_step_vb<4>(mode, a, block, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t LBM_CAT(launch_staged_, LBM_SFX)(int mode, const StepArgs &a, unsigned grid, unsigned block,
                                             size_t smem, cudaStream_t s)
{
    if (grid == 0) return cudaSuccess;
    switch (mode) {
    case MODE_STEP: pull_staged_kernel<LBM_S, MODE_STEP><<<grid, block, smem, s>>>(a); break;
    case MODE_STEP_MACRO: pull_staged_kernel<LBM_S, MODE_STEP_MACRO><<<grid, block, smem, s>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

const void *LBM_CAT(staged_kernel_ptr_, LBM_SFX)(int mode)
{
    switch (mode) {
    case MODE_STEP: return (const void *)pull_staged_kernel<LBM_S, MODE_STEP>;
    case MODE_STEP_MACRO: return (const void *)pull_staged_kernel<LBM_S, MODE_STEP_MACRO>;
    default: return nullptr;
    }
}

cudaError_t LBM_CAT(launch_init_, LBM_SFX)(const InitArgs &a, cudaStream_t s)
{
    const unsigned block = 256;
    // four consecutive x-sites per thread (dim % 4 == 0), and the sites near the
    // walls: 12 d of most planes, all d^2 of six (a thread each up to 90^3, then
    // in turns: empty blocks elsewhere would cost more)
    const unsigned d = (unsigned)a.dim, nb = (d * d / 4 + block - 1) / block;
    const unsigned ns = std::min((d * d + block - 1) / block, std::max((12 * d + block - 1) / block, 32u));
    init_kernel<LBM_S><<<dim3(nb + ns, d), block, 0, s>>>(a, nb);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || a.noise_sigma == 0.0 || a.dim < 5) return e;
    const size_t m = (size_t)(a.dim - 4);
    noise_kernel<LBM_S><<<dim3((unsigned)((m * m + block - 1) / block), (unsigned)m), block, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t LBM_CAT(launch_dump_, LBM_SFX)(const DumpArgs &a, cudaStream_t s)
{
    const unsigned block = 256;
    const size_t grid = (a.count / (a.four ? 4 : 1) + block - 1) / block;  // a.count is a multiple of 4
    if (grid == 0) return cudaSuccess;
    if (a.four) dump_f_kernel<LBM_S, LBM_T><<<(unsigned)grid, block, 0, s>>>(a);
    else dump_f_any_kernel<LBM_S, LBM_T><<<(unsigned)grid, block, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t LBM_CAT(launch_load_, LBM_SFX)(const DumpArgs &a, cudaStream_t s)
{
    const unsigned block = 256;
    const size_t grid = (a.count / (a.four ? 4 : 1) + block - 1) / block;  // a.count is a multiple of 4
    if (grid == 0) return cudaSuccess;
    if (a.four) load_f_kernel<LBM_S, LBM_T><<<(unsigned)grid, block, 0, s>>>(a);
    else load_f_any_kernel<LBM_S, LBM_T><<<(unsigned)grid, block, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace lbm
