// f64 exact path: instantiations and launchers.  This file is compiled with
// --fmad=false so that every f64 multiply-add follows the reference's
// operation order (no contraction), as the oracle and the Rust code do.
#include "lkg_score_warp.cuh"

namespace lkg {

template <int G>
static size_t exact_smem() {
    return (size_t)(WK_THREADS / 32) * (sizeof(WSlots<G>) + sizeof(ComplexDev) + sizeof(WExact<G>));
}

// WK_BLOCKS_EXACT blocks (1 KB more each, in units of 128 bytes) within the
// largest shared-memory share but one: beyond it the SM's L1 halves, and 200
// dna poses take 356 us instead of 335
static_assert(((((WK_THREADS / 32) * (sizeof(WSlots<16>) + sizeof(ComplexDev) + sizeof(WExact<16>)) + 1024) + 127) / 128) *
                      128 * WK_BLOCKS_EXACT <= 196 * 1024,
              "the f64 kernel's shared memory leaves L1 its room");

template <int G, bool IFACE, bool NP>
static cudaError_t launch_exact_gi(const LaunchParams& p, int blocks, cudaStream_t s) {
    const size_t sm = exact_smem<G>();
    cudaError_t e = cudaFuncSetAttribute(k_score_warp<G, IFACE, NP, false, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_score_warp<G, IFACE, NP, false, true><<<blocks, WK_THREADS, sm, s>>>(p);
    return cudaGetLastError();
}
template <int G>
static cudaError_t launch_exact_g(const LaunchParams& p, int blocks, cudaStream_t s) {
    if (p.iface)
        return p.parts ? launch_exact_gi<G, true, true>(p, blocks, s) : launch_exact_gi<G, true, false>(p, blocks, s);
    return p.parts ? launch_exact_gi<G, false, true>(p, blocks, s) : launch_exact_gi<G, false, false>(p, blocks, s);
}

cudaError_t launch_score_exact(const LaunchParams& p, int blocks, cudaStream_t s) {
    if (p.atom_elec) return cudaErrorInvalidValue;   // per-atom outputs are k_score_tiles<float>'s
    if (p.group <= 0 || p.tile % p.group) return cudaErrorInvalidValue;
    switch (p.group) {
        case 4: return launch_exact_g<4>(p, blocks, s);
        case 16: return launch_exact_g<16>(p, blocks, s);
        case 32: return launch_exact_g<32>(p, blocks, s);
        default: return cudaErrorInvalidValue;   // groups of 8 are searched as 16
    }
}

cudaError_t launch_desolv_exact(const LaunchParams& p, int threads, int blocks, int hcap, cudaStream_t s) {
    size_t sm = desolv_smem_bytes(hcap, true);
    cudaError_t e = cudaFuncSetAttribute(k_score_desolv<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_score_desolv<double><<<blocks, threads, sm, s>>>(p);
    return cudaGetLastError();
}

template <int G>
static int occ_exact_g() {
    int n = 0;
    const size_t sm = exact_smem<G>();
    cudaFuncSetAttribute(k_score_warp<G, false, false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_score_warp<G, false, false, false, true>, WK_THREADS, sm);
    return n;
}
int max_blocks_score_exact(int group) {
    switch (group) {
        case 4: return occ_exact_g<4>();
        case 16: return occ_exact_g<16>();
        case 32: return occ_exact_g<32>();
        default: return 0;
    }
}
int max_blocks_desolv_exact(int threads, int hcap) {
    int n = 0;
    size_t sm = desolv_smem_bytes(hcap, true);
    cudaFuncSetAttribute(k_score_desolv<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_score_desolv<double>, threads, sm);
    return n;
}

}  // namespace lkg
