// Warp-independent fused scorer: dna / pydock / vdw and the
// reference-compatible flag combinations in both precisions (f32 pair math, or
// EXACT: f64 in the reference's operation order), and the fast cpydock kernel.
//
// Every warp fetches its own work units from the global counter; there is
// no block-level barrier inside the loop, so a warp that meets a crowded
// interface never holds up the warps beside it.  A work unit is a tile of
// `p.tile` ligand atoms of one pose, in small launches a part of one (`p.sub`
// groups), in groups of G consecutive atoms (spatially compact: the ligand is
// ordered by recursive coordinate bisection in groups of G) whose bounding
// sphere (centre, radius rho, in the ligand frame) is computed on the host, as
// is the sphere of every quad of 4 consecutive atoms.  Per group:
//   1. lanes 0..G-1 transform their atom in f64 (kept as an f32 value plus
//      the rounding residual), add the far-field term q * phi(x'), and park
//      position and parameters in shared memory, two neighbouring atoms
//      interleaved (a slot pair);
//   2. the receptor rows (z, y cells of edge h) within 10 A + rho of the
//      posed centre are enumerated 32 at a time (one per lane), trimmed in x
//      to sub-cells of edge h / xsub, and turned into contiguous atom spans;
//   3. 32 candidates at a time (coalesced float4 loads, the next chunk loaded
//      while this one is tested) are tested against the spheres of the
//      group's quads (10 A + the quad's radius) and join the candidate list
//      of every quad they reach (a ballot and a popcount place them);
//   4. a full list, and at the group's end every list, is scored densely:
//      lane = (candidate, slot pair) with the slot pair in registers, every
//      listed candidate against all 4 atoms of the quad, the exact d^2 <= 100
//      test masking the sums.
// The lists of 4 atoms hold 1.8-1.9 candidate tests per near pair (CPU model
// at the batched workload's and a protein's atom densities; lists of 8 atoms
// 2.4, of 16 atoms 3.3), so the pair terms are computed on every test, on
// packed f32 pairs, without collecting the hits first.
// A group's sums are reduced over the warp at the group's end and added in
// group order: a pose's score does not depend on which warp took which part.
#pragma once
#include <type_traits>

#include "lkg_score.cuh"

namespace lkg {

constexpr int WK_THREADS = 128;   // 4 independent warps per block

// candidates a quad's list holds: lists are scored when one holds more than
// W_LIST - 64 (two chunks add at most 64).  Long enough that most groups are
// scored once, at their end, short enough to leave L1 its room.  3000 vdw poses
// of a 1300-atom ligand on 12,600 atoms at protein density, ms at 128 / 160 /
// 192 / 256 / 384: groups of 4 (one list): 2.94 / 2.89 / 2.84 / 2.80 / 2.76;
// groups of 16 (four): 2.04 / 1.99 / 2.00 / 2.02 / 2.18; groups of 32 (eight):
// 2.35 / 2.45 / 2.41 / 2.65 / 3.59, 2.44 at 96.  Groups of 8 (cpydock, 300
// atoms): 0.94 at 192 and at 256.
template <int G> constexpr int W_LIST = G <= 8 ? 256 : (G == 32 ? 128 : 192);

// resident blocks per SM the register budget is sized for: 72 registers (a
// few spills in the cold parts).  Sixteen complexes of 2,000 poses: 12.5 ms at
// 5 blocks, 12.4 at 6, 12.1 at 7, 12.5 at 8.  Groups of 32, whose lists leave
// room for no more: 5 (3000 vdw poses of 300 atoms on 5000 at chain density, ms
// at 5 / 6 / 7 blocks: 0.255 / 0.266 / 0.289 with 7 A cells, 0.291 / 0.313 /
// 0.360 with 2.5 A; 1300 atoms on 12,600 at protein density 2.17 / 2.20 / 2.34).
template <int G> constexpr int WK_BLOCKS = G == 32 ? 5 : 7;
// f64 mode: bound by the latency of its f64 chains, so more warps win over
// fewer spills (200 poses: 440 us at 4 blocks, 399 at 5, 387 at 6, 370 at 7,
// 360 at 8)
constexpr int WK_BLOCKS_EXACT = 8;

// per-warp desolvation state of the two slot sets (cpydock): the slot
// atoms' f64 positions, their running minimum d^2 to non-excluded receptor
// atoms (f64 bits; non-negative doubles order like their bit patterns), and
// the hits within 6.4 A that wait for it (slot << 26 | receptor index, bit 31
// when the receptor atom's minimum is wanted too): fewer than 32 wait when a
// step of 64 tests adds its own
template <int G>
struct WDes {
    double lx[2 * G], ly[2 * G], lz[2 * G];
    unsigned long long lmin[2 * G];
    unsigned hit[96];
};

// interface words a warp collects in shared memory before merging them into
// the pose's bits (larger sets go to HBM directly)
constexpr int W_IBUF = 32;

// two neighbouring ligand atoms, interleaved: every field is a packed f32
// pair as the pair math takes it
struct __align__(16) WPair {
    float x[2], y[2], z[2];      // f64 position rounded to f32
    float rx[2], ry[2], rz[2];   // and its rounding residual
    float q[2], sv[2], r[2];     // charge, sqrt eps, radius
    float h[2];                  // 0.75 for a heavy atom, else 0
};

template <int G>
struct WSlots {
    Rot rot;                          // pose of the current work unit
    float scan, stretch;              // and its search radius around an atom, its factor on lengths (w_pose)
    WPair pair[G / 2];
    float4 quad[(G + 3) / 4];         // candidate test of each quad's sphere: -2 c', R^2 - |c'|^2 (c' = c - group centre)
    unsigned list[(G + 3) / 4][W_LIST<G> + 16];   // receptor indices of each quad's candidates (and padding)
    int first[(G + 3) / 4], cnt[(G + 3) / 4];   // the part of each list that is scored
    float one[2];                     // 1, 1 (see w_d2)
    double* part;                     // the unit's group partials (split tiles), or null
    int row[32];                      // per non-empty row of the current 32: first atom - the row's candidate offset
    int ltag[G];                      // IFACE: restraint bit of the slot atom, -1 = none
    float lf[G];                      // DESOLV: largest f32 d^2 of interest (-1: atom excluded)
    unsigned* ibits;                  // IFACE: interface bits of the current pose in HBM (null: none)
    unsigned* iset;                   // IFACE: where pairs set them: ibuf, or ibits when the pose has more words
    unsigned ibuf[W_IBUF];            // IFACE: the unit's bits, merged into ibits once at the unit's end
};

// Staged candidates (the plain kernel's TMA variant, selected per context):
// a window of STAGE_WIN receptor atoms (their float4 positions) copied from
// the row spans into shared memory by bulk copies (cp.async.bulk, no
// multicast) that complete on the warp's mbarrier.
constexpr int STAGE_WIN = 64;
struct WStage {
    float4 a[STAGE_WIN];
    unsigned long long bar;
    unsigned phase;   // parity of the barrier's current phase
};

__device__ __forceinline__ uint32_t w_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// bounded wait for phase `parity` of the mbarrier at `bar` (false: ran out)
__device__ __forceinline__ bool w_bar_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred P1;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, P1;\n\t}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// Receptor-side minima of the fast cpydock kernel: one 64-bit word per slot,
// the minimum d^2 quantised to 37 bits (0 .. SOLV2_D in steps of 3e-10 A^2)
// above the 27-bit receptor index, so one atomicMin updates a slot (the key
// bits are equal) and a slot costs 8 bytes of shared memory instead of 12.
// Only pairs with d^2 <= SOLV2_D are inserted; the receptor term's
// sqrt(d^2) then moves by < 1e-10 A.
// Spill: a pose that touches more receptor atoms within 6.4 A than the
// shared table holds (a ligand sunk into a large receptor) continues in the
// block's own table in global memory, of more slots than the complex has
// receptor atoms, so an insert there always finds its key or an empty slot.
// A key enters the global table only after its PROBES slots of the shared
// table were found taken by others, and taken slots stay taken, so the two
// tables hold disjoint keys and the receptor sum runs over both.  The block empties the
// global slots it used when it sums them.
struct MinHash64 {
    static constexpr unsigned long long EMPTY = ~0ull;
    static constexpr unsigned long long KEY_MASK = (1ull << 27) - 1;
    static constexpr double SCALE = (double)((1ull << 37) - 1) / SOLV2_D;
    // slots of the shared table a key may take.  Without a limit a pose that
    // filled the table probed all of it (2048 slots) for each key that it then
    // spilled: 1500 poses with a 12,000-atom ligand sunk into a 101,000-atom
    // receptor took 49.6 ms, now 5.9 (16 slots: 6.6, and 8 % more than 64
    // where the table is three quarters full; 32: 6.3)
    static constexpr int PROBES = 64;
    unsigned long long* slot;
    int cap;
    unsigned long long* spill;   // the block's global table (all EMPTY between poses), or null
    int spill_cap;
    int* spilled;                // shared flag: the pose used the global table
    __device__ void init(char* smem, int cap_, unsigned long long* spill_, int spill_cap_, int* spilled_) {
        cap = cap_;
        slot = reinterpret_cast<unsigned long long*>(smem);
        spill = spill_;
        spill_cap = spill_cap_;
        spilled = spilled_;
        for (int s = threadIdx.x; s < cap; s += blockDim.x) slot[s] = EMPTY;
        if (threadIdx.x == 0) *spilled = 0;
    }
    // linear probing over tab[0..n) (n a power of two); false when full (the
    // shared table: when the key's PROBES slots are).
    // GLOBAL: the table is in global memory, where the atomics act in L2:
    // plain reads there bypass L1 (__ldcg), which could hold a stale line
    template <bool GLOBAL>
    __device__ static bool put(unsigned long long* tab, int n, int k, unsigned long long w) {
        unsigned h = ((unsigned)k * 2654435761u) & (unsigned)(n - 1);
        const int most = GLOBAL ? n : (n < PROBES ? n : PROBES);
        for (int probe = 0; probe < most; ++probe) {
            unsigned long long v = GLOBAL ? __ldcg(tab + h) : tab[h];
            if (v == EMPTY) {
                v = atomicCAS(tab + h, EMPTY, w);
                if (v == EMPTY) return true;
            }
            if ((v & KEY_MASK) == (unsigned long long)k) {
                atomicMin(tab + h, w);
                return true;
            }
            h = (h + 1) & (unsigned)(n - 1);
        }
        return false;
    }
    // k < 2^26 (the receptor index limit); 0 <= d2 <= SOLV2_D
    __device__ bool insert(int k, double d2) {
        const unsigned long long w = (__double2ull_rn(d2 * SCALE) << 27) | (unsigned long long)k;
        if (put<false>(slot, cap, k, w)) return true;
        if (!spill) return false;
        *spilled = 1;
        return put<true>(spill, spill_cap, k, w);
    }
    __device__ static int key_of(unsigned long long v) { return v == EMPTY ? -1 : (int)(v & KEY_MASK); }
    __device__ static double value_of(unsigned long long v) { return fmin((double)(v >> 27) / SCALE, SOLV2_D); }
    __device__ int key(int s) const { return key_of(slot[s]); }
    __device__ double value(int s) const { return value_of(slot[s]); }
};

// IFACE: start a unit of pose bits `bits` (lane 0; the caller syncs the
// warp after): collect in the warp's buffer when the pose fits in it
template <int G>
__device__ __forceinline__ void w_iface_begin(WSlots<G>& W, const ComplexDev& c, unsigned* bits) {
    W.ibits = bits;
    W.iset = !bits ? nullptr : (c.iface_words <= W_IBUF ? W.ibuf : bits);
}

// IFACE: merge the warp's buffer into the pose's bits and clear it (all
// lanes); the buffer is all zero between units
template <int G>
__device__ __forceinline__ void w_iface_flush(WSlots<G>& W, const ComplexDev& c) {
    __syncwarp();
    if (W.iset == W.ibuf)
        for (int w = (int)(threadIdx.x & 31); w < c.iface_words; w += 32) {
            const unsigned v = W.ibuf[w];
            if (v) { atomicOr(W.ibits + w, v); W.ibuf[w] = 0u; }
        }
    __syncwarp();
}

// 1 / x and 1 / sqrt(x) by the MUFU approximations alone (PTX rcp.approx /
// rsqrt.approx, flush-to-zero): the pair distances are far from f32
// denormals (d^2 >= ~1 A^2 for any real pair, <= 100 here), where these
// are within a few ulp, the budget of the f32 pair math
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Packed pairs of f32 (Blackwell's f32x2 FADD / FMUL / FFMA: one instruction
// computes both lanes of the pair, each rounded as the scalar operation)
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { F2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// one receptor atom, 32 bytes: (x, y, z, q), (sqrt eps, r, heavy, excluded);
// atom nr is out of reach of everything (it pads the candidate lists)
struct WAtom {
    float4 a, p;
};
__device__ __forceinline__ WAtom w_atom(const float4* __restrict__ rpk, unsigned k) {
    WAtom r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.p.x), "=f"(r.p.y), "=f"(r.p.z), "=f"(r.p.w)
        : "l"(rpk + 2 * (size_t)k));
    return r;
}

// the lane index, read once (a plain threadIdx.x & 31 is read again at every
// use when registers are short)
__device__ __forceinline__ int w_lane() {
    unsigned l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return (int)l;
}

// The unit's pose, its factor on lengths, and the search radius of its atoms.
// A quaternion (w, v) is used as given: the matrix keeps v's axis and turns the
// plane across it by a matrix of norm sqrt(1 + 4 |v|^2 (|q|^2 - 1)), so the
// ligand's spheres grow by at most that: up to 2e-6 (the f32 arithmetic here is
// off by 1e-6 at most near unit quaternions) by the spheres' own margin of 4e-6.
// The search radius is SCAN_R grown by what f32 takes from the positions.  The receptor's and the centres' are rounded (2^-24
// of a coordinate each), as are the distances to the cell rows (under 12
// roundings of a coordinate; 2^-21 is 8 on the radius, 16 on its square).  1e-4 A
// at 200 A, and at most 1 A, so that a pose at infinity does not search the whole
// receptor: enough for coordinates up to 7e5 A.
template <int G>
__device__ __forceinline__ void w_pose(WSlots<G>& W, const ComplexDev& c, const double* pq) {
    W.rot = pose_matrix(pq);
    const float qw = (float)pq[0], qx = (float)pq[1], qy = (float)pq[2], qz = (float)pq[3];
    const float v2 = qx * qx + qy * qy + qz * qz, e = 4.f * v2 * (qw * qw + v2 - 1.f);
    float s = 1.f;
    if (e > 4e-6f && e < 3e38f) s = sqrtf(1.f + e);
    W.stretch = s;
    const float t = fabsf((float)pq[4]) + fabsf((float)pq[5]) + fabsf((float)pq[6]);
    W.scan = SCAN_R + fminf(0x1p-21f * (t + s * c.lext), 1.f);
}

// the descriptor of a unit's complex into shared memory by n threads (its
// fields are read all through a unit; from global memory each read waited)
__device__ __forceinline__ void w_descriptor(ComplexDev* dst, const ComplexDev* src, int lane, int n) {
    static_assert(sizeof(ComplexDev) % 8 == 0, "copied in 8-byte words");
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(src);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(dst);
    for (int i = lane; i < (int)(sizeof(ComplexDev) / 8); i += n) d[i] = __ldg(s + i);
}

constexpr unsigned long long W_NOMIN = 0x7fefffffffffffffull;   // largest finite double

// lower bound of the distance from (x, y, z) to the nearest receptor atom
// (ComplexDev::rlb; rlb_m outside its grid)
__device__ __forceinline__ float w_receptor_bound(const ComplexDev& c, float x, float y, float z) {
    const int ix = (int)floorf((x - c.rlbox) * c.rlb_inv);
    const int iy = (int)floorf((y - c.rlboy) * c.rlb_inv);
    const int iz = (int)floorf((z - c.rlboz) * c.rlb_inv);
    if (ix < 0 || iy < 0 || iz < 0 || ix >= c.rlbx || iy >= c.rlby || iz >= c.rlbz) return c.rlb_m;
    return __ldg(c.rlb + ((size_t)iz * c.rlby + iy) * c.rlbx + ix);
}


// The f64 mode's slots: a group's ligand atoms as the reference holds them.
template <int G>
struct WExact {
    double x[G], y[G], z[G], q[G], sv[G], r[G], eps[G], h[G];
};

// The warp's sums over its groups (cpydock: per lane; else per group, reduced).
struct WAcc {
    double elec = 0.0, vdw = 0.0, solv = 0.0;
    int np = 0;
};

// cpydock: the first n (<= 32) waiting hits, one a lane, update both atoms'
// minimum distance in f64 (cpydock.rs:615-668), the ligand atom's in its slot,
// the receptor atom's in the block's hash
template <int G>
__device__ __forceinline__ void w_minima(const ComplexDev& c, WDes<G>* D, MinHash64* hash, int* status, int first,
                                         int n) {
    const int lane = threadIdx.x & 31;
    if (lane >= n) return;
    const unsigned e = D->hit[first + lane];
    const int l = (int)(e >> 26 & 31u), k = (int)(e & 0x3ffffffu);
    const double4 a = c.rpos64[k];
    const double ex = D->lx[l] - a.x, ey = D->ly[l] - a.y, ez = D->lz[l] - a.z;
    const double d2 = ex * ex + ey * ey + ez * ez;
    atomicMin(&D->lmin[l], (unsigned long long)__double_as_longlong(d2));
    if ((e >> 31) && d2 <= SOLV2_D && !hash->insert(k, d2)) atomicOr(status, 1);
}

// d^2 of a receptor atom and both slots of a pair, from the compensated
// differences (l - a) + residual.  CHAIN (cpydock and interface kernels): one
// fused chain; else (dx^2 + dy^2) + dz^2 with the first sum rounded on its own
// (`one` is 1, from memory: a plain packed add of two products is contracted)
template <bool CHAIN>
__device__ __forceinline__ F2 w_d2(const WPair& P, const WAtom& A, F2 one) {
    const F2 dx = add2(f2(P.x[0] - A.a.x, P.x[1] - A.a.x), f2(P.rx[0], P.rx[1]));
    const F2 dy = add2(f2(P.y[0] - A.a.y, P.y[1] - A.a.y), f2(P.ry[0], P.ry[1]));
    const F2 dz = add2(f2(P.z[0] - A.a.z, P.z[1] - A.a.z), f2(P.rz[0], P.rz[1]));
    return CHAIN ? fma2(dz, dz, fma2(dx, dx, mul2(dy, dy))) : fma2(dz, dz, fma2(mul2(dy, dy), one, mul2(dx, dx)));
}

// The listed pairs whose f32 d^2 lies within NEAR_BAND of the cutoff, which
// w_dense leaves out: in or out as f64 decides.  Out of line: one test in some
// ten thousand, so the lists of about one group in thirty are read again.
template <int G, bool CHAIN>
__device__ __noinline__ void w_band(const ComplexDev& c, const WSlots<G>& W, int lane, unsigned flags,
                                    WAcc& r) {
    for (int quad = 0; quad < (G + 3) / 4; ++quad)
    for (int i = lane >> 1; i < W.cnt[quad]; i += 16) {
        const WPair& P = W.pair[quad * 2 + (lane & 1)];
        const unsigned k = W.list[quad][W.first[quad] + i];
        const WAtom A{__ldg(c.rpk + 2 * (size_t)k), __ldg(c.rpk + 2 * (size_t)k + 1)};
        float d20, d21;
        f2_get(w_d2<CHAIN>(P, A, f2(W.one[0], W.one[1])), d20, d21);
        for (int h = 0; h < 2; ++h) {
            const float d2 = h ? d21 : d20;
            if (!(fabsf(d2 - 100.f) < NEAR_BAND) || k >= (unsigned)c.nr ||
                !near_exact(c, (int)k, P.x[h], P.rx[h], P.y[h], P.ry[h], P.z[h], P.rz[h]))
                continue;
            ++r.np;
            const float ir2 = rcp_approx(d2);
            if (flags & F_ELEC) r.elec += (double)fminf(fmaxf(P.q[h] * A.a.w * ir2, -ES_CAP_F), ES_CAP_F);
            const float rr = P.r[h] + A.p.y, t = rr * rr * ir2, p6 = t * t * t;
            float vp = fminf(P.sv[h] * A.p.x * p6 * (p6 - 2.f), 1.0f);
            if (flags & F_CLASH)
                vp = fmaf(6.f, fmaxf(P.h[h] * fabsf(A.p.z) * rr - d2 * rsqrt_approx(d2), 0.f), vp);
            r.vdw += (double)vp;
        }
    }
}

// The first n (<= 32) waiting pairs with a tagged atom that can lie within
// 3.9 A, one a lane: re-tested in f64 (the slot position as f32 value +
// residual, ~2^-48 relative), which sets the pose's interface bits.
template <int G, bool DESOLV>
__device__ __forceinline__ void w_tags(const ComplexDev& c, const WSlots<G>& W, const WDes<G>* D, const unsigned* hit,
                                       int lane, int set, int n) {
    if (lane >= n || !W.iset) return;
    const unsigned e = hit[lane];
    const int l = (int)(e >> 26), k = (int)(e & 0x3ffffffu);
    const double4 a64 = c.rpos64[k];
    double ex, ey, ez;
    if (DESOLV) {
        ex = D->lx[set + l] - a64.x;
        ey = D->ly[set + l] - a64.y;
        ez = D->lz[set + l] - a64.z;
    } else {
        const WPair& P = W.pair[l >> 1];
        const int h = l & 1;
        ex = ((double)P.x[h] + (double)P.rx[h]) - a64.x;
        ey = ((double)P.y[h] + (double)P.ry[h]) - a64.y;
        ez = ((double)P.z[h] + (double)P.rz[h]) - a64.z;
    }
    if (ex * ex + ey * ey + ez * ez <= IFACE2_D) {
        const int2 rt = __ldg(c.rtag + k);
        iface_set(W.iset, rt.x);
        iface_set(W.iset, rt.y);
        iface_set(W.iset, W.ltag[l]);
    }
}

// Scores n listed candidates (from list[first]) of quad `quad` densely: 16
// candidates a step, lane = (candidate, slot pair), the slot pair in
// registers, two steps side by side (two receptor atoms in flight, two
// independent chains).  Per test the reference formulas on packed f32 pairs
// (both slots of the pair).  off: the smallest |d^2 - 100| seen.  ELEC /
// CLASH: the complex's terms.  The list is padded to a whole step.
template <int G, bool DESOLV, bool IFACE, bool NP, bool ELEC, bool CLASH>
__device__ __forceinline__ void w_dense(const ComplexDev& c, WSlots<G>& W, WDes<G>* D, MinHash64* hash, int* status,
                                        int lane, int set, int quad, int first, int n, WAcc& acc, float& off,
                                        int& nhit, int& old_hits, unsigned* thit, int& ntag) {
    constexpr unsigned FULL = 0xffffffffu;
    const int half = lane & 1;
    const WPair P = W.pair[quad * 2 + half];
    unsigned* const list = W.list[quad] + first;
    const float4* rpk = c.rpk;
    const F2 one = f2(W.one[0], W.one[1]);
    const int slot0 = quad * 4 + half * 2;
    // IFACE: the slot is tagged (untagged receptor atoms matter then)
    const bool tag0 = IFACE && W.ltag[slot0] >= 0, tag1 = IFACE && W.ltag[slot0 + 1] >= 0;
    float lf0 = 0.f, lf1 = 0.f;
    bool need0 = false, need1 = false;   // DESOLV: the slot's own minimum is wanted
    if (DESOLV) {
        lf0 = W.lf[slot0]; lf1 = W.lf[slot0 + 1];
        need0 = lf0 > SOLV2_F * 1.0005f; need1 = lf1 > SOLV2_F * 1.0005f;
    }
    auto step = [&](const WAtom& A, unsigned k) {
        const F2 d2 = w_d2<DESOLV || IFACE>(P, A, one);
        float d20, d21, t0, t1;
        f2_get(d2, d20, d21);
        f2_get(sub2(d2, f2(100.f, 100.f)), t0, t1);
        const F2 ir2 = f2(rcp_approx(d20), rcp_approx(d21));
        float e0 = 0.f, e1 = 0.f, v0, v1;
        if (ELEC) {
            f2_get(mul2(f2(P.q[0] * A.a.w, P.q[1] * A.a.w), ir2), e0, e1);
            e0 = fminf(fmaxf(e0, -ES_CAP_F), ES_CAP_F);
            e1 = fminf(fmaxf(e1, -ES_CAP_F), ES_CAP_F);
        }
        const F2 sv = f2(P.sv[0] * A.p.x, P.sv[1] * A.p.x);
        const F2 rr = f2(P.r[0] + A.p.y, P.r[1] + A.p.y);
        const F2 t = mul2(mul2(rr, rr), ir2);
        const F2 p6 = mul2(mul2(t, t), t);
        f2_get(mul2(mul2(sv, p6), sub2(p6, f2(2.f, 2.f))), v0, v1);
        v0 = fminf(v0, 1.0f);
        v1 = fminf(v1, 1.0f);
        if (CLASH) {
            const float hz = fabsf(A.p.z);   // the sign marks a tagged atom
            float g0, g1, m0, m1;
            f2_get(mul2(d2, f2(rsqrt_approx(d20), rsqrt_approx(d21))), g0, g1);
            f2_get(mul2(f2(P.h[0] * hz, P.h[1] * hz), rr), m0, m1);   // 0 unless both are heavy
            v0 = fmaf(6.f, fmaxf(__fsub_rn(m0, g0), 0.f), v0);
            v1 = fmaf(6.f, fmaxf(__fsub_rn(m1, g1), 0.f), v1);
        }
        // selected before the sums: a branch or a predicated f64 add cost more
        const bool in0 = t0 <= -NEAR_BAND, in1 = t1 <= -NEAR_BAND;
        if (ELEC) acc.elec = (acc.elec + (double)(in0 ? e0 : 0.f)) + (double)(in1 ? e1 : 0.f);
        acc.vdw = (acc.vdw + (double)(in0 ? v0 : 0.f)) + (double)(in1 ? v1 : 0.f);
        if (NP) acc.np += (int)in0 + (int)in1;
        off = fminf(off, fminf(fabsf(t0), fabsf(t1)));
        // pairs near enough with a tagged atom (the receptor's sign on its
        // heavy flag, or a tagged slot) wait for w_tags
        if (IFACE) {
            const bool rt = __float_as_uint(A.p.z) >> 31;
            const bool g0 = (rt || tag0) && d20 <= IFACE2_F, g1 = (rt || tag1) && d21 <= IFACE2_F;
            const unsigned b0 = __ballot_sync(FULL, g0), b1 = __ballot_sync(FULL, g1);
            if (b0 | b1) {
                const unsigned lt_mask = (1u << lane) - 1u;
                const int n0 = __popc(b0);
                const unsigned e = ((unsigned)slot0 << 26) | k;
                if (g0) thit[ntag + __popc(b0 & lt_mask)] = e;
                if (g1) thit[ntag + n0 + __popc(b1 & lt_mask)] = e + (1u << 26);
                ntag += n0 + __popc(b1);
                __syncwarp();
                while (ntag >= 32) {   // the last 32 first: the rest stays at the front
                    ntag -= 32;
                    w_tags<G, DESOLV>(c, W, D, thit + ntag, lane, set, 32);
                    __syncwarp();
                }
            }
        }
        if (DESOLV) {
            const bool want = A.p.w == 0.f, may = A.p.w != 1.f;
            const bool s0 = d20 <= lf0 && may && (want || need0), s1 = d21 <= lf1 && may && (want || need1);
            const unsigned b0 = __ballot_sync(FULL, s0), b1 = __ballot_sync(FULL, s1);
            if (b0 | b1) {
                const unsigned lt_mask = (1u << lane) - 1u;
                const int n0 = __popc(b0);
                const unsigned e = ((unsigned)(set + slot0) << 26) | k | (want ? 0x80000000u : 0u);
                if (s0) D->hit[nhit + __popc(b0 & lt_mask)] = e;
                if (s1) D->hit[nhit + n0 + __popc(b1 & lt_mask)] = e + (1u << 26);
                nhit += n0 + __popc(b1);
                __syncwarp();
                int head = 0;
                for (; nhit - head >= 32; head += 32) w_minima<G>(c, D, hash, status, head, 32);
                if (head > 0) {   // the rest moves to the front
                    const unsigned v = head + lane < nhit ? D->hit[head + lane] : 0u;
                    __syncwarp();
                    D->hit[lane] = v;
                    nhit -= head;
                    old_hits -= head;
                    __syncwarp();
                }
            }
        }
    };
    int i = 0;
    for (; i + 16 < n; i += 32) {
        const unsigned ka = list[i + (lane >> 1)], kb = list[i + 16 + (lane >> 1)];
        const WAtom A = w_atom(rpk, ka), B = w_atom(rpk, kb);
        step(A, ka);
        step(B, kb);
    }
    if (i < n) {
        const unsigned ka = list[i + (lane >> 1)];
        step(w_atom(rpk, ka), ka);
    }
}

// The f64 mode of w_dense: the listed candidates in the reference's arithmetic
// (compiled without contraction), 16 a step, lane = (candidate, two slots).
// The lists only have to hold every pair within the cutoff; each pair is in or
// out by its own f64 d^2.
template <int G, bool IFACE, bool NP>
__device__ __forceinline__ void w_dense_exact(const ComplexDev& c, const WSlots<G>& W, const WExact<G>& X,
                                              unsigned* iset, int lane, int quad, int first, int n, WAcc& acc) {
    const int slot0 = quad * 4 + (lane & 1) * 2;
    for (int i = lane >> 1; i < n; i += 16) {
        const int k = (int)W.list[quad][first + i];
        const double4 a = c.rpos64[k];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int l = slot0 + h;
            const double dx = X.x[l] - a.x, dy = X.y[l] - a.y, dz = X.z[l] - a.z;
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (!(d2 <= 100.0)) continue;
            if (NP) ++acc.np;
            pair_exact(c.flags, c.lj_form, X.q[l], X.sv[l], X.r[l], X.eps[l], X.h[l] != 0.0, a, c.rpar64[k], d2,
                       acc.elec, acc.vdw);
            if (IFACE && iset && d2 <= IFACE2_D) {
                const int2 rt = __ldg(c.rtag + k);
                iface_set(iset, rt.x);
                iface_set(iset, rt.y);
                iface_set(iset, W.ltag[l]);
            }
        }
    }
}

// Scores groups group_of(first), group_of(first + step), ... (indices < end) of
// one pose whose rotation is in W.rot.  Plain and interface kernels: after each group its
// sums, reduced over the warp, are added to acc.elec (lanes 0-15: the
// electrostatics, lanes 16-31: the vdW), so acc is the sum of the groups'
// sums in order; with W.part, each group's sums also go to its own 4 doubles
// there.  DESOLV: acc holds the lane's own sums, and each slot atom's
// g(min d^2) * des is added to acc.solv once its hits are all evaluated.
template <int G, bool DESOLV, bool IFACE, bool NP, bool STAGE, bool EXACT, class GroupOf>
__device__ __forceinline__ void w_groups(const ComplexDev& c, WSlots<G>& W, WDes<G>* D, MinHash64* hash, int* status,
                                         int lane, int first, int end, int step, GroupOf group_of, WAcc& acc,
                                         WStage* S = nullptr, WExact<G>* X = nullptr, bool far_sep = false,
                                         unsigned* thit = nullptr) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NQ = (G + 3) / 4;
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned flags = c.flags;
    const int nl = c.nl;
    unsigned* const iset = IFACE ? W.iset : nullptr;   // set by the caller for the unit
    int nhit = 0;                 // DESOLV: hits waiting for their minima
    int old_hits = 0;             // DESOLV: the first of them, of groups before the previous one (may go below 0)
    int jdes0 = -1, jdes1 = -1;   // DESOLV: this lane's slot atom in set 0 / set 1
    auto minima_rest = [&]() {
        __syncwarp();
        w_minima<G>(c, D, hash, status, 0, nhit);
        nhit = 0;
        __syncwarp();
    };
    auto finalize = [&](int set) {   // DESOLV: the slot set's minima are final
        const int j = set ? jdes1 : jdes0;
        if (lane < G && j >= 0) {
            const double2 ls = c.lsolv64[j];
            acc.solv += solv_term(__longlong_as_double((long long)D->lmin[set + lane]), ls.y) * ls.x;
        }
        if (set) jdes1 = -1; else jdes0 = -1;
    };
    int it = 0;
    for (int gk = first; gk < end; gk += step, ++it) {
        const int grp = group_of(gk);
        const int set = DESOLV ? (it & 1) * G : 0;
        __syncwarp();
        if (DESOLV) {
            // slot set `set` last served the group before the previous one,
            // whose last hits may still wait
            if (old_hits > 0) minima_rest();
            old_hits = nhit;
            finalize(set);
        }
        WAcc gsum;   // the group's near pairs and far field
        // 1. the group's ligand atoms (lanes 0..G-1), the spheres of its quads
        //    and its own (the lanes above; a second round with groups of 32)
        float gx, gy, gz, R;
        {
            const int j = grp * G + lane;
            const bool atom = lane < G && j < nl;
            // from the f64 base coordinates, as the reference transforms them
            double4 b = make_double4(0.0, 0.0, 0.0, 0.0);
            constexpr int Q0 = G < 32 ? G : 0;   // lane of the first quad
            const int qi = grp * NQ + lane - Q0;
            const bool quad = lane >= Q0 && lane < Q0 + NQ && qi * 4 < nl;
            float rad = 0.f;
            auto sphere = [&]() {
                if (lane >= Q0 && lane <= Q0 + NQ) {
                    const float4 s = lane == Q0 + NQ ? __ldg(c.lgrp + grp) : (quad ? __ldg(c.lquad + qi) : make_float4(0.f, 0.f, 0.f, 0.f));
                    b = make_double4((double)s.x, (double)s.y, (double)s.z, 0.0);
                    rad = fmaf(W.stretch, s.w, W.scan);
                }
            };
            if (atom) b = c.lpos64[j];
            if (G < 32) sphere();
            double xd, yd, zd;
            apply(W.rot, b.x, b.y, b.z, xd, yd, zd);
            float x = (float)xd, y = (float)yd, z = (float)zd;
            if (lane < G) {
                const float q = (float)b.w;
                if constexpr (EXACT) {
                    const double4 lp = atom ? c.lpar64[j] : make_double4(0.0, 0.0, 0.0, 0.0);
                    X->x[lane] = atom ? xd : 1e30;   // never within reach of a receptor atom
                    X->y[lane] = atom ? yd : 1e30;
                    X->z[lane] = atom ? zd : 1e30;
                    X->q[lane] = b.w; X->sv[lane] = lp.x; X->r[lane] = lp.y; X->eps[lane] = lp.z; X->h[lane] = lp.w;
                } else {
                const float4 lp4 = atom ? __ldg(c.lpar + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                WPair& P = W.pair[lane >> 1];
                const int h = lane & 1;
                P.rx[h] = (float)(xd - (double)x);
                P.ry[h] = (float)(yd - (double)y);
                P.rz[h] = (float)(zd - (double)z);
                P.x[h] = atom ? x : 1e30f;   // never within reach of a receptor atom
                P.y[h] = atom ? y : 1e30f;
                P.z[h] = atom ? z : 1e30f;
                P.q[h] = q; P.sv[h] = lp4.x; P.r[h] = lp4.y;
                P.h[h] = lp4.z != 0.f ? 0.75f : 0.f;
                if (DESOLV) {
                    D->lx[set + lane] = xd; D->ly[set + lane] = yd; D->lz[set + lane] = zd;
                    D->lmin[set + lane] = W_NOMIN;
                    // (two thresholds, both above 6.4^2: the larger one marks an
                    // atom whose own minimum is wanted)
                    const bool need = atom && solv_counts(c.lsolv64[j]);
                    W.lf[lane] = lp4.w != 0.f ? -1.f : (need ? SOLV2_F * 1.001f : SOLV2_F * 1.0004f);
                    if (set) jdes1 = atom ? j : -1; else jdes0 = atom ? j : -1;
                }
                }
                if (IFACE) W.ltag[lane] = (atom && c.ltag) ? __ldg(c.ltag + j) : -1;
                // far field with the reference's f64 interpolation (a per-atom
                // cost; f32 here would add up over thousands of charged atoms)
                // (the cpydock kernel takes it from k_far_poses instead when
                // that pass ran: far_sep)
                if (atom && (flags & F_FAR) && !(DESOLV && far_sep) && (EXACT ? b.w != 0.0 : q != 0.f))
                    gsum.elec = b.w * sample_phi(c, xd, yd, zd);
            }
            if (G == 32) {
                sphere();
                apply(W.rot, b.x, b.y, b.z, xd, yd, zd);
                x = (float)xd; y = (float)yd; z = (float)zd;
            }
            gx = __shfl_sync(FULL, x, Q0 + NQ);
            gy = __shfl_sync(FULL, y, Q0 + NQ);
            gz = __shfl_sync(FULL, z, Q0 + NQ);
            R = __shfl_sync(FULL, rad, Q0 + NQ);
            if (lane >= Q0 && lane < Q0 + NQ) {
                // |a' - c'|^2 <= r^2 as |a'|^2 - 2 a'.c' <= r^2 - |c'|^2 in the
                // group frame (the rounding is in the quad's radius); a quad
                // past the ligand never passes
                const float lx = (float)(xd - (double)gx), ly = (float)(yd - (double)gy), lz = (float)(zd - (double)gz);
                W.quad[lane - Q0] = quad ? make_float4(-2.f * lx, -2.f * ly, -2.f * lz,
                                                       rad * rad - (lx * lx + ly * ly + lz * lz))
                                         : make_float4(0.f, 0.f, 0.f, -3e30f);
            }
        }
        // 2. receptor rows within reach of the group sphere
        const float R2 = R * R;
        const int cz0 = max(0, (int)floorf((gz - R - c.oz) * c.inv_h));
        const int cz1 = min(c.ncz - 1, (int)floorf((gz + R - c.oz) * c.inv_h));
        const int cy0 = max(0, (int)floorf((gy - R - c.oy) * c.inv_h));
        const int cy1 = min(c.ncy - 1, (int)floorf((gy + R - c.oy) * c.inv_h));
        const int nyr = cy1 - cy0 + 1, nzr = cz1 - cz0 + 1;
        const int nbox = (nyr > 0 && nzr > 0) ? nyr * nzr : 0;
        const float inv_nyr = 1.0f / (float)max(nyr, 1);
        int cnt[NQ];   // list lengths
#pragma unroll
        for (int s = 0; s < NQ; ++s) cnt[s] = 0;
        // 3. 32 candidates (relative to the group centre): listed for every
        //    quad whose sphere they are in
        auto chunk = [&](const float4 a, const int ridx) {
            const float ax = a.x - gx, ay = a.y - gy, az = a.z - gz;
            const float aa = ax * ax + ay * ay + az * az;
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                const float4 t = W.quad[s];
                const bool in = fmaf(ax, t.x, fmaf(ay, t.y, fmaf(az, t.z, aa))) <= t.w;
                const unsigned b = __ballot_sync(FULL, in);
                if (in) W.list[s][cnt[s] + __popc(b & lt_mask)] = (unsigned)ridx;
                cnt[s] += __popc(b);
            }
        };
        auto full = [&]() {   // two more chunks may not fit
            int m = cnt[0];
#pragma unroll
            for (int s = 1; s < NQ; ++s) m = max(m, cnt[s]);
            return m > W_LIST<G> - 64;
        };
        const float4 far_away = make_float4(3e30f, 3e30f, 3e30f, 0.f);
        int r0 = -32;                                     // the current 32 rows
        int st = 0, len = 0, excl = 0, total = 0;         // this lane's row: first atom, atoms, candidates before it; all rows' candidates
        int k0 = 0, rows = 0;                             // next candidate, rows that start before it
        bool more = true;
        // candidate kk belongs to the last non-empty row that starts at or
        // before it: the starts within a chunk of 32 as a bit mask, the rows
        // before the chunk counted in `rows`
        auto locate = [&](int kc) {   // receptor index of candidate kc + lane (chunks in order)
            const unsigned d = (unsigned)(excl - kc);
            const unsigned m = __reduce_or_sync(FULL, (len > 0 && d < 32u) ? 1u << d : 0u);
            const int ord = rows + __popc(m & (lt_mask | (1u << lane))) - 1;
            rows += __popc(m);
            return W.row[ord] + kc + lane;
        };
        do {
            while (!full()) {
                if (k0 >= total) {
                    r0 += 32;
                    if (r0 >= nbox) { more = false; break; }
                    const int r = r0 + lane;
                    st = len = 0;
                    if (r < nbox) {
                        // r = zz * nyr + yy; (r + 0.5) / nyr is at least 0.5 / nyr
                        // away from an integer, far above the f32 rounding error
                        const int zz = (int)(((float)r + 0.5f) * inv_nyr), yy = r - zz * nyr;
                        const int cz = cz0 + zz, cy = cy0 + yy;
                        const float zlo = c.oz + cz * c.h, ylo = c.oy + cy * c.h;
                        const float dzm = fmaxf(0.f, fmaxf(zlo - gz, gz - (zlo + c.h)));
                        const float dym = fmaxf(0.f, fmaxf(ylo - gy, gy - (ylo + c.h)));
                        const float rem = R2 - dzm * dzm - dym * dym;
                        if (rem >= 0.f) {
                            const float wx = sqrtf(rem);
                            const int cx0 = max(0, (int)floorf((gx - wx - c.ox) * c.inv_hx));
                            const int cx1 = min(c.ncx - 1, (int)floorf((gx + wx - c.ox) * c.inv_hx));
                            if (cx0 <= cx1) {
                                const int row = (cz * c.ncy + cy) * c.ncx;
                                st = __ldg(c.cell_start + row + cx0);
                                len = __ldg(c.cell_start + row + cx1 + 1) - st;
                            }
                        }
                    }
                    int inc = len;   // inclusive prefix of the span lengths
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(FULL, inc, o);
                        if (lane >= o) inc += v;
                    }
                    total = __shfl_sync(FULL, inc, 31);
                    excl = inc - len;
                    k0 = rows = 0;
                    const unsigned ne = __ballot_sync(FULL, len > 0);
                    __syncwarp();
                    if (len > 0) W.row[__popc(ne & lt_mask)] = st - excl;
                    __syncwarp();
                    if (total == 0) continue;
                }
                if (!STAGE) {
                    // two chunks in flight, through L1; from rpk, whose lines
                    // the scoring reads again
                    const bool two = k0 + 32 < total;
                    const int ra = locate(k0);
                    const float4 a = k0 + lane < total ? __ldg(c.rpk + 2 * (size_t)ra) : far_away;
                    if (two) {
                        const int rb = locate(k0 + 32);
                        const float4 b = k0 + 32 + lane < total ? __ldg(c.rpk + 2 * (size_t)rb) : far_away;
                        chunk(a, ra);
                        chunk(b, rb);
                    } else {
                        chunk(a, ra);
                    }
                    k0 += 64;
                } else {
                    // windows of STAGE_WIN candidates: every row span's part of
                    // the window is bulk-copied into shared memory by its lane
                    const uint32_t bar = w_smem_u32(&S->bar);
                    const int wn = min(STAGE_WIN, total - k0);
                    const int lo = max(excl, k0), hi = min(excl + len, k0 + wn);
                    __syncwarp();   // the previous window is read
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                                     :: "r"(bar), "r"((uint32_t)wn * 16u) : "memory");
                    __syncwarp();
                    if (hi > lo) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                            :: "r"(w_smem_u32(S->a + (lo - k0))),
                               "l"(reinterpret_cast<uint64_t>(c.rpos + st + (lo - excl))),
                               "r"((uint32_t)(hi - lo) * 16u), "r"(bar) : "memory");
                    }
                    const unsigned ph = S->phase;
                    if (!w_bar_wait(bar, ph)) {
                        // ran out: report, and wait (bounded again) for the copies in flight
                        if (lane == 0) atomicOr(status, 8);
                        w_bar_wait(bar, ph);
                    }
                    __syncwarp();
                    if (lane == 0) S->phase = ph ^ 1u;
                    __syncwarp();
                    for (int kc = 0; kc < wn; kc += 32) {
                        const int ridx = locate(k0 + kc);
                        chunk(kc + lane < wn ? S->a[kc + lane] : far_away, ridx);
                    }
                    k0 += STAGE_WIN;
                }
            }
            // 4. the lists, scored: whole steps of 16 of the longer ones while
            //    the group goes on (the end of a list first, so its rest stays
            //    at the front), all at its end
            float off = 1e30f;
            int ntag = 0;   // IFACE: tagged pairs waiting
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                // the length to score, and padding past the list's end
                const int m = !more ? cnt[s] : (cnt[s] >= 32 ? cnt[s] & ~15 : 0);
                if (!EXACT && lane < 16) W.list[s][cnt[s] + lane] = (unsigned)c.nr;
                if (lane == s) { W.cnt[s] = m; W.first[s] = cnt[s] - m; }
                cnt[s] -= m;
            }
            __syncwarp();
            if constexpr (EXACT) {
#pragma unroll 1
                for (int s = 0; s < NQ; ++s)
                    w_dense_exact<G, IFACE, NP>(c, W, *X, iset, lane, s, W.first[s], W.cnt[s], gsum);
            } else {
            auto lists = [&](auto elec, auto clash) {
#pragma unroll 1
                for (int s = 0; s < NQ; ++s)
                    w_dense<G, DESOLV, IFACE, NP, decltype(elec)::value, decltype(clash)::value>(
                        c, W, D, hash, status, lane, set, s, W.first[s], W.cnt[s], gsum, off, nhit, old_hits, thit, ntag);
            };
            using T = std::true_type;
            using F = std::false_type;
            if (DESOLV) {
                if (flags & F_ELEC) lists(T(), F()); else lists(F(), F());
            } else switch (flags & (F_ELEC | F_CLASH)) {
                case F_ELEC | F_CLASH: lists(T(), T()); break;
                case F_ELEC: lists(T(), F()); break;
                case F_CLASH: lists(F(), T()); break;
                default: lists(F(), F()); break;
            }
            if (__any_sync(FULL, off < NEAR_BAND)) {
                WAcc r;
                w_band<G, DESOLV || IFACE>(c, W, lane, flags, r);
                gsum.elec += r.elec;
                gsum.vdw += r.vdw;
                if (NP) gsum.np += r.np;
            }
            if (IFACE) {
                __syncwarp();
                w_tags<G, DESOLV>(c, W, D, thit, lane, set, ntag);
            }
            }
            __syncwarp();
        } while (more);
        if (NP) acc.np += gsum.np;
        if (DESOLV) {
            acc.elec += gsum.elec;
            acc.vdw += gsum.vdw;
        } else {
            // the group's sums over the warp: electrostatics in lanes 0-15,
            // vdW in lanes 16-31
            const bool hi = lane >= 16;
            double keep = hi ? gsum.vdw : gsum.elec;
            keep += __shfl_xor_sync(FULL, hi ? gsum.elec : gsum.vdw, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(FULL, keep, o);
            acc.elec += keep;
            if (W.part) {
                double* gp = W.part + 4 * (size_t)(gk - first);
                if ((lane & 15) == 0) gp[lane >> 4] = keep;
                if (NP) {
                    const int npg = (int)__reduce_add_sync(FULL, (unsigned)gsum.np);
                    if (lane == 0) gp[3] = (double)npg;
                }
            }
        }
    }
    if (DESOLV) {
        minima_rest();
        finalize(0);
        finalize(G);
    }
}

// STAGE: the candidates reach shared memory by bulk copies (WStage) instead
// of L1 loads (selected per context; the measured alternative)
// NP: near pairs are counted (launches with parts)
// EXACT: f64 pair math in the reference's operation order
template <int G, bool IFACE, bool NP, bool STAGE = false, bool EXACT = false>
__global__ void __launch_bounds__(WK_THREADS, EXACT ? WK_BLOCKS_EXACT : WK_BLOCKS<G>) k_score_warp(const __grid_constant__ LaunchParams p) {
    static_assert(G == 4 || G == 16 || G == 32, "group size");
    static_assert(!(STAGE && (IFACE || EXACT)), "the staged variant is the plain kernel's");
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char wk_smem[];
    const int lane = w_lane();
    WSlots<G>& W = reinterpret_cast<WSlots<G>*>(wk_smem)[threadIdx.x >> 5];
    // descriptor of the current unit's complex
    ComplexDev& c = reinterpret_cast<ComplexDev*>(wk_smem + (WK_THREADS / 32) * sizeof(WSlots<G>))[threadIdx.x >> 5];
    WStage* S = STAGE ? reinterpret_cast<WStage*>(wk_smem + (WK_THREADS / 32) * (sizeof(WSlots<G>) + sizeof(ComplexDev))) +
                            (threadIdx.x >> 5)
                      : nullptr;
    WExact<G>* X = EXACT ? reinterpret_cast<WExact<G>*>(wk_smem + (WK_THREADS / 32) * (sizeof(WSlots<G>) + sizeof(ComplexDev))) +
                               (threadIdx.x >> 5)
                         : nullptr;
    // IFACE: tagged pairs waiting for w_tags
    __shared__ unsigned s_thit[IFACE && !EXACT ? WK_THREADS / 32 : 1][96];
    unsigned* const thit = IFACE && !EXACT ? s_thit[threadIdx.x >> 5] : nullptr;
    if (STAGE) {
        if (lane == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(w_smem_u32(&S->bar)), "r"(1));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            S->phase = 0u;
        }
        __syncwarp();
    }
    if (IFACE) W.ibuf[lane] = 0u;
    if (lane < 2) W.one[lane] = p.one;
    __syncwarp();
    int cur = -1;   // complex whose descriptor c holds
    // the first unit of every warp is fixed (spread over the blocks first), the
    // others come from the counter
    const long long nwarps = (long long)gridDim.x * (WK_THREADS / 32);
    for (bool first = true;; first = false) {
        long long w = (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        if (!first) {
            if (p.total_work <= nwarps) break;
            unsigned long long wq = 0;
            if (lane == 0) wq = atomicAdd(p.work_counter, 1ull);
            w = nwarps + (long long)__shfl_sync(FULL, wq, 0);
        }
        if (w >= p.total_work) break;
        const int b = find_item(p.item_work0, p.n_items, w);
        const int cid = __ldg(p.item_complex + b);
        if (cid != cur) {
            __syncwarp();
            w_descriptor(&c, p.cx + cid, lane, 32);
            cur = cid;
            __syncwarp();
        }
        const long long local = w - __ldg(p.item_work0 + b);
        const int ngrp = (c.nl + G - 1) / G, gpt = p.tile / G;
        // units of a pose, and this unit's groups: a tile's, or p.sub of them
        const int gpu = p.sub ? p.sub : gpt;
        const int nunits = (ngrp + gpu - 1) / gpu;
        // (poses x units of one item fit 32 bits except in huge batches)
        const int pose = local >> 32 ? (int)(local / nunits) : (int)((unsigned)local / (unsigned)nunits);
        const int unit = (int)(local - (long long)pose * nunits);
        const long long g = (long long)__ldg(p.item_pose0 + b) + pose;
        if (p.pose_mask && !p.pose_mask[g]) continue;   // pose skipped: keeps its score
        __syncwarp();   // readers of the previous unit's pose are done
        if (lane == 0) {
            w_pose(W, c, pose_of(p, g));
            if (IFACE) w_iface_begin(W, c, iface_bits(p, c, g));
            else if (c.iface_words) atomicOr(p.status, 2);   // a launch without room for the bits
        }
        __syncwarp();
        const int g0 = unit * gpu, g1 = min(g0 + gpu, ngrp);
        // partials: one per tile, or one per group when the tiles are split
        // (a tile's sum is then made from its groups' in the same order, so
        // the score's bits do not depend on the split)
        const size_t first_part = p.sub ? __ldg(p.item_group0 + b) + (long long)pose * ngrp : w - unit;
        if (lane == 0) W.part = p.sub ? p.partials + 4 * (first_part + g0) : nullptr;
        __syncwarp();
        WAcc acc;
        w_groups<G, false, IFACE, NP, STAGE, EXACT>(c, W, nullptr, nullptr, p.status, lane, g0, g1, 1,
                                                    [](int k) { return k; }, acc, S, X, false, thit);
        if (IFACE && W.ibits) w_iface_flush(W, c);
        double* const pose_part = p.partials + 4 * first_part;
        if (!p.sub) {
            double* const part = pose_part + 4 * (size_t)unit;
            if ((lane & 15) == 0) part[lane >> 4] = acc.elec;   // electrostatics, vdW
            if (NP) {
                const int npl = (int)__reduce_add_sync(FULL, (unsigned)acc.np);
                if (lane == 0) part[3] = (double)npl;
            }
        }
        __threadfence();   // partials (and interface bits) before the unit is published
        __syncwarp();
        int done = 0;
        if (lane == 0) done = atomicAdd(p.pose_counter + g, 1);
        done = __shfl_sync(FULL, done, 0);
        if (done == nunits - 1) {
            __threadfence();
            // lane i sums tiles i, i + 32, ..., then a fixed tree
            double e = 0.0, vv = 0.0, nps = 0.0;
            if (p.sub) {
                for (int t = lane * gpt; t < ngrp; t += 32 * gpt) {
                    double te = 0.0, tv = 0.0;
                    for (int k = t; k < min(t + gpt, ngrp); ++k) {
                        te += __ldcg(pose_part + 4 * k);
                        tv += __ldcg(pose_part + 4 * k + 1);
                        if (NP) nps += __ldcg(pose_part + 4 * k + 3);
                    }
                    e += te;
                    vv += tv;
                }
            } else {
                for (int t = lane; t < nunits; t += 32) {
                    e += __ldcg(pose_part + 4 * t);
                    vv += __ldcg(pose_part + 4 * t + 1);
                    if (NP) nps += __ldcg(pose_part + 4 * t + 3);
                }
            }
            e = warp_sum(e);
            vv = warp_sum(vv);
            if (NP) nps = warp_sum(nps);
            if (lane == 0) {
                write_pose(p, c, g, e, vv, 0.0, nps, IFACE ? W.ibits : nullptr);
                p.pose_counter[g] = 0;
            }
        }
    }
    __syncthreads();   // every warp of the block has left the work loop
    finish_launch(p);
}

// cpydock: one block per pose (the receptor-side minima live in the block's
// shared-memory hash); the pose's groups within the receptor's reach are listed
// first (a lane a group), and warp k takes the near groups k, k + NW, ... (a
// fixed assignment: the sums do not depend on scheduling).  Block layout of the
// dynamic shared memory: hash (hcap x 8 B), then NW x WSlots, NW x WDes.
// 8 warps a block, three blocks an SM (24 warps resident, 80 registers):
// the block's warps wait for one another at the end of every pose, and
// with 8 warps a pose instead of 12 that wait is shorter (a 12,000-atom
// ligand on a 101,000-atom receptor: 30.9 against 32.3 ms a step; 4 warps
// at 5 blocks: 34.2 ms).
constexpr int WD_THREADS = 256;
constexpr int WD_BLOCKS = 3;
// groups whose reach is tested at a time (most groups of a large ligand at the
// interface are too far from the receptor: in a CPU model of a 12,000-atom
// ligand on a 101,000-atom receptor 84-89 % of the groups of 16)
constexpr int WD_NEAR = 1024;

// whether a receptor atom can lie within reach of group gi (its sphere, by the
// pose's factor, grown by `scan`), by the receptor's distance bound at the posed
// centre
__device__ __forceinline__ bool w_near(const ComplexDev& c, const Rot& rot, float scan, float stretch, int gi) {
    const float4 gs = __ldg(c.lgrp + gi);
    const float R = fmaf(stretch, gs.w, scan);
    if (!c.rlb || !c.skip_far || !(R < c.rlb_m)) return true;
    double x, y, z;
    apply(rot, (double)gs.x, (double)gs.y, (double)gs.z, x, y, z);
    return !(w_receptor_bound(c, (float)x, (float)y, (float)z) > R);
}

template <int G>
__host__ __device__ constexpr size_t wd_smem(int hcap) {
    return (size_t)hcap * sizeof(unsigned long long) + (size_t)(WD_THREADS / 32) * (sizeof(WSlots<G>) + sizeof(WDes<G>));
}

template <int G, bool IFACE, bool NP>
__global__ void __launch_bounds__(WD_THREADS, WD_BLOCKS) k_score_warp_desolv(const __grid_constant__ LaunchParams p) {
    constexpr int NW = WD_THREADS / 32;
    extern __shared__ __align__(16) unsigned char wd_smem_raw[];
    __shared__ long long s_work;
    __shared__ double s_red[4][32];
    __shared__ long long s_fix[32];
    __shared__ int s_spilled;
    __shared__ ComplexDev s_c;
    __shared__ unsigned s_near[WD_NEAR / 32];
    __shared__ unsigned short s_list[WD_NEAR];
    __shared__ unsigned s_thit[IFACE ? NW : 1][96];
    unsigned* const thit = IFACE ? s_thit[threadIdx.x >> 5] : nullptr;
    const int lane = w_lane(), wid = threadIdx.x >> 5;
    unsigned long long* const spill =
        p.spill ? reinterpret_cast<unsigned long long*>(p.spill + (size_t)blockIdx.x * p.spill_cap * SPILL_SLOT_BYTES)
                : nullptr;
    for (;;) {
        if (threadIdx.x == 0) s_work = (long long)atomicAdd(p.work_counter, 1ull);
        __syncthreads();
        const long long w = s_work;
        __syncthreads();
        if (w >= p.total_work) break;
        const int b = find_item(p.item_work0, p.n_items, w);
        const ComplexDev* cg = p.cx + __ldg(p.item_complex + b);
        const int pose = (int)(w - __ldg(p.item_work0 + b));
        const long long g = (long long)__ldg(p.item_pose0 + b) + pose;
        if (p.pose_mask && !p.pose_mask[g]) continue;   // block-uniform: pose skipped
        if (threadIdx.x < 32) w_descriptor(&s_c, cg, lane, 32);
        __syncthreads();
        const ComplexDev& c = s_c;
        MinHash64 hash;
        hash.init(reinterpret_cast<char*>(wd_smem_raw), c.hcap, spill, p.spill_cap, &s_spilled);
        unsigned char* base = wd_smem_raw + (size_t)c.hcap * sizeof(unsigned long long);
        WSlots<G>& W = reinterpret_cast<WSlots<G>*>(base)[wid];
        WDes<G>* D = reinterpret_cast<WDes<G>*>(base + (size_t)NW * sizeof(WSlots<G>)) + wid;
        if (lane < 2) W.one[lane] = p.one;
        if (IFACE) W.ibuf[lane] = 0u;   // the slots move with the complex's hash size
        if (lane == 0) {
            w_pose(W, c, pose_of(p, g));
            if (IFACE) w_iface_begin(W, c, iface_bits(p, c, g));
            else if (c.iface_words) atomicOr(p.status, 2);
        }
        __syncthreads();   // hash cleared, poses set
        WAcc acc;
        const bool far_sep = p.far != nullptr;
        const int ngrp = (c.nl + G - 1) / G;
        for (int g0 = 0; g0 < ngrp; g0 += WD_NEAR) {
            // which of up to WD_NEAR groups a receptor atom can reach, a lane
            // a group (an inline far field wants them all)
            const int words = min(WD_NEAR, ngrp - g0 + 31) / 32;
            for (int i = wid; i < words; i += NW) {
                const int gi = g0 + i * 32 + lane;
                const bool near = gi < ngrp && (((c.flags & F_FAR) && !far_sep) || w_near(c, W.rot, W.scan, W.stretch, gi));
                const unsigned m = __ballot_sync(0xffffffffu, near);
                if (lane == 0) s_near[i] = m;
            }
            __syncthreads();
            // the near groups in order: lane i counts word i's, each warp
            // writes its words' out
            const unsigned mine = lane < words ? s_near[lane] : 0u;
            int inc = __popc(mine);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const int total = __shfl_sync(0xffffffffu, inc, 31);
            for (int i = wid; i < words; i += NW) {
                const unsigned m = __shfl_sync(0xffffffffu, mine, i);
                const int before = __shfl_sync(0xffffffffu, inc, i) - __popc(m);
                if (m >> lane & 1u) s_list[before + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(i * 32 + lane);
            }
            __syncthreads();
            // warp k scores the near groups k, k + NW, ...
            w_groups<G, true, IFACE, NP, false, false>(c, W, D, &hash, p.status, lane, wid, total, NW,
                                         [&](int k) { return g0 + s_list[k]; }, acc, nullptr, nullptr, far_sep,
                                                       thit);
            if (g0 + WD_NEAR < ngrp) __syncthreads();   // the list is read
        }
        if (IFACE && W.ibits) w_iface_flush(W, c);   // before the block's barrier below
        __syncthreads();   // every pair has updated the hash
        // receptor side: fixed-point (2^-40) sum over hash slots; slot order
        // depends on insertion races, integer sums do not
        long long fix = 0;
        for (int s = threadIdx.x; s < c.hcap; s += blockDim.x) {
            const int k = hash.key(s);
            if (k < 0) continue;
            const double2 rs = c.rsolv64[k];
            fix += __double2ll_rn(solv_term(hash.value(s), rs.y) * rs.x * 1099511627776.0);
        }
        if (s_spilled)   // block-uniform: read after the barrier above
            for (int s = threadIdx.x; s < p.spill_cap; s += blockDim.x) {
                const unsigned long long v = __ldcg(spill + s);
                if (v == MinHash64::EMPTY) continue;
                __stcg(spill + s, MinHash64::EMPTY);   // empty again for the block's next pose
                const int k = MinHash64::key_of(v);
                const double2 rs = c.rsolv64[k];
                fix += __double2ll_rn(solv_term(MinHash64::value_of(v), rs.y) * rs.x * 1099511627776.0);
            }
        fix = warp_sum(fix);
        if (lane == 0) s_fix[wid] = fix;
        double v[4] = {acc.elec, acc.vdw, acc.solv, (double)acc.np};
        block_sum<4>(v, s_red);   // contains __syncthreads: s_fix is complete
        if (threadIdx.x == 0) {
            long long f = 0;
            for (int i = 0; i < NW; ++i) f += s_fix[i];
            const double far = p.far ? __ldcg(p.far + g) : 0.0;   // k_far_poses' far field, when it ran
            write_pose(p, c, g, p.solv_only ? 0.0 : v[0] + far, p.solv_only ? 0.0 : v[1],
                       v[2] + (double)f * (1.0 / 1099511627776.0), v[3], IFACE ? W.ibits : nullptr);
        }
        __syncthreads();
    }
    finish_launch(p);
}

// The far field of the cpydock launch group as its own pass, before the
// fused kernel: one block per pose, each thread a fixed stride of ligand
// atoms (the f64 transform of the f64 base coordinates and the reference's
// f64 interpolation, as the fused kernel does it), then a block sum in a
// fixed order into far[pose] (deterministic).  Inside the fused kernel the
// 8 grid gathers of every charged atom waited on memory with only 24 warps
// per SM resident; here every thread has independent gathers in flight.
// Skipped (masked) poses are left alone.
constexpr int FAR_THREADS = 256;
static __global__ void __launch_bounds__(FAR_THREADS, 4) k_far_poses(const __grid_constant__ LaunchParams p) {
    __shared__ double s_red[4][32];
    for (long long w = blockIdx.x; w < p.total_work; w += gridDim.x) {
        const int b = find_item(p.item_work0, p.n_items, w);
        const ComplexDev& c = p.cx[__ldg(p.item_complex + b)];
        const long long g = (long long)__ldg(p.item_pose0 + b) + (w - __ldg(p.item_work0 + b));
        if (p.pose_mask && !p.pose_mask[g]) continue;   // block-uniform
        double v[1] = {0.0};
        if (c.flags & F_FAR) {
            const Rot rot = pose_matrix(pose_of(p, g));
            for (int j = threadIdx.x; j < c.nl; j += FAR_THREADS) {
                if (__ldg(&c.lpos[j].w) == 0.f) continue;
                const double4 b64 = c.lpos64[j];
                double xd, yd, zd;
                apply(rot, b64.x, b64.y, b64.z, xd, yd, zd);
                v[0] += b64.w * sample_phi(c, xd, yd, zd);
            }
        }
        block_sum<1>(v, s_red);
        if (threadIdx.x == 0) p.far[g] = v[0];
    }
}

}  // namespace lkg
