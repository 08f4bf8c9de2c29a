// ns.cu — the two neighbour passes of the weakly-compressible delta-SPH step.
//
// Reference counterparts: SPH_NS_simpleversion (src/equation/ns.cu:5-28) launching
// computeBoundary_Delta_acoustic_D (pass 1, src/equation/ns.cu:30-131) and
// computeGovering_equationD (pass 2, src/equation/ns.cu:134-249).
//
// Layout.  Particles are in cell-sorted order; each is one record of two vec4,
// rec[2i] = (x, y, z, p) and rec[2i+1] = (vx, vy, vz, ±rho) with the sign of rho marking a
// fluid (+) or boundary (-) particle, so everything a neighbour contributes to pass 1 is one
// aligned 32-byte sector in FP32.  Pass 1 writes the record pass 2 gathers, nrec[2i] =
// (x, y, z, q), nrec[2i+1] = (vx, vy, vz, ±rho'), where q = p' - rho0 cs h dofv: the
// acoustic-damper term of a fluid-fluid pair, rho0 cs h (dofv_i + dofv_j), splits into an i part
// and a j part, and the j part is folded into the neighbour's pressure (boundary particles
// have dofv = 0, so q = p').  It also writes self[i] = (p', rho', dofv, 0) for the particle's
// own side.
//
// Cells are walked as x-strips: with cells at least as wide as the list cutoff the 27 cells
// around a particle's cell are nine strips of three cells (x-1 .. x+1) of one (y, z) row,
// consecutive in the sorted order, so each strip is one contiguous slot range
// [cell_start[row + x-1], cell_start[row + x+2]) — the dense cell_start array gives empty cells
// the start of the next non-empty one.  With cells of a half or a third of the cutoff
// (KParams::reach 2 or 3) the walk covers 25 strips of five cells or 49 strips of seven.
//
// Neighbour list.  About 15% of the ~475 candidates of a 27-cell walk lie inside the
// support radius, and the lanes of a warp (particles of two or three adjacent cells) almost
// always have at least one hit per candidate, so a pass that tests and evaluates in one loop
// pays the full pair body for every candidate.  k_nbr_build therefore walks the candidates
// once per list build and stores the hits of the particle at work position t (all fluid slots
// first, then the walls; NbrList::order), in walk order, in column t of its warp's slot block
// (nbr_col); both passes then iterate only true neighbours, in the same order, so the sums are the
// same as a walking pass.  The passes wait for the gathers (each lane another record): the slots
// are interleaved in groups of four per lane, so that a warp's list read touches four lines per
// four steps, and padded to whole groups, so that the four gathers of a group are issued together
// without a branch.  Large FP32 runs share each list and gather between two particles
// (ns_twin.cu).  A particle with more hits than the list capacity is marked and walks the cells
// itself (same order again).
//
// With a Verlet skin the list is built with the cutoff kh(1 + s) (NbrList::cut2, else
// kh2_list) on cells kh(1 + skin) wide, s <= skin, and kept while the displacements since the
// build stay within the bound the solver's rebuild test checks; both passes still test r < kh
// on the current positions, and k_nbr_build keeps the build positions (xb) that pass 2
// measures each particle's displacement against.
//
// Precision.  Every kernel is instantiated for the three policies of sph_internal.h: FP32
// (records of float4), FP64 (records of two 32-byte double vectors) and mixed.  The mixed
// policy stores positions as FP32 offsets from the origin of the particle's cell at the last
// list build; a pair's relative position is (o_i - o_j) - (c_j - c_i) cell, exact to a few
// ulp of the cell size instead of a few ulp of the domain size, with c_j - c_i stored in the
// list slot (or known to the cell walk); its integrator advances FP64 positions and the FP64
// density perturbation rho - rho0.  A fourth policy adds compensated (Neumaier) accumulation
// of the density and force sums (measured on the 765,828-particle case: no accuracy gain over
// plain FP32 sums on relative positions, +14% time).
//
// Kernel algebra (same quantities as the reference, simplified): with r = x_i - x_j,
// q = |r|/h, t = 1 - q/2, the Wendland C2 gradient is grad W = c_fr t^3 r with
// c_fr = -5 adh / h^2, which is the reference's per-component expression
// adh(-2 t^3 (2q+1) + 2 t^4) r/(h|r|) after factoring.
#include <cuda_runtime.h>

#include <type_traits>

#include "ns_pair.cuh"
#include "sph_internal.h"

namespace sph {

namespace {
// List modes of the one-lane passes (template LIST): no list (cell walks), a list of plain
// windows, or one of interleaved windows (KParams::list_win).  The mode is a template
// parameter: a runtime choice between the two loops cost pass 2 1%.
enum { LIST_NONE = 0, LIST_PLAIN = 1, LIST_WIN = 2 };

// Whether the passes take a particle's listed neighbours two at a time in two-lane FP32
// instructions (fluid_two): FP32 pair arithmetic with plain sums.
template <class P>
constexpr bool kPairTwo = std::is_same<typename P::T, float>::value && !P::kComp;

// The records of a chunk's four slots, and the pairs of a fluid particle with them in list order.
template <class P>
__device__ __forceinline__ void load_chunk(const float4* __restrict__ R, const int4& q,
                                           float4 (&a)[4], float4 (&v)[4]) {
    const int e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int c = 0; c < 4; c++) ld_rec(R, P::kCodes ? slot_index(e[c]) : e[c], a[c], v[c]);
}
template <class P, class Acc>
__device__ __forceinline__ void pair_chunk(const KParamsT<float>& k, const int4& q,
                                           const float4 (&a)[4], const float4 (&v)[4], Acc& acc) {
    const int e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int c = 0; c < 4; c += 2)
        acc.fluid_two(k, a[c], v[c], P::kCodes ? (unsigned)e[c] : 0u, a[c + 1], v[c + 1],
                      P::kCodes ? (unsigned)e[c + 1] : 0u);
}

// Listed neighbours of a fluid particle, a chunk of four at a time: the four record gathers are
// issued together and the pairs evaluated without a branch, in list order.  DEEP: the records of the
// next chunk are in flight while the current one is evaluated (twice the registers), for runs too
// small to fill the SMs with warps, where the latency of a gather is all there is to hide.
template <class P, bool WIN, bool DEEP, class Acc>
__device__ __forceinline__ void visit_fluid(const KParamsT<float>& k, const NbrList& nl,
                                            const float4* __restrict__ R, int t, int cnt,
                                            Acc& acc) {
    const int* __restrict__ col = nl.idx + nbr_col(nl, t);
    if constexpr (DEEP) {
        const int pad = pad_slot<P>(k.n);
        auto slots = [&](int c) {
            return chunk_first<WIN>(c) < cnt ? ld_slots(col + ((size_t)c << 7))
                                             : make_int4(pad, pad, pad, pad);
        };
        if (cnt <= 0) return;
        int4 q0 = slots(0), q1 = slots(1), q2 = slots(2);
        float4 a0[4], v0[4], a1[4], v1[4];
        load_chunk<P>(R, q0, a0, v0);
#pragma unroll 1
        for (int c = 0; chunk_first<WIN>(c) < cnt; c += 2) {
            load_chunk<P>(R, q1, a1, v1);
            const int4 q3 = slots(c + 3);
            pair_chunk<P>(k, q0, a0, v0, acc);
            q0 = q2;
            load_chunk<P>(R, q0, a0, v0);
            q2 = slots(c + 4);
            pair_chunk<P>(k, q1, a1, v1, acc);
            q1 = q3;
        }
    } else {
        for_each_chunk<WIN>(col, cnt, 0, 1, [&](const int4& q) {
            float4 a[4], v[4];
            load_chunk<P>(R, q, a, v);
            pair_chunk<P>(k, q, a, v, acc);
        });
    }
}

// Neighbours of slot i (work position t; r2 < kh2) with their records R[2j], R[2j+1]: from the list
// (pairs in the skin beyond the support radius are skipped), or by walking the cells over
// X[XSTRIDE * j] when i overflowed the list.  f(j, a, b, dx, dy, dz, r2, vol); with kPairTwo the list
// of a fluid particle goes through acc.fluid_two instead.
template <class P, int LIST, int XSTRIDE, bool DEEP, class Acc, class F>
__device__ __forceinline__ void visit_records(const KParamsT<typename P::T>& k,
                                              const int* __restrict__ cs,
                                              const unsigned* __restrict__ keys,
                                              const NbrList& nl,
                                              const vec4_t<typename P::T>* __restrict__ X,
                                              const vec4_t<typename P::T>* __restrict__ R,
                                              const typename P::T* __restrict__ vol, int t, int i,
                                              Acc& acc, F&& f) {
    using T = typename P::T;
    using V = vec4_t<T>;
    if constexpr (LIST != LIST_NONE) {
        const int cnt = __ldg(nl.count + t);
        if (cnt <= nl.cap) {
            if constexpr (kPairTwo<P>) {
                if (acc.fi) {
                    visit_fluid<P, LIST == LIST_WIN, DEEP>(k, nl, R, t, cnt, acc);
                    return;
                }
            }
            auto one = [&](int e) {
                const int j = P::kCodes ? slot_index(e) : e;
                V a, b;
                ld_rec(R, j, a, b);
                T dx, dy, dz;
                rel_pos<P>(k, acc.pi, a, P::kCodes ? (unsigned)e : 0u, dx, dy, dz);
                const T r2 = dist2(dx, dy, dz);
                if (inside(r2, k.kh2)) f(j, a, b, dx, dy, dz, r2, ld_vol(vol, j));
            };
            for_each_chunk<LIST == LIST_WIN>(nl.idx + nbr_col(nl, t), cnt, 0, 1,
                                             [&](const int4& q) {
                one(q.x);
                one(q.y);
                one(q.z);
                one(q.w);
            });
            return;
        }
    }
    walk_pairs<P, XSTRIDE>(k, cs, keys, X, i, acc.pi, k.kh2,
                           [&](int j, unsigned, const V&, T dx, T dy, T dz, T r2) {
        V a, b;
        ld_rec(R, j, a, b);
        f(j, a, b, dx, dy, dz, r2, ld_vol(vol, j));
    });
}

// Neighbour-list build: every boundary particle keeps its fluid neighbours (all that pass 1
// needs), every fluid particle all of them; with walls_all, boundary particles keep all.
// Slots are warp-interleaved (nbr_col): the passes read them coalesced, the build writes them
// scattered within its warp's block, which L2 merges before they reach HBM.
template <class P, bool WIN>
__device__ __forceinline__ void nbr_build_one(const KParamsT<typename P::T>& k,
                                              const vec4_t<typename P::T>* __restrict__ X,
                                              const unsigned* __restrict__ keys,
                                              const int* __restrict__ cs, const NbrList& nl,
                                              int walls_all, unsigned* err, int4* stage, int t) {
    using T = typename P::T;
    const int i = work_slot(nl, t);
    T cut2 = nl.cut2 ? (T)__ldg(nl.cut2) : k.kh2_list;
    if (nl.iw) {
        // per-instance decisions: the particles of the instances that rebuild, each at its
        // instance's list cutoff; the others keep their lists
        const unsigned* w = nl.iw + IW_STRIDE * (__ldg(nl.inst + i) + 1);
        if (!w[IW_REBUILD]) return;
        cut2 = (T)__uint_as_float(w[IW_CUT2]);
    }
    const vec4_t<T> pi = X[i];
    if (nl.xb) nl.xb[i] = as_float4(pi);
    const bool keep_all = fluid_rec(pi.w) || walls_all;
    if (!keep_all && nl.rank && !inactive_key(k, keys[i])) {
        // a boundary particle with no fluid in the cells it walks has an empty list
        int cx, cy, cz;
        cell_of_key(k.gx, k.gy, keys[i], cx, cy, cz);
        if (!near_fluid(k, cs, nl.rank, cx, cy, cz)) {
            nl.count[t] = 0;
            return;
        }
    }
    SlotWriter<WIN> w(nl.idx + nbr_col(nl, t), nl.cap, stage);
    if constexpr (P::kCodes) {
        // i's offsets moved into each run's anchor frame once per run instead of decoding the
        // code for every candidate.  That rounds differently from the passes' decode, so the
        // cutoff is widened by 2^-16: every pair the passes would put inside it is listed, and
        // the passes test r < kh with their own decode, so they still evaluate exactly the
        // pairs of a cell walk.
        const unsigned key = keys[i];
        if (!inactive_key(k, key)) {
            int cx, cy, cz;
            cell_of_key(k.gx, k.gy, key, cx, cy, cz);
            const T cut2w = cut2 * (T(1) + T(1.0 / 65536.0));
            const StripWindow win = strip_window<P>(k, pi, cx, cy, cz, cut2w);
            for_each_run<true>(k, cs, cx, cy, cz, [&](int j0, int j1, unsigned code) {
                float fx, fy, fz;
                code_steps(code, fx, fy, fz);
                const float sx = fma_rn(-fx, k.reach_cell, pi.x);
                const float sy = fma_rn(-0.25f * fy, k.reach_cell, pi.y);
                const float sz = fma_rn(-0.0625f * fz, k.reach_cell, pi.z);
#pragma unroll 4
                for (int j = j0; j < j1; j++) {
                    const vec4_t<T> pj = ld_pos(X, (size_t)j);
                    const T r2 = dist2(sub_rn(sx, pj.x), sub_rn(sy, pj.y), sub_rn(sz, pj.z));
                    if (r2 < cut2w && j != i && (keep_all || fluid_rec(pj.w)))
                        w.put(make_slot(j, code));
                }
            }, win);
        }
    } else {
        // the cell walk of walk_pairs, narrowed to the cells the cutoff sphere reaches (the
        // same slots pass the distance test, in the same order)
        const unsigned key = keys[i];
        if (!inactive_key(k, key)) {
            int cx, cy, cz;
            cell_of_key(k.gx, k.gy, key, cx, cy, cz);
            const StripWindow win = strip_window<P>(k, pi, cx, cy, cz, cut2);
            for_each_run<false>(k, cs, cx, cy, cz, [&](int j0, int j1, unsigned) {
#pragma unroll 4
                for (int j = j0; j < j1; j++) {
                    const vec4_t<T> pj = ld_pos(X, (size_t)j);
                    T dx, dy, dz;
                    rel_pos<P>(k, pi, pj, 0u, dx, dy, dz);
                    const T r2 = dist2(dx, dy, dz);
                    if (r2 < cut2 && j != i && (keep_all || fluid_rec(pj.w))) w.put(j);
                }
            }, win);
        }
    }
    w.flush(pad_slot<P>(k.n));
    nl.count[t] = w.cnt;
    raise_flags(err, w.cnt > nl.cap ? SPH_FLAG_NEIGHBOR_OVERFLOW : 0u);
}

template <class P, bool GS, bool WIN>
__global__ void __launch_bounds__(NS_MAX_THREADS)
k_nbr_build(KParamsT<typename P::T> k, const vec4_t<typename P::T>* __restrict__ X,
            const unsigned* __restrict__ keys, const int* __restrict__ cs, NbrList nl,
            vec4_t<typename P::T>* rec, vec4_t<typename P::T>* nrec, int walls_all, unsigned* err,
            const unsigned* gate) {
    __shared__ int4 s_stage[SlotWriter<WIN>::kStage * NS_MAX_THREADS];
    if (gated_off(gate)) return;
    int4* stage = s_stage;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 == 0) {
        pad_record<typename P::T>(rec, k.n);
        pad_record<typename P::T>(nrec, k.n);
    }
    if constexpr (GS) {
        for (int i = i0; i < k.n; i += gridDim.x * blockDim.x)
            nbr_build_one<P, WIN>(k, X, keys, cs, nl, walls_all, err, stage, i);
    } else if (i0 < k.n) {
        nbr_build_one<P, WIN>(k, X, keys, cs, nl, walls_all, err, stage, i0);
    }
}

template <class P, bool WRITE_SUMS, int LIST, bool DEEP>
__device__ __forceinline__ void pass1_one(const KParamsT<typename P::T>& k,
                                          const ParticleSetT<typename P::T>& in,
                                          const unsigned* __restrict__ keys,
                                          const int* __restrict__ cs, const NbrList& nl,
                                          const Pass1OutT<typename P::T>& out,
                                          float* __restrict__ rhop_sum, float* __restrict__ w_sum,
                                          int t) {
    using T = typename P::T;
    using V = vec4_t<T>;
    const int i = work_slot(nl, t);
    Pass1Acc<P> acc;
    acc.load(in.rec, i);
    // a particle whose list overflowed walks the records' positions, a pass without lists the dense
    // ones of this half step's rebuild
    visit_records<P, LIST, LIST == LIST_NONE ? 1 : 2, DEEP>(k, cs, keys, nl,
                              LIST == LIST_NONE ? in.xyz : in.rec, in.rec, in.vol, t, i, acc,
                              [&](int, const V& aj, const V& vj, T dx, T dy, T dz, T r2, T vol) {
        acc.pair(k, aj, vj, dx, dy, dz, r2, vol);
    });
    acc.template finish<WRITE_SUMS>(k, out, rhop_sum, w_sum, i);
}

// Registers of pass 1: room for the four records of a chunk in flight, or (DEEP) two chunks.
template <class P, bool DEEP>
constexpr int kPass1Regs = DEEP ? 144 : std::is_same<typename P::T, double>::value ? 96 : 72;

template <class P, bool WRITE_SUMS, int LIST, bool GS, bool DEEP = false>
__global__ void __maxnreg__((kPass1Regs<P, DEEP>))
k_pass1(KParamsT<typename P::T> k, ParticleSetT<typename P::T> in,
        const unsigned* __restrict__ keys, const int* __restrict__ cs, NbrList nl,
        Pass1OutT<typename P::T> out, float* __restrict__ rhop_sum, float* __restrict__ w_sum) {
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (GS) {
        for (int i = i0; i < k.n; i += gridDim.x * blockDim.x)
            pass1_one<P, WRITE_SUMS, LIST, DEEP>(k, in, keys, cs, nl, out, rhop_sum, w_sum, i);
    } else if (i0 < k.n) {
        pass1_one<P, WRITE_SUMS, LIST, DEEP>(k, in, keys, cs, nl, out, rhop_sum, w_sum, i0);
    }
}
template <class P, int MODE, int LIST, bool DEEP>
__device__ __forceinline__ void pass2_one(const KParamsT<typename P::T>& k, int t,
                                          const ParticleSetT<typename P::T>& in,
                                          const unsigned* __restrict__ keys,
                                          const int* __restrict__ cs, const NbrList& nl,
                                          const Pass1OutT<typename P::T>& p1,
                                          float* __restrict__ rho_dt, float* __restrict__ vel_dt,
                                          int wall_rates, const ParticleSetT<typename P::T>& out,
                                          unsigned* __restrict__ out_hash, unsigned* err,
                                          DispBox& box, unsigned* disp) {
    using T = typename P::T;
    using V = vec4_t<T>;
    const int i = work_slot(nl, t);
    Pass2Acc<P, MODE> acc;
    acc.load(k, p1, i, wall_rates);
    if (acc.active)
        visit_records<P, LIST, 2, DEEP>(k, cs, keys, nl, p1.nrec, p1.nrec, p1.vol, t, i, acc,
                                  [&](int j, const V& aj, const V& vj, T dx, T dy, T dz, T r2,
                                      T vol) {
            acc.pair(k, p1, j, aj, vj, dx, dy, dz, r2, vol);
        });
    pass2_finish<P, MODE>(k, i, acc, in, keys, nl, rho_dt, vel_dt, wall_rates, out, out_hash,
                          err, box, disp);
}


template <class P, int MODE, int LIST, bool GS>
__global__ void __launch_bounds__(NS_MAX_THREADS)
k_pass2(KParamsT<typename P::T> k, ParticleSetT<typename P::T> in,
        const unsigned* __restrict__ keys, const int* __restrict__ cs, NbrList nl,
        Pass1OutT<typename P::T> p1, float* __restrict__ rho_dt, float* __restrict__ vel_dt,
        int wall_rates, ParticleSetT<typename P::T> out, unsigned* __restrict__ out_hash,
        unsigned* err, unsigned* disp) {
    DispBox box;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (GS) {
        for (int i = i0; i < k.n; i += gridDim.x * blockDim.x)
            pass2_one<P, MODE, LIST, false>(k, i, in, keys, cs, nl, p1, rho_dt, vel_dt, wall_rates,
                                            out, out_hash, err, box, disp);
    } else if (i0 < k.n) {
        pass2_one<P, MODE, LIST, false>(k, i0, in, keys, cs, nl, p1, rho_dt, vel_dt, wall_rates,
                                        out, out_hash, err, box, disp);
    }
    if (MODE == MODE_RATES || disp == nullptr) return;
    // the block's displacement box; blockDim is a multiple of 32, every thread gets here
    __shared__ unsigned s_box[6 * (NS_MAX_THREADS / 32)];
    __shared__ int s_inst[NS_MAX_THREADS / 32];
    reduce_disp(k, box, disp, s_box, s_inst);
}

// The same kernel held to CAP registers (one particle per thread): room for a chunk's four records
// in flight with the most warps that leaves.  At 133,968 particles (linear EOS) 80 registers run
// in 29 us, 64 in 35, 48 in 49, against 44 for one gather at a time in 40; at 380,000 80 run in
// 45 us, 96 in 55.  More than 100 registers: the deep form (visit_fluid).  The kernel on cell-local
// offsets keeps 72 (380,000 particles: 77 us, 79 at 80, 83 at 64).
template <class P, int MODE, int LIST, int CAP>
__global__ void __maxnreg__(CAP)
k_pass2_cap(KParamsT<typename P::T> k, ParticleSetT<typename P::T> in,
        const unsigned* __restrict__ keys, const int* __restrict__ cs, NbrList nl,
        Pass1OutT<typename P::T> p1, float* __restrict__ rho_dt, float* __restrict__ vel_dt,
        int wall_rates, ParticleSetT<typename P::T> out, unsigned* __restrict__ out_hash,
        unsigned* err, unsigned* disp) {
    DispBox box;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < k.n)
        pass2_one<P, MODE, LIST, (CAP > 100)>(k, t, in, keys, cs, nl, p1, rho_dt, vel_dt,
                                              wall_rates, out, out_hash, err, box, disp);
    if (MODE == MODE_RATES || disp == nullptr) return;
    // the block's displacement box; blockDim is a multiple of 32, every thread gets here
    __shared__ unsigned s_box[6 * (NS_MAX_THREADS / 32)];
    __shared__ int s_inst[NS_MAX_THREADS / 32];
    reduce_disp(k, box, disp, s_box, s_inst);
}

// Launch shape of a neighbour kernel: KParams::threads per block, KParams::ppt particles per
// thread.
template <class KP>
inline dim3 ns_grid(const KP& k) {
    const long per_block = (long)k.threads * (k.ppt > 0 ? k.ppt : 1);
    const long b = ((long)k.n + per_block - 1) / per_block;
    return dim3((unsigned)(b > 0 ? b : 1));
}

template <class P, int LIST, bool GS>
void pass1_launch_gs(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& in,
                     const unsigned* keys, const int* cs, const NbrList& nl,
                     const Pass1OutT<typename P::T>& o, float* rhop_sum, float* w_sum,
                     cudaStream_t s) {
    const dim3 b = ns_grid(k);
    if constexpr (P::kId == SPH_PREC_FP32) {
        if (rhop_sum && w_sum) {
            k_pass1<P, true, LIST, GS><<<b, k.threads, 0, s>>>(k, in, keys, cs, nl, o, rhop_sum,
                                                               w_sum);
            return;
        }
    }
    k_pass1<P, false, LIST, GS><<<b, k.threads, 0, s>>>(k, in, keys, cs, nl, o, nullptr,
                                                        nullptr);
}

// Below this many particles the passes run their deep form.  27,288 particles, five steps: FP32 292
// us against 328, cell-local offsets 318 against 380; at 133,968 it has too few warps left (ten
// steps 1.20 ms against 1.11).
constexpr int DEEP_MAX_PARTICLES = 60000;

template <class P, int LIST>
void pass1_launch(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& in,
                  const unsigned* keys, const int* cs, const NbrList& nl,
                  const Pass1OutT<typename P::T>& o, float* rhop_sum, float* w_sum,
                  cudaStream_t s) {
    if constexpr (LIST == LIST_PLAIN && kPairTwo<P>) {
        if (k.ppt <= 1 && k.n < DEEP_MAX_PARTICLES && !rhop_sum && !w_sum) {
            k_pass1<P, false, LIST, false, true><<<ns_grid(k), k.threads, 0, s>>>(
                k, in, keys, cs, nl, o, nullptr, nullptr);
            return;
        }
    }
    if (k.ppt > 1)
        pass1_launch_gs<P, LIST, true>(k, in, keys, cs, nl, o, rhop_sum, w_sum, s);
    else
        pass1_launch_gs<P, LIST, false>(k, in, keys, cs, nl, o, rhop_sum, w_sum, s);
}

template <class P, int MODE, bool GS>
void pass2_launch_gs(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& in,
                     const unsigned* keys, const int* cs, const NbrList* nl,
                     const Pass1OutT<typename P::T>& p1, float* rho_dt, float* vel_dt,
                     int wall_rates, ParticleSetT<typename P::T> out, unsigned* out_hash,
                     unsigned* err, unsigned* disp, cudaStream_t s) {
    const dim3 b = ns_grid(k);
    if (!nl) {
        k_pass2<P, MODE, LIST_NONE, GS><<<b, k.threads, 0, s>>>(k, in, keys, cs, NbrList{}, p1,
                                                                 rho_dt, vel_dt, wall_rates, out,
                                                                 out_hash, err, nullptr);
        return;
    }
    auto with_list = [&](auto mode) {
        constexpr int L = decltype(mode)::value;
        if constexpr (MODE != MODE_RATES && !GS && (P::kId == SPH_PREC_FP32 || P::kMixed)) {
            if constexpr (L == LIST_PLAIN && kPairTwo<P>) {
                if (k.n < DEEP_MAX_PARTICLES) {
                    k_pass2_cap<P, MODE, L, 168><<<b, k.threads, 0, s>>>(
                        k, in, keys, cs, *nl, p1, rho_dt, vel_dt, wall_rates, out, out_hash, err,
                        disp);
                    return;
                }
            }
            constexpr int cap = P::kCodes ? 72 : 80;
            k_pass2_cap<P, MODE, L, cap><<<b, k.threads, 0, s>>>(
                k, in, keys, cs, *nl, p1, rho_dt, vel_dt, wall_rates, out, out_hash, err, disp);
        } else {
            k_pass2<P, MODE, L, GS><<<b, k.threads, 0, s>>>(k, in, keys, cs, *nl, p1, rho_dt,
                                                             vel_dt, wall_rates, out, out_hash,
                                                             err, disp);
        }
    };
    // the rates (sph_ns) run on the drop-in's own list, which has plain windows
    if constexpr (MODE != MODE_RATES) {
        if (k.list_win) {
            with_list(std::integral_constant<int, LIST_WIN>{});
            return;
        }
    }
    with_list(std::integral_constant<int, LIST_PLAIN>{});
}

template <class P, int MODE>
void pass2_launch(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& in,
                  const unsigned* keys, const int* cs, const NbrList* nl,
                  const Pass1OutT<typename P::T>& p1, float* rho_dt, float* vel_dt,
                  int wall_rates, ParticleSetT<typename P::T> out, unsigned* out_hash,
                  unsigned* err, unsigned* disp, cudaStream_t s) {
    if (k.ppt > 1)
        pass2_launch_gs<P, MODE, true>(k, in, keys, cs, nl, p1, rho_dt, vel_dt, wall_rates, out,
                                       out_hash, err, disp, s);
    else
        pass2_launch_gs<P, MODE, false>(k, in, keys, cs, nl, p1, rho_dt, vel_dt, wall_rates,
                                        out, out_hash, err, disp, s);
}

}  // namespace

double lattice_neighbours(const sph_params& p, double skin) {
    const double r = (double)p.kh * (1.0 + skin) / (double)p.dx;
    return 4.18879020478639 * r * r * r;
}

int nbr_capacity_for(const sph_params& p, double skin) {
    // 1.5x the particles of a lattice inside the list sphere, rounded up to 16
    int cap = (int)(1.5 * lattice_neighbours(p, skin)) + 16;
    cap = (cap + 15) & ~15;
    return cap < 32 ? 32 : cap;
}

template <class P>
cudaError_t launch_nbr_build(const KParamsT<typename P::T>& k,
                             const ParticleSetT<typename P::T>& in, const unsigned* keys,
                             const int* cs, const NbrList& nl, vec4_t<typename P::T>* nrec,
                             int walls_all, unsigned* err, cudaStream_t s, const unsigned* gate) {
    if (k.n <= 0) return cudaSuccess;
    const dim3 g = ns_grid(k);
    if (k.ppt > 1) {
        if (k.list_win)
            k_nbr_build<P, true, true><<<g, k.threads, 0, s>>>(k, in.xyz, keys, cs, nl, in.rec, nrec,
                                                                walls_all, err, gate);
        else
            k_nbr_build<P, true, false><<<g, k.threads, 0, s>>>(k, in.xyz, keys, cs, nl, in.rec, nrec,
                                                                 walls_all, err, gate);
    } else {
        if (k.list_win)
            k_nbr_build<P, false, true><<<g, k.threads, 0, s>>>(k, in.xyz, keys, cs, nl, in.rec, nrec,
                                                                 walls_all, err, gate);
        else
            k_nbr_build<P, false, false><<<g, k.threads, 0, s>>>(k, in.xyz, keys, cs, nl, in.rec, nrec,
                                                                  walls_all, err, gate);
    }
    return cudaGetLastError();
}

template <class P>
cudaError_t launch_pass1(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& in,
                         const unsigned* keys, const int* cs, const NbrList* nl,
                         const Pass1OutT<typename P::T>& out, float* rhop_sum, float* w_sum,
                         cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    if (nl && k.lanes > 1 && !rhop_sum && !w_sum)
        return launch_pass1_groups<P>(k, in, keys, cs, *nl, out, s);
    if (nl && k.list_win)
        pass1_launch<P, LIST_WIN>(k, in, keys, cs, *nl, out, rhop_sum, w_sum, s);
    else if (nl)
        pass1_launch<P, LIST_PLAIN>(k, in, keys, cs, *nl, out, rhop_sum, w_sum, s);
    else
        pass1_launch<P, LIST_NONE>(k, in, keys, cs, NbrList{}, out, rhop_sum, w_sum, s);
    return cudaGetLastError();
}

cudaError_t launch_pass2_rates(const KParams& k, const ParticleSet& in, const unsigned* keys,
                               const int* cs, const NbrList* nl, const Pass1Out& p1,
                               float* rho_dt, float* vel_dt, int wall_rates, cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    pass2_launch<PrecF32, MODE_RATES>(k, in, keys, cs, nl, p1, rho_dt, vel_dt, wall_rates,
                                      ParticleSet{}, nullptr, nullptr, nullptr, s);
    return cudaGetLastError();
}

template <class P>
cudaError_t launch_pass2_step(const KParamsT<typename P::T>& k, HalfStep half,
                              const ParticleSetT<typename P::T>& in, const unsigned* keys,
                              const int* cs, const NbrList* nl,
                              const Pass1OutT<typename P::T>& p1,
                              ParticleSetT<typename P::T> out, unsigned* out_hash, unsigned* err,
                              unsigned* disp, cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    if (half == HALF_PREDICT)
        pass2_launch<P, MODE_PRED>(k, in, keys, cs, nl, p1, nullptr, nullptr, 0, out, out_hash,
                                   err, disp, s);
    else
        pass2_launch<P, MODE_CORR>(k, in, keys, cs, nl, p1, nullptr, nullptr, 0, out, out_hash,
                                   err, disp, s);
    return cudaGetLastError();
}

#define SPH_NS_INSTANTIATE(P)                                                                  \
    template cudaError_t launch_nbr_build<P>(const KParamsT<P::T>&, const ParticleSetT<P::T>&, \
                                             const unsigned*, const int*, const NbrList&,      \
                                             vec4_t<P::T>*, int, unsigned*, cudaStream_t,      \
                                             const unsigned*);                                 \
    template cudaError_t launch_pass1<P>(const KParamsT<P::T>&, const ParticleSetT<P::T>&,     \
                                         const unsigned*, const int*, const NbrList*,          \
                                         const Pass1OutT<P::T>&, float*, float*, cudaStream_t);\
    template cudaError_t launch_pass2_step<P>(                                                 \
        const KParamsT<P::T>&, HalfStep, const ParticleSetT<P::T>&, const unsigned*,           \
        const int*, const NbrList*, const Pass1OutT<P::T>&, ParticleSetT<P::T>, unsigned*,    \
        unsigned*, unsigned*, cudaStream_t);
SPH_NS_INSTANTIATE(PrecF32)
SPH_NS_INSTANTIATE(PrecF64)
SPH_NS_INSTANTIATE(PrecMix)
SPH_NS_INSTANTIATE(PrecMixC)
SPH_NS_INSTANTIATE(PrecMixA)
#undef SPH_NS_INSTANTIATE

}  // namespace sph
