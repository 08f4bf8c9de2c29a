// ns_twin.cu — the neighbour list and both passes with two particles per thread, for the FP32 pair
// arithmetic (FP32, and mixed precision on FP32 positions).
//
// Same pairs, same arithmetic and same order of every particle's sums as ns.cu (bit for bit);
// another assignment of work to threads.  Thread u takes work positions 2u and 2u + 1 over one
// list: the union of their neighbours in cell-walk order, about 1.3 times as long as either's.
// Every record gathered serves both (two-lane instructions, one lane per particle, each sum under
// the predicate of its own distance), so a particle costs 0.65 gathers per neighbour instead of
// one: the passes with one particle per thread are bound by the L1 data stage and the latency of
// those gathers.
//
// The two particles lie one above the other (the same x in rows y = 2m and 2m + 1; k_work_order
// merges the rows): the lanes of a warp then still gather neighbouring records, 9.3 L1 wavefronts
// a request.  Two neighbours of one row per thread have the same union but put the lanes two
// records apart: 17 wavefronts, and pass 1 at 467 instead of 361 us (4.96M particles).
//
// Measured, pass 1 / pass 2 against one particle per thread with one gather in flight: 4.96M
// particles 520 / 609 -> 361 / 582 us, a disordered surge of 6.70M 1020 / 1078 -> 750 / 927 us (with
// the copies that pass 2 no longer writes, 357 / 555 of 4.96M).  What is left is latency: pass 2
// issues in 62% of cycles with 19 warps per SM (a cap of 104 registers, 96 used), L1 data stage 48%
// (pass 1: 60%, 22 warps, 73%).  Slower: 80 registers (630 us, the gathers of a chunk no longer
// issued together), records of the next half chunk loaded during the current one (640-690 us),
// lists prefetched into L2 ahead of their use (level).
//
// The two particles must be of one simulation: candidates are told apart by distance alone, and
// batched instances hold positions in a frame of their own each.  The work order of a batch gives each
// instance's fluid and each one's walls an even number of positions, so no thread holds two instances.
// (A list of each particle in its half of the column, for the threads on a seam, kept the pairs but not
// the time: such a thread reads two lists one after the other, and its warp waits.  16 tanks of 25,000
// particles 0.22 ms a step, 0.15 with even positions.)
#include <cuda_runtime.h>

#include <type_traits>

#include "ns_pair.cuh"
#include "sph_internal.h"

namespace sph {

namespace {

// The two particles of thread u: slots a and b (b = a when u has one particle only).  BATCH: of a padded
// work order, where no slot is -1 (none of a thread past the last instance).
struct Twin {
    int a, b;
    bool two;
};
template <bool BATCH>
__device__ __forceinline__ Twin twin_of(const NbrList& nl, int u, int n) {
    Twin w;
    w.a = work_slot(nl, 2 * u);
    if constexpr (BATCH) {
        const int b = work_slot(nl, 2 * u + 1);
        w.two = b >= 0;
        w.b = w.two ? b : w.a;
    } else {
        w.two = 2 * u + 1 < n;
        w.b = w.two ? work_slot(nl, 2 * u + 1) : w.a;
    }
    return w;
}
// Column of thread u's list: as nbr_col, with the slots of its two particles.
__device__ __forceinline__ size_t twin_col(const NbrList& nl, int u) {
    return (size_t)(u >> 5) * ((size_t)nl.cap << 6) + ((size_t)(u & 31) << 2);
}
// nl.count of a thread: the entries of its shared list, TWIN_WALKS when they do not fit it.
constexpr int TWIN_WALKS = -1;

// ---------------------------------------------------------------- list build
// One particle's side of the build: its cell and the part of a strip its cutoff sphere reaches.
struct TwinWalk {
    int cx, cy, cz;
    bool on;  // takes part in the neighbour search
    StripWindow win;
    template <class KP>
    __device__ __forceinline__ bool strip(const KP& k, int y, int z, int& xl, int& xh) const {
        const int r = k.reach;
        if (!on || abs(z - cz) > r || abs(y - cy) > r) return false;
        xl = max(cx - r, 0);
        xh = min(cx + r, k.gx - 1);
        return win(y, z, xl, xh);
    }
};

template <class P>
__device__ __forceinline__ TwinWalk twin_walk(const KParamsT<float>& k, const float4& p,
                                              unsigned key, float cut2) {
    TwinWalk w;
    w.on = !inactive_key(k, key);
    cell_of_key(k.gx, k.gy, w.on ? key : 0u, w.cx, w.cy, w.cz);
    w.win = strip_window<P>(k, p, w.cx, w.cy, w.cz, cut2);
    return w;
}

constexpr int TWIN_BUILD_THREADS = 128;

// Appends slots to a column without a branch per candidate: every candidate is written to the next
// free entry of the thread's ring in shared memory (RING entries, TWIN_BUILD_THREADS words apart)
// and a hit moves that entry on; drain() stores whole chunks of four.  At most CHUNK candidates may
// be offered between two drains.
struct RingWriter {
    static constexpr int RING = 16, CHUNK = 8;
    int* __restrict__ col;
    int cap;
    int* ring;
    int cnt = 0, out = 0;
    __device__ __forceinline__ RingWriter(int* c, int cp, int* r)
        : col(c), cap(cp), ring(r + threadIdx.x) {}
    __device__ __forceinline__ int& entry(int e) {
        return ring[(e & (RING - 1)) * TWIN_BUILD_THREADS];
    }
    __device__ __forceinline__ void offer(int j, bool hit) {
        entry(cnt) = j;
        cnt += hit;
    }
    __device__ __forceinline__ void store() {
        if (out < cap)  // cap is a multiple of 16
            *reinterpret_cast<int4*>(col + ((size_t)out << 5)) =
                make_int4(entry(out), entry(out + 1), entry(out + 2), entry(out + 3));
        out += 4;
    }
    __device__ __forceinline__ void drain() {
#pragma unroll 1
        while (cnt - out >= 4) store();
    }
    // the last, partial chunk, filled up with `pad`
    __device__ __forceinline__ void flush(int pad) {
        drain();
        if (cnt == out) return;
        for (int e = cnt; e < out + 4; e++) entry(e) = pad;
        store();
    }
};

// The shared lists.  Bound by instructions (62% issue, 40% of the ALU pipe; about 390 candidates a
// warp for 100 listed slots).  4.96M particles, 1.60 ms with a window per particle and strip and a
// branch per candidate; 1.27 with one walk over the rows and cells either sphere reaches; 1.16 with
// branch-free candidates on top; 1.05 with near_fluid on the fluid ranks.
//
// BATCH: batched instances, on a padded work order (twin_of).
template <class P, bool BATCH>
__global__ void __launch_bounds__(TWIN_BUILD_THREADS)
k_nbr_build_twin(KParamsT<float> k, const float4* __restrict__ X,
                 const unsigned* __restrict__ keys, const int* __restrict__ cs, NbrList nl,
                 float4* rec, float4* nrec, unsigned* err, const unsigned* gate) {
    __shared__ int s_ring[RingWriter::RING * TWIN_BUILD_THREADS];
    if (gated_off(gate)) return;
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u == 0) {
        pad_record<float>(rec, k.n);
        pad_record<float>(nrec, k.n);
    }
    if (2 * u >= (BATCH ? k.positions : k.n)) return;
    const float cut2 = nl.cut2 ? __ldg(nl.cut2) : k.kh2_list;
    const Twin tw = twin_of<BATCH>(nl, u, k.n);
    if (BATCH && tw.a < 0) return;
    const int a = tw.a, b = tw.b;
    const float4 pa = X[a], pb = X[b];
    if (nl.xb) {
        nl.xb[a] = pa;
        nl.xb[b] = pb;
    }
    const bool alla = fluid_rec(pa.w), allb = fluid_rec(pb.w);
    const TwinWalk wa = twin_walk<P>(k, pa, keys[a], cut2), wb = twin_walk<P>(k, pb, keys[b], cut2);
    if (!alla && !allb && nl.rank && !(wa.on && near_fluid(k, cs, nl.rank, wa.cx, wa.cy, wa.cz)) &&
        !(wb.on && near_fluid(k, cs, nl.rank, wb.cx, wb.cy, wb.cz))) {
        nl.count[u] = 0;
        return;
    }
    const int r = k.reach;
    // two particles next to each other in one layer, each inside its cell
    const bool near = wa.on && wb.on && wa.cz == wb.cz && abs(wa.cy - wb.cy) <= 1 &&
                      abs(wa.cx - wb.cx) <= 2 && wa.win.rc2 >= 0.f && wb.win.rc2 >= 0.f;
    // one(j, position) for the candidates of slots j0 .. j1 - 1, chunk() after at most CHUNK
    auto take = [&](int j, int j1, auto&& one, auto&& chunk) {
#pragma unroll 1
        while (j < j1) {
            const int je = min(j + RingWriter::CHUNK, j1);
#pragma unroll 1
            for (; j + 1 < je; j += 2) {
                const float4 p = ld_pos(X, (size_t)j), q = ld_pos(X, (size_t)j + 1);
                one(j, p);
                one(j + 1, q);
            }
            if (j < je) {
                one(j, ld_pos(X, (size_t)j));
                j++;
            }
            chunk();
        }
    };
    // every candidate of either particle in (z, y, x) order of the cells
    auto visit = [&](auto&& one, auto&& chunk) {
        if (near) {
            // one walk over the cells either cutoff sphere reaches
            const float rc2 = wa.win.rc2;
            const float uxl = fminf(wa.win.ux, wb.win.ux), uxh = fmaxf(wa.win.ux, wb.win.ux);
            const float uyl = fminf(wa.win.uy, wb.win.uy), uyh = fmaxf(wa.win.uy, wb.win.uy);
            const float uzl = fminf(wa.win.uz, wb.win.uz), uzh = fmaxf(wa.win.uz, wb.win.uz);
            const int xl0 = max(min(wa.cx, wb.cx) - r, 0);
            const int xh0 = min(max(wa.cx, wb.cx) + r, k.gx - 1);
            const int yl0 = max(min(wa.cy, wb.cy) - r, 0);
            const int yh0 = min(max(wa.cy, wb.cy) + r, k.gy - 1);
            const int z1 = min(wa.cz + r, k.gz - 1);
            int z = max(wa.cz - r, 0) - 1, y = 0, y1 = -1;
            float w2z = 0.f;
            // the slots of the next strip the spheres reach (widened as StripWindow does)
            auto next = [&](int& j0, int& j1) {
                for (;;) {
                    while (++y > y1) {
                        if (++z > z1) return false;
                        const float fz = (float)(z - wa.win.zb);
                        const float dz = fmaxf(0.f, fmaxf(fz - uzh, uzl - fz - 1.f));
                        w2z = rc2 - dz * dz;
                        const float wy = pair_sqrt(fmaxf(w2z, 0.f)) + 1e-3f;
                        y = max(yl0, (int)floorf(uyl - wy)) - 1;
                        y1 = w2z < 0.f ? y : min(yh0, (int)floorf(uyh + wy));
                    }
                    const float fy = (float)y;
                    const float dy = fmaxf(0.f, fmaxf(fy - uyh, uyl - fy - 1.f));
                    const float wx = pair_sqrt(fmaxf(w2z - dy * dy, 0.f)) + 1e-3f;
                    const int xl = max(xl0, (int)floorf(uxl - wx));
                    const int xh = min(xh0, (int)floorf(uxh + wx));
                    if (xl > xh) continue;
                    const int row = (z * k.gy + y) * k.gx;
                    j0 = max(__ldg(cs + row + xl), 0);
                    j1 = min(__ldg(cs + row + xh + 1), k.n);  // bounds guard only
                    return true;
                }
            };
            // the next strip's slots are looked up while the candidates of this one are tested
            int j0 = 0, j1 = 0;
            bool more = next(j0, j1);
#pragma unroll 1
            while (more) {
                const int i0 = j0, i1 = j1;
                more = next(j0, j1);
                take(i0, i1, one, chunk);
            }
            return;
        }
        if (!wa.on && !wb.on) return;
        // the strips of either particle, each particle's cells of a strip
        auto run = [&](int row, int x0, int x1) {
            take(max(__ldg(cs + row + x0), 0), min(__ldg(cs + row + x1 + 1), k.n), one, chunk);
        };
        const int za = wa.on ? wa.cz : wb.cz, zb = wb.on ? wb.cz : wa.cz;
        const int z1 = min(max(za, zb) + r, k.gz - 1);
#pragma unroll 1
        for (int z = max(min(za, zb) - r, 0); z <= z1; z++) {
            const bool ina = wa.on && abs(z - wa.cz) <= r, inb = wb.on && abs(z - wb.cz) <= r;
            if (!ina && !inb) {  // between two particles far apart
                z = max(za, zb) - r - 1;
                continue;
            }
            const int ya = ina ? wa.cy : wb.cy, yb = inb ? wb.cy : wa.cy;
            const int y1 = min(max(ya, yb) + r, k.gy - 1);
#pragma unroll 1
            for (int y = max(min(ya, yb) - r, 0); y <= y1; y++) {
                if (abs(y - ya) > r && abs(y - yb) > r) {
                    y = max(ya, yb) - r - 1;
                    continue;
                }
                int la, ha, lb, hb;
                const bool sa = wa.strip(k, y, z, la, ha), sb = wb.strip(k, y, z, lb, hb);
                if (!sa && !sb) continue;
                const int row = (z * k.gy + y) * k.gx;
                int l = sa ? la : lb, h = sa ? ha : hb, l2 = 1, h2 = 0;
                if (sa && sb) {
                    l = min(la, lb);
                    h = max(ha, hb);
                    if (max(la, lb) > min(ha, hb) + 1) {  // two separate runs of one strip
                        l2 = max(la, lb);
                        h2 = h;
                        h = min(ha, hb);
                    }
                }
#pragma unroll 1
                for (;;) {
                    run(row, l, h);
                    if (l2 > h2) break;
                    l = l2;
                    h = h2;
                    h2 = l2 - 1;
                }
            }
        }
    };
    // the candidates inside either cutoff.  A particle itself passes its own test (r^2 = 0) and may
    // be listed: it adds nothing to its sums.
    RingWriter w(nl.idx + twin_col(nl, u), 2 * nl.cap, s_ring);
    auto dist = [&](const float4& p, float& r2a, float& r2b) {
        float ax, ay, az, bx, by, bz;
        rel_pos<P>(k, pa, p, 0u, ax, ay, az);
        rel_pos<P>(k, pb, p, 0u, bx, by, bz);
        r2a = dist2(ax, ay, az);
        r2b = dist2(bx, by, bz);
    };
    const float ca = alla ? cut2 : -1.f, cb = allb ? cut2 : -1.f;  // cutoffs for boundary candidates
    visit(
        [&](int j, const float4& p) {
            float r2a, r2b;
            dist(p, r2a, r2b);
            const bool fj = fluid_rec(p.w);
            w.offer(j, r2a < (fj ? cut2 : ca) || r2b < (fj ? cut2 : cb));
        },
        [&]() { w.drain(); });
    w.flush(pad_slot<P>(k.n));
    // A particle overflows when its own neighbours do: counted only when the shared list is longer than
    // one particle's room, from the list just written where it is whole (a third of the candidates of
    // another walk), else from the candidates.  Only a list that is not whole sends its particles to
    // their cells: a whole one has both, overflowed or not (765,828 disordered particles with 96 slots,
    // which many overflow: a step 0.67 ms when those walked, 0.51 now).
    bool over = false;
    if (w.cnt > nl.cap) {
        int na = 0, nb = 0;
        auto count = [&](int j, const float4& p) {
            float r2a, r2b;
            dist(p, r2a, r2b);
            const bool fj = fluid_rec(p.w);
            na += j != a && r2a < (fj ? cut2 : ca);
            nb += j != b && r2b < (fj ? cut2 : cb);
        };
        if (w.cnt <= 2 * nl.cap) {
#pragma unroll 1
            for (int c = 0; c < w.cnt; c += 4) {
                const int4 q = *reinterpret_cast<const int4*>(w.col + ((size_t)c << 5));
                const int e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int l = 0; l < 4; l++)
                    if (c + l < w.cnt) count(e[l], ld_pos(X, (size_t)e[l]));
            }
        } else {
            visit(count, [] {});
        }
        over = na > nl.cap || nb > nl.cap;
    }
    nl.count[u] = w.cnt > 2 * nl.cap ? TWIN_WALKS : w.cnt;
    raise_flags(err, over ? SPH_FLAG_NEIGHBOR_OVERFLOW : 0u);
}

// ---------------------------------------------------------------- passes
// The records of thread u's list, four gathers issued together: one(a, v) for each in order.
template <class F>
__device__ __forceinline__ void visit_twin(const NbrList& nl, const float4* __restrict__ R, int u,
                                           int cnt, F&& one) {
    for_each_chunk<false>(nl.idx + twin_col(nl, u), cnt, 0, 1, [&](const int4& q) {
        const int e[4] = {q.x, q.y, q.z, q.w};
        float4 a[4], v[4];
#pragma unroll
        for (int c = 0; c < 4; c++) ld_rec(R, e[c], a[c], v[c]);
#pragma unroll
        for (int c = 0; c < 4; c++) one(a[c], v[c]);
    });
}

// The cells of two particles that do not fit their list, when they are of one cell or of neighbouring
// ones: one box of cells holds the walks of both, and a candidate that only one of them walks lies
// outside the other's support radius.
struct TwinCells {
    int xl, xh, yl, yh, zl, zh;
    bool near;
};
__device__ __forceinline__ TwinCells twin_cells(const KParamsT<float>& k,
                                                const unsigned* __restrict__ keys, const Twin& tw) {
    TwinCells w;
    const unsigned ka = keys[tw.a], kb = keys[tw.b];
    w.near = !inactive_key(k, ka) && !inactive_key(k, kb);
    if (!w.near) return w;
    int ax, ay, az, bx, by, bz;
    cell_of_key(k.gx, k.gy, ka, ax, ay, az);
    cell_of_key(k.gx, k.gy, kb, bx, by, bz);
    const int r = k.reach;
    w.near = abs(ax - bx) <= 1 && abs(ay - by) <= 1 && abs(az - bz) <= 1;
    w.xl = max(min(ax, bx) - r, 0), w.xh = min(max(ax, bx) + r, k.gx - 1);
    w.yl = max(min(ay, by) - r, 0), w.yh = min(max(ay, by) + r, k.gy - 1);
    w.zl = max(min(az, bz) - r, 0), w.zh = min(max(az, bz) + r, k.gz - 1);
    return w;
}

// one(a, v) for the records of those cells, the candidates of a row of cells four at a time, the last
// four filled up with the padding record n.  Bound by the latency of one candidate's arithmetic after
// another, on few warps: 32,000 particles at one point among 765,828 take 13.2 ms a step; 48.7 with
// the two walked one after the other, a candidate at a time, 41.3 with one particle per thread.  Passing
// over candidates that neither needs costs the list path its registers.
template <class F>
__device__ __forceinline__ void walk_twin(const KParamsT<float>& k, const int* __restrict__ cs,
                                          const TwinCells& w, const float4* __restrict__ R,
                                          F&& one) {
#pragma unroll 1
    for (int z = w.zl; z <= w.zh; z++) {
#pragma unroll 1
        for (int y = w.yl; y <= w.yh; y++) {
            const int row = (z * k.gy + y) * k.gx;
            const int j0 = max(__ldg(cs + row + w.xl), 0);
            const int j1 = min(__ldg(cs + row + w.xh + 1), k.n);  // bounds guard only
#pragma unroll 1
            for (int j = j0; j < j1; j += 4) {
                float4 a[4], v[4];
#pragma unroll
                for (int c = 0; c < 4; c++) ld_rec(R, j + c < j1 ? j + c : k.n, a[c], v[c]);
#pragma unroll
                for (int c = 0; c < 4; c++) one(a[c], v[c]);
            }
        }
    }
}

// Pass-1 sums of two fluid particles and one neighbour (Pass1Acc::pair of each).
template <class P>
__device__ __forceinline__ void pass1_twin(const KParamsT<float>& k, Pass1Acc<P>& A,
                                           Pass1Acc<P>& B, const float4& aj, const float4& vj) {
    float ax, ay, az, bx, by, bz;
    rel_pos<P>(k, A.pi, aj, 0u, ax, ay, az);
    rel_pos<P>(k, B.pi, aj, 0u, bx, by, bz);
    const float r2a = dist2(ax, ay, az), r2b = dist2(bx, by, bz);
    const F2 rr = pack2(pair_sqrt(r2a), pair_sqrt(r2b));
    const F2 t = fma2_rn(F2{k.m_half2}, mul2_rn(rr, F2{k.inv_h2}), F2{k.one2});
    const F2 fr = mul2_rn(mul2_rn(F2{k.c_fr2}, mul2_rn(t, t)), t);
    const F2 vdotr = pack2(dot_rn(A.vi, vj, ax, ay, az), dot_rn(B.vi, vj, bx, by, bz));
    float ua, ub;
    unpack2(mul2_rn(fr, vdotr), ua, ub);
    const float m = mul_rn(k.mass, pair_rcp(vj.w));
    add_if(r2a, k.kh2, vj.w, -ua, m, A.dofv.s);
    add_if(r2b, k.kh2, vj.w, -ub, m, B.dofv.s);
}

// Pass-2 sums of two fluid particles and one neighbour (Pass2Acc::pair of each).
template <class P, int MODE>
__device__ __forceinline__ void pass2_twin(const KParamsT<float>& k, Pass2Acc<P, MODE>& A,
                                           Pass2Acc<P, MODE>& B, const float4& aj,
                                           const float4& vj) {
    float ax, ay, az, sa, bx, by, bz, sb;
    rel_pos_s<P>(k, A.pi, -A.presi, aj, 0u, ax, ay, az, sa);
    rel_pos_s<P>(k, B.pi, -B.presi, aj, 0u, bx, by, bz, sb);
    const float r2a = dist2(ax, ay, az), r2b = dist2(bx, by, bz);
    const F2 r2 = pack2(r2a, r2b);
    const float rhoj = dabs(vj.w);
    const F2 rr = pack2(pair_sqrt(r2a), pair_sqrt(r2b));
    const F2 t = fma2_rn(F2{k.m_half_inv_h2}, rr, F2{k.one2});
    float wa, wb, ea, eb;
    unpack2(mul2_rn(mul2_rn(F2{k.c_fr_mass2}, mul2_rn(t, t)), t), wa, wb);
    const float rj = pair_rcp(rhoj);
    wa = mul_rn(wa, rj);
    wb = mul_rn(wb, rj);
    const F2 vdotr = pack2(dot_rn(A.vi, vj, ax, ay, az), dot_rn(B.vi, vj, bx, by, bz));
    unpack2(add2_rn(r2, F2{k.eta2_2}), ea, eb);
    const F2 inv = pack2(pair_rcp(ea), pair_rcp(eb));
    const F2 dr = pack2(sub_rn(A.rhoi, rhoj), sub_rn(B.rhoi, rhoj));
    const F2 diff = mul2_rn(mul2_rn(mul2_rn(dr, F2{k.delta_h_cs2}), r2), inv);
    unpack2(fma2_rn(pack2(A.rhoi, B.rhoi), vdotr, diff), ea, eb);
    float va, vb;
    unpack2(fma2_rn(mul2_rn(F2{k.visc2}, vdotr), inv, pack2(A.damp_i, B.damp_i)), va, vb);
    const bool fj = fluid_rec(vj.w);
    const float ca = mul_rn(wa, fj ? add_rn(sa, va) : sa), cb = mul_rn(wb, fj ? add_rn(sb, vb) : sb);
    add_if(r2a, k.kh2, wa, ea, ca, ax, ay, az, A.sd.s, A.sx.s, A.sy.s, A.sz.s);
    add_if(r2b, k.kh2, wb, eb, cb, bx, by, bz, B.sd.s, B.sx.s, B.sy.s, B.sz.s);
}

template <class P, bool BATCH>
__global__ void __maxnreg__(80)
k_pass1_twin(KParamsT<float> k, ParticleSet in, const unsigned* __restrict__ keys,
             const int* __restrict__ cs, NbrList nl, Pass1Out out) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * u >= (BATCH ? k.positions : k.n)) return;
    const Twin tw = twin_of<BATCH>(nl, u, k.n);
    if (BATCH && tw.a < 0) return;
    Pass1Acc<P> A, B;
    A.load(in.rec, tw.a);
    B.load(in.rec, tw.b);
    const int cnt = __ldg(nl.count + u);
    if (cnt >= 0) {
        if (A.fi || B.fi) {
            visit_twin(nl, in.rec, u, cnt, [&](const float4& aj, const float4& vj) {
                pass1_twin<P>(k, A, B, aj, vj);
            });
            if (!A.fi) A.dofv.s = 0.f;
            if (!B.fi) B.dofv.s = 0.f;
        }
        if (!A.fi || !B.fi) {
            visit_twin(nl, in.rec, u, cnt, [&](const float4& aj, const float4& vj) {
                float dx, dy, dz;
                rel_pos<P>(k, A.pi, aj, 0u, dx, dy, dz);
                float r2 = dist2(dx, dy, dz);
                if (!A.fi && r2 < k.kh2) A.pair(k, aj, vj, dx, dy, dz, r2, 0.f);
                rel_pos<P>(k, B.pi, aj, 0u, dx, dy, dz);
                r2 = dist2(dx, dy, dz);
                if (!B.fi && r2 < k.kh2) B.pair(k, aj, vj, dx, dy, dz, r2, 0.f);
            });
        }
    } else {
        const TwinCells w = twin_cells(k, keys, tw);
        if (w.near && A.fi && B.fi) {
            walk_twin(k, cs, w, in.rec, [&](const float4& aj, const float4& vj) {
                pass1_twin<P>(k, A, B, aj, vj);
            });
        } else {
#pragma unroll 1
            for (int m = 0; m < 2; m++) {
                Pass1Acc<P> C = m ? B : A;
                walk_pairs<P, 2>(k, cs, keys, in.rec, m ? tw.b : tw.a, C.pi, k.kh2,
                                 [&](int j, unsigned, const float4&, float dx, float dy, float dz,
                                     float r2) {
                    float4 aj, vj;
                    ld_rec(in.rec, j, aj, vj);
                    C.pair(k, aj, vj, dx, dy, dz, r2, 0.f);
                });
                if (m) B = C;
                else A = C;
            }
        }
    }
    A.template finish<false>(k, out, nullptr, nullptr, tw.a);
    if (tw.two) B.template finish<false>(k, out, nullptr, nullptr, tw.b);
}

// The caps leave both at ten blocks of 64 per SM: 96 registers of 104, in a batch 94 of 96 (96 of 104
// there cost six dam breaks of 5.0M particles 0.8% of their steps).
template <class P, int MODE, bool BATCH>
__global__ void __maxnreg__(BATCH ? 96 : 104)
k_pass2_twin(KParamsT<float> k, ParticleSet in, const unsigned* __restrict__ keys,
             const int* __restrict__ cs, NbrList nl, Pass1Out p1, float* __restrict__ rho_dt,
             float* __restrict__ vel_dt, ParticleSet out, unsigned* __restrict__ out_hash,
             unsigned* err, unsigned* disp) {
    DispBox box;
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * u < (BATCH ? k.positions : k.n) && (!BATCH || work_slot(nl, 2 * u) >= 0)) {
        const Twin tw = twin_of<BATCH>(nl, u, k.n);
        Pass2Acc<P, MODE> A, B;
        A.load(k, p1, tw.a, 0);
        B.load(k, p1, tw.b, 0);
        if (A.active || B.active) {
            const int cnt = __ldg(nl.count + u);
            if (cnt >= 0) {
                visit_twin(nl, p1.nrec, u, cnt, [&](const float4& aj, const float4& vj) {
                    pass2_twin<P, MODE>(k, A, B, aj, vj);
                });
            } else {
                const TwinCells w = twin_cells(k, keys, tw);
                if (w.near && A.active && B.active) {
                    walk_twin(k, cs, w, p1.nrec, [&](const float4& aj, const float4& vj) {
                        pass2_twin<P, MODE>(k, A, B, aj, vj);
                    });
                } else {
#pragma unroll 1
                    for (int m = 0; m < 2; m++) {
                        Pass2Acc<P, MODE> C = m ? B : A;
                        if (C.active)
                            walk_pairs<P, 2>(k, cs, keys, p1.nrec, m ? tw.b : tw.a, C.pi, k.kh2,
                                             [&](int j, unsigned, const float4&, float dx, float dy,
                                                 float dz, float r2) {
                                float4 aj, vj;
                                ld_rec(p1.nrec, j, aj, vj);
                                C.pair(k, p1, j, aj, vj, dx, dy, dz, r2, 0.f);
                            });
                        if (m) B = C;
                        else A = C;
                    }
                }
            }
        }
#pragma unroll 1
        for (int m = 0; m < (tw.two ? 2 : 1); m++) {
            const Pass2Acc<P, MODE> C = m ? B : A;
            pass2_finish<P, MODE>(k, m ? tw.b : tw.a, C, in, keys, nl, rho_dt, vel_dt, 0, out,
                                  out_hash, err, box, disp);
        }
    }
    if (MODE == MODE_RATES || disp == nullptr) return;
    // the block's displacement box; blockDim is a multiple of 32, every thread gets here
    __shared__ unsigned s_box[6 * (NS_MAX_THREADS / 32)];
    reduce_disp_box(box, disp, s_box);
}

inline int twin_blocks(int positions, int threads) {
    return (positions + 2 * threads - 1) / (2 * threads);
}

}  // namespace

template <class P>
cudaError_t launch_nbr_build_twin(const KParams& k, const ParticleSet& in, const unsigned* keys,
                                  const int* cs, const NbrList& nl, float4* nrec, unsigned* err,
                                  cudaStream_t s, const unsigned* gate) {
    if (k.n <= 0) return cudaSuccess;
    const int blocks = twin_blocks(k.positions, TWIN_BUILD_THREADS);
    if (k.inst_cells)
        k_nbr_build_twin<P, true><<<blocks, TWIN_BUILD_THREADS, 0, s>>>(k, in.xyz, keys, cs, nl,
                                                                         in.rec, nrec, err, gate);
    else
        k_nbr_build_twin<P, false><<<blocks, TWIN_BUILD_THREADS, 0, s>>>(k, in.xyz, keys, cs, nl,
                                                                          in.rec, nrec, err, gate);
    return cudaGetLastError();
}

template <class P>
cudaError_t launch_pass1_twin(const KParams& k, const ParticleSet& in, const unsigned* keys,
                              const int* cs, const NbrList& nl, const Pass1Out& out,
                              cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    const int blocks = twin_blocks(k.positions, k.threads);
    if (k.inst_cells)
        k_pass1_twin<P, true><<<blocks, k.threads, 0, s>>>(k, in, keys, cs, nl, out);
    else
        k_pass1_twin<P, false><<<blocks, k.threads, 0, s>>>(k, in, keys, cs, nl, out);
    return cudaGetLastError();
}

template <class P>
cudaError_t launch_pass2_twin(const KParams& k, HalfStep half, const ParticleSet& in,
                              const unsigned* keys, const int* cs, const NbrList& nl,
                              const Pass1Out& p1, ParticleSet out, unsigned* out_hash,
                              unsigned* err, unsigned* disp, cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    const int blocks = twin_blocks(k.positions, k.threads);
    auto launch = [&](auto mode, auto batch) {
        k_pass2_twin<P, decltype(mode)::value, decltype(batch)::value>
            <<<blocks, k.threads, 0, s>>>(k, in, keys, cs, nl, p1, nullptr, nullptr, out, out_hash,
                                          err, disp);
    };
    auto either = [&](auto mode) {
        if (k.inst_cells) launch(mode, std::true_type{});
        else launch(mode, std::false_type{});
    };
    if (half == HALF_PREDICT) either(std::integral_constant<int, MODE_PRED>{});
    else either(std::integral_constant<int, MODE_CORR>{});
    return cudaGetLastError();
}

cudaError_t launch_pass2_rates_twin(const KParams& k, const ParticleSet& in, const unsigned* keys,
                                    const int* cs, const NbrList& nl, const Pass1Out& p1,
                                    float* rho_dt, float* vel_dt, cudaStream_t s) {
    if (k.n <= 0) return cudaSuccess;
    k_pass2_twin<PrecF32, MODE_RATES, false><<<twin_blocks(k.positions, k.threads), k.threads, 0, s>>>(
        k, in, keys, cs, nl, p1, rho_dt, vel_dt, ParticleSet{}, nullptr, nullptr, nullptr);
    return cudaGetLastError();
}

#define SPH_NS_TWIN_INSTANTIATE(P)                                                             \
    template cudaError_t launch_nbr_build_twin<P>(const KParams&, const ParticleSet&,          \
                                                  const unsigned*, const int*, const NbrList&, \
                                                  float4*, unsigned*, cudaStream_t,            \
                                                  const unsigned*);                            \
    template cudaError_t launch_pass1_twin<P>(const KParams&, const ParticleSet&,              \
                                              const unsigned*, const int*, const NbrList&,     \
                                              const Pass1Out&, cudaStream_t);                  \
    template cudaError_t launch_pass2_twin<P>(const KParams&, HalfStep, const ParticleSet&,    \
                                              const unsigned*, const int*, const NbrList&,     \
                                              const Pass1Out&, ParticleSet, unsigned*,         \
                                              unsigned*, unsigned*, cudaStream_t);
SPH_NS_TWIN_INSTANTIATE(PrecF32)
SPH_NS_TWIN_INSTANTIATE(PrecMixA)
#undef SPH_NS_TWIN_INSTANTIATE

}  // namespace sph
