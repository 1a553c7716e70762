// Region form of a pass: one cooperative launch runs every time step of a
// forward or backward pass, one block per region of the padded grid.
//
// What bounds it.  A step of one launch per time step is a chain of
// latencies (launch gap, tile copies, L2 reads of level n-1 and c2, the
// slowest tile) around little work.  Here the wavefield levels, c2 and the
// C-PML memory variables of a region stay in the shared memory of the block
// that owns it for the whole pass; a step reads no global memory but the
// snapshot (backward), image and injection values, and regions exchange only
// the 3-cell rings of level n+1.
//
// Exchange.  Every edge position of a region is one 16-byte packet: the 3
// cells next to the edge and the step's tag, written with one 128-bit
// relaxed store and polled with 128-bit relaxed loads.  A packet is its own
// flag (the accesses are single-copy atomic), so a step waits for one store
// and one load through L2 (500 cycles one way on a die, 800-900 across the
// two), with no fence and no separate flag.  Packets alternate between two
// planes by step parity; a region overwrites a plane only two steps later,
// which it cannot reach before every neighbour has read the plane, since it
// needs that neighbour's next packets first.  Waits are bounded.  A step
// updates the cells that need no ring while the packets are on their way.
//
// Regions.  Interior, C-PML strips (the full strip thickness, cut along the
// strip) and corners are cut separately, so that a block runs one kind of
// update and phi's strip-local stencils never cross a region.  Shared arrays
// are (fast, slow): the fast axis is z, and x in the z-strips, so that both
// kinds of strip run the same float4 update with the slow axis across the
// strip.  The planner bisects the largest region cost over the cuts of each
// part with at most one region per multiprocessor.
//
// Measured on the B200 (a shot, against one launch per step): 1200 x 1136
// window, 8000 steps 89.0 ms against 164.5 (forward step 10.4 -> 5.0 us,
// backward 9.4 -> 6.1); 200 x 249, 3000 steps 13.0 against 53.4; 331 x 321
// with C-PML on all sides, 1501 steps 6.4 against 39.9; 36 x 64, 260 steps
// 1.22 against 4.51.  12 warps of up to 168 registers: 16 warps spill the
// column loops (model of the first window 24.3 against 19.5 ms), and two
// blocks a multiprocessor halve a region's cells but double its packets
// (first window 125 ms).
//
// The arithmetic of every cell is the step kernels' in their order, so the
// results are the same bit for bit; the pass starts from and leaves the same
// global state as the launches it replaces.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>
#include <vector>

#include "rtm_device.cuh"
#include "rtm_internal.h"

namespace psdm {
namespace {

constexpr int kT = kRegThreads;

// Packet of 3 cells and the step's tag, in one access.
__device__ __forceinline__ void st_packet(uint4* p, float a, float b, float c, unsigned int tag) {
    asm volatile(
        "{\n .reg .b128 t;\n .reg .b64 lo, hi;\n mov.b64 lo, {%1, %2};\n mov.b64 hi, {%3, %4};\n"
        " mov.b128 t, {lo, hi};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
        "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(tag)
        : "memory");
}
__device__ __forceinline__ uint4 ld_packet(const uint4* p) {
    uint4 v;
    asm volatile(
        "{\n .reg .b128 t;\n .reg .b64 lo, hi;\n ld.relaxed.gpu.global.b128 t, [%4];\n"
        " mov.b128 {lo, hi}, t;\n mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}
// Polls a packet until its tag is `tag`; gives up after ~2 s, which it tells
// the other blocks, or when another block has given up.
__device__ __forceinline__ bool wait_packet(const uint4* p, unsigned int tag, int* abort, uint4& v) {
    v = ld_packet(p);
    if (v.w == tag) return true;
    uint64_t t0 = 0;
    for (int it = 1;; ++it) {
        v = ld_packet(p);
        if (v.w == tag) return true;
        if ((it & 63) == 0) {
            const uint64_t t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (ld_relaxed(abort) != 0) return false;
            if (t - t0 > 2000000000ull) {
                atomicExch(abort, 1);
                return false;
            }
        }
    }
}

// Packed arithmetic of the updates.  A product is an FMA with -0 added
// (read from the launch's arguments, so that it stays one): a packed multiply
// may be fused into a following packed add, and an FMA cannot, so the sums of
// products may be packed too.  A difference is an FMA with -1.  Both round as
// the multiply and the subtraction do, signs of zeros included.
struct Consts {
    float2 c[4];   // second-derivative taps
    float2 n0, m1; // -0, -1
};
__device__ __forceinline__ float2 mul_p(const Consts& k, const float2& x, const float2& c) {
    return __ffma2_rn(x, c, k.n0);
}
__device__ __forceinline__ float2 sub_p(const Consts& k, const float2& x, const float2& y) {
    return __ffma2_rn(y, k.m1, x);
}
__device__ __forceinline__ float2 sum4p(const Consts& k, const float2& t0, const float2& t1, const float2& t2,
                                        const float2& t3) {
    return __fadd2_rn(__fadd2_rn(__fadd2_rn(mul_p(k, t0, k.c[0]), mul_p(k, t1, k.c[1])), mul_p(k, t2, k.c[2])),
                      mul_p(k, t3, k.c[3]));
}
__device__ __forceinline__ float2 dbl(const float2& x) { return __fadd2_rn(x, x); }

// Second derivatives of the rows of one float4 c along the fast axis, zm and
// zp the float4s before and after it.  Tap sums of pairs that start on an odd
// row are scalar: building the pairs would cost more.
__device__ __forceinline__ void fast_deriv2(const Consts& k, const float4& zm, const float4& c, const float4& zp,
                                            float2& a, float2& b) {
    const float2 a1 = make_float2(__fadd_rn(c.y, zm.w), __fadd_rn(c.z, c.x));
    const float2 b1 = make_float2(__fadd_rn(c.w, c.y), __fadd_rn(zp.x, c.z));
    const float2 a3 = make_float2(__fadd_rn(c.w, zm.y), __fadd_rn(zp.x, zm.z));
    const float2 b3 = make_float2(__fadd_rn(zp.y, zm.w), __fadd_rn(zp.z, c.x));
    a = sum4p(k, dbl(lo2(c)), a1, __fadd2_rn(hi2(c), hi2(zm)), a3);
    b = sum4p(k, dbl(hi2(c)), b1, __fadd2_rn(lo2(zp), lo2(c)), b3);
}

// (p3 - p1) * 0.5 / dt of one float4, correctly rounded as div_dt does.  The
// halved differences are scaled by -2^64, so that the reciprocal with its FMA
// correction (q1) is exact for every nonzero one, and the quotients scaled
// back with one rounding.  The residual is taken with its sign turned (q0 dt
// - x), so that the correction of a zero is -0 and the zero keeps its sign (a
// halved difference of the smallest subnormal rounds to one).  A quotient half
// way between two subnormals (diff = half a step) takes the sign of q1's exact
// residual; an overflow of the scaled form (diff is NaN) takes div_dt.  Testing
// for small differences (below 2^-90) instead sent a band of about 20 cells
// ahead of the wavefront through div_dt, and that set the pace of the whole
// pass.
__device__ __forceinline__ float4 snapshot4(const StepArgs& a, const Consts& kc, const float4& out, const float4& pm) {
    const float2 half = make_float2(0.5f, 0.5f), nup = make_float2(-0x1p64f, -0x1p64f),
                 dn = make_float2(0x1p-64f, 0x1p-64f);
    const float2 nr = make_float2(-a.inv_dt, -a.inv_dt), dt = make_float2(a.dt, a.dt);
    float2 h[2], q[2], q1[2], nx[2], diff[2];
    h[0] = __fmul2_rn(sub_p(kc, lo2(out), lo2(pm)), half);
    h[1] = __fmul2_rn(sub_p(kc, hi2(out), hi2(pm)), half);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        nx[k] = __fmul2_rn(h[k], nup);
        const float2 q0 = __fmul2_rn(nx[k], nr);
        const float2 e = __ffma2_rn(q0, dt, nx[k]);
        q1[k] = __ffma2_rn(e, nr, q0);
        q[k] = __fmul2_rn(q1[k], dn);
        diff[k] = __ffma2_rn(q[k], nup, q1[k]);  // exact
    }
    const float tie = 0x1p-86f;  // half a subnormal step
    const bool rare = !(fabsf(diff[0].x) < tie && fabsf(diff[0].y) < tie && fabsf(diff[1].x) < tie &&
                        fabsf(diff[1].y) < tie);
    if (rare || !a.fast_div) {
        const float d[4] = {diff[0].x, diff[0].y, diff[1].x, diff[1].y};
        if (!a.fast_div || !(d[0] == d[0] && d[1] == d[1] && d[2] == d[2] && d[3] == d[3]))
            return make_float4(div_dt(a, h[0].x), div_dt(a, h[0].y), div_dt(a, h[1].x), div_dt(a, h[1].y));
        float v[4] = {q[0].x, q[0].y, q[1].x, q[1].y};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float2 e = __ffma2_rn(q1[k], dt, nx[k]);  // sign of (q1 - true)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float ej = j == 0 ? e.x : e.y, dj = d[2 * k + j];
                if (fabsf(dj) == tie && ej != 0.f && signbit(ej) != signbit(dj))
                    v[2 * k + j] = __fadd_rn(v[2 * k + j], copysignf(0x1p-149f, dj));
            }
        }
        return make_float4(v[0], v[1], v[2], v[3]);
    }
    return make_float4(q[0].x, q[0].y, q[1].x, q[1].y);
}

// New level of one float4 of interior rows: win = the 7 x-neighbour columns
// (centre win[3]), zm / zp = the float4s above and below, pm = level n-1.
// SRC: an injected source is added to the sum of the second derivatives, as
// the generic cell does; quads without one add zeros, which changes no
// result (the sum's sign of zero is lost in the last add, whose other term is
// never -0).
template <bool SRC>
__device__ __forceinline__ float4 interior_update(const Consts& k, const float4 (&win)[7], const float4& zm,
                                                  const float4& zp, const float4& pm, const float4& c2,
                                                  const float4& src) {
    const float4& c = win[3];
    float2 dz[2], o[2];
    fast_deriv2(k, zm, c, zp, dz[0], dz[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#define XR(j) (h == 0 ? lo2(win[3 + (j)]) : hi2(win[3 + (j)]))
        const float2 dx = sum4p(k, dbl(XR(0)), __fadd2_rn(XR(1), XR(-1)), __fadd2_rn(XR(2), XR(-2)),
                                __fadd2_rn(XR(3), XR(-3)));
        float2 lap = __fadd2_rn(dx, dz[h]);
        if (SRC) lap = __fadd2_rn(lap, h == 0 ? lo2(src) : hi2(src));
        const float2 base = sub_p(k, dbl(XR(0)), h == 0 ? lo2(pm) : hi2(pm));
        o[h] = __fadd2_rn(base, mul_p(k, h == 0 ? lo2(c2) : hi2(c2), lap));
#undef XR
    }
    return make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
}

// The imaging update of one float4 (emit4's arithmetic): the new image value.
__device__ __forceinline__ float4 image4(const StepArgs& a, const Consts& k, float w, const float4& out,
                                         const float4& pm, float4 F, const float4& img) {
    float2 f[2] = {lo2(F), hi2(F)}, r[2];
    const float2 half = make_float2(0.5f, 0.5f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (w != 1.f) f[h] = __fmul2_rn(f[h], make_float2(w, w));
        const float2 d = sub_p(k, h == 0 ? lo2(out) : hi2(out), h == 0 ? lo2(pm) : hi2(pm));
        float2 inc = mul_p(k, __fmul2_rn(half, d), f[h]);
        if (a.ss != 1.f) inc = mul_p(k, inc, make_float2(a.ss, a.ss));
        r[h] = __fadd2_rn(h == 0 ? lo2(img) : hi2(img), inc);
    }
    return make_float4(r[0].x, r[0].y, r[1].x, r[1].y);
}

extern __shared__ __align__(16) float g_smem[];

// Shared memory of a region's pass, as offsets into g_smem.  Every column of
// a region's arrays has the launch's pitch P, so that the column loops address
// their neighbours with constants.
struct RegSmem {
    // two levels, ns + 6 columns of P, the region's cell (f, s) at (s + 3) P + f + 4
    int np;                      // floats of a level; level 0 at offset 0
    int c2, nq;                  // (f, s) at s (P - 8) + f, as the arrays below; floats of such an array
    int phi, nphi, chi;          // strips and corners (corners: along the slow axis, phi with the slow ring)
    int psi, xsi;                // corners: phi and chi along the fast axis
    int img;                     // interior, backward: the image
    int src;                     // injected values of two steps, float4 of row quad slot k and column s at (k ns + s) 4
    int A, B;                    // C-PML factors by slow position (strips) or factor index (corners)
    int side, ns;                // free-surface histories by slow position, two levels
};

// What a block keeps in shared memory beside its arrays.
struct RegShared {
    RegBlock b;
    RegLoad ld;
    RegSmem m;
    RegVar v[2];  // values of this step and the next
    unsigned int amax;
    signed char slot[kRegMaxQuads];
};

// A region's packets: each thread keeps the descriptors of its first two each
// way.  The first one received is requested while the thread's last columns
// are updated, so that a packet that is there by then costs no round trip.
template <int P, bool PHI>
struct Mail {
    uint4* board;
    const RegPair* pub;
    const int* rcv;
    int npk, npub, nrcv, rcv_first;
    RegPair p0, p1;
    int r0, r1;
    uint4 v;
    bool asked;

    __device__ __forceinline__ void init(const RegBlock& b, const RegJob& job, int tid) {
        board = static_cast<uint4*>(job.board);
        npk = job.npk;
        npub = b.npub;
        nrcv = b.nrcv;
        rcv_first = b.rcv_first;
        pub = job.pub + b.pub0;
        rcv = job.rcv + b.rcv0;
        p0 = tid < npub ? pub[tid] : RegPair{0, 0};
        p1 = tid + kT < npub ? pub[tid + kT] : RegPair{0, 0};
        r0 = tid < nrcv ? rcv[tid] : 0;
        r1 = tid + kT < nrcv ? rcv[tid + kT] : 0;
        asked = false;
    }
    // plane of the packets published in the step of parity `par`
    __device__ __forceinline__ void request(int par, int tid, bool due) {
        asked = due && tid < nrcv;
        if (asked) v = ld_packet(board + par * npk + rcv_first + tid);
    }
    __device__ __forceinline__ bool take(float* lev, float* phi, int d, const uint4* at, unsigned int tag, int* abort,
                                         bool early) {
        uint4 w = v;
        bool ok = true;
        if (!early || w.w != tag) ok = wait_packet(at, tag, abort, w);
        float* to = (PHI && (d & kRegPhi)) ? phi : lev;
        const int off = d & kRegOffMask, st = (PHI && (d & kRegPhi)) ? P - 8 : ((d & kRegSlow) ? P : 1);
        to[off] = __uint_as_float(w.x);
        to[off + st] = __uint_as_float(w.y);
        to[off + 2 * st] = __uint_as_float(w.z);
        return ok;
    }
    __device__ __forceinline__ bool receive(float* lev, float* phi, int par, unsigned int tag, int* abort, int tid) {
        const uint4* at = board + par * npk + rcv_first;
        bool ok = true;
        if (tid < nrcv) ok = take(lev, phi, r0, at + tid, tag, abort, asked);
        if (tid + kT < nrcv) ok = take(lev, phi, r1, at + tid + kT, tag, abort, false) && ok;
        for (int j = tid + 2 * kT; j < nrcv; j += kT) ok = take(lev, phi, rcv[j], at + j, tag, abort, false) && ok;
        return ok;
    }
    __device__ __forceinline__ void put(const float* lev, const float* phi, const RegPair& d, uint4* plane,
                                        unsigned int tag) {
        const float* from = (PHI && (d.y & kRegPhi)) ? phi : lev;
        const int off = d.y & kRegOffMask, st = (PHI && (d.y & kRegPhi)) ? P - 8 : ((d.y & kRegSlow) ? P : 1);
        st_packet(plane + d.x, from[off], from[off + st], from[off + 2 * st], tag);
    }
    __device__ __forceinline__ void send(const float* lev, const float* phi, int par, unsigned int tag, int tid) {
        uint4* plane = board + par * npk;
        if (tid < npub) put(lev, phi, p0, plane, tag);
        if (tid + kT < npub) put(lev, phi, p1, plane, tag);
        for (int j = tid + 2 * kT; j < npub; j += kT) put(lev, phi, pub[j], plane, tag);
    }
};

// The next step's values, fetched at the start of a step and stored before its
// last barrier by the first threads.
constexpr int kVarWords = (int)(sizeof(RegVar) / 4);
__device__ __forceinline__ int fetch_var(const RegVar* var, int i, int tid) {
    return tid < kVarWords ? __ldg(reinterpret_cast<const int*>(var + i) + tid) : 0;
}
__device__ __forceinline__ void store_var(RegVar* v, int word, int tid) {
    if (tid < kVarWords) reinterpret_cast<int*>(v)[tid] = word;
}

// Receivers of a region at the start of a step (forward): level n is the
// previous step's p3.
template <int MODE>
__device__ __forceinline__ void gather(const RegParams& rp, const RegJob& job, const RegShared& sh, const float* lev,
                                       int nrec, int rec_t, int tid) {
    if constexpr (MODE == 0) {
        if (rec_t < 0) return;
        for (int j = tid; j < nrec; j += kT) {
            const RegPair r = rp.rec[sh.ld.rec0 + j];
            job.a.rec_out[(size_t)r.x * job.a.rec_ld + rec_t] = lev[r.y];
        }
    }
}

// Snapshot, image and compensation values of one float4, requested ahead.
struct Ahead {
    float4 F, I, C;
    uint2 R;
};
// A step's snapshot or imaging operands.
struct Emit {
    void* field;  // null: none this step
    void* aux;    // forward: largest magnitude or null; mode 2: inverse scale
    float w, isc;
    float* image;  // in global memory
    float* comp;
};
// IMG: the image is in shared memory.
template <int MODE, bool IMG>
__device__ __forceinline__ void load_ahead(const Emit& t, int fi, Ahead& h) {
    if (MODE == 1) {
        h.F = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(t.field) + fi));
        if (!IMG) h.I = *reinterpret_cast<const float4*>(t.image + fi);
    }
    if (MODE == 2) {
        h.R = load16x4_raw(t.field, fi);
        h.I = *reinterpret_cast<const float4*>(t.image + fi);
        h.C = *reinterpret_cast<const float4*>(t.comp + fi);
    }
}

// Image and compensation of one float4 with a 16-bit snapshot (emit4's order).
__device__ __forceinline__ void image16(const StepArgs& a, const Emit& t, int fi, const float4& out, const float4& pm,
                                        const Ahead& h) {
    const float4 F4 = unpack16x4(h.R, a.kind16, t.isc);
    float Iv[4] = {h.I.x, h.I.y, h.I.z, h.I.w}, Cv[4] = {h.C.x, h.C.y, h.C.z, h.C.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float F = comp(F4, e);
        if (t.w != 1.f) F = __fmul_rn(F, t.w);
        float inc = __fmul_rn(__fmul_rn(0.5f, __fsub_rn(comp(out, e), comp(pm, e))), F);
        if (a.ss != 1.f) inc = __fmul_rn(inc, a.ss);
        kahan(Iv[e], Cv[e], inc);
    }
    *reinterpret_cast<float4*>(t.image + fi) = make_float4(Iv[0], Iv[1], Iv[2], Iv[3]);
    *reinterpret_cast<float4*>(t.comp + fi) = make_float4(Cv[0], Cv[1], Cv[2], Cv[3]);
}

// Snapshot or imaging update of one float4 at offset fi (gi: in the shared
// image).  rows: valid rows of the quad.
template <int MODE, bool IMG>
__device__ __forceinline__ void emit_quad(const StepArgs& a, const Consts& kc, const Emit& t,
                                          const float4& out, const float4& pm, int rows, int fi, float4* gi,
                                          const Ahead& h, float& amax_t) {
    if (t.field == nullptr) return;
    if (MODE == 0) {
        float4 D = snapshot4(a, kc, out, pm);
        if (rows < 4) {  // rows past the interior: the pad rows stay zero
            if (rows < 2) D.y = 0.f;
            if (rows < 3) D.z = 0.f;
            D.w = 0.f;
        }
        *reinterpret_cast<float4*>(static_cast<float*>(t.field) + fi) = D;
        if (t.aux != nullptr)
            amax_t = fmaxf(amax_t, fmaxf(fmaxf(fabsf(D.x), fabsf(D.y)), fmaxf(fabsf(D.z), fabsf(D.w))));
    } else if (MODE == 1) {
        if (IMG)
            *gi = image4(a, kc, t.w, out, pm, h.F, *gi);
        else
            *reinterpret_cast<float4*>(t.image + fi) = image4(a, kc, t.w, out, pm, h.F, h.I);
    } else {
        image16(a, t, fi, out, pm, h);
    }
}

// The i-th boundary quad of a region: the row quads outside [qa, qb) over all
// columns, then the columns outside [sa, sb) of the others.
__device__ __forceinline__ void boundary_quad(const RegBlock& b, int i, int& q, int& s) {
    const int nqi = b.qb - b.qa, nband = b.nq - nqi, rows = nband * b.ns;
    if (i < rows) {
        s = i / nband;
        q = i - s * nband;
        if (q >= b.qa) q += nqi;
    } else {
        s = (i - rows) / nqi;
        q = b.qa + (i - rows) - s * nqi;
        if (s >= b.sa) s += b.sb - b.sa;
    }
}

// All steps of an interior region.  Inner cells (whose stencils do not touch
// the ring) are updated while the ring's packets are on their way: a thread
// slides down C columns of one row quad, or takes single quads where that is
// only one or two columns (C = 0).  Then the ring, the boundary quads,
// and the packets of the new level.  SPECIAL: the region holds injection
// points or the free surface.  Returns false when a wait gave up.
template <int MODE, bool IMG, bool SPECIAL, int P>
__device__ __forceinline__ bool run_interior(const RegParams& rp, const RegJob& job, RegShared& sh, const Consts& kc) {
    constexpr int P4 = P / 4, Q4 = (P - 8) / 4;
    constexpr int kAhead = MODE == 1 ? 2 : 1;  // columns of snapshot values in flight
    const StepArgs& a = rp.job[0].a;
    const RegBlock& b = sh.b;
    const int tid = threadIdx.x, nsteps = job.nsteps, np = sh.m.np, nslot = sh.ld.nslot, ninj = sh.ld.ninj,
              nrec = sh.ld.nrec, ldf = job.a.ldf, items = b.items, nbound = b.nbound, C = b.C, nqi = b.qb - b.qa;
    const float4* c24 = reinterpret_cast<const float4*>(g_smem + sh.m.c2);
    float4* img4 = reinterpret_cast<float4*>(g_smem + sh.m.img);
    float* src = g_smem + sh.m.src;
    const int nsrc = nslot * b.ns * 4;
    const bool zero_top = SPECIAL && b.fsrow;
    const float* trace = job.a.inj_trace;
    const int inj_ld = job.a.inj_ld;
    Emit em;
    em.image = job.a.image;
    em.comp = job.a.comp;
    em.isc = 1.f;
    Mail<P, false> mail;
    mail.init(b, job, tid);
    // this thread's first boundary quad
    int bq = 0, bs = 0;
    if (tid < nbound) boundary_quad(b, tid, bq, bs);
    for (int i = 0; i < nsteps; ++i) {
        const int cur = i & 1;
        const bool more = i + 1 < nsteps;
        const RegVar& v = sh.v[cur];
        const float4* pc = reinterpret_cast<const float4*>(g_smem + cur * np);
        float4* pn = reinterpret_cast<float4*>(g_smem + (cur ^ 1) * np);
        const int inj_n = ninj > 0 ? v.inj_next : -1;
        em.field = v.field;
        em.aux = v.aux;
        em.w = v.w;
        if (MODE == 2) em.isc = em.field != nullptr ? __ldg(static_cast<const float*>(em.aux)) : 1.f;
        const int vnext = more ? fetch_var(job.var, i + 1, tid) : 0;
        float inj_v = 0.f;
        if (SPECIAL && inj_n >= 0 && tid < ninj)
            inj_v = __ldg(trace + (size_t)rp.inj[sh.ld.inj0 + tid].y * inj_ld + inj_n);
        if (nrec > 0) gather<MODE>(rp, job, sh, g_smem + cur * np, nrec, v.rec_t, tid);
        if (MODE == 1 && v.next != nullptr) {
            // the next step's snapshot into L2, a 128-byte line a thread
            const int lines = (b.nq + 7) >> 3;
            for (int j = tid; j < lines * b.ns; j += kT) {
                const int s = j / lines;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const float*>(v.next) + b.f0 + s * ldf +
                                                              32 * (j - s * lines)));
            }
        }
        const float4* src4 = reinterpret_cast<const float4*>(src + cur * nsrc);
        float amax_t = 0.f;
        mail.asked = false;
        // one quad, all its operands from shared memory
        auto single = [&](int q, int s, const Ahead& h) {
            const float4* w = pc + s * P4 + 1 + q;
            float4* po = pn + (s + 3) * P4 + 1 + q;
            float4 win[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) win[k] = w[k * P4];
            const float4 pm = po[0];
            float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (SPECIAL && sh.slot[q] >= 0) sv = src4[sh.slot[q] * b.ns + s];
            float4 out =
                interior_update<SPECIAL>(kc, win, w[3 * P4 - 1], w[3 * P4 + 1], pm, c24[s * Q4 + q], sv);
            if (zero_top && q == 0) out.x = 0.f;
            emit_quad<MODE, IMG>(a, kc, em, out, pm, b.nf - 4 * q, b.f0 + s * ldf + 4 * q, img4 + s * Q4 + q, h,
                                 amax_t);
            po[0] = out;
        };
        // ---- inner cells
        for (int j = tid; C == 0 && j < items; j += kT) {
            const int col = j / nqi, q = b.qa + j - col * nqi, s = b.sa + col;
            if (j + kT >= items) mail.request(cur ^ 1, tid, i > 0);
            Ahead h;
            if (MODE != 0 && em.field != nullptr) load_ahead<MODE, IMG>(em, b.f0 + s * ldf + 4 * q, h);
            single(q, s, h);
        }
        for (int it = tid; C > 0 && it < items; it += kT) {
            const int ch = it / nqi, q = b.qa + it - ch * nqi, s0 = b.sa + ch * C, n = min(C, b.sb - s0);
            const float4* w = pc + s0 * P4 + 1 + q;
            float4* po = pn + (s0 + 3) * P4 + 1 + q;
            const float4* cp = c24 + s0 * Q4 + q;
            float4* gi = img4 + s0 * Q4 + q;
            const float4* sp = nullptr;
            if (SPECIAL && sh.slot[q] >= 0) sp = src4 + sh.slot[q] * b.ns + s0;
            int fi = b.f0 + s0 * ldf + 4 * q;
            const bool emit = MODE != 0 && em.field != nullptr;
            Ahead h0, h1;
            if (emit) {
                load_ahead<MODE, IMG>(em, fi, h0);
                if (kAhead > 1 && n > 1) load_ahead<MODE, IMG>(em, fi + ldf, h1);
            }
            const int ask = i > 0 && it + kT >= items ? max(n - 2, 0) : -1;
            float4 win[7];
#pragma unroll
            for (int k = 0; k < 6; ++k) win[k] = w[k * P4];
            float4 nw = w[6 * P4], nzm = w[3 * P4 - 1], nzp = w[3 * P4 + 1];
#pragma unroll 1
            for (int j0 = 0; j0 < n; j0 += 7) {
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    if (j0 + k >= n) break;
                    if (j0 + k == ask) mail.request(cur ^ 1, tid, true);
                    win[6] = nw;
                    const float4 zm = nzm, zp = nzp, pm = po[k * P4], c2 = cp[k * Q4];
                    // the next column's operands (past the last one: of the ring, unused)
                    nw = w[(k + 7) * P4];
                    nzm = w[(k + 4) * P4 - 1];
                    nzp = w[(k + 4) * P4 + 1];
                    const Ahead h = h0;
                    if (kAhead > 1) h0 = h1;
                    if (emit && j0 + k + kAhead < n)
                        load_ahead<MODE, IMG>(em, fi + kAhead * ldf, kAhead > 1 ? h1 : h0);
                    float4 out = interior_update<SPECIAL>(
                        kc, win, zm, zp, pm, c2, SPECIAL && sp != nullptr ? sp[j0 + k] : make_float4(0.f, 0.f, 0.f, 0.f));
                    if (zero_top && q == 0) out.x = 0.f;
                    emit_quad<MODE, IMG>(a, kc, em, out, pm, 4, fi, gi + k * Q4, h, amax_t);
                    po[k * P4] = out;
#pragma unroll
                    for (int x = 0; x < 6; ++x) win[x] = win[x + 1];
                    fi += ldf;
                }
                w += 7 * P4;
                po += 7 * P4;
                cp += 7 * Q4;
                gi += 7 * Q4;
            }
        }
        Ahead bh;
        if (MODE != 0 && em.field != nullptr && tid < nbound)
            load_ahead<MODE, IMG>(em, b.f0 + bs * ldf + 4 * bq, bh);
        // ---- the ring of level n
        bool ok = true;
        if (i > 0)
            ok = mail.receive(g_smem + cur * np, nullptr, cur ^ 1, rp.epoch + (unsigned int)i - 1u, rp.abort, tid);
        if (__syncthreads_or(!ok)) return false;
        // ---- boundary cells
        for (int j = tid; j < nbound; j += kT) {
            int q = bq, s = bs;
            if (j != tid) {
                boundary_quad(b, j, q, s);
                if (MODE != 0 && em.field != nullptr) load_ahead<MODE, IMG>(em, b.f0 + s * ldf + 4 * q, bh);
            }
            single(q, s, bh);
        }
        if (MODE == 0 && em.aux != nullptr) {
            const unsigned int w = __reduce_max_sync(0xffffffffu, __float_as_uint(amax_t));
            if ((tid & 31) == 0 && w != 0u) atomicMax(&sh.amax, w);
        }
        if (more) store_var(&sh.v[cur ^ 1], vnext, tid);
        if (SPECIAL && inj_n >= 0)
            for (int j = tid; j < ninj; j += kT) {
                const RegPair d = rp.inj[sh.ld.inj0 + j];
                src[(cur ^ 1) * nsrc + d.x] = j == tid ? inj_v : trace[(size_t)d.y * inj_ld + inj_n];
            }
        __syncthreads();
        if (MODE == 0 && tid == 0 && sh.amax != 0u) {
            atomicMax(static_cast<unsigned int*>(em.aux), sh.amax);
            sh.amax = 0u;
        }
        // ---- level n+1's edges to the neighbours
        if (more) mail.send(g_smem + (cur ^ 1) * np, nullptr, cur, rp.epoch + (unsigned int)i, tid);
    }
    return true;
}

// A strip's arrays and factors of one step, beside the levels.
struct StripStep {
    const float4* pc;
    float4* pn;
    const float4* c2;
    const float4* ph;  // phi at level n
    float4* pho;       // phi at level n+1
    float4* ch;
    const float* A;  // C-PML factors by slow position
    const float* B;
    const float* side;  // free-surface histories at level n (null: not this region), and n-1 -> n+1
    float* side_m;
};

// One float4 of a C-PML strip: the slow axis runs across the strip (kx or kz
// by slow position), the fast axis along it.  X: level n around the stencil
// centre, F: phi around the strip-local one (F[3] unused).
template <int P>
__device__ __forceinline__ void strip_update(const Consts& kc, const float2 (&k1)[4], const StripStep& u, int q, int s,
                                             const float4 (&X)[7], const float4 (&F)[7], const float4& c,
                                             const float4& zm, const float4& zp, const float4& phc) {
    constexpr int P4 = P / 4, Q4 = (P - 8) / 4;
    const bool hist = u.side != nullptr && q == 0;
    const int g = s * Q4 + q, gp = (s + 3) * P4 + 1 + q;
    const float4 pm = u.pn[gp], chc = u.ch[g], c2 = u.c2[g];
    const float2 A2 = make_float2(u.A[s], u.A[s]), B2 = make_float2(u.B[s], u.B[s]);
    auto deriv1 = [&](const float2& p1, const float2& m1, const float2& p2, const float2& m2, const float2& p3,
                      const float2& m3) {
        return __fadd2_rn(__fadd2_rn(mul_p(kc, sub_p(kc, p1, m1), k1[1]), mul_p(kc, sub_p(kc, p2, m2), k1[2])),
                          mul_p(kc, sub_p(kc, p3, m3), k1[3]));
    };
    float2 pp[2] = {lo2(c), hi2(c)}, pl[2] = {lo2(pm), hi2(pm)}, df[2];
    fast_deriv2(kc, zm, c, zp, df[0], df[1]);
    if (hist) {
        pp[0].x = u.side[s];
        pl[0].x = u.side_m[s];
    }
    float2 o[2], phn[2], chn[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#define XR(k) (h == 0 ? lo2(X[3 + (k)]) : hi2(X[3 + (k)]))
#define FR(k) (h == 0 ? lo2(F[3 + (k)]) : hi2(F[3 + (k)]))
        const float2 ds = sum4p(kc, dbl(XR(0)), __fadd2_rn(XR(1), XR(-1)), __fadd2_rn(XR(2), XR(-2)),
                                __fadd2_rn(XR(3), XR(-3)));
        const float2 d1 = deriv1(XR(1), XR(-1), XR(2), XR(-2), XR(3), XR(-3));
        const float2 dph = deriv1(FR(1), FR(-1), FR(2), FR(-2), FR(3), FR(-3));
#undef XR
#undef FR
        const float2 ph = h == 0 ? lo2(phc) : hi2(phc), ch = h == 0 ? lo2(chc) : hi2(chc),
                     cv = h == 0 ? lo2(c2) : hi2(c2);
        phn[h] = __fadd2_rn(mul_p(kc, A2, ph), mul_p(kc, B2, d1));
        chn[h] = __fadd2_rn(mul_p(kc, A2, ch), mul_p(kc, B2, __fadd2_rn(ds, dph)));
        const float2 prop = __fadd2_rn(dph, chn[h]);
        const float2 base = sub_p(kc, dbl(pp[h]), pl[h]);
        o[h] = __fadd2_rn(base, mul_p(kc, cv, __fadd2_rn(__fadd2_rn(ds, df[h]), prop)));
    }
    if (hist) {  // free-surface row: the private history keeps p3, the grid gets 0
        u.side_m[s] = o[0].x;
        o[0].x = 0.f;
    }
    u.pn[gp] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
    u.pho[g] = make_float4(phn[0].x, phn[0].y, phn[1].x, phn[1].y);
    u.ch[g] = make_float4(chn[0].x, chn[0].y, chn[1].x, chn[1].y);
}

// All steps of a C-PML strip region, in run_interior's phases.  Inner quads
// are those at slow positions whose stencil centres are not clamped.
template <int MODE, int P>
__device__ __forceinline__ bool run_strip(const RegParams& rp, const RegJob& job, RegShared& sh, const Consts& kc) {
    constexpr int P4 = P / 4, Q4 = (P - 8) / 4;
    const StepArgs& a = rp.job[0].a;
    const RegBlock& b = sh.b;
    const int tid = threadIdx.x, nsteps = job.nsteps, np = sh.m.np, nq = sh.m.nq, ns = b.ns, nrec = sh.ld.nrec,
              items = b.items, nbound = b.nbound, C = b.C, nqi = b.qb - b.qa;
    const bool hist = b.fsrow && !a.disk;
    float2 k1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) k1[k] = make_float2(a.cf1[k], a.cf1[k]);
    StripStep u;
    u.c2 = reinterpret_cast<const float4*>(g_smem + sh.m.c2);
    u.ch = reinterpret_cast<float4*>(g_smem + sh.m.chi);
    u.A = g_smem + sh.m.A;
    u.B = g_smem + sh.m.B;
    Mail<P, false> mail;
    mail.init(b, job, tid);
    int bq = 0, bs = 0;
    if (tid < nbound) boundary_quad(b, tid, bq, bs);
    for (int i = 0; i < nsteps; ++i) {
        const int cur = i & 1;
        const bool more = i + 1 < nsteps;
        u.pc = reinterpret_cast<const float4*>(g_smem + cur * np);
        u.pn = reinterpret_cast<float4*>(g_smem + (cur ^ 1) * np);
        u.ph = reinterpret_cast<const float4*>(g_smem + sh.m.phi + cur * nq);
        u.pho = reinterpret_cast<float4*>(g_smem + sh.m.phi + (cur ^ 1) * nq);
        u.side = hist ? g_smem + sh.m.side + cur * ns : nullptr;
        u.side_m = g_smem + sh.m.side + (cur ^ 1) * ns;
        const int vnext = more && nrec > 0 ? fetch_var(job.var, i + 1, tid) : 0;
        if (nrec > 0) gather<MODE>(rp, job, sh, g_smem + cur * np, nrec, sh.v[cur].rec_t, tid);
        mail.asked = false;
        // any quad: stencil centres clamped at the grid's edge (p) and at both edges of the strip (phi)
        auto single = [&](int q, int s) {
            const int cp = b.low ? max(s, 3) : min(s, ns - 4), cf = clampi(s, 3, ns - 4);
            const float4* w = u.pc + cp * P4 + 1 + q;
            const float4* f = u.ph + (cf - 3) * Q4 + q;
            float4 X[7], F[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                X[k] = w[k * P4];
                F[k] = k == 3 ? make_float4(0.f, 0.f, 0.f, 0.f) : f[k * Q4];
            }
            const float4* zc = u.pc + (s + 3) * P4 + 1 + q;
            strip_update<P>(kc, k1, u, q, s, X, F, zc[0], zc[-1], zc[1], u.ph[s * Q4 + q]);
        };
        // ---- inner quads: a thread slides both stencils across C positions of one quad, or takes single quads
        for (int j = tid; C == 0 && j < items; j += kT) {
            const int s = j / nqi;
            if (j + kT >= items) mail.request(cur ^ 1, tid, i > 0);
            single(b.qa + j - s * nqi, b.sa + s);
        }
        for (int it = tid; C > 0 && it < items; it += kT) {
            const int ch = it / nqi, q = b.qa + it - ch * nqi, s0 = b.sa + ch * C, n = min(C, b.sb - s0);
            const float4* w = u.pc + s0 * P4 + 1 + q;
            const float4* f = u.ph + (s0 - 3) * Q4 + q;
            float4 X[7], F[7];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                X[k] = w[k * P4];
                F[k] = f[k * Q4];
            }
            const int ask = i > 0 && it + kT >= items ? n - 1 : -1;
#pragma unroll 1
            for (int j0 = 0; j0 < n; j0 += 7) {
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    if (j0 + k >= n) break;
                    if (j0 + k == ask) mail.request(cur ^ 1, tid, true);
                    X[6] = w[(k + 6) * P4];
                    F[6] = f[(k + 6) * Q4];
                    strip_update<P>(kc, k1, u, q, s0 + j0 + k, X, F, X[3], w[(k + 3) * P4 - 1], w[(k + 3) * P4 + 1],
                                    F[3]);
#pragma unroll
                    for (int x = 0; x < 6; ++x) {
                        X[x] = X[x + 1];
                        F[x] = F[x + 1];
                    }
                }
                w += 7 * P4;
                f += 7 * Q4;
            }
        }
        // ---- the ring of level n
        bool ok = true;
        if (i > 0)
            ok = mail.receive(g_smem + cur * np, nullptr, cur ^ 1, rp.epoch + (unsigned int)i - 1u, rp.abort, tid);
        if (__syncthreads_or(!ok)) return false;
        // ---- boundary quads
        for (int j = tid; j < nbound; j += kT) {
            int q = bq, s = bs;
            if (j != tid) boundary_quad(b, j, q, s);
            single(q, s);
        }
        if (more && nrec > 0) store_var(&sh.v[cur ^ 1], vnext, tid);
        __syncthreads();
        // ---- level n+1's edges to the neighbours
        if (more) mail.send(g_smem + (cur ^ 1) * np, nullptr, cur, rp.epoch + (unsigned int)i, tid);
    }
    return true;
}

// A corner region's arrays in one step: columns [so, so + ns) of the dn x dn
// corner, fast axis z.
struct CornerStep {
    int dn, so;
    bool low, lowf;
    const float* pc;
    float* pn;
    const float* phx;  // phi along the slow axis, with the slow ring, levels n and n+1
    float* phxo;
    float* chx;
    const float* phz;
    float* phzo;
    float* chz;
    const float* c2;
    const float* A;  // by factor index
    const float* B;
};

template <int P>
__device__ __forceinline__ void corner_cell(const StepArgs& a, const CornerStep& u, int f, int s) {
    constexpr int Q = P - 8;
    const int dn = u.dn, so = u.so;
    const float* c1 = a.cf1;
    const float* c2 = a.cf2;
    const int sg = s + so;  // column of the corner
    const int cs = (u.low ? max(sg, 3) : min(sg, dn - 4)) - so;
    const int cz = u.lowf ? max(f, 3) : min(f, dn - 4);
    const float* colx = u.pc + (cs + 3) * P + f + 4;
    const float* colz = u.pc + (s + 3) * P + cz + 4;
    const int k = max(u.low ? dn - sg : sg + 1, u.lowf ? dn - f : f + 1);  // factor index max(kx, kz)
    const int g = s * Q + f, gx = g + 3 * Q, gp = (s + 3) * P + f + 4;
    const float* px = u.phx + (clampi(sg, 3, dn - 4) - so + 3) * Q + f;
    const float* pz = u.phz + s * Q + clampi(f, 3, dn - 4);
    const float A = u.A[k - 1], B = u.B[k - 1], c2v = u.c2[g], pl = u.pn[gp], p0 = u.pc[gp];
    const float ox = u.phx[gx], oz = u.phz[g], hx = u.chx[g], hz = u.chz[g];
#define AX(k) colx[(k) * P]
#define AZ(k) colz[(k)]
    const float d2x = D2(AX, c2), d2z = D2(AZ, c2);
    const float d1x = D1(AX, c1), d1z = D1(AZ, c1);
#undef AX
#undef AZ
#define PX(k) px[(k) * Q]
#define PZ(k) pz[(k)]
    const float dpx = D1(PX, c1), dpz = D1(PZ, c1);
#undef PX
#undef PZ
    const float cx = __fadd_rn(__fmul_rn(A, hx), __fmul_rn(B, __fadd_rn(d2x, dpx)));
    const float propx = __fadd_rn(dpx, cx);
    const float cz2 = __fadd_rn(__fmul_rn(A, hz), __fmul_rn(B, __fadd_rn(d2z, dpz)));
    const float propz = __fadd_rn(dpz, cz2);
    const float base = __fadd_rn(-pl, __fmul_rn(2.f, p0));
    const float p3 = __fadd_rn(base, __fmul_rn(c2v, __fadd_rn(__fadd_rn(d2x, d2z), propx)));
    u.phxo[gx] = __fadd_rn(__fmul_rn(A, ox), __fmul_rn(B, d1x));
    u.phzo[g] = __fadd_rn(__fmul_rn(A, oz), __fmul_rn(B, d1z));
    u.chx[g] = cx;
    u.chz[g] = cz2;
    u.pn[gp] = __fadd_rn(p3, __fmul_rn(c2v, propz));
}

// All steps of a corner region, in run_interior's phases, one cell an item.
template <int MODE, int P>
__device__ __forceinline__ bool run_corner(const RegParams& rp, const RegJob& job, RegShared& sh) {
    const StepArgs& a = rp.job[0].a;
    const RegBlock& b = sh.b;
    const int tid = threadIdx.x, nsteps = job.nsteps, np = sh.m.np, nq = sh.m.nq, nphi = sh.m.nphi, nrec = sh.ld.nrec,
              items = b.items, nbound = b.nbound, fa = b.fa, fn = b.fb - fa, sa = b.sa, sn = b.sb - sa;
    const int nband = b.nf - fn, rows = nband * b.ns;
    CornerStep u;
    u.dn = b.nf;
    u.so = b.soff;
    u.low = b.low != 0;
    u.lowf = b.lowf != 0;
    u.chx = g_smem + sh.m.chi;
    u.chz = g_smem + sh.m.xsi;
    u.c2 = g_smem + sh.m.c2;
    u.A = g_smem + sh.m.A;
    u.B = g_smem + sh.m.B;
    Mail<P, true> mail;
    mail.init(b, job, tid);
    for (int i = 0; i < nsteps; ++i) {
        const int cur = i & 1;
        const bool more = i + 1 < nsteps;
        u.pc = g_smem + cur * np;
        u.pn = g_smem + (cur ^ 1) * np;
        u.phx = g_smem + sh.m.phi + cur * nphi;
        u.phxo = g_smem + sh.m.phi + (cur ^ 1) * nphi;
        u.phz = g_smem + sh.m.psi + cur * nq;
        u.phzo = g_smem + sh.m.psi + (cur ^ 1) * nq;
        const int vnext = more && nrec > 0 ? fetch_var(job.var, i + 1, tid) : 0;
        if (nrec > 0) gather<MODE>(rp, job, sh, u.pc, nrec, sh.v[cur].rec_t, tid);
        mail.asked = false;
#pragma unroll 1
        for (int j = tid; j < items; j += kT) {
            const int s = j / fn;
            if (j + kT >= items) mail.request(cur ^ 1, tid, i > 0);
            corner_cell<P>(a, u, fa + j - s * fn, sa + s);
        }
        bool ok = true;
        if (i > 0)
            ok = mail.receive(g_smem + cur * np, g_smem + sh.m.phi + cur * nphi, cur ^ 1,
                              rp.epoch + (unsigned int)i - 1u, rp.abort, tid);
        if (__syncthreads_or(!ok)) return false;
        // rows outside [fa, fb) of every column, then the other rows of the columns outside [sa, sb)
#pragma unroll 1
        for (int j = tid; j < nbound; j += kT) {
            int f, s;
            if (j < rows) {
                s = j / nband;
                f = j - s * nband;
                if (f >= fa) f += fn;
            } else {
                s = (j - rows) / fn;
                f = fa + (j - rows) - s * fn;
                if (s >= sa) s += sn;
            }
            corner_cell<P>(a, u, f, s);
        }
        if (more && nrec > 0) store_var(&sh.v[cur ^ 1], vnext, tid);
        __syncthreads();
        if (more) mail.send(u.pn, u.phxo, cur, rp.epoch + (unsigned int)i, tid);
    }
    return true;
}

// fn(f, s) over the fast range [fa, fb) and slow range [sa, sb), f fastest.
template <class F>
__device__ __forceinline__ void for_cells(int fa, int fb, int sa, int sb, const F& fn) {
    const int n = fb - fa, total = n * (sb - sa);
    for (int i = threadIdx.x; i < total; i += kT) {
        const int s = i / n;
        fn(fa + i - s * n, sa + s);
    }
}

// The pass of one region a block.  IMG: the image stays in shared memory
// (MODE 1).  P: pitch of the shared columns.
template <int MODE, bool IMG, int P>
__global__ void __launch_bounds__(kT, 1) region_kernel(const __grid_constant__ RegParams rp) {
    constexpr int Q = P - 8;
    __shared__ __align__(16) RegShared sh;
    const int tid = threadIdx.x;
    for (int w = tid; w < (int)(sizeof(RegLoad) / 4); w += kT)
        reinterpret_cast<int*>(&sh.ld)[w] = reinterpret_cast<const int*>(rp.loads + blockIdx.x)[w];
    if (tid == 0) sh.amax = 0u;
    __syncthreads();
    // The constants of the arithmetic (a) are those of every job; the job's
    // own pointers and sizes are ja's.
    const StepArgs& a = rp.job[0].a;
    const RegJob& job = rp.job[sh.ld.job];
    if (job.nsteps <= 0) return;
    for (int w = tid; w < (int)(sizeof(RegBlock) / 4); w += kT)
        reinterpret_cast<int*>(&sh.b)[w] = reinterpret_cast<const int*>(job.blocks + sh.ld.region)[w];
    __syncthreads();
    const StepArgs& ja = job.a;
    const RegBlock& b = sh.b;
    RegSmem& m = sh.m;
    store_var(&sh.v[0], fetch_var(job.var, 0, tid), tid);
    for (int q = tid; q < b.nq; q += kT) sh.slot[q] = rp.slots[sh.ld.slot0 + q];
    const int nf = b.nf, ns = b.ns, type = b.type;
    const bool strip = type == kRegStrip, corner = type == kRegCorner;
    const bool alongx = corner || !b.fastx;  // the slow axis of phi is x
    if (tid == 0) {
        int o = 0;
        auto take = [&o](int n) {
            const int at = o;
            o += n;
            return at;
        };
        m.np = P * (ns + 6);
        m.nq = Q * ns;
        m.nphi = Q * (corner ? ns + 6 : ns);
        m.ns = ns;
        take(2 * m.np);
        m.c2 = take(m.nq);
        m.phi = take(strip || corner ? 2 * m.nphi : 0);
        m.chi = take(strip || corner ? m.nq : 0);
        m.psi = take(corner ? 2 * m.nq : 0);
        m.xsi = take(corner ? m.nq : 0);
        m.img = take(type == kRegInterior && IMG ? m.nq : 0);
        const int nfac = strip ? ns : (corner ? nf : 0);
        m.A = take(nfac);
        m.B = take(nfac);
        m.side = take(strip ? 2 * ns : 0);
        m.src = (o + 3) & ~3;
    }
    __syncthreads();
    // Global state of the first step.  Levels with their rings (0 outside the
    // grid); rows above a free surface are part of the ring and stay zero.
    {
        const long long gf = b.fastx ? ja.ldz : 1, gs = b.fastx ? 1 : ja.ldz;
        const long long g0 = (long long)b.x0 * ja.ldz + b.z0;
        const int nfast = b.fastx ? ja.nxt : ja.ldz, nslow = b.fastx ? ja.ldz : ja.nxt;
        const int fo = b.fastx ? b.x0 : b.z0, so = b.fastx ? b.z0 : b.x0;
        for (int l = 0; l < 2; ++l) {
            const float* lv = l == 0 ? ja.p : ja.pm;
            float* to = g_smem + l * m.np;
            for_cells(-4, P - 4, -3, ns + 3, [&](int f, int s) {
                const bool in = f < nf + 4 && f + fo >= 0 && f + fo < nfast && s + so >= 0 && s + so < nslow;
                to[(s + 3) * P + f + 4] = in ? lv[g0 + f * gf + s * gs] : 0.f;
            });
        }
        float* z = g_smem + m.c2;  // zero the arrays without ring, pads included
        for (int i = tid; i < m.src - m.c2 + 2 * sh.ld.nslot * ns * 4; i += kT) z[i] = 0.f;
        __syncthreads();
        for_cells(0, nf, 0, ns, [&](int f, int s) {
            const long long g = g0 + f * gf + s * gs;
            const int i = s * Q + f;
            g_smem[m.c2 + i] = ja.c2[g];
            if (type == kRegInterior) {
                if (IMG) g_smem[m.img + i] = ja.image[b.f0 + (size_t)s * ja.ldf + f];
                return;
            }
            g_smem[m.chi + i] = (alongx ? ja.chix : ja.chiz)[g];
            if (strip) g_smem[m.phi + i] = (alongx ? ja.phix_in : ja.phiz_in)[g];
            if (corner) {
                g_smem[m.psi + i] = ja.phiz_in[g];
                g_smem[m.xsi + i] = ja.chiz[g];
            }
        });
        if (corner)  // with the ring that lies in the corner
            for_cells(0, nf, -3, ns + 3, [&](int f, int s) {
                if (s + b.soff >= 0 && s + b.soff < nf)
                    g_smem[m.phi + (s + 3) * Q + f] = ja.phix_in[(long long)(b.x0 + s) * ja.ldz + b.z0 + f];
            });
        if (type != kRegInterior)
            for (int s = tid; s < (strip ? ns : nf); s += kT) {
                const int k = corner ? s + 1 : (b.low ? ns - s : s + 1);
                g_smem[m.A + s] = ja.fA[k - 1];
                g_smem[m.B + s] = ja.fB[k - 1];
                if (strip && b.fsrow) {
                    g_smem[m.side + s] = ja.side_p[b.x0 + s];
                    g_smem[m.side + ns + s] = ja.side_pm[b.x0 + s];
                }
            }
        if (sh.v[0].inj_t >= 0)
            for (int j = tid; j < sh.ld.ninj; j += kT) {
                const RegPair d = rp.inj[sh.ld.inj0 + j];
                g_smem[m.src + d.x] = ja.inj_trace[(size_t)d.y * ja.inj_ld + sh.v[0].inj_t];
            }
    }
    __syncthreads();
    Consts kc;
#pragma unroll
    for (int k = 0; k < 4; ++k) kc.c[k] = make_float2(a.cf2[k], a.cf2[k]);
    kc.n0 = make_float2(rp.neg0, rp.neg0);
    kc.m1 = make_float2(-1.f, -1.f);
    bool ok;
    if (type == kRegInterior) {
        ok = sh.ld.nslot > 0 || b.fsrow ? run_interior<MODE, IMG, true, P>(rp, job, sh, kc)
                                        : run_interior<MODE, IMG, false, P>(rp, job, sh, kc);
    } else if (strip) {
        ok = run_strip<MODE, P>(rp, job, sh, kc);
    } else {
        ok = run_corner<MODE, P>(rp, job, sh);
    }
    if (!ok) {
        if (tid == 0) atomicCAS(a.err, 0, 3);
        return;
    }
    // The state as launches of one step leave it: the levels, phi of the last
    // level, chi, the histories and the image.
    const int last = job.nsteps & 1;
    const long long gf = b.fastx ? ja.ldz : 1, gs = b.fastx ? 1 : ja.ldz;
    const long long g0 = (long long)b.x0 * ja.ldz + b.z0;
    for_cells(0, nf, 0, ns, [&](int f, int s) {
        const long long g = g0 + f * gf + s * gs;
        const int i = s * Q + f, ip = (s + 3) * P + f + 4;
        const_cast<float*>(ja.p)[g] = g_smem[ip];
        ja.pm[g] = g_smem[m.np + ip];
        if (type == kRegInterior) {
            if (IMG) ja.image[b.f0 + (size_t)s * ja.ldf + f] = g_smem[m.img + i];
            return;
        }
        float* ph = alongx ? (last ? ja.phix_out : const_cast<float*>(ja.phix_in))
                           : (last ? ja.phiz_out : const_cast<float*>(ja.phiz_in));
        ph[g] = g_smem[m.phi + last * m.nphi + (corner ? i + 3 * Q : i)];
        (alongx ? ja.chix : ja.chiz)[g] = g_smem[m.chi + i];
        if (corner) {
            (last ? ja.phiz_out : const_cast<float*>(ja.phiz_in))[g] = g_smem[m.psi + last * m.nq + i];
            ja.chiz[g] = g_smem[m.xsi + i];
        }
    });
    if (b.fsrow && strip)
        for (int s = tid; s < ns; s += kT) {
            const_cast<float*>(ja.side_p)[b.x0 + s] = g_smem[m.side + s];
            ja.side_pm[b.x0 + s] = g_smem[m.side + ns + s];
        }
}

// ---- planner ----------------------------------------------------------------

struct Shape {
    int type, nf, ns;
};

int quads(int n) { return (n + 3) / 4; }

// Inner and boundary items of a region whose edges in `nb` (bit 0 low slow, 1
// high slow, 2 low fast, 3 high fast) have neighbours.
void item_shape(RegBlock* r, int nb) {
    r->nq = quads(r->nf);
    r->sa = (nb & 1) ? std::min(3, r->ns) : 0;
    r->sb = std::max(r->sa, r->ns - ((nb & 2) ? 3 : 0));
    r->fa = (nb & 4) ? std::min(3, r->nf) : 0;
    r->fb = std::max(r->fa, r->nf - ((nb & 8) ? 3 : 0));
    // whole row quads whose stencils end inside the region
    r->qa = (nb & 4) ? 1 : 0;
    r->qb = std::max(r->qa, (nb & 8) ? (r->nf - 3) / 4 : r->nq);
    if (r->type == kRegStrip) {  // the clamped positions at both edges of the strip are single quads
        r->sa = 3;
        r->sb = std::max(3, r->ns - 3);
    }
    r->C = 0;
    if (r->type == kRegCorner) {
        r->items = (r->fb - r->fa) * (r->sb - r->sa);
        r->nbound = r->nf * r->ns - r->items;
        return;
    }
    const int nqi = r->qb - r->qa, nsi = r->sb - r->sa;
    r->items = nqi * nsi;
    r->nbound = r->nq * r->ns - r->items;
    if (r->items > 0) {
        const int nch = std::max(1, std::min(nsi, kT / nqi));
        r->C = (nsi + nch - 1) / nch;
        // single quads where a column would be one or two long: a column's first quad costs 1050 cycles more than a
        // single one's (200 x 249 window, 3000 steps: 19.8 -> 15.0 ms, 331 x 321 9.6 -> 7.0)
        if (r->C <= 2)
            r->C = 0;
        else
            r->items = nqi * ((nsi + r->C - 1) / r->C);
    }
}

size_t region_floats(int P_, int type, int nf, int ns, int nslot, bool img) {
    const size_t P = P_, Q = P - 8;
    size_t n = 2 * P * (ns + 6) + Q * ns;
    if (type == kRegInterior && img) n += Q * ns;
    if (type == kRegStrip) n += 3 * Q * ns + 4 * (size_t)ns;
    if (type == kRegCorner) n += 2 * Q * (ns + 6) + 4 * Q * ns + 2 * (size_t)nf;
    return ((n + 3) & ~(size_t)3) + 2 * (size_t)nslot * ns * 4;
}

// Estimated cycles of a region's step: warp instructions over the four
// schedulers, at least the chain of its longest thread, in both phases, and
// its packets: the fixed round trip, a chain of one packet per kT, and a share
// per packet.  That share (7 cycles) was taken where the windows that are all
// latency stop gaining: 331 x 321 with C-PML on all sides 7.4, 7.0, 7.0 and
// 6.4 ms with 1.7, 2.5, 4 and 7; 200 x 249 15.0, 15.0, 12.8 and 12.9.
double region_cost(int type, int nf, int ns) {
    RegBlock r{};
    r.type = type;
    r.nf = nf;
    r.ns = ns;
    item_shape(&r, 15);
    // cycles measured on the B200: a warp's share of an item's issue and shared
    // memory time, the chain of the longest thread, and the phases' fixed parts
    auto phase = [](int items, double warp, double chain, double fixed) {
        return items > 0 ? std::max(std::ceil(items / 32.0) * warp, std::ceil(items / (double)kT) * chain) + fixed : 0.0;
    };
    const double pk = 2.0 * (nf + ns);  // packets each way
    const double mail = 700 + 300 * std::ceil(pk / kT) + 7.0 * pk;
    if (type == kRegCorner) return phase(r.items, 75, 860, 100) + phase(r.nbound, 60, 500, 500) + mail;
    if (type == kRegStrip)
        return (r.C > 0 ? phase(r.items, r.C * 85.0, r.C * 950.0, 550) : phase(r.items, 90, 900, 250)) +
               phase(r.nbound, 80, 800, 350) + mail;
    return (r.C > 0 ? phase(r.items, r.C * 52.0, r.C * 560.0, 1050) : phase(r.items, 70, 700, 250)) +
           phase(r.nbound, 70, 700, 250) + mail;
}

struct Part {  // a rectangle of the padded grid cut into a x b regions
    int type, fastx, low, lowf;
    int zr, x, h, w;  // device row, column, rows, columns
    int a = 1, b = 1; // cuts along the fast and slow axes
    int nfast() const { return fastx ? w : h; }
    int nslow() const { return fastx ? h : w; }
};

// Largest piece of n cells cut into k pieces of whole quads (fast) or cells.
int piece_fast(int n, int k) { return 4 * ((quads(n) + k - 1) / k); }
int piece_slow(int n, int k) { return (n + k - 1) / k; }

// Fewest regions of a part with cost <= target that fit in shared memory
// (img: with the image beside); sets its cuts.  0 if there are none.
int cut_part(Part* p, int P, double target, size_t max_floats, int budget, bool img) {
    const int nf = p->nfast(), ns = p->nslow();
    int best = 0;
    // interior: both ways; strips: along the strip; corners: in columns of at least
    // 7, so that the clamped stencils at the grid's edge (columns 0 to 6) and of phi at the corner's
    // inner edge lie in one region: those cells are updated before the ring arrives
    const int amax = p->type == kRegCorner ? 1 : std::max(1, std::min(quads(nf) / 2, budget));
    for (int ka = 1; ka <= amax; ++ka) {
        const int f = std::min(nf, piece_fast(nf, ka));
        if (f > P - 8) continue;
        const int bmax = p->type == kRegInterior ? std::max(1, std::min(ns / 3, budget / ka))
                                                 : (p->type == kRegCorner ? std::max(1, std::min(ns / 7, budget)) : 1);
        auto good = [&](int kb) {
            const int s = piece_slow(ns, kb);
            return region_floats(P, p->type, f, s, img ? 1 : 0, img) + 64 <= max_floats &&
                   region_cost(p->type, f, s) <= target;
        };
        int lo = 1, hi = bmax;
        if (best > 0) hi = std::min(hi, (best - 1) / ka);
        if (hi < 1 || !good(hi)) continue;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (good(mid)) hi = mid; else lo = mid + 1;
        }
        best = ka * lo;
        p->a = ka;
        p->b = lo;
    }
    return best;
}

// The parts of a padded grid; false if a region of it could be narrower than
// a packet.
bool grid_parts(const Grid& g, int fs, int max_regions, std::vector<Part>* out) {
    // packets carry 3 cells of one region, so every region is 3 cells wide;
    // strips are at least 8
    if (g.ny < 3 || g.nx < 3 || g.dn < 8 || max_regions < 1) return false;
    const int dn = g.dn, d0 = dn + g.zoff, zb = d0 + g.ny, xr = dn + g.nx;
    std::vector<Part>& parts = *out;
    parts.clear();
    parts.push_back({kRegInterior, 0, 0, 0, d0, dn, g.ny, g.nx});
    parts.push_back({kRegStrip, 0, 1, 0, d0, 0, g.ny, dn});
    parts.push_back({kRegStrip, 0, 0, 0, d0, xr, g.ny, dn});
    parts.push_back({kRegStrip, 1, 0, 0, zb, dn, dn, g.nx});
    parts.push_back({kRegCorner, 0, 1, 0, zb, 0, dn, dn});
    parts.push_back({kRegCorner, 0, 0, 0, zb, xr, dn, dn});
    if (!fs) {
        parts.push_back({kRegStrip, 1, 1, 0, g.zoff, dn, dn, g.nx});
        parts.push_back({kRegCorner, 0, 1, 1, g.zoff, 0, dn, dn});
        parts.push_back({kRegCorner, 0, 0, 1, g.zoff, xr, dn, dn});
    }
    return true;
}

// The cheapest largest region of the parts with columns of P; < 0 if they do
// not fit.
double cheapest_cut(std::vector<Part>& parts, int P, int max_regions, size_t max_floats, bool img) {
    auto total = [&](double target) {
        int n = 0;
        for (Part& p : parts) {
            const int k = cut_part(&p, P, target, max_floats, max_regions, img);
            if (k == 0) return 1 << 20;
            n += k;
        }
        return n;
    };
    double lo = 0, hi = 1e7;
    if (total(hi) > max_regions) return -1.0;
    for (int it = 0; it < 30 && hi - lo > 10; ++it) {
        const double mid = it < 8 ? std::sqrt(std::max(lo, 100.0) * hi) : 0.5 * (lo + hi);
        (total(mid) <= max_regions ? hi : lo) = mid;
    }
    return hi;
}

// A pass whose image stays in global memory, in units of one that keeps it in
// shared memory: regions that leave room for the image are taken unless they
// cost that much more.  Measured, a shot of 2000 steps whose cheapest regions
// have no room against those with: 1100 x 1200 27.0 -> 22.4 ms, 1200 x 1000
// 24.6 -> 20.6, 1300 x 1000 25.2 -> 22.1; the backward step alone is 25 %
// longer without (1200 x 1136).
constexpr double kImageOut = 1.12;

// The pitch and form of the cheapest cut; its cost (< 0: none fits).
double best_cut(std::vector<Part>& parts, int max_regions, size_t max_floats, int pitch, int* P_out, bool* img_out) {
    double best = -1.0, weighed = 0.0;
    for (int P : kRegPitches)
        for (bool img : {true, false}) {
            if (pitch != 0 && P != pitch) continue;
            const double c = cheapest_cut(parts, P, max_regions, max_floats, img), w = c * (img ? 1.0 : kImageOut);
            if (c >= 0 && (best < 0 || w < weighed)) {
                best = c;
                weighed = w;
                *P_out = P;
                *img_out = img;
            }
        }
    return best;
}

}  // namespace

double region_step_cost(const Grid& g, int fs, int max_regions, size_t max_floats, int* blocks) {
    std::vector<Part> parts;
    int P = 0;
    bool img = false;
    const double best = grid_parts(g, fs, max_regions, &parts)
                            ? best_cut(parts, max_regions, max_floats, 0, &P, &img) : -1.0;
    if (blocks != nullptr) {
        *blocks = 0;
        if (best >= 0)
            for (Part& p : parts) *blocks += cut_part(&p, P, best, max_floats, max_regions, img);
    }
    return best;
}

bool plan_regions(const Grid& g, int fs, int max_regions, size_t max_floats, RegPlan* plan, int pitch) {
    *plan = RegPlan{};
    std::vector<Part> parts;
    if (!grid_parts(g, fs, max_regions, &parts)) return false;
    const int dn = g.dn, d0 = dn + g.zoff;
    bool img = false;
    const double best = best_cut(parts, max_regions, max_floats, pitch, &plan->pitch, &img);
    if (best < 0) return false;
    for (Part& p : parts) cut_part(&p, plan->pitch, best, max_floats, max_regions, img);
    plan->cost = best;
    size_t most = 0;
    // The region of a cell: its part by the bands of rows and columns, and the
    // piece by the position in the part (a table of all cells took 7 of the 9 ms
    // of a plan of 1200 x 1136).
    struct Pieces {
        int first = 0;
        std::vector<short> fast, slow;
    };
    std::vector<Pieces> pieces(parts.size());
    int part_of[3][3] = {{-1, -1, -1}, {-1, -1, -1}, {-1, -1, -1}};
    auto band = [dn](int i, int n) { return i < dn ? 0 : i < dn + n ? 1 : 2; };
    for (size_t k = 0; k < parts.size(); ++k) {
        const Part& p = parts[k];
        const int nf = p.nfast(), ns = p.nslow(), nq = quads(nf);
        Pieces& pc = pieces[k];
        pc.first = (int)plan->blocks.size();
        pc.fast.resize(nf);
        pc.slow.resize(ns);
        part_of[band(p.zr - g.zoff, g.ny)][band(p.x, g.nx)] = (int)k;
        for (int ib = 0; ib < p.b; ++ib)
            for (int ia = 0; ia < p.a; ++ia) {
                const int q0 = (int)((long long)nq * ia / p.a), q1 = (int)((long long)nq * (ia + 1) / p.a);
                const int f0 = 4 * q0, f1 = std::min(4 * q1, nf);
                const int s0 = (int)((long long)ns * ib / p.b), s1 = (int)((long long)ns * (ib + 1) / p.b);
                if (f1 - f0 < 3 || s1 - s0 < 3) return false;
                RegBlock r{};
                r.type = p.type;
                r.fastx = p.fastx;
                r.low = p.low;
                r.lowf = p.lowf;
                r.z0 = p.zr + (p.fastx ? s0 : f0);
                r.x0 = p.x + (p.fastx ? f0 : s0);
                r.nf = f1 - f0;
                r.ns = s1 - s0;
                r.P = plan->pitch;
                r.Q = r.P - 8;
                r.fsrow = fs && !p.fastx && r.z0 == d0;
                r.f0 = (r.x0 - dn) * g.ldf + (r.z0 - d0);  // interior only
                for (int f = f0; f < f1; ++f) pc.fast[f] = (short)ia;
                for (int v = s0; v < s1; ++v) pc.slow[v] = (short)ib;
                r.soff = s0;
                most = std::max(most, region_floats(r.P, r.type, r.nf, r.ns, 0, false));
                plan->blocks.push_back(r);
            }
    }
    plan->floats = most;
    auto owner = [&](int z, int x) {  // of a live device cell; -1 above a free surface
        const int k = part_of[band(z - g.zoff, g.ny)][band(x, g.nx)];
        if (k < 0) return -1;
        const Part& p = parts[k];
        const int f = p.fastx ? x - p.x : z - p.zr, v = p.fastx ? z - p.zr : x - p.x;
        return pieces[k].first + pieces[k].slow[v] * p.a + pieces[k].fast[f];
    };
    // Packets: each edge position of a region with a neighbour receives one,
    // numbered along the region's edges; the neighbour publishes it.
    const int n = (int)plan->blocks.size();
    std::vector<std::vector<RegPair>> pub(n);
    auto local = [](const RegBlock& r, int z, int x) {  // shared offset of device cell (z, x)
        const int f = r.fastx ? x - r.x0 : z - r.z0, s = r.fastx ? z - r.z0 : x - r.x0;
        return (s + 3) * r.P + f + 4;
    };
    int npk = 0;
    for (int id = 0; id < n; ++id) {
        RegBlock& r = plan->blocks[id];
        r.rcv0 = (int)plan->rcv.size();
        r.rcv_first = npk;
        int nb = 0;  // edges with neighbours
        const int h = r.fastx ? r.ns : r.nf, w = r.fastx ? r.nf : r.ns;
        for (int edge = 0; edge < 4; ++edge) {
            const bool alongx = edge < 2;  // left / right edges: packets run along x
            const int len = alongx ? h : w;
            for (int t = 0; t < len; ++t) {
                // the adjacent cell outside, and the first (lowest) of the packet's 3 cells
                int z, x, pz, px;
                if (edge == 0) { z = r.z0 + t; x = r.x0 - 1; pz = z; px = x - 2; }
                else if (edge == 1) { z = r.z0 + t; x = r.x0 + w; pz = z; px = x; }
                else if (edge == 2) { x = r.x0 + t; z = r.z0 - 1; px = x; pz = z - 2; }
                else { x = r.x0 + t; z = r.z0 + h; px = x; pz = z; }
                const int lz = z - g.zoff;
                if (x < 0 || x >= g.nxt || lz < 0 || lz >= g.nyt) continue;
                const int o = owner(z, x);
                if (o < 0) continue;  // rows above a free surface
                const RegBlock& from = plan->blocks[o];
                const bool slow_r = alongx != (bool)r.fastx, slow_n = alongx != (bool)from.fastx;
                plan->rcv.push_back(local(r, pz, px) | (slow_r ? kRegSlow : 0));
                pub[o].push_back(RegPair{npk, local(from, pz, px) | (slow_n ? kRegSlow : 0)});
                ++npk;
                nb |= 1 << ((edge & 1) + (slow_r ? 0 : 2));
                if (r.type == kRegCorner && from.type == kRegCorner) {  // a cut of a corner: phi too
                    auto phi = [](const RegBlock& k, int z, int x) { return (x - k.x0 + 3) * k.Q + z - k.z0; };
                    plan->rcv.push_back(phi(r, pz, px) | kRegSlow | kRegPhi);
                    pub[o].push_back(RegPair{npk, phi(from, pz, px) | kRegSlow | kRegPhi});
                    ++npk;
                }
            }
        }
        r.nrcv = npk - r.rcv_first;
        item_shape(&r, nb);
    }
    plan->npk = npk;
    for (int id = 0; id < n; ++id) {
        RegBlock& r = plan->blocks[id];
        r.pub0 = (int)plan->pub.size();
        r.npub = (int)pub[id].size();
        plan->pub.insert(plan->pub.end(), pub[id].begin(), pub[id].end());
    }
    return true;
}

bool region_loads(const RegPlan& plan, const Grid& g, size_t max_floats, int ninj, const int* inj_cell,
                  const int* inj_trace, int nrec, const int* rec_cell, RegLists* out) {
    const int n = (int)plan.blocks.size();
    *out = RegLists{};
    out->loads.assign(n, RegLoad{});
    out->floats = plan.floats;
    auto owner_of = [&](int z, int x) {
        for (int id = 0; id < n; ++id) {
            const RegBlock& r = plan.blocks[id];
            const int h = r.fastx ? r.ns : r.nf, w = r.fastx ? r.nf : r.ns;
            if (z >= r.z0 && z < r.z0 + h && x >= r.x0 && x < r.x0 + w) return id;
        }
        return -1;
    };
    std::vector<std::vector<int>> inj(n), rec(n);
    for (int j = 0; j < ninj; ++j) {
        const int id = owner_of(inj_cell[j] % g.ldz, inj_cell[j] / g.ldz);
        if (id < 0 || plan.blocks[id].type != kRegInterior) return false;
        inj[id].push_back(j);
    }
    for (int j = 0; j < nrec; ++j) {
        // a cell in no region is never updated: its trace stays zero
        const int id = owner_of(rec_cell[j] % g.ldz, rec_cell[j] / g.ldz);
        if (id >= 0) rec[id].push_back(j);
    }
    for (int id = 0; id < n; ++id) {
        const RegBlock& r = plan.blocks[id];
        RegLoad& l = out->loads[id];
        l.region = id;
        l.slot0 = (int)out->slots.size();
        std::vector<signed char> slot(quads(r.nf), -1);
        l.inj0 = (int)out->inj.size();
        for (int j : inj[id]) {
            const int f = inj_cell[j] % g.ldz - r.z0, s = inj_cell[j] / g.ldz - r.x0;
            if (slot[f / 4] < 0) {
                if (l.nslot == 127) return false;
                slot[f / 4] = (signed char)l.nslot++;
            }
            out->inj.push_back(RegPair{(slot[f / 4] * r.ns + s) * 4 + f % 4, inj_trace[j]});
        }
        l.ninj = (int)inj[id].size();
        l.rec0 = (int)out->rec.size();
        for (int j : rec[id]) {
            const int z = rec_cell[j] % g.ldz - r.z0, x = rec_cell[j] / g.ldz - r.x0;
            out->rec.push_back(RegPair{j, ((r.fastx ? z : x) + 3) * r.P + (r.fastx ? x : z) + 4});
        }
        l.nrec = (int)rec[id].size();
        out->slots.insert(out->slots.end(), slot.begin(), slot.end());
        out->floats = std::max(out->floats, region_floats(r.P, r.type, r.nf, r.ns, l.nslot, false));
        out->floats_img = std::max(out->floats_img, region_floats(r.P, r.type, r.nf, r.ns, l.nslot, true));
        if (out->floats > max_floats) return false;
    }
    return true;
}

namespace {

// Allow the current device's kernel all of its shared memory; the dynamic
// shared floats of a block, 0 on failure.
template <int MODE, bool IMG, int P>
size_t region_max_floats_t() {
    const auto kern = region_kernel<MODE, IMG, P>;
    cudaFuncAttributes fa;
    int dev = 0, optin = 0, nb = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&fa, kern) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    const int dyn = (optin - (int)fa.sharedSizeBytes) & ~15;
    if (dyn <= 0 || cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kT, dyn) != cudaSuccess || nb < 1)
        return 0;
    return (size_t)dyn / sizeof(float);
}

template <int MODE, bool IMG, int P>
int launch_regions_t(const RegParams& rp, int nblocks, size_t floats, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = floats * sizeof(float);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, region_kernel<MODE, IMG, P>, rp);
}

template <int P>
size_t region_max_floats_p() {
    return std::min(std::min(region_max_floats_t<0, false, P>(), region_max_floats_t<1, false, P>()),
                    std::min(region_max_floats_t<1, true, P>(), region_max_floats_t<2, false, P>()));
}

template <int P>
int launch_regions_p(int mode, bool img, const RegParams& rp, int nblocks, size_t floats, cudaStream_t st) {
    if (mode == 0) return launch_regions_t<0, false, P>(rp, nblocks, floats, st);
    if (mode == 1 && img) return launch_regions_t<1, true, P>(rp, nblocks, floats, st);
    if (mode == 1) return launch_regions_t<1, false, P>(rp, nblocks, floats, st);
    return launch_regions_t<2, false, P>(rp, nblocks, floats, st);
}

// The snapshots that snapshot4 makes of levels p3 and p1, n cells, n a
// multiple of 4.
__global__ void snapshot_quotients_kernel(const StepArgs a, float neg0, const float* p3, const float* p1, float* q,
                                          int n) {
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    Consts kc{};
    kc.n0 = make_float2(neg0, neg0);
    kc.m1 = make_float2(-1.f, -1.f);
    *reinterpret_cast<float4*>(q + i) = snapshot4(a, kc, *reinterpret_cast<const float4*>(p3 + i),
                                                  *reinterpret_cast<const float4*>(p1 + i));
}

}  // namespace

int launch_snapshot_quotients(float dt, float inv_dt, int fast_div, float div_lo, float div_hi, const float* p3,
                              const float* p1, float* q, int n, void* stream) {
    if (n <= 0 || n % 4) return (int)cudaErrorInvalidValue;
    StepArgs a{};
    a.dt = dt;
    a.inv_dt = inv_dt;
    a.fast_div = fast_div;
    a.div_lo = div_lo;
    a.div_hi = div_hi;
    snapshot_quotients_kernel<<<(n / 4 + 127) / 128, 128, 0, (cudaStream_t)stream>>>(a, -0.0f, p3, p1, q, n);
    return (int)cudaGetLastError();
}

size_t region_max_floats() {
    static std::mutex lock;
    static std::map<int, size_t> known;  // by device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> hold(lock);
    auto it = known.find(dev);
    if (it == known.end())
        it = known.emplace(dev, std::min(region_max_floats_p<kRegPitches[0]>(), region_max_floats_p<kRegPitches[1]>()))
                 .first;
    return it->second;
}

int launch_regions(int mode, bool img, int pitch, const RegParams& rp, int nblocks, size_t floats, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (pitch == kRegPitches[0]) return launch_regions_p<kRegPitches[0]>(mode, img, rp, nblocks, floats, st);
    return launch_regions_p<kRegPitches[1]>(mode, img, rp, nblocks, floats, st);
}

}  // namespace psdm
