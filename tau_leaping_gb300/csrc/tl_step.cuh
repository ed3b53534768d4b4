// tl_step.cuh - one step of one realization for the fast and scores builds.
//
// The same method, streams and sums as do_step() (tl_device.cuh), which the
// general build, the plain form and the parity kernels keep: for one group
// kind the trajectories are bit-identical.  What differs is how the state and
// the tables lie in memory, because the path is bound by instruction issue:
//
//  * X[]: every population as FP32 with its criticality (x < n_c) in the sign
//    bit, then |x - 1| with the 2S criticality (x < 2 n_c) for the species of
//    2S channels, then the constant 1.  A propensity is the product
//    c |X_p| |X_q| for every order, with c halved for 2S (an exact scaling),
//    and its channel is critical when either sign is set: two loads and two
//    multiplies, no conversion, no case per order.
//  * Table entries hold byte offsets and the stoichiometry's FP32 bits, so an
//    entry costs two integer instructions to take apart.  Rows are padded to
//    four entries (the padding reads a zero propensity), and a row of a
//    species that reacts nowhere is left out.
//  * A leap adds its firings to D[] (int32) by shared-memory atomics, channel
//    by channel as they are drawn, instead of every row gathering over all its
//    channels: most channels of a leap do not fire.  The propensities stay in
//    place, so a rejected leap needs no second pass over the channels.
//  * Long Poisson draws go through a queue (fast_fire), which lies over X[]:
//    a leap does not read X between its step bound and its commit.
//  * Direct-method steps draw their channel on exact integers (lane groups) or
//    on FP32 with a margin (one thread); the FP64 form decides the cases
//    neither can (ssa_select).
// Measured on GB300 against do_step() with in-place draws (4000 to 60 000
// realizations, ms): toy network 109.7 -> 63.3 on 16 lanes and 47.3 -> 29.8 on
// warps, 45 x 83 network with int64 populations 127.0 -> 83.3, 12 x 20 network
// in direct-method steps 9.55 -> 3.15, 1024-species chain 4.60 -> 3.36, colloid
// of 250 species 5.14 -> 3.44, of 400 species (global propensities) 2.74 -> 1.78.
#pragma once

#include <type_traits>

#include "tl_device.cuh"
#include "tl_shared.h"

namespace tl {

// One thread for one realization of a model that the registers of a few lanes
// do not hold (tl_tiny.cuh).  Every sum runs over the channels in order, as
// there, so a realization's trajectory is the same on either.
struct GThin {
    static constexpr int kWidth = 1;
    TL_D int rank() const { return 0; }
    TL_D int size() const { return 1; }
    TL_D void sync() const {}
    TL_D bool leader() const { return true; }
    TL_D float minf(float v) const { return v; }
    TL_D bool any(bool p) const { return p; }
    template <class T>
    TL_D T bcast(T v, int) const {
        return v;
    }
};

template <class G>
struct is_thin {
    static constexpr bool value = false;
};
template <>
struct is_thin<GThin> {
    static constexpr bool value = true;
};

// Four warps for one realization of a warp-group model in a small ensemble,
// where the latency of one realization's steps sets the time.  Passes are
// spread over 128 threads; every sum runs as a warp group forms it (each warp
// forms all of them: sum_group), so the results are the warp group's.  One
// named barrier per team.
struct GTeam {
    static constexpr int kWidth = 128;
    int tid, lane, warp, bar;
    float* red;      // one value per warp
    long long* box;  // a broadcast value
    static TL_D GTeam make(int bar, float* red, long long* box) {
        const int t = (int)threadIdx.x & 127;
        return GTeam{t, t & 31, t >> 5, bar, red, box};
    }
    TL_D int rank() const { return tid; }
    TL_D int size() const { return 128; }
    TL_D void sync() const { asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory"); }
    TL_D bool leader() const { return tid == 0; }
    TL_D bool any(bool p) const {
        unsigned r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.or.pred q, %2, 128, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(r)
            : "r"(p ? 1u : 0u), "r"(bar)
            : "memory");
        return r != 0u;
    }
    // (other barriers lie between two calls)
    TL_D float minf(float v) const {
#pragma unroll
        for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) red[warp] = v;
        sync();
        return fminf(fminf(red[0], red[1]), fminf(red[2], red[3]));
    }
    TL_D long long bcast(long long v, int) const {
        if (tid == 0) *box = v;
        sync();
        const long long r = *box;
        sync();
        return r;
    }
};
TL_D GWarp queue_group(const GTeam& g) { return GWarp{g.lane}; }

// The lanes over which a group's sums run.
template <class Grp>
TL_D const Grp& sum_group(const Grp& g) {
    return g;
}
TL_D GWarp sum_group(const GTeam& g) { return GWarp{g.lane}; }

template <class Grp>
struct many_warps {
    static constexpr bool value = Grp::kWidth == 0 || Grp::kWidth == 128;
};

// Where one realization's state and the tables lie.  Only offsets are kept:
// an array's address is formed from them and the launch parameters where it is
// used, which costs an operand of the constant bank and no register.
// STAGED: the tables at the start of (or `tab` bytes into) shared memory, else
// in global memory.  GLOBAL: the slot's propensities, and where `state` is set
// the whole slot, in global memory.
extern __shared__ __align__(16) unsigned char tl_smem[];

template <class P, bool STAGED, bool GLOBAL>
struct Lay {
    using Pop = P;
    const SimParams& p;
    uint32_t slot;             // byte offset of the slot in shared memory
    uint32_t tab;              // byte offset of the tables in shared memory
    unsigned char* g_state;    // GLOBAL: the state, in either memory
    unsigned char* g_big;      // GLOBAL: a[]
    const uint32_t* rk;        // Philox round keys, in the launch parameters where one key serves the launch

    TL_D unsigned char* state(int off) const { return GLOBAL ? g_state + off : tl_smem + (slot + (uint32_t)off); }
    TL_D unsigned char* big(int off) const {
        return GLOBAL ? g_big + off : tl_smem + (slot + (uint32_t)(p.f_big + off));
    }
    template <class T>
    TL_D const T* table(int off) const {
        if constexpr (STAGED) return reinterpret_cast<const T*>(tl_smem + (tab + (uint32_t)off));
        else return reinterpret_cast<const T*>(p.blob + off);
    }
    TL_D P* x() const { return reinterpret_cast<P*>(state(0)); }
    TL_D int* D() const { return reinterpret_cast<int*>(state(p.f_D)); }
    TL_D float* X() const { return reinterpret_cast<float*>(state(p.f_X)); }
    TL_D unsigned short* q() const { return reinterpret_cast<unsigned short*>(state(p.f_X)); }
    TL_D float* a() const { return reinterpret_cast<float*>(big(0)); }
    TL_D int* k() const { return reinterpret_cast<int*>(big(p.f_a)); }  // counts of the leap, scored runs only
    TL_D const uint32_t* chan() const { return table<uint32_t>(p.t_chan); }
    TL_D const uint2* row() const { return table<uint2>(p.t_row); }
    TL_D const uint4* ent() const { return table<uint4>(p.t_ent); }
    TL_D const uint4* col() const { return table<uint4>(p.t_col); }
    TL_D const uint32_t* cp() const { return table<uint32_t>(p.t_cp); }  // p.t_cp < 0: one chunk per channel
    TL_D const unsigned short* sp() const { return table<unsigned short>(p.t_sp); }
    // scores of realization w, scored runs only
    TL_D float* score(long long w) const {
        return p.score_global ? p.scores + (size_t)w * p.M : reinterpret_cast<float*>(big(2 * p.f_a));
    }
};

template <class T>
TL_D T& at_byte(T* p, uint32_t off) {
    return *reinterpret_cast<T*>(reinterpret_cast<char*>(p) + off);
}
template <class T>
TL_D const T& at_byte(const T* p, uint32_t off) {
    return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + off);
}

// |f| with the sign bit of s
TL_D float with_sign(float f, int s) {
    return __uint_as_float((__float_as_uint(f) & 0x7fffffffu) | ((uint32_t)s & 0x80000000u));
}
// FP32 -> FP64 and FP64 >= on integers: GB300 runs FP64 at 1/64 of the FP32
// rate, and a step needs one addition of it.
TL_D double widen(float f) {
    const uint32_t b = __float_as_uint(f);
    if (b - 0x00800000u < 0x7f000000u)  // normal and positive
        return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
    return (double)f;
}
TL_D bool reached(double t, double limit) {  // both >= 0
    return __double_as_longlong(t) >= __double_as_longlong(limit);
}

// Species i holds x: its entries of X.  Populations and thresholds are >= 0,
// so the sign of x - n_c is the criticality.
template <class Lay>
TL_D void set_species32(const Lay& L, int i, int x) {
    const int nc = L.p.nc;
    L.X()[i] = with_sign((float)x, x - nc);
    const unsigned s3 = L.sp()[i];
    if (s3) L.X()[s3] = with_sign((float)(x - 1), x - 2 * nc);
}
template <class Lay>
__device__ __noinline__ void set_species64(const Lay L, int i, long long x) {
    const int nc = L.p.nc;
    L.X()[i] = with_sign((float)x, x < (long long)nc ? (int)0x80000000 : 0);
    const unsigned s3 = L.sp()[i];
    if (s3) L.X()[s3] = with_sign((float)(x - 1), x < (long long)(2 * nc) ? (int)0x80000000 : 0);
}
template <class Lay>
TL_D void set_species(const Lay& L, int i, int x) {
    set_species32(L, i, x);
}
// int64 -> FP32 runs at the reduced FP64 rate; a population that fits int32
// (the usual case) rounds to the same float from there
template <class Lay>
TL_D void set_species(const Lay& L, int i, long long x) {
    if ((long long)(int)x == x) set_species32(L, i, (int)x);
    else set_species64(L, i, x);
}

// Channel j's propensity, and in the sign bit whether it is critical.
template <class Grp, class Lay>
TL_D float signed_prop(const SimParams& p, const Lay& L, const float* rate, int j) {
    uint32_t o0, o1;
    if (Grp::kWidth == 0 && p.chan8) {
        const uint2 r = reinterpret_cast<const uint2*>(L.chan())[j];
        o0 = r.x;
        o1 = r.y;
    } else {
        const uint32_t r = L.chan()[j];
        o0 = r & 0xffffu;
        o1 = r >> 16;
    }
    const float f0 = at_byte(L.X(), o0), f1 = at_byte(L.X(), o1);
    const float v = __ldg(rate + j) * fabsf(f0) * fabsf(f1);
    const uint32_t cr = (__float_as_uint(f0) | __float_as_uint(f1)) & 0x80000000u;
    return __uint_as_float(__float_as_uint(v) | cr);
}

// Propensities into a[] and the lane's partial sums; one thread forms the sums
// over all channels in order.  Critical channels are stored negative, or with
// ZERO as 0, which spares every net entry of the step bound a max: what reads
// their propensities forms them again (select_critical, direct steps).
template <bool ZERO, class Grp, class Lay>
TL_D void fast_props(const Grp& g, const SimParams& p, const Lay& L, const float* rate, float& pa, float& pac) {
    float s = 0.f, sc = 0.f;
    constexpr int kUnroll = is_thin<Grp>::value ? 4 : 2;
#pragma unroll kUnroll
    for (int j = g.rank(); j < p.M; j += g.size()) {
        const float sv = signed_prop<Grp>(p, L, rate, j);
        const float v = fabsf(sv);
        const bool cr = is_crit(sv);
        L.a()[j] = ZERO && cr ? 0.f : sv;
        if constexpr (!is_thin<Grp>::value && Grp::kWidth != 128) {
            s += v;
            sc += cr ? v : 0.f;
        }
    }
    g.sync();
    if constexpr (Grp::kWidth == 128) {
        // the partial sums of a warp group's lane
#pragma unroll 4
        for (int j = sum_group(g).rank(); j < p.M; j += 32) {
            const float v = L.a()[j];
            s += fabsf(v);
            sc += fmaxf(-v, 0.f);
        }
    }
    if constexpr (is_thin<Grp>::value) {
        // a[] is padded with zeros to whole blocks of four
        for (int j = 0; j < p.M; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(L.a() + j);
            s += fabsf(v.x);
            sc += fmaxf(-v.x, 0.f);
            s += fabsf(v.y);
            sc += fmaxf(-v.y, 0.f);
            s += fabsf(v.z);
            sc += fmaxf(-v.z, 0.f);
            s += fabsf(v.w);
            sc += fmaxf(-v.w, 0.f);
        }
    }
    pa = s;
    pac = sc;
}

// select_channel among the critical channels where a[] holds 0 for them: the
// lane that owns the target forms its channels' propensities again.
template <class Grp, class Lay>
__device__ __noinline__ int select_critical(const Grp g, const SimParams& p, const Lay L, const float* rate, float pac,
                                            double target) {
    const double part = (double)pac, excl = g.excl_scan(part);
    int owner = g.first(part > 0.0 && target < excl + part);
    if (owner < 0) owner = g.last(part > 0.0);
    int sel = -1;
    if (g.rank() == owner) {
        const float limit = __double2float_rd(target - excl);
        float acc = 0.f;
#pragma unroll 1
        for (int j = g.rank(); j < p.M; j += g.size()) {
            const float v = signed_prop<Grp>(p, L, rate, j);
            if (!(v < 0.f)) continue;
            acc -= v;
            sel = j;
            if (limit < acc) break;
        }
    }
    return g.bcast(sel, owner < 0 ? 0 : owner);
}

// One entry's term of mu and sigma^2.
TL_D void add_moments(float v, float aj, float& mu, float& s2) {
    const float t = v * aj;
    mu += t;
    s2 += v * t;
}
// WIDE: models of 2^18 channels and more, beyond the 20-bit offsets.  ZERO:
// critical channels are stored as 0, else negative and max(a, 0) drops them.
template <bool WIDE, bool ZERO>
TL_D void add_entry(const float* a, uint32_t e, float& mu, float& s2) {
    float v, aj;
    if constexpr (WIDE) {
        v = unpack_vf((int)e);
        aj = a[e >> 3];
    } else {
        v = __uint_as_float(e << 20);
        aj = at_byte(a, e >> 12);
    }
    add_moments(v, ZERO ? aj : fmaxf(aj, 0.f), mu, s2);
}

// The CGP bound of a species (species_bound's values, without its branches:
// g is 1, 2 or 2 + 1/(x - 1), with 3 below x = 2; a moment of 0, or below
// FP32's normal range, bounds nothing).
TL_D float row_bound(const SimParams& p, float xi, int kind, float mu, float s2) {
    float gi = kind == 1 ? 1.f : 2.f;
    if (kind == 3) gi = 2.f + __frcp_rn(fmaxf(xi - 1.f, 1.f));
    const float num = fmaxf(p.eps * (xi * fast_rcp(gi)), 1.f);
    return fminf(num * fast_rcp(fabsf(mu)), num * num * fast_rcp(s2));
}

// The CGP step bound (CSRMatrixPacked.cu:311-358).
template <bool kWide, bool ZERO, class Grp, class Lay>
TL_D float fast_tau_rows(const Grp& g, const SimParams& p, const Lay& L) {
    float tmin = kInfF;
    if constexpr (Grp::kWidth == 0) {
        if (p.row_warp) {
            // long rows: one warp per row, lanes stride the entries
#pragma unroll 1
            for (int ii = g.warp; ii < p.n_rows; ii += g.nwarps) {
                const uint2 rec = L.row()[ii];
                const uint32_t* e = reinterpret_cast<const uint32_t*>(L.ent() + (rec.x & 0xfffffu));
                const int n = 4 * (int)(rec.x >> 20);
                float mu = 0.f, s2 = 0.f;
                for (int q = g.lane; q < n; q += 32) add_entry<kWide, ZERO>(L.a(), e[q], mu, s2);
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    mu += __shfl_xor_sync(0xffffffffu, mu, o);
                    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
                }
                const float xi = fabsf(L.X()[rec.y & 0x0fffffffu]);
                tmin = fminf(tmin, row_bound(p, xi, (int)(rec.y >> 28), mu, s2));
            }
            return g.minf(tmin);
        }
    }
#pragma unroll 1
    for (int ii = g.rank(); ii < p.n_rows; ii += g.size()) {
        const uint2 rec = L.row()[ii];
        const uint4* e = L.ent() + (rec.x & 0xfffffu);
        const int n = (int)(rec.x >> 20);
        float mu = 0.f, s2 = 0.f;
#pragma unroll 1
        for (int q = 0; q < n; ++q) {
            const uint4 w = e[q];
            add_entry<kWide, ZERO>(L.a(), w.x, mu, s2);
            add_entry<kWide, ZERO>(L.a(), w.y, mu, s2);
            add_entry<kWide, ZERO>(L.a(), w.z, mu, s2);
            add_entry<kWide, ZERO>(L.a(), w.w, mu, s2);
        }
        const float xi = fabsf(L.X()[rec.y & 0x0fffffffu]);
        tmin = fminf(tmin, row_bound(p, xi, (int)(rec.y >> 28), mu, s2));
    }
    return g.minf(tmin);
}

template <bool ZERO, class Grp, class Lay>
TL_D float fast_tau(const Grp& g, const SimParams& p, const Lay& L) {
    if constexpr (Grp::kWidth == 0)
        if (p.ent_wide) return fast_tau_rows<true, ZERO>(g, p, L);
    return fast_tau_rows<false, ZERO>(g, p, L);
}

// Calls f(byte offset of the species in an int array, stoichiometry) for channel j's net entries.
template <class Lay, class F>
TL_D void for_column(const Lay& L, int j, F f) {
    const SimParams& p = L.p;
    int c0 = j, n = 1;
    if (p.t_cp >= 0) {
        c0 = (int)L.cp()[j];
        n = (int)L.cp()[j + 1] - c0;
    }
#pragma unroll 1
    for (int q = 0; q < n; ++q) {
        const uint4 w = L.col()[c0 + q];
        const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (e[i] & 0xfffu) f(e[i] >> 12, (int)(e[i] << 20) >> 20);
    }
}

// k firings of channel j.
template <class Grp, class Lay>
TL_D void fire_channel(const Lay& L, int j, int k) {
    for_column(L, j, [&](uint32_t off, int v) {
        if constexpr (Grp::kWidth == 1) at_byte(L.D(), off) += v * k;
        else atomicAdd(&at_byte(L.D(), off), v * k);
    });
}


// Four species at a time: x, D and X are padded to whole blocks of four (the
// padding holds 0 and no channel reads it).
template <class Pop>
struct Four {
    Pop v[4];
};
TL_D Four<int> load_four(const int* p, int i4) {
    const int4 t = reinterpret_cast<const int4*>(p)[i4];
    return {{t.x, t.y, t.z, t.w}};
}
TL_D Four<long long> load_four(const long long* p, int i4) {
    const longlong2 t = reinterpret_cast<const longlong2*>(p)[2 * i4], u = reinterpret_cast<const longlong2*>(p)[2 * i4 + 1];
    return {{t.x, t.y, u.x, u.y}};
}
TL_D void store_four(int* p, int i4, const Four<int>& f) {
    reinterpret_cast<int4*>(p)[i4] = make_int4(f.v[0], f.v[1], f.v[2], f.v[3]);
}
TL_D void store_four(long long* p, int i4, const Four<long long>& f) {
    reinterpret_cast<longlong2*>(p)[2 * i4] = make_longlong2(f.v[0], f.v[1]);
    reinterpret_cast<longlong2*>(p)[2 * i4 + 1] = make_longlong2(f.v[2], f.v[3]);
}
TL_D int add_pop(int x, int d) { return (int)((unsigned)x + (unsigned)d); }
TL_D long long add_pop(long long x, int d) { return x + d; }

template <class Lay>
TL_D void set_four(const Lay& L, int i4, const Four<int>& x) {
    const int nc = L.p.nc;
    reinterpret_cast<float4*>(L.X())[i4] =
        make_float4(with_sign((float)x.v[0], x.v[0] - nc), with_sign((float)x.v[1], x.v[1] - nc),
                    with_sign((float)x.v[2], x.v[2] - nc), with_sign((float)x.v[3], x.v[3] - nc));
    const uint2 s3 = reinterpret_cast<const uint2*>(L.sp())[i4];
    const unsigned at[4] = {s3.x & 0xffffu, s3.x >> 16, s3.y & 0xffffu, s3.y >> 16};
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (at[e]) L.X()[at[e]] = with_sign((float)(x.v[e] - 1), x.v[e] - 2 * nc);
}
template <class Lay>
TL_D void set_four(const Lay& L, int i4, const Four<long long>& x) {
    // all four within int32, as they nearly always are
    const auto fits = [](long long v) { return (long long)(int)v == v; };
    if (fits(x.v[0]) && fits(x.v[1]) && fits(x.v[2]) && fits(x.v[3])) {
        set_four(L, i4, Four<int>{{(int)x.v[0], (int)x.v[1], (int)x.v[2], (int)x.v[3]}});
    } else {
#pragma unroll 1
        for (int e = 0; e < 4; ++e) set_species64(L, 4 * i4 + e, x.v[e]);
    }
}

// All of X from x.  D is zero.
template <class Grp, class Lay>
TL_D void fast_refresh(const Grp& g, const SimParams& p, const Lay& L) {
#pragma unroll 1
    for (int i = g.rank(); i < p.N; i += g.size()) set_species(L, i, L.x()[i]);
    if (g.leader()) L.X()[p.x_one] = 1.f;
}

// After a rejected leap: D to zero, and where select_critical reads X, which
// the queue lay over, X again.  Out of line: rejections are rare.
template <bool ZERO, class Grp, class Lay>
__device__ __noinline__ void undo_leap(const Grp g, const SimParams& p, const Lay L) {
#pragma unroll 1
    for (int i = g.rank(); i < p.N; i += g.size()) L.D()[i] = 0;
    if constexpr (ZERO) fast_refresh(g, p, L);
    g.sync();
}

// The firing counts of one leap into D (and k[] in scored runs), for groups
// of lanes.  Instruction issue bounds this pass, and most of it would go into
// lanes that wait for a neighbour's long draw, were each lane to make its
// channels' draws one at a time.
//  * A channel whose mean lies in [0, 10) compares the shared word's
//    u = 1 - q with F0 = exp(-mu) and F1 = F0 (1 + mu), both from one fast
//    exponential and without a branch.  kFireMargin bounds what the fast forms
//    and poisson_first's own tests together can be off (under 2.3e-6: the
//    truncated word 1.8e-7, the exponential 3.5e-7, poisson_p1 / p2 1.3e-6 and the
//    sums), so outside the margin both give the same count.
//  * Every other draw (k >= 2, within the margin, means >= 10) and every
//    channel with k = 1 is marked in the lane's masks.  After at most
//    q_rounds turns the lanes list their marked channels in a queue and take
//    them in turn: inversions and single firings from the front,
//    transformed-rejection draws (PTRS) from the back, so that a pass runs one
//    kind on all lanes and a channel's firing is spread over the lanes with
//    its draw.  A PTRS lane moves on to its next draw after an accepted
//    attempt instead of waiting for the warp's last one.
// a[], k[] and the columns are padded to whole blocks of four channels: the
// padding holds 0 and has no entries.  Its mean of 0 lies within the margin where
// the word is below 5e-6 of its range, so it can be marked: its draw is 0 firings of no
// entries.  (A test for it in the queue's loop cost the 45 x 83 network 1.5 %.)
constexpr float kFireMargin = 5e-6f;

// One attempt of a queued draw of mean < 10 (poisson_first).  Attempt 0 is on
// the shared word w: k <= 1 by the exact tests unless k >= 2 is settled, else
// the sequential search.  Where the FP32 sums stop growing below u, attempts
// 1 to 16 search on fresh uniforms w (poisson_inversion).  False: try again.
TL_D bool queued_inversion(float mu, uint32_t w, int attempt, int& k) {
    float u, pk, F;
    const float e = expf(-mu);
    if (attempt == 0) {
        const float qf = ((float)w + 0.5f) * 2.3283064365386963e-10f;
        u = 1.f - qf;
        if (fmaf(e, mu, e) - u > -kFireMargin) {
            k = 0;
            if (qf >= poisson_p1(mu)) return true;
            k = 1;
            if (qf >= poisson_p2(mu)) return true;
        }
        pk = e * mu;
        F = e + pk;
        k = 1;
    } else {
        u = u01f(w);
        pk = F = e;
        k = 0;
        if (u <= F) return true;
    }
    // Four terms a turn: the sums grow until they stay at one value, so the
    // last two tell whether they stopped below u (once the terms fall, k > mu,
    // a sum that repeats repeats for good).  One term a turn leaves a warp with
    // the latency of a reciprocal and a branch for each.
    float kf = (float)k;
#pragma unroll 1
    for (;;) {
        const float q1 = mu * fast_rcp(kf + 1.f), q2 = mu * fast_rcp(kf + 2.f), q3 = mu * fast_rcp(kf + 3.f),
                    q4 = mu * fast_rcp(kf + 4.f);
        const float p1 = pk * q1, p2 = p1 * q2, p3 = p2 * q3, p4 = p3 * q4;
        const float F1 = F + p1, F2 = F1 + p2, F3 = F2 + p3, F4 = F3 + p4;
        if (u <= F4) {
            k = (int)kf + 1 + (u > F1 ? 1 : 0) + (u > F2 ? 1 : 0) + (u > F3 ? 1 : 0);
            return true;
        }
        if (F4 == F3) break;
        kf += 4.f;
        pk = p4;
        F = F4;
    }
    k = (int)mu;  // u above the representable mass
    return attempt == 16;
}

template <class Grp, class Lay, bool SENS>
TL_D void fast_fire(const Grp& g, const SimParams& p, const Lay& L, float tauf, int jc, uint32_t step,
                    uint32_t r, uint32_t set) {
    const auto qg = queue_group(g);
    constexpr int kTurn = 4 * decltype(queue_group(g))::kWidth;  // channels of a queue group's turn
    const int cap = p.q_rounds * kTurn;
    unsigned short* q = L.q();
    if constexpr (many_warps<Grp>::value) q += g.warp * (cap + 2);
    const float* a = L.a();
    const int G4 = (p.M + 3) >> 2;
    for (int b0 = g.rank() - qg.rank(); b0 < G4;) {
        const int j_first = 4 * b0;
        unsigned inv = 0, big = 0, one = 0;  // this lane's marked channels, four bits a turn
        int sh = 0;
#pragma unroll 1
        for (int m = 0; m < p.q_rounds && b0 < G4; ++m, b0 += g.size(), sh += 4) {
            const int g4 = b0 + qg.rank();
            if (g4 >= G4) continue;
            const float4 v4 = *reinterpret_cast<const float4*>(a + 4 * g4);
            const float av[4] = {v4.x, v4.y, v4.z, v4.w};
            float mu[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) mu[e] = fmaxf(av[e], 0.f) * tauf;  // critical channels: 0
            U4 gw{0u, 0u, 0u, 0u};
            if (fminf(fminf(mu[0], mu[1]), fminf(mu[2], mu[3])) < 10.f)
                gw = group_words(L.rk, (uint32_t)g4, step, r, set);
            unsigned all = 0, far = 0, fired = 0;
            const bool any_far = fmaxf(fmaxf(mu[0], mu[1]), fmaxf(mu[2], mu[3])) >= 10.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float ex = fast_ex2(mu[e] * -1.44269504f);
                // 2 - (1 - q) from the word's top 23 bits
                const float v = __uint_as_float((word_of(gw, e) >> 9) + 0x3f800000u);
                const float d0 = v + (ex - 2.f);          // F0 - u
                const float d1 = fmaf(ex, mu[e], d0);     // F1 - u >= F0 - u
                if (fminf(d1, fabsf(d0)) < kFireMargin) all |= 1u << e;
                fired |= __float_as_uint(d0) >> 31 << e;
            }
            if (any_far) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (mu[e] >= 10.f) far |= 1u << e;
                all |= far;
            }
            inv |= (all & ~far) << sh;
            big |= far << sh;
            fired &= ~all;
            one |= fired << sh;
            if constexpr (SENS)
                *reinterpret_cast<int4*>(L.k() + 4 * g4) =
                    make_int4(fired & 1, fired >> 1 & 1, fired >> 2 & 1, fired >> 3);
        }
        if (!qg.any((inv | big | one) != 0u)) continue;
        // list the marked channels: positions from one scan of the counts
        const unsigned mine =
            (unsigned)__popc(inv) | (unsigned)__popc(one) << 10 | (unsigned)__popc(big) << 20;
        const unsigned upto = qg.incl_scan(mine);
        const unsigned total = qg.bcast(upto, qg.size() - 1), before = upto - mine;
        const int n_inv = (int)(total & 1023u), n_front = n_inv + (int)(total >> 10 & 1023u), n_big = (int)(total >> 20);
        const auto list = [&](unsigned marks, int at, int by) {
            while (marks) {
                const int bit = __ffs(marks) - 1;
                marks &= marks - 1;
                q[at] = (unsigned short)((bit >> 2) * kTurn + qg.rank() * 4 + (bit & 3));
                at += by;
            }
        };
        list(inv, (int)(before & 1023u), 1);
        list(one, n_inv + (int)(before >> 10 & 1023u), 1);
        list(big, cap - 1 - (int)(before >> 20), -1);
        int* next = reinterpret_cast<int*>(q + cap);
        if (qg.rank() == 0) *next = 0;
        qg.sync();
        const auto channel = [&](int id) {
            if constexpr (many_warps<Grp>::value) return j_first + (id / kTurn) * 4 * g.size() + id % kTurn;
            else return j_first + id;
        };
        for (int i = qg.rank(); i < n_front; i += qg.size()) {
            const int j = channel(q[i]);
            int k = 1;
            if (i < n_inv) {
                const float mu = fmaxf(a[j], 0.f) * tauf;
                U4 w = group_words(L.rk, (uint32_t)j >> 2, step, r, set);
                uint32_t word = word_of(w, j & 3);
                for (int it = 0; !queued_inversion(mu, word, it, k); ++it) {
                    w = philox10(U4{(uint32_t)j, step, r, (set << 8) + (uint32_t)(it >> 2)}, p.k0, p.k1);
                    word = word_of(w, it & 3);
                }
                if constexpr (SENS) L.k()[j] = k;
            }
            fire_channel<Grp>(L, j, k);
        }
        // PTRS draws need one to several attempts: a lane that is done with
        // one takes the next that no lane has.  (A counter for the others too
        // cost the colloid model 14 %.)
        if (n_big) {
            int it = 0;  // attempts so far on this draw
            for (int i = atomicAdd(next, 1); i < n_big;) {
                const int j = channel(q[cap - 1 - i]);
                const float mu = a[j] * tauf;
                const U4 w = philox10rk(U4{(uint32_t)j, step, r, (set << 8) + (uint32_t)(it >> 1)}, L.rk);
                const bool odd = it & 1;
                int k;
                bool ok = Ptrs(mu).attempt(u01f(odd ? w.z : w.x), u01f(odd ? w.w : w.y), k);
                if (++it == kPtrsTries && !ok) {
                    k = (int)(mu + 0.5f);
                    ok = true;
                }
                if (ok) {
                    if constexpr (SENS) L.k()[j] = k;
                    fire_channel<Grp>(L, j, k);
                    it = 0;
                    i = atomicAdd(next, 1);
                }
            }
        }
        qg.sync();
    }
    // the critical channel that fires, by the lane that owns its block
    if (jc >= 0 && (jc >> 2) % g.size() == g.rank()) {
        if constexpr (SENS) L.k()[jc] = 1;
        fire_channel<Grp>(L, jc, 1);
    }
}

// The count of channel j in a leap, drawn in place: thread groups and the
// lanes of small models.
TL_D int poisson_channel(float aj, float tauf, int j, int jc, uint32_t step, uint32_t r, uint32_t set,
                         const uint32_t* rk) {
    const float mu = fmaxf(aj, 0.f) * tauf;
    int k = is_crit(aj) && j == jc ? 1 : 0;
    if (mu > 0.f) {
        const bool ptrs = mu >= 10.f;
        bool ok = false;
        for (int it = 0; !ok; ++it) {
            // the shared block of first words, or the private stream: two
            // uniforms for a PTRS attempt, one for an inversion's
            const bool shared = !ptrs && it == 0;
            const int at = ptrs ? 2 * it : it - 1;
            const U4 w = philox10rk(shared ? U4{(uint32_t)j >> 2, step, r, (set << 8) | 0xFFu}
                                           : U4{(uint32_t)j, step, r, (set << 8) + (uint32_t)(at >> 2)},
                                    rk);
            if (ptrs) {
                const bool odd = it & 1;
                ok = Ptrs(mu).attempt(u01f(odd ? w.z : w.x), u01f(odd ? w.w : w.y), k);
                if (it == kPtrsTries - 1 && !ok) {
                    k = (int)(mu + 0.5f);
                    ok = true;
                }
            } else {
                const uint32_t word = word_of(w, shared ? j & 3 : at & 3);
                // P(K >= 1) as computed never exceeds mu
                ok = shared && ((float)word + 0.5f) * 2.3283064365386963e-10f >= mu;
                if (!ok) ok = queued_inversion(mu, word, it, k);
            }
        }
    }
    return k;
}

template <class Lay, bool SENS>
TL_D void thin_fire(const SimParams& p, const Lay& L, float tauf, int jc, uint32_t step, uint32_t r, uint32_t set) {
    for (int j = 0; j < p.M; ++j) {
        const int k = poisson_channel(L.a()[j], tauf, j, jc, step, r, set, L.rk);
        if constexpr (SENS) L.k()[j] = k;
        if (k) fire_channel<GThin>(L, j, k);
    }
}

// x + D: any population negative?  (or past the population type, in *over)
template <class Grp, class Lay>
TL_D bool fast_check(const Grp& g, const SimParams& p, const Lay& L, bool& over) {
    using Pop = typename Lay::Pop;
    const int n4 = (p.N + 3) >> 2;
    Pop sign = 0;
#pragma unroll 1
    for (int i = g.rank(); i < n4; i += g.size()) {
        const Four<Pop> x = load_four(L.x(), i);
        const Four<int> d = load_four(L.D(), i);
#pragma unroll
        for (int e = 0; e < 4; ++e) sign |= add_pop(x.v[e], d.v[e]);
    }
    const bool bad = g.any(sign < 0);
    over = false;
    if (sizeof(Pop) == 4 && bad) {
        bool of = false;  // a sum that wrapped: |D| < 2^31, and not from below zero
#pragma unroll 1
        for (int i = g.rank(); i < p.N; i += g.size())
            of |= L.x()[i] >= 0 && L.D()[i] > 0 && add_pop(L.x()[i], L.D()[i]) < 0;
        over = g.any(of);
    }
    return bad;
}

template <class Grp, class Lay>
TL_D void fast_commit(const Grp& g, const SimParams& p, const Lay& L) {
    using Pop = typename Lay::Pop;
    const int n4 = (p.N + 3) >> 2;
#pragma unroll 1
    for (int i = g.rank(); i < n4; i += g.size()) {
        Four<Pop> x = load_four(L.x(), i);
        const Four<int> d = load_four(L.D(), i);
#pragma unroll
        for (int e = 0; e < 4; ++e) x.v[e] = add_pop(x.v[e], d.v[e]);
        store_four(L.x(), i, x);
        store_four(L.D(), i, Four<int>{{0, 0, 0, 0}});
        set_four(L, i, x);
    }
    if (g.leader()) L.X()[p.x_one] = 1.f;
}

// The same for one thread.
template <class Lay>
TL_D bool thin_commit(const SimParams& p, const Lay& L, bool& over) {
    using Pop = typename Lay::Pop;
    bool bad = false;
    over = false;
    for (int i = 0; i < p.N; ++i) {
        const Pop x = L.x()[i];
        const int d = L.D()[i];
        const bool b = add_pop(x, d) < 0;
        bad |= b;
        over |= sizeof(Pop) == 4 && b && d > 0 && x >= 0;
    }
    if (bad) return true;
    for (int i = 0; i < p.N; ++i) {
        const Pop nx = add_pop(L.x()[i], L.D()[i]);
        L.x()[i] = nx;
        L.D()[i] = 0;
        set_species(L, i, nx);
    }
    L.X()[p.x_one] = 1.f;
    return false;
}

// A leap that may hold more than 10^8 firings, whose sums could leave int32:
// the counts are drawn in place and added in 64 bits, over D and X together.
// Returns as fast_check and commits where that allows it.
constexpr float kWideLeap = 1e8f;

template <class Grp, class Lay, bool SENS>
TL_D bool wide_leap(const Grp& g, const SimParams& p, const Lay& L, float tauf, int jc, uint32_t step, uint32_t r,
                    uint32_t set, bool& over) {
    using Pop = typename Lay::Pop;
    unsigned long long* D64 = reinterpret_cast<unsigned long long*>(L.D());
#pragma unroll 1
    for (int i = g.rank(); i < p.N; i += g.size()) D64[i] = 0ull;
    g.sync();
#pragma unroll 1
    for (int j = g.rank(); j < p.M; j += g.size()) {
        const float aj = L.a()[j];
        int k = 0;
        if (is_crit(aj)) {
            k = j == jc ? 1 : 0;
        } else {
            const U4 gw = group_words(L.rk, (uint32_t)j >> 2, step, r, set);
            ChanRng rng;
            rng.init((uint32_t)j, step, r, set, L.rk);
            k = poisson_first(aj * tauf, word_of(gw, j & 3), rng);
        }
        if constexpr (SENS) L.k()[j] = k;
        for_column(L, j, [&](uint32_t off, int v) { atomicAdd(&D64[off >> 2], (unsigned long long)((long long)v * k)); });
    }
    g.sync();
    bool bad = false, of = false;
#pragma unroll 1
    for (int i = g.rank(); i < p.N; i += g.size()) {
        const long long nx = (long long)L.x()[i] + (long long)D64[i];
        of |= sizeof(Pop) == 4 && nx > 2147483647LL;
        bad |= nx < 0 || of;
    }
    over = g.any(of);
    bad = g.any(bad);
    if (!bad)
#pragma unroll 1
        for (int i = g.rank(); i < p.N; i += g.size()) L.x()[i] = (Pop)((long long)L.x()[i] + (long long)D64[i]);
    g.sync();
    // the padding of D too: the 64-bit sums lay over it
#pragma unroll 1
    for (int i = g.rank(); i < ((p.N + 3) & ~3); i += g.size()) L.D()[i] = 0;
    if (!bad) fast_refresh(g, p, L);
    g.sync();
    return bad;
}

// ---------------------------------------------------------------------------
// Direct-method steps: the channel with probability a_j / a0 and a0 in FP32.
// ---------------------------------------------------------------------------
// One thread: one running sum in channel order, target u * a0 with u of 52
// bits.  FP32 decides every channel whose running sum is further from the
// target than the products' rounding (2^-23 a0, margin 4e-7 a0); the FP64
// target decides the others.
template <class Lay>
TL_D int thin_select(const SimParams& p, const Lay& L, float part, uint32_t w_hi, uint32_t w_lo) {
    const float t = ((float)(w_hi >> 6) * 1.4901161193847656e-08f) * part;  // 2^-26
    const float m = 4e-7f * part, above = t + m, below = t - m;
    float acc = 0.f;
    int sel = -1, last = -1;
    bool close = false;
    // four channels a turn without a branch; the padding is 0
#pragma unroll 1
    for (int j = 0; j < p.M && sel < 0; j += 4) {
        const float4 v4 = *reinterpret_cast<const float4*>(L.a() + j);
        const float v[4] = {fabsf(v4.x), fabsf(v4.y), fabsf(v4.z), fabsf(v4.w)};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            acc += v[e];
            const bool some = v[e] > 0.f;
            close |= some && acc >= below && acc <= above;
            if (some && sel < 0 && acc > above) sel = j + e;
            if (some) last = j + e;
        }
    }
    if (close) {
        const float tf = __double2float_rd(u01d(w_hi, w_lo) * (double)part);
        acc = 0.f;
        sel = -1;
#pragma unroll 1
        for (int j = 0; j < p.M && sel < 0; ++j) {
            const float v = fabsf(L.a()[j]);
            acc += v;
            if (v > 0.f && tf < acc) sel = j;
        }
    }
    return sel >= 0 ? sel : last;
}

// Lane groups.  The lanes' partial sums are put on one integer grid, the lsb
// of the largest one's exponent - 24; when every partial lies on it, the FP64
// sums of the general form are exact too, and 64-bit integers give a0, the
// cumulative sums and the target.  Where a partial falls off the grid, the
// target lies within the FP64 product's rounding of a lane's boundary, or the
// search inside a lane of several channels comes within FP32 rounding, the
// FP64 form decides (select_channel_impl).  GB300's FP64 rate is 1/64 of FP32:
// the FP64 butterfly and scan took 82 % of that pipe on a 12 x 20 network.
// S to FP32, to nearest even, for 2^32 <= S < 2^53 (the largest partial alone
// is 2^47): the conversion instruction runs at the FP64 rate.
TL_D float round53(unsigned long long S) {
    const int lz = __clz((int)(S >> 32));
    const unsigned long long X = S << lz;  // top bit at 63
    uint32_t m = (uint32_t)(X >> 40);
    const unsigned long long rest = X & ((1ull << 40) - 1), half = 1ull << 39;
    m += rest > half || (rest == half && (m & 1u)) ? 1u : 0u;
    return (float)m * __uint_as_float((uint32_t)(127 + 40 - lz) << 23);
}

template <class Grp, class Lay>
__device__ __noinline__ int ssa_select_fp64(const Grp g, const SimParams& p, const Lay& L, float part, uint32_t w_hi,
                                            uint32_t w_lo, float& a0f) {
    const double a0 = g.sumd((double)part);
    a0f = (float)a0;
    return select_channel_impl<Grp, double>(g, p.M, L.a(), part, u01d(w_hi, w_lo) * a0, 0);
}

template <class Grp, class Lay>
TL_D int ssa_select(const Grp& g, const SimParams& p, const Lay& L, float part, uint32_t w_hi, uint32_t w_lo,
                    float& a0f) {
    const uint32_t bits = __float_as_uint(part);
    const int e = (int)(bits >> 23);
    const int emax = (int)g.max_int(e);
    const int eb = emax - 24;
    const bool off = bits != 0u && e < eb;
    if (emax < 60 || emax > 250 || g.any(off)) return ssa_select_fp64(g, p, L, part, w_hi, w_lo, a0f);
    const uint32_t mant = bits ? (bits & 0x7fffffu) | 0x800000u : 0u;
    const int up = e - eb;  // 0..24 where mant != 0
    const float unit = __uint_as_float((uint32_t)(eb - 23) << 23);  // value of the grid's lsb; eb >= 36
    if (p.M <= g.size()) {
        // One channel a lane.  The total from the sums of the halves; the
        // target and the cumulative sums from their top 27 bits: P is short of
        // the true sum by less than 32 units (2^22 of the grid), T of the
        // target by less than 4, so outside that window both place the target.
        const uint32_t hi = mant ? mant >> (24 - up) : 0u, lo = mant ? mant << up & 0xffffffu : 0u;
        const unsigned long long S = ((unsigned long long)g.sum_uint(hi) << 24) + g.sum_uint(lo);
        a0f = round53(S) * unit;
        const int T = (int)__umulhi((w_hi & ~63u) | w_lo >> 26, (uint32_t)(S >> 22) << 1) >> 1;
        const int P = (int)g.incl_scan(hi << 2 | lo >> 22);
        const bool some = mant != 0u;
        if (g.any(some && P - T > -32 && P - T < 4)) return ssa_select_fp64(g, p, L, part, w_hi, w_lo, a0f);
        const int first = g.first(some && P > T);
        return first >= 0 ? first : g.last(some);
    }
    const unsigned long long F = (unsigned long long)mant << (mant ? up : 0);
    // u = k2 2^-53 and, below, T = floor(u S)
    const unsigned long long k2 = (((unsigned long long)(w_hi >> 6) << 26 | (w_lo >> 6)) << 1) | 1ull;
    // inclusive scan; the last lane holds the total
    unsigned long long P = F;
#pragma unroll
    for (int o = 1; o < Grp::kWidth; o <<= 1) {
        const unsigned long long n = g.shfl_up(P, o);
        if (g.rank() >= o) P += n;
    }
    const unsigned long long S = g.bcast(P, g.size() - 1);
    a0f = round53(S) * unit;
    const unsigned long long T = __umul64hi(k2 << 11, S);
    // general form: target < excl + part = P with target = u * S rounded to FP64
    bool close = F != 0ull && T + 1ull == P;
    const int first = g.first(F != 0ull && T < P);
    const int Ls = first >= 0 ? first : g.last(F != 0ull);
    int sel = -1;
    if (g.rank() == Ls && !close) {
        const float tf = __ull2float_rn(T + F - P) * unit;  // target - excl
        float acc = 0.f;
        for (int j = g.rank(); j < p.M; j += g.size()) {
            const float v = fabsf(L.a()[j]);
            if (!(v > 0.f)) continue;
            acc += v;
            sel = j;
            if (j + g.size() < p.M) {  // not the lane's last channel
                if (fabsf(acc - tf) <= 4e-7f * part) {
                    close = true;
                    break;
                }
                if (tf < acc) break;
            }
        }
    }
    if (g.any(close)) return ssa_select_fp64(g, p, L, part, w_hi, w_lo, a0f);
    return g.bcast(sel, Ls);
}


// ---------------------------------------------------------------------------
// One step (model.cu:301-413): a tau-leap with rejection and halving, or a
// block of direct-method steps.
// ---------------------------------------------------------------------------
// Every leap attempt and every direct-method step advances the Philox step
// counter once: accepted() = step - rej in 64 bits, leaps = accepted - ssa.
struct FastState {
    double t;
    double t_next;  // grid time kpt; done may be set before the last point: the state holds
    int kpt;        // next grid point to record
    uint32_t step;
    uint32_t rej, ssa;
    uint32_t epochs;   // wraps of step before this leap or block
    uint32_t ex_from;  // the lanes hold the critical waiting times (unit rate) of the steps from here
    float ex;
    bool wide;     // the next step is a wide leap
    bool done;
};

// Index of realization r of a set in this call's samples and scores.
TL_D size_t realization_index(const SimParams& p, int set, uint32_t r) {
    return (size_t)((long long)set * p.R + ((long long)r - p.r_off));
}

template <class Grp, class Lay>
TL_D void fast_record(const Grp& g, const SimParams& p, const Lay& L, int set, uint32_t r, int kpt) {
    using Pop = typename Lay::Pop;
    Pop* samp = reinterpret_cast<Pop*>(p.samples) + realization_index(p, set, r) * (p.n_int + 1) * p.K;
    samp += (size_t)kpt * p.K;
#pragma unroll 1
    for (int q = g.rank(); q < p.K; q += g.size()) samp[q] = L.x()[p.tracked[q]];
}

// Records the state at the next grid point.
template <class Grp, class Lay>
TL_D void record_next(const Grp& g, const SimParams& p, const Lay& L, int set, uint32_t r, FastState& st) {
    fast_record(g, p, L, set, r, st.kpt++);
    if (st.kpt <= p.n_int) st.t_next = grid_time<double>(p, set, st.kpt);
}

// score_m += term(m, a_m, k_m) / c_m over the group's channels; counts: k_m
// is read (0 otherwise).  Four channels at a time where every array is aligned
// for it: gradients of the toy network 32.4 -> 31.6 ms.
template <class Grp, class Lay, class F>
TL_D void add_scores(const Grp& g, const SimParams& p, const Lay& L, int set, uint32_t r, bool counts, F term) {
    float* score = L.score((long long)realization_index(p, set, r));
    const float* c0 = p.rates + (size_t)set * p.M;
    if ((p.M & 3) == 0 && !is_thin<Grp>::value) {
#pragma unroll 1
        for (int b = g.rank(); 4 * b < p.M; b += g.size()) {
            const float4 c4 = __ldg(reinterpret_cast<const float4*>(c0) + b);
            const float4 a4 = reinterpret_cast<const float4*>(L.a())[b];
            const int4 k4 = counts ? reinterpret_cast<const int4*>(L.k())[b] : make_int4(0, 0, 0, 0);
            float4 s4 = reinterpret_cast<const float4*>(score)[b];
            if (c4.x > 0.f) s4.x += term(4 * b, a4.x, k4.x) / c4.x;
            if (c4.y > 0.f) s4.y += term(4 * b + 1, a4.y, k4.y) / c4.y;
            if (c4.z > 0.f) s4.z += term(4 * b + 2, a4.z, k4.z) / c4.z;
            if (c4.w > 0.f) s4.w += term(4 * b + 3, a4.w, k4.w) / c4.w;
            reinterpret_cast<float4*>(score)[b] = s4;
        }
        return;
    }
#pragma unroll 1
    for (int m = g.rank(); m < p.M; m += g.size()) {
        const float c = __ldg(c0 + m);
        if (c > 0.f) score[m] += term(m, L.a()[m], counts ? L.k()[m] : 0) / c;
    }
}

// The same block for a warp whose lanes hold a channel and a species each (up
// to 32 of both): the populations stay in registers and a step exchanges them
// by shuffles, without the two barriers and the dozen shared-memory accesses
// of the general block.  Issue and FP64 latency bound it; 12 x 20 network, 5000
// realizations: 1957 -> 1607 us of kernel time (general block: 285 instructions a step).
template <class Lay, bool SENS>
TL_D void direct_steps_lanes(const GWarp& g, const SimParams& p, const Lay& L, int set, uint32_t r, float pa,
                             FastState& st) {
    using Pop = typename Lay::Pop;
    const int lane = g.lane, one = 4 * p.x_one;
    const bool channel = lane < p.M, species = lane < p.N;
    // the channel's factors: |x| of species src0, then of src1, |x - 1| of src0, or 1
    const uint32_t rec = channel ? L.chan()[lane] : (uint32_t)one << 16 | (uint32_t)one;
    const int o0 = (int)(rec & 0xffffu), o1 = (int)(rec >> 16);
    const bool none = o0 == one, single = o1 == one, twice = !single && o1 >= 4 * ((p.N + 3) & ~3);
    const int src0 = none ? 0 : o0 >> 2, src1 = single || twice ? 0 : o1 >> 2;
    const float rate = channel ? __ldg(p.frates + (size_t)set * p.M + lane) : 0.f;
    float c = 0.f, score = 0.f;
    if (SENS && p.scores && channel) {
        c = __ldg(p.rates + (size_t)set * p.M + lane);
        score = L.score((long long)realization_index(p, set, r))[lane];
    }
    Pop x = species ? L.x()[lane] : (Pop)0;
    U4 w{0u, 0u, 0u, 0u};
    float ex = 0.f;
    for (int q = 0;;) {
        if ((q & 31) == 0) {
            w = step_words(L.rk, st.step + (uint32_t)lane, r, (uint32_t)set);
            ex = -logf(u01f(w.x));
        }
        float a0;
        const int j = ssa_select(g, p, L, pa, g.bcast(w.z, q & 31), g.bcast(w.w, q & 31), a0);
        const float dtf = g.bcast(ex, q & 31) / a0;
        const double t_new = st.t + widen(dtf);
        if (reached(t_new, st.t_next)) {
            if (species) L.x()[lane] = x;
            g.sync();
            while (st.kpt <= p.n_int && reached(t_new, st.t_next)) record_next(g, p, L, set, r, st);
            g.sync();
            if (st.kpt > p.n_int) {
                if (SENS && c > 0.f) score -= pa * (float)(p.t_final[set] - st.t) / c;
                st.done = true;
                break;
            }
        }
        if (SENS && c > 0.f) score += ((lane == j ? 1.f : 0.f) - pa * dtf) / c;
        // the fired channel's entries, to the lanes of their species
        if (j >= 0) {
            const uint4 e = L.col()[j];
            int d = 0;
            if ((int)(e.x >> 14) == lane) d = (int)(e.x << 20) >> 20;
            if ((int)(e.y >> 14) == lane && (e.y & 0xfffu)) d = (int)(e.y << 20) >> 20;
            if ((int)(e.z >> 14) == lane && (e.z & 0xfffu)) d = (int)(e.z << 20) >> 20;
            if ((int)(e.w >> 14) == lane && (e.w & 0xfffu)) d = (int)(e.w << 20) >> 20;
            x = add_pop(x, d);
        }
        st.t = t_new;
        st.step++;
        st.ssa++;
        ++q;
        if (q == p.ssa_block || (p.max_steps > 0 && accepted(st.epochs + wrapped(st.step, q), st.step, st.rej) >= p.max_steps)) break;
        // propensities: products of |x|, as everywhere (a channel that lists a
        // species twice can take it below zero)
        const float f = fabsf(popf(x));
        const float f0 = g.bcast(f, src0), fs = g.bcast(f, src1), f2 = g.bcast(popf((Pop)(x - 1)), src0);
        const float f1 = single ? 1.f : twice ? fabsf(f2) : fs;
        pa = rate * (none ? 1.f : f0) * f1;
        if (channel) L.a()[lane] = pa;  // ssa_select's FP64 form reads it
        g.sync();
        if (!g.any(pa > 0.f)) {
            st.done = true;
            break;
        }
    }
    if (species) {
        L.x()[lane] = x;
        set_species(L, lane, x);
    }
    if (SENS && p.scores && channel) L.score((long long)realization_index(p, set, r))[lane] = score;
    g.sync();
}

// A block of direct-method steps (CGP 2006 step 2; model.cu:334-345) from the
// propensities in a[] (pa: the lane's partial sum).  The lanes draw the words
// of a run of steps at once, each its own step's, and hand them out: every
// lane drawing every step's took 20 % of the instructions.
template <class Grp, class Lay, bool SENS>
TL_D void direct_steps(const Grp& g, const SimParams& p, const Lay& L, int set, uint32_t r, float pa,
                       FastState& st) {
    using Pop = typename Lay::Pop;
    constexpr bool kThin = is_thin<Grp>::value;
    if constexpr (std::is_same<Grp, GWarp>::value)
        if (p.M <= 32 && p.N <= 32 && p.t_cp < 0) {
            direct_steps_lanes<Lay, SENS>(g, p, L, set, r, pa, st);
            return;
        }
    const auto qg = queue_group(g);
    const float* rate = p.frates + (size_t)set * p.M;
    U4 w{0u, 0u, 0u, 0u};
    float ex = 0.f;
    for (int q = 0;;) {
        if ((q & (qg.size() - 1)) == 0) {
            w = step_words(L.rk, st.step + (uint32_t)qg.rank(), r, (uint32_t)set);
            ex = -logf(u01f(w.x));
        }
        const int from = q & (qg.size() - 1);
        const uint32_t w_hi = qg.bcast(w.z, from), w_lo = qg.bcast(w.w, from);
        int j;
        float a0;  // total for the waiting time
        if constexpr (kThin) {
            a0 = pa;
            j = thin_select(p, L, pa, w_hi, w_lo);
        } else if constexpr (Grp::kWidth == 0) {
            const double total = g.sumd((double)pa);
            a0 = (float)total;
            j = select_channel<Grp, double>(g, p, L.a(), pa, u01d(w_hi, w_lo) * total, 0);
        } else {
            j = ssa_select(sum_group(g), p, L, pa, w_hi, w_lo, a0);
        }
        // the waiting time in FP32 (FP64 keeps only the time sum)
        const float dtf = qg.bcast(ex, from) / a0;
        const double t_new = st.t + widen(dtf);
        while (st.kpt <= p.n_int && reached(t_new, st.t_next)) record_next(g, p, L, set, r, st);
        if (st.kpt > p.n_int) {
            if (SENS && p.scores) {
                const float rem = (float)(p.t_final[set] - st.t);
                add_scores(g, p, L, set, r, false, [&](int, float a, int) { return -(fabsf(a) * rem); });
            }
            st.done = true;
            g.sync();
            return;
        }
        if (SENS && p.scores)
            add_scores(g, p, L, set, r, false,
                       [&](int m, float a, int) { return (m == j ? 1.f : 0.f) - fabsf(a) * dtf; });
        g.sync();
        if (j >= 0) {
            // the channel's entries, one lane each
            int c0 = j, n = 1;
            if (p.t_cp >= 0) {
                c0 = (int)L.cp()[j];
                n = (int)L.cp()[j + 1] - c0;
            }
            constexpr int kBy = Grp::kWidth == 1 ? 1 : 4;  // lanes
            if (g.rank() < kBy)
#pragma unroll 1
                for (int e = 4 * c0 + g.rank(); e < 4 * (c0 + n); e += kBy) {
                    const uint32_t en = reinterpret_cast<const uint32_t*>(L.col())[e];
                    if (!(en & 0xfffu)) continue;
                    const int i = (int)(en >> 14);
                    const Pop nx = L.x()[i] + (Pop)((int)(en << 20) >> 20);
                    L.x()[i] = nx;
                    set_species(L, i, nx);
                }
        }
        g.sync();
        st.t = t_new;
        st.step++;
        st.ssa++;
        ++q;
        if (q == p.ssa_block || (p.max_steps > 0 && accepted(st.epochs + wrapped(st.step, q), st.step, st.rej) >= p.max_steps)) return;
        float pac;
        fast_props<false>(g, p, L, rate, pa, pac);
        if (!g.any(pa > 0.f)) {
            st.done = true;
            return;
        }
    }
}

template <class Grp, class Lay, bool SENS, bool WIDE>
TL_D void fast_step(const Grp& g, const SimParams& p, const Lay& L, int set, uint32_t r, FastState& st) {
    using Pop = typename Lay::Pop;
    constexpr bool kThin = is_thin<Grp>::value;
    const float* rate = p.frates + (size_t)set * p.M;  // halved for 2S
    float pa, pac;
    // Scores read a critical channel's propensity, and teams form their sums
    // from a[].  Warps and CTAs gain (4000 realizations of the toy network
    // 27.7 -> 27.15 ms, 250 species of the colloid 3.39 -> 3.34 ms), 8 lanes lose
    // (50001 realizations of the 45 x 83 network 77.9 -> 78.7 ms: four realizations
    // share the warp that selects).  16 lanes keep the negative form too, though zeros
    // would gain there (60000 of the toy network 57.8 -> 56.7 ms).
    constexpr bool kZero = !SENS && !WIDE && (Grp::kWidth == 32 || Grp::kWidth == 0);
    fast_props<kZero>(g, p, L, rate, pa, pac);
    float a0f;
    if constexpr (kThin) a0f = pa;
    else a0f = sum_group(g).sumf(pa);
    if (!(a0f > 0.f)) {
        st.done = true;  // nothing can fire: the state holds to t_final
        return;
    }
    float tau1 = fast_tau<kZero>(g, p, L);

    if (!WIDE && tau1 * a0f < p.ssa_factor) {
        if constexpr (kZero) fast_props<false>(g, p, L, rate, pa, pac);
        direct_steps<Grp, Lay, SENS>(g, p, L, set, r, pa, st);
        return;
    }

    if (!WIDE && tau1 * a0f >= kWideLeap && a0f * (float)(st.t_next - st.t) >= kWideLeap) {
        st.wide = true;  // nothing has changed: wide_step starts over
        return;
    }

    // ---- tau-leap with negative-population rejection (CGP 2006 steps 3-5) ----
    double t_new;    // time after the leap (unless clamped to the next grid time)
    float tau_used;  // the leap's tau
    bool clamp;
    float a0cf;
    if constexpr (kThin) a0cf = pac;
    else a0cf = sum_group(g).sumf(pac);
    for (int attempt = 0;; ++attempt) {
        // the step's scalar words are needed only when a channel is critical
        // and each lane draws another step's
        float tau2 = kInfF;
        if (a0cf > 0.f) {
            const auto qg = queue_group(g);
            if (st.step - st.ex_from >= (uint32_t)qg.size()) {
                st.ex_from = st.step;
                st.ex = -logf(u01f(step_words(L.rk, st.step + (uint32_t)qg.rank(), r, (uint32_t)set).x));
            }
            tau2 = qg.bcast(st.ex, (int)(st.step - st.ex_from)) / a0cf;
        }
        float tauf = fminf(tau1, tau2);
        bool fire = tau2 < tau1;
        t_new = st.t + widen(tauf);
        clamp = reached(t_new, st.t_next);
        if (clamp) {
            tauf = (float)(st.t_next - st.t);
            fire = false;
        }
        tau_used = tauf;
        int jc = -1;
        if (fire) {
            const U4 w = step_words(L.rk, st.step, r, (uint32_t)set);
            if constexpr (kThin) {
                const double a0c = (double)pac;
                jc = select_channel<G1, double>(G1{}, p, L.a(), pac, u01d(w.z, w.w) * a0c, 1);
            } else {
                const auto sg = sum_group(g);
                const double a0c = sg.sumd((double)pac);
                const double target = u01d(w.z, w.w) * a0c;
                if constexpr (kZero) jc = select_critical(g, p, L, rate, pac, target);
                else jc = select_channel<std::decay_t<decltype(sum_group(g))>, double>(sg, p, L.a(), pac, target, 1);
            }
        }
        bool over = false, bad;
        if constexpr (WIDE) {
            bad = wide_leap<Grp, Lay, SENS>(g, p, L, tauf, jc, st.step, r, (uint32_t)set, over);
        } else {
            if constexpr (kThin) {
                thin_fire<Lay, SENS>(p, L, tauf, jc, st.step, r, (uint32_t)set);
                g.sync();
                bad = thin_commit(p, L, over);
            } else {
                fast_fire<Grp, Lay, SENS>(g, p, L, tauf, jc, st.step, r, (uint32_t)set);
                g.sync();
                bad = fast_check(g, p, L, over);
                if (!bad) fast_commit(g, p, L);
            }
            if (bad) undo_leap<kZero>(g, p, L);
        }
        if (over) {
            if (g.leader()) atomicOr((unsigned*)(p.ctr + 5), kErrOverflow);
            st.done = true;
            return;
        }
        if (!bad) break;
        // reject: halve tau1, fresh counters, same state and propensities
        st.step++;
        st.rej++;
        tau1 *= 0.5f;
        if (attempt + 1 > p.max_halv) {
            if (g.leader()) atomicOr((unsigned*)(p.ctr + 5), kErrHalving);
            st.done = true;
            return;
        }
    }
    if (SENS && p.scores) {
        // score_j += (k_j - a_j*tau)/c_j with a_j of the pre-leap state
        add_scores(g, p, L, set, r, true, [&](int, float a, int k) { return (float)k - fabsf(a) * tau_used; });
    }
    g.sync();
    st.step++;
    if (clamp) {
        st.t = st.t_next;
        record_next(g, p, L, set, r, st);
        if (st.kpt > p.n_int) st.done = true;
    } else {
        st.t = t_new;
    }
}

// The same step as a wide leap, out of line.
template <class Grp, class Lay, bool SENS>
__device__ __noinline__ void wide_step(const Grp g, const SimParams& p, const Lay L, int set, uint32_t r,
                                       FastState* st) {
    st->wide = false;
    fast_step<Grp, Lay, SENS, true>(g, p, L, set, r, *st);
}

// One realization from x0 to t_final.  The step counts go straight to the
// run's counters (one atomic each), so no totals stay live across the loop.
template <class Grp, class Lay, bool SENS>
TL_D void fast_realization(const Grp& g, const SimParams& p, const Lay& L, long long w) {
    using Pop = typename Lay::Pop;
    const int set = p.S == 1 ? 0 : (int)(w / p.R);
    const uint32_t r = (uint32_t)(p.r_off + w - (long long)set * p.R);
    const Pop* x0 = reinterpret_cast<const Pop*>(p.x0);
#pragma unroll 1
    for (int i = g.rank(); i < ((p.N + 3) & ~3); i += g.size()) {
        L.x()[i] = i < p.N ? x0[i] : (Pop)0;
        L.D()[i] = 0;
    }
    // the padding of a[]: the rest of the last block of four, and the block
    // that the padding of the rows reads
    for (int j = p.M + g.rank(); j < ((p.M + 3) & ~3) + 4; j += g.size()) L.a()[j] = 0.f;
    if (SENS && p.scores)
        for (int j = g.rank(); j < p.M; j += g.size()) L.score(w)[j] = 0.f;
    g.sync();
    fast_refresh(g, p, L);
    fast_record(g, p, L, set, r, 0);
    g.sync();
    FastState st{0.0, grid_time<double>(p, set, 1), 1, 0u, 0u, 0u, 0u, 0u - 32u, 0.f, false, false};  // ex: not drawn yet
    bool trunc = false;
    while (!st.done) {
        const uint32_t from = st.step;
        fast_step<Grp, Lay, SENS, false>(g, p, L, set, r, st);
        if (st.wide) {
            FastState tmp = st;
            wide_step<Grp, Lay, SENS>(g, p, L, set, r, &tmp);
            st = tmp;
        }
        st.epochs += wrapped_past(st.step, from);  // (once a leap or block: counting at each step took 0.7 % on 16 lanes)
        if (!st.done && p.max_steps > 0 && accepted(st.epochs, st.step, st.rej) >= p.max_steps) {
            st.done = true;
            trunc = true;
        }
    }
    // a realization that ends early holds its state on the rest of the grid
#pragma unroll 1
    while (st.kpt <= p.n_int) fast_record(g, p, L, set, r, st.kpt++);
    g.sync();
    if (SENS && p.scores && !p.score_global) {
        float* to = p.scores + realization_index(p, set, r) * p.M;
        for (int j = g.rank(); j < p.M; j += g.size()) to[j] = L.score(0)[j];
    }
    if (g.leader()) {
        const long long leaps = accepted(st.epochs, st.step, st.rej) - (long long)st.ssa;
        if (leaps) atomicAdd(p.ctr + 1, (unsigned long long)leaps);
        if (st.ssa) atomicAdd(p.ctr + 2, (unsigned long long)st.ssa);
        if (st.rej) atomicAdd(p.ctr + 3, (unsigned long long)st.rej);
        if (trunc) atomicAdd(p.ctr + 4, 1ull);
    }
    g.sync();
}

}  // namespace tl
