// tl_tiny.cuh - realizations of small models in the registers of W lanes.
//
// Models of up to W channels and W species (W = 4, 8, 16): lane j holds
// channel j and lane i species i, with its row of the stoichiometry, so that a
// step exchanges values by shuffles and touches no shared memory.  What bounds
// these models is the latency of one realization's chain of dependent steps
// (10^4 realizations keep a tenth of the GPU's warp slots busy), and most of
// that chain was loads: tables, populations and propensities in shared memory
// with a barrier after each pass.  Sums run over the channels in order, as one
// thread forms them, so the results are those of the thread group.
#pragma once

#include "tl_launch.h"
#include "tl_step.cuh"

namespace tl {

template <int W>
struct TinyGroup {
    int lane, base;
    unsigned mask;
    static TL_D TinyGroup make() {
        TinyGroup g;
        const int l = (int)(threadIdx.x & 31);
        g.lane = l & (W - 1);
        g.base = l & ~(W - 1);
        g.mask = ((1u << W) - 1u) << g.base;
        return g;
    }
    template <class T>
    TL_D T from(T v, int src) const {
        return __shfl_sync(mask, v, src, W);
    }
    TL_D bool any(bool p) const { return (__ballot_sync(mask, p) & mask) != 0u; }
    TL_D float minf(float v) const {
#pragma unroll
        for (int o = W / 2; o; o >>= 1) v = fminf(v, __shfl_xor_sync(mask, v, o, W));
        return v;
    }
};

template <int W, class Pop>
struct TinyLane {
    // channel
    int src0, src1, order;
    // species
    float vf[W];          // its row of the stoichiometry
    uint32_t vb[W / 4];   // the same as bytes
    int kind;
    Pop x;
    float xa, xb;         // FP32 x and |x - 1| with the criticalities in the sign

    TL_D int v(int j) const { return (int)(int8_t)(vb[j >> 2] >> (8 * (j & 3))); }
    TL_D void load(const TinyTable* t, int lane) {
        const uint32_t c = t->chan[lane];
        src0 = (int)(c & 0xffu);
        src1 = (int)(c >> 8 & 0xffu);
        order = (int)(c >> 16);
        const uint32_t* row = reinterpret_cast<const uint32_t*>(t->v[lane]);
#pragma unroll
        for (int q = 0; q < W / 4; ++q) vb[q] = row[q];
#pragma unroll
        for (int j = 0; j < W; ++j) vf[j] = (float)v(j);
        kind = (int)t->gkind[lane];
    }
    TL_D void set(Pop nx, int nc) {
        x = nx;
        if ((Pop)(int)nx == nx) {  // int64 -> FP32 runs at the FP64 rate
            const int xi = (int)nx;
            xa = with_sign((float)xi, xi - nc);
            xb = with_sign((float)(xi - 1), xi - 2 * nc);
        } else {
            xa = (float)nx;  // far above any threshold
            xb = (float)(nx - 1);
        }
    }
};

// The state at grid point kpt: the lane of each tracked species writes it.
template <int W, class Pop>
TL_D void tiny_record(const TinyGroup<W>& g, const SimParams& p, const TinyLane<W, Pop>& L, int set, uint32_t r,
                      int kpt) {
    Pop* samp = reinterpret_cast<Pop*>(p.samples) + (realization_index(p, set, r) * (p.n_int + 1) + kpt) * p.K;
#pragma unroll 1
    for (int q = 0; q < p.K; ++q)
        if (__ldg(p.tracked + q) == g.lane) samp[q] = L.x;
}

// The channel at `target` on the running sum over the channels (thin_select);
// crit: over the critical ones only, always on the FP64 target.
template <int W>
TL_D int tiny_select(const float* av, float part, uint32_t w_hi, uint32_t w_lo, bool crit) {
    const float t = ((float)(w_hi >> 6) * 1.4901161193847656e-08f) * part;  // 2^-26
    const float m = 4e-7f * part, above = t + m, below = t - m;
    float acc = 0.f;
    int sel = -1, last = -1;
    bool close = crit;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const float v = fabsf(av[j]);
        acc += v;
        const bool some = v > 0.f;
        close |= some && acc >= below && acc <= above;
        if (some && sel < 0 && acc > above) sel = j;
        if (some) last = j;
    }
    if (close) {
        const float tf = __double2float_rd(u01d(w_hi, w_lo) * (double)part);
        acc = 0.f;
        sel = last = -1;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const float v = crit ? fmaxf(-av[j], 0.f) : fabsf(av[j]);
            acc += v;
            if (v > 0.f && sel < 0 && tf < acc) sel = j;
            if (v > 0.f) last = j;
        }
    }
    return sel >= 0 ? sel : last;
}

template <int W, class Pop, bool SENS>
TL_D void tiny_realization(const TinyGroup<W>& g, const SimParams& p, const uint32_t* rk, TinyLane<W, Pop>& L,
                           long long w_index) {
    const int set = p.S == 1 ? 0 : (int)(w_index / p.R);
    const uint32_t r = (uint32_t)(p.r_off + w_index - (long long)set * p.R);
    const bool channel = g.lane < p.M, species = g.lane < p.N;
    const float rate = channel ? __ldg(p.frates + (size_t)set * p.M + g.lane) : 0.f;  // halved for 2S
    float c = 0.f, score = 0.f;
    if (SENS && p.scores && channel) c = __ldg(p.rates + (size_t)set * p.M + g.lane);
    L.set(species ? reinterpret_cast<const Pop*>(p.x0)[g.lane] : (Pop)0, p.nc);
    tiny_record(g, p, L, set, r, 0);
    double t = 0.0, t_next = grid_time<double>(p, set, 1);
    int kpt = 1;
    uint32_t step = 0, rej = 0, ssa = 0, epochs = 0, last = 0, w_from = 0u - 32u;
    U4 w{0u, 0u, 0u, 0u};  // the lanes hold the scalar words of the steps from w_from
    float ex = 0.f;        // and their waiting times at unit rate
    int ssa_left = 0;
    bool trunc = false;
    // a[] of every channel in every lane, the critical ones negative
    float av[W], aj = 0.f, pa = 0.f, pac = 0.f, tau1 = 0.f;
    const auto words = [&]() {
        if (step - w_from >= (uint32_t)W) {
            w_from = step;
            w = step_words(rk, step + (uint32_t)g.lane, r, (uint32_t)set);
            ex = -logf(u01f(w.x));
        }
    };
    const auto record_next = [&]() {
        tiny_record(g, p, L, set, r, kpt++);
        if (kpt <= p.n_int) t_next = grid_time<double>(p, set, kpt);
    };
    const auto add_score = [&](float term) {
        if (SENS && c > 0.f) score += term / c;
    };
    for (;;) {
        epochs += wrapped_past(step, last);
        last = step;
        if (p.max_steps > 0 && accepted(epochs, step, rej) >= p.max_steps) {
            trunc = true;
            break;
        }
        // propensities and criticalities
        {
            const float f0 = g.from(L.xa, L.src0), f1a = g.from(L.xa, L.src1), f1b = g.from(L.xb, L.src1);
            const float f1 = L.order == 2 ? f1a : L.order == 3 ? f1b : 1.f;
            const float e0 = L.order == 0 ? 1.f : f0;
            const float v = rate * fabsf(e0) * fabsf(f1);
            aj = __uint_as_float(__float_as_uint(v) | ((__float_as_uint(e0) | __float_as_uint(f1)) & 0x80000000u));
        }
        pa = pac = 0.f;
#pragma unroll
        for (int j = 0; j < W; ++j) av[j] = g.from(aj, j);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            pa += fabsf(av[j]);
            pac += fmaxf(-av[j], 0.f);
        }
        if (!(pa > 0.f)) break;  // nothing can fire: the state holds to t_final
        if (ssa_left == 0) {
            float mu = 0.f, s2 = 0.f;
#pragma unroll
            for (int j = 0; j < W; ++j)  // no entry: 0, whatever the propensity
                add_moments(L.vf[j], L.vf[j] != 0.f ? fmaxf(av[j], 0.f) : 0.f, mu, s2);
            tau1 = g.minf(L.kind ? row_bound(p, fabsf(L.xa), L.kind, mu, s2) : kInfF);
            if (tau1 * pa < p.ssa_factor) ssa_left = p.ssa_block;
        }
        if (ssa_left > 0) {
            // ---- direct-method step ----
            words();
            const int from = (int)(step - w_from);
            const int j = tiny_select<W>(av, pa, g.from(w.z, from), g.from(w.w, from), false);
            const float dt = g.from(ex, from) / pa;
            const double t_new = t + widen(dt);
            while (kpt <= p.n_int && reached(t_new, t_next)) record_next();
            if (kpt > p.n_int) {
                const float rem = (float)(p.t_final[set] - t);
                add_score(-(fabsf(aj) * rem));
                break;
            }
            add_score((g.lane == j ? 1.f : 0.f) - fabsf(aj) * dt);
            int d = 0;
#pragma unroll
            for (int q = 0; q < W; ++q) d = q == j ? L.v(q) : d;
            L.set(L.x + (Pop)d, p.nc);
            t = t_new;
            ++step;
            ++ssa;
            --ssa_left;
            continue;
        }
        // ---- tau-leap with negative-population rejection ----
        double t_new;
        float tauf;
        bool clamp, stop = false;
        int k;
        long long nx;
        for (int attempt = 0;; ++attempt) {
            float tau2 = kInfF;
            if (pac > 0.f) {
                words();
                tau2 = g.from(ex, (int)(step - w_from)) / pac;
            }
            tauf = fminf(tau1, tau2);
            bool fire = tau2 < tau1;
            t_new = t + widen(tauf);
            clamp = reached(t_new, t_next);
            if (clamp) {
                tauf = (float)(t_next - t);
                fire = false;
            }
            int jc = -1;
            if (fire) {
                const int from = (int)(step - w_from);
                jc = tiny_select<W>(av, pac, g.from(w.z, from), g.from(w.w, from), true);
            }
            k = channel ? poisson_channel(aj, tauf, g.lane, jc, step, r, (uint32_t)set, rk) : 0;
            long long d = 0;
#pragma unroll
            for (int j = 0; j < W; ++j) d += (long long)L.v(j) * (long long)g.from(k, j);
            nx = (long long)L.x + d;
            const bool of = sizeof(Pop) == 4 && nx > 2147483647LL;
            if (g.any(of)) {
                if (g.lane == 0) atomicOr((unsigned*)(p.ctr + 5), kErrOverflow);
                stop = true;
                break;
            }
            if (!g.any(nx < 0)) break;
            // reject: halve tau1, fresh counters, same state and propensities
            ++step;
            ++rej;
            tau1 *= 0.5f;
            if (attempt + 1 > p.max_halv) {
                if (g.lane == 0) atomicOr((unsigned*)(p.ctr + 5), kErrHalving);
                stop = true;
                break;
            }
        }
        if (stop) break;
        add_score((float)k - fabsf(aj) * tauf);
        L.set((Pop)nx, p.nc);
        ++step;
        if (clamp) {
            t = t_next;
            record_next();
            if (kpt > p.n_int) break;
        } else {
            t = t_new;
        }
    }
    // a realization that ends early holds its state on the rest of the grid
#pragma unroll 1
    while (kpt <= p.n_int) tiny_record(g, p, L, set, r, kpt++);
    if (SENS && p.scores && channel) p.scores[realization_index(p, set, r) * p.M + g.lane] = score;
    if (g.lane == 0) {
        const long long leaps = accepted(epochs + wrapped_past(step, last), step, rej) - (long long)ssa;
        if (leaps) atomicAdd(p.ctr + 1, (unsigned long long)leaps);
        if (ssa) atomicAdd(p.ctr + 2, (unsigned long long)ssa);
        if (rej) atomicAdd(p.ctr + 3, (unsigned long long)rej);
        if (trunc) atomicAdd(p.ctr + 4, 1ull);
    }
}

}  // namespace tl
