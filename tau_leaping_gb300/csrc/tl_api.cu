// tl_api.cu - the C ABI (include/tl.h): model upload, run configuration,
// the autotuner, kernel launches and result reduction.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "tl_device.cuh"
#include "tl_internal.h"
#include "tl_launch.h"
#include "tl_shared.h"

namespace tl {

static thread_local std::string g_last_error;
static thread_local int g_device = 0;

void set_last_error(const std::string& s) { g_last_error = s; }

static tl_status cuda_fail(cudaError_t e, const char* what) {
    set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
    cudaGetLastError();  // clear a non-sticky error
    return e == cudaErrorMemoryAllocation ? TL_ERR_OUT_OF_MEMORY
           : e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver ? TL_ERR_NO_DEVICE
                                                                          : TL_ERR_CUDA;
}

#define TLC(expr)                                          \
    do {                                                   \
        cudaError_t _e = (expr);                           \
        if (_e != cudaSuccess) return cuda_fail(_e, #expr); \
    } while (0)

static size_t al16(size_t b) { return (b + 15) & ~(size_t)15; }

// Grow-only device scratch owned by the model.
static tl_status scratch_get(tl_model* m, size_t bytes, void** out) {
    if (bytes > m->scratch_bytes) {
        if (m->scratch) cudaFree(m->scratch);
        m->scratch = nullptr;
        m->scratch_bytes = 0;
        TLC(cudaMalloc(&m->scratch, bytes));
        m->scratch_bytes = bytes;
    }
    *out = m->scratch;
    return TL_OK;
}

struct Carver {
    size_t off = 0;
    size_t take(size_t b) {
        const size_t o = off;
        off = (off + b + 255) & ~(size_t)255;
        return o;
    }
};

// Whether halving a rate is exact: not near FP32's ends.
static bool halves_exactly(float c) { return c == 0.f || (c >= 7.8886e-31f && c <= 1.1529e18f); }

// One set's rates in FP32, as given and halved for 2S channels (the fast
// builds).  False where halving might not be exact.
static bool fill_rates(const HostModel& h, const double* c, float* plain, float* halved) {
    bool exact = true;
    for (int j = 0; j < h.M; ++j) {
        const float cf = (float)c[j];
        const bool twice = h.order[(size_t)j] == 3;
        if (plain) plain[j] = cf;
        if (halved) halved[j] = twice ? 0.5f * cf : cf;
        if (twice && !halves_exactly(cf)) exact = false;
    }
    return exact;
}

// Tables of the fast and scores builds, in the layout tl_step.cuh reads:
//  chan  per channel the byte offsets in X of its two factors: 16 bits each,
//        or 32 where X is past 64 KB
//  row   per reacting species, longest row first: {first chunk | chunks << 20,
//        species | g kind << 28}, a chunk being four entries
//  ent   row entries: byte offset in a[] << 12 | the stoichiometry's FP32 bits
//        >> 20, from 2^18 channels on (col << 3) | ((v + 2) & 7); padding
//        reads the zero block behind the last channel
//  col   per channel, chunks of four net entries: byte offset of the species
//        in an int array << 12 | stoichiometry & 0xfff, 0 stoichiometry = none
//  cp    first chunk of each channel, where a channel needs more than one
//        (col and cp hold whole blocks of four channels, as a[] does: the
//        firing pass may mark a channel of the padding, which has no entries)
//  sp    per species the index in X of its |x - 1|, 0 if it has none
//  tiny  a TinyTable, for models of up to 16 channels and species
static void fast_layout(const HostModel& h, DevModel& d) {
    const int N = h.N, M = h.M;
    d.x2.assign((size_t)N, 0);
    d.n_2s = 0;
    for (int j = 0; j < M; ++j)
        if (h.order[(size_t)j] == 3 && !d.x2[(size_t)h.s0[(size_t)j]]) {
            d.x2[(size_t)h.s0[(size_t)j]] = 1;
            ++d.n_2s;
        }
    const int Np = (N + 3) & ~3;  // X pads the species to whole blocks of four
    int next = Np;
    for (int i = 0; i < N; ++i)
        if (d.x2[(size_t)i]) d.x2[(size_t)i] = next++;
    const int one = Np + d.n_2s;
    const int pad = (M + 3) & ~3;  // the zero block behind a[]
    d.chan8 = (size_t)one * 4 > 0xffff;
    d.ent_wide = M + 8 > (1 << 18);
    d.fast_ok = false;
    if (N >= (1 << 18) || next > 0xffff || M >= (1 << 28) - 8) return;
    size_t ent_chunks = 0, col_chunks = 0;
    int max_chunks = 0, max_col = 0;
    for (int i = 0; i < N; ++i) {
        const int n = (h.net_rp[(size_t)i + 1] - h.net_rp[(size_t)i] + 3) / 4;
        if (h.gkind[(size_t)i]) ent_chunks += (size_t)n;
        max_chunks = std::max(max_chunks, n);
    }
    for (int j = 0; j < M; ++j) max_col = std::max(max_col, h.net_cp[(size_t)j + 1] - h.net_cp[(size_t)j]);
    if (ent_chunks >= (1u << 20) || max_chunks >= (1 << 12)) return;
    for (int j = 0; j < M; ++j)
        col_chunks += (size_t)(h.net_cp[(size_t)j + 1] - h.net_cp[(size_t)j] + 3) / 4;
    d.n_rows = 0;
    for (int i = 0; i < N; ++i) d.n_rows += h.gkind[(size_t)i] != 0;
    if (max_col <= 4) col_chunks = (size_t)pad;
    size_t off = 0;
    const auto sect = [&](size_t bytes) {
        const size_t o = off;
        off += al16(bytes);
        return (int)o;
    };
    d.t_chan = sect((size_t)M * (d.chan8 ? 8 : 4));
    d.t_row = sect((size_t)d.n_rows * 8);
    d.t_ent = sect(ent_chunks * 16);
    d.t_col = sect(col_chunks * 16);
    d.t_cp = max_col > 4 ? sect((size_t)(pad + 1) * 4) : -1;
    d.t_sp = sect((size_t)Np * 2);
    const bool tiny = N <= 16 && M <= 16;
    d.t_tiny = tiny ? sect(sizeof(TinyTable)) : 0;
    if (off >= (1u << 31)) return;
    d.f_stage_bytes = (int)std::max<size_t>(off, 16);
    d.fast_ok = true;
}

void fast_tables(const HostModel& h, DevModel& d, std::vector<unsigned char>& out) {
    if (!d.fast_ok) fast_layout(h, d);
    if (!d.fast_ok) return;
    const int N = h.N, M = h.M;
    const std::vector<int>& x2 = d.x2;
    const int one = ((N + 3) & ~3) + d.n_2s, pad = (M + 3) & ~3;
    const bool tiny = N <= 16 && M <= 16;
    out.assign((size_t)d.f_stage_bytes, 0);
    uint32_t* chan = reinterpret_cast<uint32_t*>(out.data() + d.t_chan);
    for (int j = 0; j < M; ++j) {
        const int o = h.order[(size_t)j], s0 = h.s0[(size_t)j], s1 = h.s1[(size_t)j];
        const uint32_t f0 = 4u * (uint32_t)(o == 0 ? one : s0);
        const uint32_t f1 = 4u * (uint32_t)(o == 2 ? s1 : o == 3 ? x2[(size_t)s0] : one);
        if (d.chan8) {
            chan[2 * (size_t)j] = f0;
            chan[2 * (size_t)j + 1] = f1;
        } else {
            chan[j] = f0 | f1 << 16;
        }
    }
    uint32_t* row = reinterpret_cast<uint32_t*>(out.data() + d.t_row);
    uint32_t* ent = reinterpret_cast<uint32_t*>(out.data() + d.t_ent);
    // a packed entry's low bits (v + 2) & 7 -> the stoichiometry's FP32 bits >> 20, and its 12 bits
    uint32_t vf[8], vi[8];
    for (int b = 0; b < 8; ++b) {
        const float f = (float)unpack_v(b);
        memcpy(&vf[b], &f, 4);
        vf[b] >>= 20;
        vi[b] = (uint32_t)unpack_v(b) & 0xfffu;
    }
    size_t e = 0;
    int nr = 0;
    for (int ii = 0; ii < N; ++ii) {
        const int i = h.rowperm[(size_t)ii];
        if (!h.gkind[(size_t)i]) continue;
        const int q0 = h.net_rp[(size_t)i], n = h.net_rp[(size_t)i + 1] - q0, chunks = (n + 3) / 4;
        const int32_t* const vc = h.net_vc.data() + q0;
        row[2 * nr] = (uint32_t)(e / 4) | (uint32_t)chunks << 20;
        row[2 * nr + 1] = (uint32_t)i | (uint32_t)h.gkind[(size_t)i] << 28;
        ++nr;
        uint32_t* const to = ent + e;
        if (d.ent_wide)
            for (int q = 0; q < n; ++q) to[q] = (uint32_t)vc[q];
        else
            for (int q = 0; q < n; ++q) to[q] = (uint32_t)(vc[q] >> 3) << 14 | vf[vc[q] & 7];
        for (int q = n; q < 4 * chunks; ++q) to[q] = d.ent_wide ? (uint32_t)pad << 3 | 2u : (uint32_t)pad << 14;
        e += 4 * (size_t)chunks;
    }
    uint32_t* col = reinterpret_cast<uint32_t*>(out.data() + d.t_col);
    uint32_t* cp = d.t_cp >= 0 ? reinterpret_cast<uint32_t*>(out.data() + d.t_cp) : nullptr;
    size_t c4 = 0;
    const int32_t* const rv = h.net_rv.data();
    for (int j = 0; j < M; ++j) {
        const int q0 = h.net_cp[(size_t)j], n = h.net_cp[(size_t)j + 1] - q0;
        if (cp) cp[j] = (uint32_t)c4;
        for (int q = 0; q < n; ++q) col[4 * c4 + (size_t)q] = (uint32_t)(rv[q0 + q] >> 3) << 14 | vi[rv[q0 + q] & 7];
        c4 += cp ? (size_t)(n + 3) / 4 : 1;
    }
    if (cp) std::fill(cp + M, cp + pad + 1, (uint32_t)c4);
    unsigned short* sp = reinterpret_cast<unsigned short*>(out.data() + d.t_sp);
    for (int i = 0; i < N; ++i) sp[i] = (unsigned short)x2[(size_t)i];
    if (tiny) {
        TinyTable* tt = reinterpret_cast<TinyTable*>(out.data() + d.t_tiny);
        for (int j = 0; j < M; ++j) {
            tt->chan[j] = (uint32_t)h.s0[(size_t)j] | (uint32_t)h.s1[(size_t)j] << 8 | (uint32_t)h.order[(size_t)j] << 16;
            for (int q = h.net_cp[(size_t)j]; q < h.net_cp[(size_t)j + 1]; ++q)
                tt->v[unpack_idx(h.net_rv[(size_t)q])][j] = (int8_t)unpack_v(h.net_rv[(size_t)q]);
        }
        for (int i = 0; i < N; ++i) tt->gkind[i] = (uint8_t)h.gkind[(size_t)i];
    }
}

// Tables of the general build and the parity entry points:
// [chan][ref order][gkind][perm][net rp][net vc][net cp][net rv] | [raw rp][raw vc]
static void general_layout(const HostModel& h, DevModel& d) {
    const size_t N = (size_t)h.N, M = (size_t)h.M;
    d.nnz_net = (int)h.net_vc.size();
    d.nnz_raw = (int)h.raw_vc.size();
    size_t off = 0;
    auto sect = [&](size_t bytes) {
        const size_t o = off;
        off += al16(bytes);
        return (int)o;
    };
    d.off_chan = sect(M * 8);
    d.off_rord = sect(M);
    d.off_gkind = sect(N);
    d.off_perm = sect(N * 4);
    d.off_rp = sect((N + 1) * 4);
    d.off_vc = sect((size_t)d.nnz_net * 4);
    d.off_cp = sect((M + 1) * 4);
    d.off_rv = sect((size_t)d.nnz_net * 4);
    d.stage_bytes = (int)off;
    d.off_raw_rp = sect((N + 1) * 4);
    d.off_raw_vc = sect((size_t)d.nnz_raw * 4);
    d.blob_bytes = off;
}

static void general_tables(const HostModel& h, const DevModel& d, std::vector<unsigned char>& hb) {
    const size_t N = (size_t)h.N, M = (size_t)h.M;
    hb.assign(d.blob_bytes, 0);
    // channel record: {s0, s1 | order << 28} (species indices < 2^28)
    int2* chan = reinterpret_cast<int2*>(hb.data() + d.off_chan);
    for (size_t j = 0; j < M; ++j) chan[j] = make_int2(h.s0[j], h.s1[j] | ((int)h.order[j] << 28));
    memcpy(hb.data() + d.off_rord, h.ref_order.data(), M);
    memcpy(hb.data() + d.off_gkind, h.gkind.data(), N);
    memcpy(hb.data() + d.off_perm, h.rowperm.data(), N * 4);
    memcpy(hb.data() + d.off_rp, h.net_rp.data(), (N + 1) * 4);
    if (d.nnz_net) memcpy(hb.data() + d.off_vc, h.net_vc.data(), (size_t)d.nnz_net * 4);
    memcpy(hb.data() + d.off_cp, h.net_cp.data(), (M + 1) * 4);
    if (d.nnz_net) memcpy(hb.data() + d.off_rv, h.net_rv.data(), (size_t)d.nnz_net * 4);
    memcpy(hb.data() + d.off_raw_rp, h.raw_rp.data(), (N + 1) * 4);
    if (d.nnz_raw) memcpy(hb.data() + d.off_raw_vc, h.raw_vc.data(), (size_t)d.nnz_raw * 4);
}

// The tables that a launch reads, on the device: each set is built and sent when
// the first such launch comes.  The memory of both is there from the first
// call on (upload), so the static entry allocates nothing here either.  First
// call of a model on GB300, ms, both sets at once -> so (and the general one
// alone, before there were two): colloid of 400 species, simulate 1.82 -> 1.04
// (0.88), on the general build 1.83 -> 0.90 (0.88), replay 2.09 -> 1.08 (0.97).
static tl_status ensure_tables(tl_model* m, bool general, bool fast, cudaStream_t st) {
    DevModel& d = m->d;
    for (const bool f : {false, true}) {
        bool& sent = f ? d.fast_sent : d.general_sent;
        if (sent || !(f ? fast && d.fast_ok : general)) continue;
        std::vector<unsigned char> hb;
        if (f) fast_tables(m->h, d, hb);
        else general_tables(m->h, d, hb);
        TLC(cudaMemcpyAsync(f ? d.fblob : d.blob, hb.data(), hb.size(), cudaMemcpyHostToDevice, st));
        TLC(cudaStreamSynchronize(st));  // hb ends here
        sent = true;
    }
    return TL_OK;
}

// The device memory of a model, its populations and rates.
static tl_status upload(tl_model* m) {
    HostModel& h = m->h;
    DevModel& d = m->d;
    const int N = h.N, M = h.M;
    general_layout(h, d);
    fast_layout(h, d);
    TLC(cudaMalloc(&d.blob, d.blob_bytes + (d.fast_ok ? (size_t)d.f_stage_bytes : 0)));
    d.fblob = d.blob + d.blob_bytes;
    const size_t w = h.pop_bits == 64 ? 8 : 4;
    TLC(cudaMalloc(&d.x0, (size_t)N * w));
    if (w == 8) {
        std::vector<long long> x(h.x0.begin(), h.x0.end());
        TLC(cudaMemcpy(d.x0, x.data(), (size_t)N * 8, cudaMemcpyHostToDevice));
    } else {
        std::vector<int> x(h.x0.begin(), h.x0.end());
        TLC(cudaMemcpy(d.x0, x.data(), (size_t)N * 4, cudaMemcpyHostToDevice));
    }
    std::vector<float> r(2 * (size_t)M);
    d.halvable = fill_rates(h, h.rate.data(), r.data(), r.data() + M);
    TLC(cudaMalloc(&d.rate, r.size() * 4));
    TLC(cudaMemcpy(d.rate, r.data(), r.size() * 4, cudaMemcpyHostToDevice));
    return TL_OK;
}

static tl_status finish_model(tl_model* m, tl_model** out) {
    std::string err;
    tl_status s = derive_tables(m->h, err);
    if (s != TL_OK) {
        set_last_error(err);
        delete m;
        return s;
    }
    m->d.device = g_device;  // device tables are uploaded on first use
    *out = m;
    return TL_OK;
}

static tl_status ensure_device(tl_model* m) {
    if (m->d.blob) return TL_OK;
    TLC(cudaSetDevice(m->d.device));
    return upload(m);
}

static MView global_view(const tl_model* m, bool raw_mu, bool raw_update) {
    const DevModel& d = m->d;
    const unsigned char* b = d.blob;
    MView v;
    v.chan = reinterpret_cast<const int2*>(b + d.off_chan);
    v.rord = reinterpret_cast<const signed char*>(b + d.off_rord);
    v.gkind = reinterpret_cast<const signed char*>(b + d.off_gkind);
    v.perm = reinterpret_cast<const int*>(b + d.off_perm);
    const int* nrp = reinterpret_cast<const int*>(b + d.off_rp);
    const int* nvc = reinterpret_cast<const int*>(b + d.off_vc);
    const int* rrp = reinterpret_cast<const int*>(b + d.off_raw_rp);
    const int* rvc = reinterpret_cast<const int*>(b + d.off_raw_vc);
    v.rp = raw_mu ? rrp : nrp;
    v.vc = raw_mu ? rvc : nvc;
    v.urp = raw_update ? rrp : nrp;
    v.uvc = raw_update ? rvc : nvc;
    v.cp = reinterpret_cast<const int*>(b + d.off_cp);
    v.rv = reinterpret_cast<const int*>(b + d.off_rv);
    return v;
}

// One group's slot: x, x' and a[]; scored runs add the firing counts.
static size_t slot_bytes(const tl_model* m, bool sens = false) {
    const size_t w = m->h.pop_bits == 64 ? 8 : 4;
    return al16((size_t)m->h.N * w) * 2 + al16((size_t)m->h.M * 4) * (sens ? 2 : 1);
}

// The slot of the fast and scores builds (tl_step.cuh): the state x, D and X,
// with the queue of long draws over X, then a[] and in scored runs the counts
// and, where they fit, the scores.  The queue takes a 16-bit channel for each
// of the four channels that a lane may mark in one turn, times the turns
// between two drains: enough for a whole leap of models up to 28 channels a
// lane, whose few long draws then fill one pass; four for wide CTA groups,
// where 128 channels a turn and warp fill a pass sooner.
struct SlotLayout {
    size_t bytes = 0;  // the whole slot
    size_t state = 0;  // its state part
    int f_D = 0, f_X = 0, f_a = 0;
    int q_rounds = 0;
    bool score_global = false;
};

static SlotLayout slot_layout(const tl_model* m, bool sens, int mode, int kind, int block, int most_rounds = kMaxRounds) {
    SlotLayout L;
    const int N = m->h.N, M = m->h.M;
    if (mode == kModeGeneral) {
        L.bytes = slot_bytes(m, sens);
        return L;
    }
    const size_t w = m->h.pop_bits == 64 ? 8 : 4;
    size_t q_bytes = 0;
    if (kind != 1) {
        const int lanes = kind ? kind : block;
        const int turns = (M + 4 * lanes - 1) / (4 * lanes);
        L.q_rounds = std::min({turns, lanes > 256 ? 4 : kMaxRounds, most_rounds});
        q_bytes = (size_t)L.q_rounds * lanes * 4 * 2 + 4 * (size_t)(kind ? 1 : block / 32);  // and a counter each
    }
    const size_t Np = ((size_t)N + 3) & ~(size_t)3;  // whole blocks of four species
    L.f_D = (int)(Np * w);
    L.f_X = L.f_D + (int)(Np * 4);
    L.state = (size_t)L.f_X + al16(std::max((Np + (size_t)m->d.n_2s + 1) * 4, q_bytes));
    L.f_a = ((M + 3) / 4 * 4 + 4) * 4;
    L.bytes = L.state + (size_t)L.f_a * (mode == kModeScores ? 3 : 1);
    return L;
}

static int max_smem_optin() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v > 0 ? v : 48 * 1024;
}

static int sm_count() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
}

// Launch plan for the fused kernel.
struct Plan {
    int kind = 32;      // 1, 32, 0
    int block = 256;
    int grid = 1;
    size_t smem = 0;
    int stage = 0;      // staged bytes (0 = constants read through L1/L2)
    int variant = TL_VARIANT_WARP;
    bool row_warp = false;
    bool gslot = false;  // CTA groups: the slot lives in global memory
    int mode = kModeFast;  // the kernel build
    int lanes = 32;        // thread groups: lanes of a warp that take realizations
    int thin = 1;          // and lanes of one realization
    bool state_global = false;  // global slots: the state as well as a[]
    bool batch = false;
    bool team = false;     // warp groups: four warps per realization
    SlotLayout slot;
};

// The kernel a plan launches (CTA groups with global slots are their own build).
static int launch_kind(const Plan& pl) {
    if (pl.gslot) return kKindCtaGlobal;
    if (pl.team) return kKindTeam;
    if (pl.kind == 1 && pl.mode != kModeGeneral) return 100 + pl.thin;
    return pl.kind;
}

// Autotuner, heuristic part: the group width follows the model size.
//  * a handful of channels: one realization per thread (all lanes busy on
//    independent realizations); small ensembles use small blocks so that
//    every SM gets work;
//  * per-realization state up to 8 KB: a group of W lanes of a warp per
//    realization, 256-thread blocks, model tables staged in shared memory.
//    W is the smallest of 8, 16 and 32 that leaves each lane at most 16
//    channels and 8 species rows, provided the ensemble fills the GPU's
//    warp-group slots at least 8 times over (smaller ensembles keep whole
//    warps, whose realizations finish sooner); scored runs keep whole warps
//    (the sub-warp kinds have no scores-only build).  Measured on GB300 over
//    eight model sizes: 32-channel chain 8 lanes 9.8e8 against a warp 4.3e8,
//    32 x 64 network 8 lanes 9.6e8 against 6.9e8, the 128 x 256 toy network
//    16 lanes 3.64e8 against 3.50e8, 128-channel chain 16 lanes = warp,
//    256 x 512 network and the 40-species colloid a warp;
//  * up to 64 KB: one 128-thread (up to 1024 channels) or 256-thread CTA per
//    realization, tables through L1/L2 (chain-sized models: 1024 species
//    and channels);
//  * larger: one 1024-thread CTA per realization (propensities of ~30k
//    channels fill most of the 227 KB of shared memory).
// The choices follow sweeps of the (variant, block, staging) plans on GB300.
static int heuristic_variant(const tl_model* m, size_t sb, long long total, int mode, int nsm) {
    const int M = m->h.M, N = m->h.N;
    if (M <= 16 && N <= 16) return TL_VARIANT_THREAD;
    if (sb > 8 * 1024) return TL_VARIANT_CTA;
    // warp groups: 256-thread CTAs, 5 per SM
    constexpr long long kWarpGroupsPerSm = 40;
    if (mode != kModeScores && total >= 8 * kWarpGroupsPerSm * (long long)nsm) {
        if (M <= 16 * 8 && N <= 8 * 8) return TL_VARIANT_LANES8;
        if (M <= 16 * 16 && N <= 8 * 16) return TL_VARIANT_LANES16;
    }
    return TL_VARIANT_WARP;
}

// What a plan depends on besides the model and the launch: the leap condition's
// eps and the time between two grid points.
struct LeapScale {
    double eps = 0.03, dt = 1.0;
};

// Whether most draws of a leap have means of 10 and more (PTRS), by the first
// leap from x0 at the model's own rates: the mean of channel j is a_j times the CGP
// bound or dt.
static bool mostly_long_draws(const HostModel& h, const LeapScale& ls) {
    const int M = h.M, N = h.N;
    std::vector<double> a((size_t)M);
    const auto pop = [&](int i) { return (double)h.x0[(size_t)i]; };
    for (int j = 0; j < M; ++j) {
        const int o = h.order[(size_t)j], s0 = h.s0[(size_t)j], s1 = h.s1[(size_t)j];
        a[(size_t)j] = h.rate[(size_t)j] * (o == 0 ? 1.0 : o == 1 ? pop(s0) : o == 2 ? pop(s0) * pop(s1) : pop(s0) * (pop(s0) - 1.0) * 0.5);
    }
    double tau = ls.dt;
    for (int i = 0; i < N; ++i) {
        if (!h.gkind[(size_t)i]) continue;
        double mu = 0.0, s2 = 0.0;
        for (int q = h.net_rp[(size_t)i]; q < h.net_rp[(size_t)i + 1]; ++q) {
            const double v = unpack_v(h.net_vc[(size_t)q]), t = v * a[(size_t)unpack_idx(h.net_vc[(size_t)q])];
            mu += t;
            s2 += v * t;
        }
        const double num = std::max(ls.eps * pop(i) / (h.gkind[(size_t)i] == 1 ? 1.0 : 2.0), 1.0);
        if (mu != 0.0) tau = std::min(tau, num / std::fabs(mu));
        if (s2 > 0.0) tau = std::min(tau, num * num / s2);
    }
    int many = 0;
    for (int j = 0; j < M; ++j) many += a[(size_t)j] * tau >= 10.0;
    return 4 * many >= 3 * M;
}

// Thread-group plans of a model of `size` channels or species at most: lanes
// per realization (W; 1: thread groups on shared memory, else tl_tiny.cuh), and
// lanes of each warp that take realizations.  One realization's chain of
// dependent steps sets the time of small and mid-sized ensembles, so W lanes
// share its draws until the ensemble is `most` warps per SM; past that the
// lanes do more as W realizations.  And the
// realizations of a warp lengthen one another's chains (they sit in different
// steps, branches and draws), so small ensembles leave lanes idle.  Measured on
// GB300 (ms; the last row: shared memory, four lanes, before tl_tiny.cuh):
//   dimer decay, t = 10   32    1000   3000   10000  30000  100000
//   W = 4, 32 lanes      1.96   1.97   1.98    2.23   3.28    9.91
//   W = 4, 8 lanes       1.36   1.38   1.59    3.38   8.49   26.3
//   W = 4, 4 lanes       1.16   1.24   1.72    5.09  14.1    45.4
//   W = 1, 32 lanes      4.39   4.44   4.45    4.45   4.89    8.12
//   shared, 32 lanes     3.08   3.11   3.12    3.45   6.94   15.9
// and a 12 x 16 network in direct-method steps, W = 16 against 1: 1.29 against
// 5.38 at 32, 4.67 against 6.91 at 10000, 20.0 against 8.03 at 50000.
static void thin_plan(int size, long long total, int nsm, long long most, int& thin, int& lanes) {
    thin = size <= 4 ? 4 : size <= 8 ? 8 : size <= 16 ? 16 : 1;
    if (total * thin > most * 32 * nsm) thin = 1;
    lanes = 32;
    if (thin > 1)
        while (lanes > thin && total * 2 * thin <= (thin == 4 ? 10LL : 3LL) * nsm * lanes) lanes /= 2;
}

// `most` for an ensemble of its own.  W = 8 and 16: some 56, more than twice the
// 24 that are resident.  W = 4: little more than one wave of them, since
// one lane needs only 4 times the steps of four.  Dimer decay, ms, W = 4 and 1
// (and one thread of the build before them): to t = 5e-4, 30000 realizations 0.80
// and 0.94 (1.00), 35000 1.07 and 0.95 (1.01), 60000 1.44 and 1.17 (1.17); t = 1,
// 30000 1.85 and 2.44 (2.74), 40000 2.67 and 2.67 (3.02), 60000 3.38 and 3.00 (3.43);
// t = 4, 40000 3.32 and 3.54 (4.24), 60000 4.21 and 3.99 (4.85).  Not where nearly
// every draw is long, which four lanes share well: cyclic chain of 4 species,
// 60000 realizations of 8 steps 0.098 and 0.122 (0.141).
static long long thin_most_warps(const HostModel& h, const LeapScale& ls) {
    return std::max(h.N, h.M) > 4 || mostly_long_draws(h, ls) ? 56 : 28;
}

// And for a batch, whose kernel has 16 warps resident.  Sets of the dimer decay
// alone, ms, W = 4 and 1: 48000 realizations to t = 0.01 1.83 and 2.10, t = 1 2.98 and
// 3.58; 65536 2.56 and 2.13, 4.17 and 3.58; with scores 2.70 and 2.71, 4.34 and 4.36;
// beside 4 x 700 toy realizations 6.63 and 6.41, 8.22 and 8.87.
static long long thin_most_warps_batch(int size, bool small_only, bool scores) {
    return size <= 4 && small_only && !scores ? 48 : 56;
}

// Four-warp teams for a warp-group ensemble of up to eight realizations an SM:
// enough channels for 128 threads, and a chain of steps that sets the time.
// Measured on GB300, toy network (128 x 256) to t = 0.002, ms, one warp a
// realization -> a team: 10.9 -> 6.1 at 152 realizations, 10.9 -> 8.5 at 1216;
// above eight realizations an SM the warps still run in one wave and a team no
// longer does.
static bool team_pays(const tl_model* m, long long total, int nsm) {
    return m->h.M >= 128 && total <= 8LL * nsm;
}

// Threads per CTA of a warp or sub-warp ensemble that runs in one wave.  The SM
// with the most warps ends last, and CTAs of eight warps share out unevenly:
// 500 of them put 32 warps on 44 of 152 SMs and 24 on the others.  Of 8 to 4
// warps a CTA (an SM has four schedulers, and each CTA stages the tables) the
// largest with the fewest warps on the fullest SM.  Measured on GB300, kernel
// ms, 256 threads -> this rule: toy network (128 x 256) to t = 0.002, 1500
// realizations 15.97 -> 14.88 (192), 2600 20.06 -> 17.77 (192), 3300 the same
// (256), 4000 25.51 -> 23.31 (224); 12 x 20 network in direct-method steps, 4000
// 1.270 -> 1.165; 45 x 83 network 13.91 -> 12.75.  Two or three warps a CTA
// saved another warp an SM and were 1-3 % slower; with several waves the sizes
// differ by +-2 % either way, and 256 stays.
static int even_block(long long total, int groups_per_warp, int nsm, int most_warps) {
    const long long warps = (total + groups_per_warp - 1) / groups_per_warp;
    int best = most_warps;
    long long most = 0;
    for (int w = most_warps; w >= 4; --w) {
        const long long ctas = (warps + w - 1) / w, full = (ctas + nsm - 1) / nsm * w;
        if (w == most_warps || full < most) {
            best = w;
            most = full;
        }
    }
    return 32 * best;
}

// Lane groups of 2 to 16 lanes that the general build runs faster.  The fast
// build's queue of long draws is one per group, and the groups of a warp drain
// theirs one after another: what 32 and 16 lanes gain, 2 to 8 lose where nearly
// every draw is long or one drain does not hold a leap.  Measured on GB300, ms,
// fast -> general build:
//   8 lanes, cyclic chains, 50 000 realizations: 32 species 0.507 -> 0.333 (int64
//     0.558 -> 0.358), 17 species 0.415 -> 0.306, 64 species 0.96 -> 0.79; networks
//     of 20 to 256 channels, up to 45 % long draws, 1.3 to 1.9 times faster on the fast one
//   16 lanes: chains of 96 to 256 species 1.1 to 1.3 times faster on the fast
//     build, 1024 species 17.4 -> 12.7 (30 000 realizations)
//   4 lanes, 4000 realizations: 64 x 128 network 4.77 against 8.83, 96 x 192 5.37 -> 3.00,
//     128 x 256 31.8 -> 16.9
//   2 lanes: dimer decay 0.80 -> 0.55, 12 x 20 1.05 -> 0.89, 30 x 60 18.6 -> 8.0, 128 x 256 124 -> 38
//     (only 8 x 12 and smaller direct-method models gain on the fast build)
static bool general_is_faster(const HostModel& h, int kind, const LeapScale& ls) {
    if (kind == 2 || (kind == 4 && h.M > 128)) return true;
    return (kind <= 8 || h.M > 512) && mostly_long_draws(h, ls);
}

static tl_status make_plan(const tl_model* m, int variant, int block_req, int mode, bool sens, bool compat_stoich,
                           bool no_stage, long long total, const LeapScale& ls, Plan& pl, bool force_gslot = false) {
    const size_t sb = slot_bytes(m, mode != kModeFast);
    const int smax = max_smem_optin() - 2048;
    const bool autov = variant == TL_VARIANT_AUTO;
    const int nsm = sm_count();
    pl = Plan{};  // nothing of a plan that pl held before (measured mode plans twice)
    if (autov) variant = heuristic_variant(m, sb, total, mode, nsm);
    pl.variant = variant;
    int groups_per_block = 1;
    if (variant == TL_VARIANT_THREAD) {
        pl.kind = 1;
        if (mode != kModeGeneral) thin_plan(std::max(m->h.N, m->h.M), total, nsm, thin_most_warps(m->h, ls), pl.thin, pl.lanes);
        int b = block_req;
        if (b <= 0) {
            // spread small ensembles over every SM
            const int per_warp = pl.lanes / pl.thin;
            const long long per_sm = ((total + per_warp - 1) / per_warp + nsm - 1) / nsm;  // warps
            b = 32 * (int)std::min<long long>(4, std::max<long long>(1, per_sm));
        }
        pl.block = b;
        groups_per_block = pl.block;  // the fit below is that of whole warps
    } else if (variant == TL_VARIANT_WARP) {
        pl.kind = 32;
        pl.block = block_req > 0 ? block_req : 256;
        groups_per_block = pl.block / 32;
    } else if (variant >= TL_VARIANT_LANES2 && variant <= TL_VARIANT_LANES16) {
        pl.kind = 2 << (variant - TL_VARIANT_LANES2);
        pl.block = block_req > 0 ? block_req : 256;
        groups_per_block = pl.block / pl.kind;
    } else if (variant == TL_VARIANT_CTA) {
        pl.kind = 0;
        // chain-sized models (up to 1024 channels): 128 threads, 8 channels
        // each (cyclic chain 1024: 3.67e7 realization-steps/s against 3.41e7
        // at 256); up to 64 KB of state: 256; larger: 1024
        pl.block = block_req > 0 ? block_req : (sb <= 64 * 1024 ? (m->h.M <= 1024 ? 128 : 256) : 1024);
        groups_per_block = 1;
    } else {
        set_last_error("unknown variant");
        return TL_ERR_INVALID_ARGUMENT;
    }
    if (pl.block % 32 || pl.block < 32 || pl.block > (pl.kind == 0 ? 1024 : 256)) {
        set_last_error("block_threads must be a multiple of 32 in [32, 256] (thread / warp groups) "
                       "or [32, 1024] (CTA groups)");
        return TL_ERR_INVALID_ARGUMENT;
    }
    // shrink the block until the slots fit
    const int asked = pl.block;
    const auto fit = [&](int mode_) {
        pl.mode = mode_;
        pl.block = asked;
        pl.slot = slot_layout(m, sens, mode_, pl.kind, pl.block);
        groups_per_block = pl.kind ? pl.block / pl.kind : 1;
        while ((size_t)groups_per_block * pl.slot.bytes > (size_t)smax && pl.kind != 0 && pl.block > 32) {
            pl.block -= 32;
            groups_per_block = pl.block / pl.kind;
        }
        // a CTA's queue is drained more often where that makes its slot fit (ms,
        // general build -> so: colloid of 312 species 0.423 -> 0.258, of 328 0.464 -> 0.333)
        for (int r = pl.slot.q_rounds - 1; r > 0 && pl.kind == 0 && !pl.gslot && pl.slot.bytes > (size_t)smax; --r) {
            const SlotLayout less = slot_layout(m, sens, mode_, pl.kind, pl.block, r);
            if (less.bytes <= (size_t)smax) pl.slot = less;
        }
        return (size_t)groups_per_block * pl.slot.bytes <= (size_t)smax;
    };
    pl.gslot = force_gslot && pl.kind == 0;
    // the packed tables hold the model (CTA groups: wide forms too)?
    const bool packed = m->d.fast_ok && (pl.kind == 0 || (!m->d.chan8 && !m->d.ent_wide));
    // the sub-warp and global-slot kinds have no scores build
    const bool sub = pl.kind > 1 && pl.kind < 32;
    if (!packed || (mode == kModeScores && (pl.gslot || sub))) mode = kModeGeneral;
    if (mode == kModeFast && sub && general_is_faster(m->h, pl.kind, ls)) mode = kModeGeneral;
    if (!fit(mode) && !pl.gslot) {
        // The general build's slot is smaller for wide models.  A CTA's propensities
        // go to global memory instead where the state stays in shared memory,
        // ms on GB300, general -> so: colloid of 332 species 0.472 -> 0.356 (152
        // realizations), chain of 15000 species 0.469 -> 0.370, 6000 x 40000 network 19.0 -> 10.7
        const bool big_only = mode == kModeFast && pl.kind == 0 && pl.slot.state <= (size_t)smax;
        if (mode == kModeGeneral || big_only || !fit(kModeGeneral)) {
            if (pl.kind != 0) {
                set_last_error("model too large for the shared-memory slot of this variant");
                return TL_ERR_UNSUPPORTED;
            }
            // one realization's state exceeds shared memory: CTA groups keep it
            // in global memory (one slot per CTA, served from L2)
            pl.gslot = true;
            fit(mode == kModeScores ? kModeGeneral : mode);
        }
    }
    if (pl.kind == 1) groups_per_block = pl.mode == kModeGeneral ? pl.block : pl.block / 32 * (pl.lanes / pl.thin);
    const bool tiny = pl.kind == 1 && pl.mode != kModeGeneral && pl.thin > 1;  // no slots: registers
    size_t slot_smem = tiny ? 0 : (size_t)groups_per_block * pl.slot.bytes;
    if (pl.gslot) {
        // fast build: a[] in global memory, the state beside it only if it
        // does not fit either
        slot_smem = pl.mode == kModeGeneral ? 0 : pl.slot.state;
        pl.state_global = slot_smem > (size_t)smax;
        if (pl.state_global) slot_smem = 0;
    }
    const int stage = (compat_stoich || no_stage || pl.gslot) ? 0
                      : pl.mode == kModeGeneral               ? m->d.stage_bytes
                      : tiny                                  ? (int)sizeof(TinyTable)
                                                              : m->d.f_stage_bytes;
    // chain-sized CTA groups leave the tables in L1/L2 (staging them would
    // cost more shared memory than the realization itself)
    const bool stage_ok = !(autov && pl.kind == 0 && sb <= 64 * 1024);
    pl.stage = (stage_ok && slot_smem + (size_t)stage <= (size_t)smax) ? stage : 0;
    pl.smem = (size_t)pl.stage + slot_smem;
    // scores beside the counts while four such CTAs fit an SM, else in global memory
    if (pl.mode == kModeScores && !tiny && pl.smem > (size_t)smax / 4) {
        pl.slot.score_global = true;
        pl.slot.bytes -= (size_t)pl.slot.f_a;
        pl.smem -= (size_t)groups_per_block * (size_t)pl.slot.f_a;
    }
    pl.row_warp = pl.kind == 0 && m->h.max_row > 32;
    int bps = 0;
    const int lk = launch_kind(pl);
    const bool staged = pl.stage > 0;
    cudaError_t e = m->h.pop_bits == 64 ? fused_occupancy<long long>(lk, pl.mode, staged, pl.block, pl.smem, &bps)
                                        : fused_occupancy<int>(lk, pl.mode, staged, pl.block, pl.smem, &bps);
    if (e != cudaSuccess) return cuda_fail(e, "occupancy");
    if (bps < 1) {
        set_last_error("the launch does not fit an SM");
        return TL_ERR_UNSUPPORTED;
    }
    if (pl.kind == 32 && pl.mode != kModeGeneral && block_req <= 0 && staged && !pl.slot.score_global &&
        team_pays(m, total, nsm)) {
        Plan t = pl;
        t.team = true;
        t.block = 128;
        t.slot = slot_layout(m, sens, pl.mode, 0, 128);
        t.smem = (size_t)t.stage + t.slot.bytes;
        int tb = 0;
        if (t.smem <= (size_t)smax) {
            e = m->h.pop_bits == 64 ? fused_occupancy<long long>(kKindTeam, t.mode, true, 128, t.smem, &tb)
                                    : fused_occupancy<int>(kKindTeam, t.mode, true, 128, t.smem, &tb);
            if (e != cudaSuccess) return cuda_fail(e, "occupancy");
        }
        if (total <= (long long)nsm * tb) {  // all realizations at once
            pl = t;
            groups_per_block = 1;
            bps = tb;
        }
    }
    const long long need = (total + groups_per_block - 1) / groups_per_block;
    pl.grid = (int)std::min<long long>((long long)nsm * bps, std::max<long long>(need, 1));
    if (pl.kind >= 2 && pl.kind <= 32 && !pl.team && block_req <= 0 && need <= (long long)nsm * bps) {
        const int block = even_block(total, 32 / pl.kind, nsm, pl.block / 32);
        Plan q;
        if (block < pl.block && make_plan(m, variant, block, mode, sens, compat_stoich, no_stage, total, ls, q) == TL_OK &&
            q.block == block && q.mode == pl.mode && (q.stage > 0) == staged && (long long)q.grid * (block / q.kind) >= total)
            pl = q;
    }
    return TL_OK;
}

struct RunBuffers {
    float* rates = nullptr;
    double* tfin = nullptr;
    double* grid = nullptr;
    int* tracked = nullptr;
    void* samples = nullptr;
    float* scores = nullptr;
    unsigned long long* ctr = nullptr;
    double* mean = nullptr;
    double* sd = nullptr;
    double* grad = nullptr;
    double* gse = nullptr;
    double* gmean = nullptr;
    void* pstate = nullptr;
    void* pslots = nullptr;
    float* a_all = nullptr;
};

// The rates of a call on the device: the model's own resident ones, or the
// call's sets as given, halved for 2S channels (fast builds), or both.
enum class RateForm { Model, Plain, Halved, Both };

// One (model, configuration) pair of a call: validation, scratch layout,
// device parameters, reduction and result.
struct Job {
    tl_model* m = nullptr;
    const tl_run_cfg* cfg = nullptr;
    tl_result* res = nullptr;
    tl_grad_result* grad = nullptr;
    int S = 1, P = 2, K = 0;
    long long R = 1, total = 1;
    bool sens = false, keep = false, plain = false, compat_stoich = false;
    int mode = kModeFast;  // the kernel build: scores and / or compatibility switches
    size_t w = 4;
    // what goes to the device, the call's rate sets first, in the forms that the
    // build reads (job_rates)
    std::unique_ptr<unsigned char[]> hin;
    size_t in_bytes = 0;
    RateForm rate_form = RateForm::Model;
    bool measure = false;
    bool wide_stats = false, fixed_scratch = false;  // (the static entry's scratch holds no sums)
    size_t o_acc = 0;
    unsigned char* base = nullptr;
    size_t o_in = 0;
    LeapScale scale;
    std::vector<double> htf;
    std::vector<double> hgrid;  // [S][P] grid times
    Plan pl;
    size_t o_rates = 0, o_tf = 0, o_grid = 0, o_tr = 0, o_samp = 0, o_sc = 0, o_ctr = 0, o_mean = 0, o_sd = 0, o_grad = 0,
           o_gse = 0, o_gm = 0, o_ps = 0, o_pslot = 0, o_aall = 0, o_gslot = 0;
    RunBuffers rb;
    SimParams p{};
    std::unique_ptr<int[]> hs;  // 32-bit samples on their way to the result
    std::vector<unsigned char> hout;
    unsigned long long hc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
};

// Bytes of the call's rate sets in J.hin.
static size_t rate_bytes(const Job& J) {
    const size_t copies = J.rate_form == RateForm::Model ? 0 : J.rate_form == RateForm::Both ? 2 : 1;
    return al16(copies * (size_t)J.S * (size_t)J.m->h.M * 4);
}
// Bytes of the rest: end times, grid, tracked species, zeroed counters.
static size_t rest_bytes(const Job& J) {
    return al16((size_t)J.S * 8) + al16((size_t)J.S * J.P * 8) + al16((size_t)std::max(J.K, 1) * 4) + 64;
}

// n rates to FP32 times `by`, in vectors.  Returns a top bit where one may be
// negative or not finite: every such double has its sign bit or, the lowest exponent bit added, gets it.
static uint64_t convert_rates(const double* __restrict from, const float* __restrict by, float* __restrict to, size_t n) {
    uint64_t any = 0;
    for (size_t j = 0; j < n; ++j) {
        uint64_t b;
        memcpy(&b, from + j, 8);
        any |= b | (b + 0x0010000000000000ull);
        to[j] = (float)from[j] * by[j];
    }
    return any;
}

// The call's rate sets into J.hin in one form, checked on the way: one pass reads
// the doubles and writes what is sent.  exact: halving is (see fill_rates).  Host time
// of a call on GB300: 0.8 ns a rate (60 000 sets of 256 rates: 12 ms); 2.4 ns with
// both forms made apart, zeroed and copied, 1.0 ns with one form zeroed and copied.
static tl_status job_rates(Job& J, RateForm form, bool& exact) {
    const HostModel& h = J.m->h;
    const size_t M = (size_t)h.M, S = (size_t)J.S;
    J.rate_form = form;
    J.in_bytes = rate_bytes(J) + rest_bytes(J);
    J.hin.reset(new unsigned char[J.in_bytes]);
    std::vector<float> by(M, 1.f);
    std::vector<int> twice;
    for (size_t j = 0; j < M && form != RateForm::Plain; ++j)
        if (h.order[j] == 3) {
            by[j] = 0.5f;
            twice.push_back((int)j);
        }
    float* const first = reinterpret_cast<float*>(J.hin.get());
    float* const halved = form == RateForm::Both ? first + S * M : first;
    uint64_t any = 0;
    exact = true;
    for (size_t s = 0; s < S; ++s) {
        const double* const c = J.cfg->rate_sets + s * M;
        float* const to = halved + s * M;
        any |= convert_rates(c, by.data(), to, M);
        for (const int j : twice) exact &= halves_exactly((float)c[j]);
        if (form == RateForm::Both) {
            float* const plain = first + s * M;
            memcpy(plain, to, M * 4);
            for (const int j : twice) plain[j] = (float)c[j];
        }
    }
    if (any >> 63)  // a bad one, or -0.0
        for (size_t q = 0; q < S * M; ++q)
            if (!std::isfinite(J.cfg->rate_sets[q]) || J.cfg->rate_sets[q] < 0.0) {
                set_last_error("rate constants must be finite and >= 0");
                return TL_ERR_NUMERIC;
            }
    return TL_OK;
}

static tl_status job_prepare(Job& J) {
    tl_model* m = J.m;
    const tl_run_cfg* cfg = J.cfg;
    if (!m || !cfg) {
        set_last_error("null model or config");
        return TL_ERR_INVALID_ARGUMENT;
    }
    const HostModel& h = m->h;
    const int N = h.N, M = h.M;
    if (!(cfg->t_final > 0.0) || !std::isfinite(cfg->t_final) || !(cfg->eps > 0.0) || cfg->n_realizations < 1 ||
        cfg->n_intervals < 1 || cfg->n_tracked < 0 || cfg->n_rate_sets < 0 || cfg->max_steps < 0) {
        set_last_error("invalid run configuration (t_final > 0, eps > 0, n >= 1, intervals >= 1)");
        return TL_ERR_INVALID_ARGUMENT;
    }
    if (cfg->n_realizations + cfg->realization_offset > 0xFFFFFFFFLL || cfg->realization_offset < 0 ||
        cfg->n_rate_sets >= (1 << 24)) {
        set_last_error("at most 2^32 realizations per set and 2^24 rate sets");
        return TL_ERR_INVALID_ARGUMENT;
    }
    if (cfg->n_tracked > 0 && !cfg->tracked) {
        set_last_error("tracked is NULL");
        return TL_ERR_INVALID_ARGUMENT;
    }
    for (int q = 0; q < cfg->n_tracked; ++q)
        if (cfg->tracked[q] < 0 || cfg->tracked[q] >= N) {
            set_last_error("tracked species index out of range");
            return TL_ERR_INVALID_ARGUMENT;
        }
    if (cfg->n_rate_sets > 0 && !cfg->rate_sets) {
        set_last_error("rate_sets is NULL");
        return TL_ERR_INVALID_ARGUMENT;
    }
    J.S = std::max(1, cfg->n_rate_sets);
    J.R = cfg->n_realizations;
    J.P = cfg->n_intervals + 1;
    J.K = cfg->n_tracked;
    J.total = J.R * J.S;
    J.sens = J.grad != nullptr;
    J.mode = (cfg->flags & TL_FLAG_COMPAT_REFERENCE) ? kModeGeneral : J.sens ? kModeScores : kModeFast;
    J.keep = (cfg->flags & TL_FLAG_KEEP_SAMPLES) != 0;
    J.plain = cfg->variant == TL_VARIANT_PLAIN;
    J.compat_stoich = (cfg->flags & TL_FLAG_COMPAT_STOICH) != 0;
    J.w = h.pop_bits == 64 ? 8 : 4;
    if (J.plain && J.sens) {
        set_last_error("the plain form has no sensitivity pass");
        return TL_ERR_UNSUPPORTED;
    }
    if (J.sens && J.K < 1) {
        set_last_error("sensitivity needs at least one tracked species");
        return TL_ERR_INVALID_ARGUMENT;
    }
    J.htf.assign((size_t)J.S, cfg->t_final);
    bool halvable = true;
    if (cfg->n_rate_sets > 0) {
        // scored and measured runs may read both forms
        const RateForm form = J.plain || J.mode == kModeGeneral        ? RateForm::Plain
                              : J.mode == kModeScores || J.measure ? RateForm::Both
                                                                       : RateForm::Halved;
        const tl_status rs = job_rates(J, form, halvable);
        if (rs != TL_OK) return rs;
    } else {
        const tl_status ds = ensure_device(m);  // the model's own rates are resident
        if (ds != TL_OK) return ds;
        halvable = m->d.halvable;
        J.in_bytes = rest_bytes(J);
        J.hin.reset(new unsigned char[J.in_bytes]);
    }
    // the packed criticalities are signs of x - n_c and x - 2 n_c, in int32
    if (!halvable || cfg->n_critical >= (1 << 30)) J.mode = kModeGeneral;
    if (cfg->n_rate_sets > 0 && cfg->t_final_sets)
        for (int s = 0; s < J.S; ++s) {
            J.htf[(size_t)s] = cfg->t_final_sets[s];
            if (!(J.htf[(size_t)s] > 0.0) || !std::isfinite(J.htf[(size_t)s])) {
                set_last_error("t_final_sets must be > 0");
                return TL_ERR_INVALID_ARGUMENT;
            }
        }
    J.scale = LeapScale{cfg->eps, J.htf[0] / (double)cfg->n_intervals};
    // grid t_k = T*k/n_int (FP64, the last point T itself)
    J.hgrid.resize((size_t)J.S * J.P);
    for (int s = 0; s < J.S; ++s)
        for (int k = 0; k < J.P; ++k)
            J.hgrid[(size_t)s * J.P + k] = k >= cfg->n_intervals
                                               ? J.htf[(size_t)s]
                                               : J.htf[(size_t)s] * (double)k / (double)cfg->n_intervals;
    return ensure_device(m);
}

// A CTA's slot in global memory: without the state where that is in shared memory.
static size_t global_slot_bytes(const Plan& pl) {
    return pl.mode == kModeGeneral || pl.state_global ? pl.slot.bytes : pl.slot.bytes - pl.slot.state;
}

// The plan's part of the launch parameters.
static void bind_plan(const tl_model* m, const Plan& pl, SimParams& p) {
    p.blob = pl.mode == kModeGeneral ? m->d.blob : m->d.fblob;
    // (a batch keeps the tables' start: its items differ)
    if (pl.kind == 1 && pl.mode != kModeGeneral && pl.thin > 1 && !pl.batch) p.blob += m->d.t_tiny;
    p.stage_bytes = pl.stage;
    p.slot_bytes = (int)(pl.gslot ? global_slot_bytes(pl) : pl.slot.bytes);
    p.f_D = pl.slot.f_D;
    p.f_X = pl.slot.f_X;
    p.f_a = pl.slot.f_a;
    p.f_big = pl.gslot && !pl.state_global ? 0 : (int)pl.slot.state;
    p.score_global = pl.slot.score_global ? 1 : 0;
    p.state_global = pl.state_global ? 1 : 0;
    p.q_rounds = pl.slot.q_rounds;
    p.lanes = pl.lanes;
    p.row_warp = pl.row_warp ? 1 : 0;
}

static void job_layout(Job& J, Carver& c) {
    const int M = J.m->h.M, N = J.m->h.N, K1 = std::max(J.K, 1);
    // what goes to the device in one copy: rate sets, end times, grid, tracked
    // species and zeroed counters, which come back with the statistics.  Only
    // a plan that fell back to the general build finds the wrong form here.
    if (J.rate_form == RateForm::Halved && J.pl.mode == kModeGeneral) {
        bool exact;
        job_rates(J, RateForm::Plain, exact);
    }
    size_t o = 0;
    const auto put = [&](size_t& at, size_t bytes) {
        at = o;
        o += al16(bytes);
    };
    put(J.o_rates, rate_bytes(J));
    put(J.o_tf, (size_t)J.S * 8);
    put(J.o_grid, (size_t)J.S * J.P * 8);
    put(J.o_tr, (size_t)K1 * 4);
    put(J.o_ctr, 8 * 8);
    put(J.o_mean, (size_t)J.S * J.P * K1 * 8);
    put(J.o_sd, (size_t)J.S * J.P * K1 * 8);
    const size_t at = c.take(o);
    for (size_t* q : {&J.o_rates, &J.o_tf, &J.o_grid, &J.o_tr, &J.o_ctr, &J.o_mean, &J.o_sd}) *q += at;
    J.o_in = at;
    J.o_samp = c.take((size_t)J.total * J.P * K1 * J.w);
    // many columns side by side: from 64 the coalesced statistics win (chain
    // of 1024: 187 -> 30 us; 33 columns of 10^4 realizations: 25 us either way)
    J.wide_stats = J.w == 4 && J.P * J.K >= 64 && J.S <= 65535 && (long long)J.S * J.P * J.K < (1LL << 30) &&
                   J.R >= 64 && !J.fixed_scratch;
    J.o_acc = J.wide_stats ? c.take((size_t)J.S * J.P * J.K * 24) : 0;
    J.o_sc = J.sens ? c.take((size_t)J.total * M * 4) : 0;
    J.o_grad = J.sens ? c.take((size_t)J.S * J.K * M * 8) : 0;
    J.o_gse = J.sens ? c.take((size_t)J.S * J.K * M * 8) : 0;
    J.o_gm = J.sens ? c.take((size_t)J.S * J.K * 8) : 0;
    J.o_ps = J.plain ? c.take((size_t)J.total * 64) : 0;
    J.o_pslot = J.plain ? c.take((size_t)J.total * 2 * al16((size_t)N * J.w)) : 0;
    J.o_aall = J.plain ? c.take((size_t)J.total * M * 4) : 0;
    J.o_gslot = (!J.plain && J.pl.gslot) ? c.take((size_t)J.pl.grid * global_slot_bytes(J.pl)) : 0;
}

static tl_status job_bind(Job& J, unsigned char* B, cudaStream_t st) {
    tl_model* m = J.m;
    const tl_run_cfg* cfg = J.cfg;
    RunBuffers& rb = J.rb;
    J.base = B;
    rb.rates = reinterpret_cast<float*>(B + J.o_rates);
    rb.tfin = reinterpret_cast<double*>(B + J.o_tf);
    rb.grid = reinterpret_cast<double*>(B + J.o_grid);
    rb.tracked = reinterpret_cast<int*>(B + J.o_tr);
    rb.samples = B + J.o_samp;
    rb.scores = J.sens ? reinterpret_cast<float*>(B + J.o_sc) : nullptr;
    rb.ctr = reinterpret_cast<unsigned long long*>(B + J.o_ctr);
    rb.mean = reinterpret_cast<double*>(B + J.o_mean);
    rb.sd = reinterpret_cast<double*>(B + J.o_sd);
    if (J.sens) {
        rb.grad = reinterpret_cast<double*>(B + J.o_grad);
        rb.gse = reinterpret_cast<double*>(B + J.o_gse);
        rb.gmean = reinterpret_cast<double*>(B + J.o_gm);
    }
    if (J.plain) {
        rb.pstate = B + J.o_ps;
        rb.pslots = B + J.o_pslot;
        rb.a_all = reinterpret_cast<float*>(B + J.o_aall);
    }
    const auto fill = [&](size_t at, const void* from, size_t bytes) {
        if (bytes) memcpy(J.hin.get() + (at - J.o_in), from, bytes);
    };
    const size_t M = (size_t)m->h.M;
    memset(J.hin.get() + (J.o_tf - J.o_in), 0, J.in_bytes - (J.o_tf - J.o_in));
    fill(J.o_tf, J.htf.data(), J.htf.size() * 8);
    fill(J.o_grid, J.hgrid.data(), J.hgrid.size() * 8);
    fill(J.o_tr, cfg->tracked, (size_t)J.K * 4);
    const bool general = J.plain || J.pl.mode == kModeGeneral;
    const tl_status ts = ensure_tables(m, general || J.measure, !general || J.measure, st);
    if (ts != TL_OK) return ts;
    TLC(cudaMemcpyAsync(B + J.o_in, J.hin.get(), J.in_bytes, cudaMemcpyHostToDevice, st));
    // (a run that reads one form finds it in both)
    const float* const plain = J.rate_form == RateForm::Model ? m->d.rate : rb.rates;
    const float* const halved = J.rate_form == RateForm::Model  ? m->d.rate + M
                                : J.rate_form == RateForm::Both ? rb.rates + (size_t)J.S * M
                                                                : rb.rates;
    SimParams& p = J.p;
    p = SimParams{};
    p.N = m->h.N;
    p.M = m->h.M;
    p.g = global_view(m, J.compat_stoich, false);
    p.x0 = m->d.x0;
    p.rates = plain;
    p.t_final = rb.tfin;
    p.grid = rb.grid;
    p.R = J.R;
    p.r_off = cfg->realization_offset;
    p.S = J.S;
    p.k0 = (uint32_t)(cfg->seed & 0xFFFFFFFFu);
    p.k1 = (uint32_t)(cfg->seed >> 32);
    round_keys(p.k0, p.k1, p.rk);
    p.eps = (float)cfg->eps;
    p.nc = cfg->n_critical > 0 ? cfg->n_critical : 5;
    p.ssa_factor = (float)(cfg->ssa_factor > 0 ? cfg->ssa_factor : 10);
    p.ssa_block = cfg->ssa_block > 0 ? cfg->ssa_block : 100;
    p.n_int = cfg->n_intervals;
    p.K = J.K;
    p.tracked = rb.tracked;
    p.samples = rb.samples;
    p.scores = rb.scores;
    p.max_steps = cfg->max_steps;
    p.flags = cfg->flags;
    p.max_halv = cfg->max_halvings > 0 ? cfg->max_halvings : 64;
    p.wait_polls = cfg->stage_wait_polls == 0 ? (1 << 22) : std::max(cfg->stage_wait_polls, 0);
    p.frates = halved;
    p.off_chan = m->d.off_chan;
    p.off_rord = m->d.off_rord;
    p.off_gkind = m->d.off_gkind;
    p.off_perm = m->d.off_perm;
    p.off_rp = m->d.off_rp;
    p.off_vc = m->d.off_vc;
    p.off_cp = m->d.off_cp;
    p.off_rv = m->d.off_rv;
    p.n_rows = m->d.n_rows;
    p.x_one = ((m->h.N + 3) & ~3) + m->d.n_2s;
    p.chan8 = m->d.chan8 ? 1 : 0;
    p.ent_wide = m->d.ent_wide ? 1 : 0;
    p.t_chan = m->d.t_chan;
    p.t_row = m->d.t_row;
    p.t_ent = m->d.t_ent;
    p.t_col = m->d.t_col;
    p.t_cp = m->d.t_cp;
    p.t_sp = m->d.t_sp;
    p.t_tiny = m->d.t_tiny;
    bind_plan(m, J.pl, p);
    p.gslots = J.pl.gslot ? B + J.o_gslot : nullptr;
    p.ctr = rb.ctr;
    p.pstate = rb.pstate;
    p.pslots = rb.pslots;
    return TL_OK;
}

// Statistics / gradient reductions and the device-to-host copies.
static tl_status job_reduce(Job& J, cudaStream_t st) {
    const int M = J.m->h.M;
    RunBuffers& rb = J.rb;
    cudaError_t le;
    if (J.K > 0) {
        le = J.wide_stats
                 ? launch_stats_wide(rb.samples, J.R, J.P * J.K, J.S, J.base + J.o_acc, rb.mean, rb.sd, sm_count(), st)
             : J.w == 8 ? launch_stats<long long>(rb.samples, J.R, J.P, J.K, J.S, rb.mean, rb.sd, st)
                      : launch_stats<int>(rb.samples, J.R, J.P, J.K, J.S, rb.mean, rb.sd, st);
        if (le != cudaSuccess) return cuda_fail(le, "statistics launch");
    }
    if (J.sens) {
        le = J.w == 8 ? launch_grad<long long>(rb.samples, rb.scores, J.R, J.P, J.K, M, J.S, rb.grad, rb.gse, rb.gmean, st)
                      : launch_grad<int>(rb.samples, rb.scores, J.R, J.P, J.K, M, J.S, rb.grad, rb.gse, rb.gmean, st);
        if (le != cudaSuccess) return cuda_fail(le, "gradient launch");
    }
    // counters, means and deviations in one copy
    const bool stats = J.res && J.K > 0 && (J.res->mean || J.res->stddev);
    const size_t SPK = (size_t)J.S * J.P * J.K;
    J.hout.resize(stats ? J.o_sd - J.o_ctr + SPK * 8 : 64);
    TLC(cudaMemcpyAsync(J.hout.data(), rb.ctr, J.hout.size(), cudaMemcpyDeviceToHost, st));
    if (J.res && J.res->samples && J.keep && J.K > 0) {
        const size_t n = (size_t)J.total * J.P * J.K;
        void* to = J.res->samples;
        if (J.w == 4) {
            J.hs.reset(new int[n]);
            to = J.hs.get();
        }
        TLC(cudaMemcpyAsync(to, rb.samples, n * J.w, cudaMemcpyDeviceToHost, st));
    }
    if (J.sens) {
        tl_grad_result* g = J.grad;
        const size_t SKM = (size_t)J.S * J.K * M;
        if (g->grad) TLC(cudaMemcpyAsync(g->grad, rb.grad, SKM * 8, cudaMemcpyDeviceToHost, st));
        if (g->grad_stderr) TLC(cudaMemcpyAsync(g->grad_stderr, rb.gse, SKM * 8, cudaMemcpyDeviceToHost, st));
        if (g->mean_final)
            TLC(cudaMemcpyAsync(g->mean_final, rb.gmean, (size_t)J.S * J.K * 8, cudaMemcpyDeviceToHost, st));
    }
    return TL_OK;
}

// After the stream is synchronised: fill the result, map error bits.
static tl_status job_finish(Job& J, double kernel_ms, int launches, double total_ms) {
    tl_result* res = J.res;
    if (J.hs) {
        const size_t n = (size_t)J.total * J.P * J.K;
        const int* src = J.hs.get();
        for (size_t q = 0; q < n; ++q) res->samples[q] = src[q];
    }
    memcpy(J.hc, J.hout.data(), 64);
    if (res && J.hout.size() > 64) {
        const size_t n = (size_t)J.S * J.P * J.K * 8;
        if (res->mean) memcpy(res->mean, J.hout.data() + (J.o_mean - J.o_ctr), n);
        if (res->stddev) memcpy(res->stddev, J.hout.data() + (J.o_sd - J.o_ctr), n);
    }
    if (res) {
        if (res->times) std::copy(J.hgrid.begin(), J.hgrid.end(), res->times);
        res->leaps = (int64_t)J.hc[1];
        res->ssa_steps = (int64_t)J.hc[2];
        res->rejections = (int64_t)J.hc[3];
        res->truncated = (int64_t)J.hc[4];
        res->kernel_ms = kernel_ms;
        res->variant_used = J.pl.variant;
        res->block_threads_used = J.pl.block;
        res->grid_used = J.pl.grid;
        res->launches = launches;
        res->total_ms = total_ms;
    }
    const unsigned eb = (unsigned)J.hc[5];
    if (eb & kErrWaitTimeout) {
        set_last_error("shared-memory staging wait timed out");
        return TL_ERR_WAIT_TIMEOUT;
    }
    if (eb & kErrOverflow) {
        set_last_error("a population left the range of the population type");
        return TL_ERR_OVERFLOW;
    }
    if (eb & (kErrHalving | kErrNumeric)) {
        set_last_error("a leap could not be made non-negative by halving tau " +
                       std::to_string(J.p.max_halv) + " times (max_halvings)");
        return TL_ERR_NUMERIC;
    }
    if (J.hc[4] > 0) {
        set_last_error("max_steps reached; truncated realizations hold their last state");
        return TL_ERR_STEP_CAP;
    }
    return TL_OK;
}

// The model's pair of timing events.
static tl_status timing_events(tl_model* m, cudaEvent_t* e0, cudaEvent_t* e1) {
    for (void*& e : m->ev)
        if (!e) {
            cudaEvent_t made = nullptr;
            TLC(cudaEventCreate(&made));
            e = made;
        }
    *e0 = (cudaEvent_t)m->ev[0];
    *e1 = (cudaEvent_t)m->ev[1];
    return TL_OK;
}

static double ms_since(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// Autotuner, measured part (TL_FLAG_AUTOTUNE_MEASURE): time every plan that
// fits on the first realizations of this very ensemble (identical streams,
// so identical work per candidate), the planned one among them (teams and even
// CTAs are planned, never asked for by a block), keep the fastest in the model
// handle, keyed by the flags that change the kernel.  The trial writes only the
// prefix of the sample buffer, which the real run then overwrites.
static tl_status autotune_measure(Job& J, cudaStream_t st) {
    tl_model* m = J.m;
    const bool planned_gslot = J.pl.gslot;
    const int planned_grid = J.pl.grid;
    const bool planned_nostage = (J.cfg->flags & TL_FLAG_NO_STAGE) != 0;
    const bool force_gslot = (J.cfg->flags & TL_FLAG_GLOBAL_SLOTS) != 0;
    unsigned char* const planned_gslots = J.p.gslots;
    // the best plan depends on how many realizations fill the GPU: key the
    // cache by the ensemble size (power-of-two bucket) as well
    int bucket = 0;
    while (bucket < 40 && (1LL << bucket) < J.total) ++bucket;
    const unsigned key = 0x80000000u | (J.sens ? 1u : 0u) | (J.compat_stoich ? 2u : 0u) | ((unsigned)bucket << 2) |
                         (unsigned)(J.cfg->flags & ~(TL_FLAG_KEEP_SAMPLES | TL_FLAG_AUTOTUNE_MEASURE)) << 8;
    if (m->tuned_key != key) {
        struct Cand {
            int variant, block;
            bool nostage;
        };
        std::vector<Cand> cands;
        if (m->h.M <= 64 && m->h.N <= 64)
            for (int b : {32, 64, 128}) cands.push_back({TL_VARIANT_THREAD, b, false});
        if (m->h.M <= 1024)
            for (int v = TL_VARIANT_LANES2; v <= TL_VARIANT_LANES16; ++v)
                for (int b : {128, 256}) cands.push_back({v, b, false});
        for (int b : {64, 128, 256})
            for (bool ns : {false, true}) cands.push_back({TL_VARIANT_WARP, b, ns});
        for (int b : {64, 128, 256, 512, 1024})
            for (bool ns : {false, true}) cands.push_back({TL_VARIANT_CTA, b, ns});
        // toy network, 152 realizations, ms: teams 9.78, CTAs 10.68, warps 13.58; 1000: 12.57, 13.34, 14.39
        cands.push_back({TL_VARIANT_AUTO, 0, planned_nostage});
        // a prefix large enough to fill the GPU under every candidate
        const long long trial = std::min<long long>(J.total, 16384);
        SimParams tp = J.p;
        tp.R = trial;
        tp.S = 1;
        cudaEvent_t e0, e1;
        TLC(cudaEventCreate(&e0));
        TLC(cudaEventCreate(&e1));
        float best = 3.4e38f;
        Cand win{-1, 0, false};
        for (const Cand& c : cands) {
            Plan pl;
            if (c.variant == TL_VARIANT_AUTO) pl = J.pl;
            else if (make_plan(m, c.variant, c.block, J.mode, J.sens, J.compat_stoich, c.nostage, trial, J.scale, pl) != TL_OK) continue;
            if (c.variant == TL_VARIANT_THREAD && c.block != pl.block) continue;
            // global slots exist for the launch the heuristic planned
            if (pl.gslot && (!planned_gslot || pl.grid > planned_grid)) continue;
            bind_plan(m, pl, tp);
            tp.gslots = pl.gslot ? planned_gslots : nullptr;
            if (cudaMemsetAsync(tp.ctr, 0, 64, st) != cudaSuccess) break;
            cudaEventRecord(e0, st);
            cudaError_t le = J.w == 8 ? launch_fused<long long>(tp, launch_kind(pl), pl.mode, pl.stage > 0, pl.block, pl.grid, pl.smem, st)
                                      : launch_fused<int>(tp, launch_kind(pl), pl.mode, pl.stage > 0, pl.block, pl.grid, pl.smem, st);
            cudaEventRecord(e1, st);
            if (le != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                win = c;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        TLC(cudaMemsetAsync(J.p.ctr, 0, 64, st));
        if (win.variant < 0) {
            set_last_error("autotuner found no plan that fits");
            return TL_ERR_UNSUPPORTED;
        }
        m->tuned_key = key;
        m->tuned_variant = win.variant;
        m->tuned_block = win.block;
        m->tuned_nostage = win.nostage ? 1 : 0;
    }
    tl_status ps = make_plan(m, m->tuned_variant, m->tuned_block, J.mode, J.sens, J.compat_stoich, m->tuned_nostage != 0,
                             J.total, J.scale, J.pl, m->tuned_variant == TL_VARIANT_AUTO && force_gslot);
    if (ps != TL_OK) return ps;
    if (J.pl.gslot && (!planned_gslot || J.pl.grid > planned_grid)) {
        // a cached global-slot plan that needs more slots than were laid out:
        // keep the planned launch
        ps = make_plan(m, TL_VARIANT_AUTO, 0, J.mode, J.sens, J.compat_stoich, planned_nostage, J.total, J.scale,
                       J.pl, force_gslot);
        if (ps != TL_OK) return ps;
    }
    bind_plan(m, J.pl, J.p);
    J.p.gslots = J.pl.gslot ? planned_gslots : nullptr;
    return TL_OK;
}

static tl_status run(tl_model* m, const tl_run_cfg* cfg, tl_result* res, tl_grad_result* grad) {
    const auto t0 = std::chrono::steady_clock::now();
    Job J;
    J.m = m;
    J.cfg = cfg;
    J.res = res;
    J.grad = grad;
    J.measure = cfg && cfg->variant == TL_VARIANT_AUTO && (cfg->flags & TL_FLAG_AUTOTUNE_MEASURE);
    tl_status ps = job_prepare(J);
    if (ps != TL_OK) return ps;
    TLC(cudaSetDevice(m->d.device));
    cudaStream_t st = (cudaStream_t)cfg->stream;
    const bool no_stage = (cfg->flags & TL_FLAG_NO_STAGE) != 0;
    if (!J.plain) {
        ps = make_plan(m, cfg->variant, cfg->block_threads, J.mode, J.sens, J.compat_stoich, no_stage, J.total, J.scale, J.pl,
                       (cfg->flags & TL_FLAG_GLOBAL_SLOTS) != 0);
        if (ps != TL_OK) return ps;
    } else {
        J.pl.variant = TL_VARIANT_PLAIN;
        J.pl.kind = 1;
        J.pl.block = 128;
        J.pl.grid = (int)((J.total + 127) / 128);
    }
    Carver c;
    job_layout(J, c);
    void* base = nullptr;
    ps = scratch_get(m, c.off, &base);
    if (ps != TL_OK) return ps;
    ps = job_bind(J, reinterpret_cast<unsigned char*>(base), st);
    if (ps != TL_OK) return ps;
    if (J.measure) {
        ps = autotune_measure(J, st);
        if (ps != TL_OK) return ps;
    }
    const SimParams& p = J.p;
    const size_t w = J.w;

    cudaEvent_t e0, e1;
    ps = timing_events(m, &e0, &e1);
    if (ps != TL_OK) return ps;
    int launches = 0;
    cudaError_t le = cudaEventRecord(e0, st);
    if (le == cudaSuccess) {
        if (!J.plain) {
            le = w == 8 ? launch_fused<long long>(p, launch_kind(J.pl), J.pl.mode, J.pl.stage > 0, J.pl.block, J.pl.grid, J.pl.smem, st)
                        : launch_fused<int>(p, launch_kind(J.pl), J.pl.mode, J.pl.stage > 0, J.pl.block, J.pl.grid, J.pl.smem, st);
            launches = 1;
        } else {
            le = w == 8 ? launch_plain_init<long long>(p, st) : launch_plain_init<int>(p, st);
            launches = 1;
            // With TL_FLAG_GRAPH the 16 step launches between two polls are
            // captured once (on a private stream) and replayed as one graph.
            cudaGraphExec_t gexec = nullptr;
            if (le == cudaSuccess && (cfg->flags & TL_FLAG_GRAPH)) {
                cudaStream_t cs = nullptr;
                le = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
                if (le == cudaSuccess) {
                    cudaGraph_t g = nullptr;
                    le = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
                    for (int q = 0; q < 16 && le == cudaSuccess; ++q)
                        le = w == 8 ? launch_plain_step<long long>(p, J.rb.a_all, cs)
                                    : launch_plain_step<int>(p, J.rb.a_all, cs);
                    const cudaError_t ec = cudaStreamEndCapture(cs, &g);
                    if (le == cudaSuccess) le = ec;
                    if (le == cudaSuccess) le = cudaGraphInstantiate(&gexec, g, 0);
                    if (g) cudaGraphDestroy(g);
                    cudaStreamDestroy(cs);
                }
            }
            unsigned long long* hdone = nullptr;
            if (le == cudaSuccess) le = cudaMallocHost(&hdone, 8);
            while (le == cudaSuccess) {
                if (gexec) {
                    le = cudaGraphLaunch(gexec, st);
                    launches += 16;
                } else {
                    for (int q = 0; q < 16 && le == cudaSuccess; ++q) {
                        le = w == 8 ? launch_plain_step<long long>(p, J.rb.a_all, st)
                                    : launch_plain_step<int>(p, J.rb.a_all, st);
                        ++launches;
                    }
                }
                if (le != cudaSuccess) break;
                le = cudaMemcpyAsync(hdone, J.rb.ctr + 6, 8, cudaMemcpyDeviceToHost, st);
                if (le == cudaSuccess) le = cudaStreamSynchronize(st);
                if (le == cudaSuccess && *hdone >= (unsigned long long)J.total) break;
                if (launches > (1 << 26)) {  // a realization that never ends
                    if (gexec) cudaGraphExecDestroy(gexec);
                    cudaFreeHost(hdone);
                    set_last_error("plain form exceeded 2^26 launches; set max_steps");
                    return TL_ERR_STEP_CAP;
                }
            }
            if (gexec) cudaGraphExecDestroy(gexec);
            if (hdone) cudaFreeHost(hdone);
            if (le == cudaSuccess) le = launch_plain_tally(p, st);
            ++launches;
        }
    }
    if (le == cudaSuccess) le = cudaEventRecord(e1, st);
    if (le != cudaSuccess) return cuda_fail(le, "simulation launch");
    ps = job_reduce(J, st);
    if (ps != TL_OK) return ps;
    TLC(cudaStreamSynchronize(st));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    return job_finish(J, ms, launches, ms_since(t0));
}

// The batch kernel's CTAs per SM: two (128 registers, no spills) while they
// hold every unit at once, three (80 registers) beyond, where more warps hide
// more of a step's latency.  Measured on GB300, ms at 2 -> 3 -> 4, gradients of
// dimer sets (16) and toy network sets (4), realizations a set: dimer 1024
// 1.63 -> 1.73 -> 1.83 (one wave), 4096 5.71 -> 4.71 -> 4.20, 16384 17.7 -> 15.8
// -> 15.0; toy 700 20.4 -> 17.6 -> 18.8, 1500 32.9 -> 30.7 -> 31.5; both, 4096
// and 700, 22.4 -> 19.6 -> 23.0; 64 x 4096 and 16 x 1024 to t = 10 and 0.1,
// 1501 -> 1247 -> 1371.
// Batches of small items on one lane each alone run best at four (64 registers)
// where three do not hold them at once: dimer sets, ms at 2 -> 4, 16 x 8192 realizations to t = 0.01 4.15 -> 3.65, t = 1 6.94 ->
// 6.04, with scores 5.47 -> 4.80 and 8.75 -> 7.46; 64 x 4096 to t = 1 11.1 -> 10.1 and
// 14.0 -> 12.7.
static int batch_minb(long long units, int warps, int nsm, bool thin_only) {
    if (thin_only && units > 3LL * warps * nsm) return TL_BATCH_THIN_MINB;
    return units > 2LL * warps * nsm ? TL_BATCH_MANY_MINB : TL_BATCH_MINB;
}

// One launch over several (model, configuration) items.  Items of small
// models run as lane units (several realizations per warp, on one or 4 to 16
// lanes each), the others as warp units (one realization per warp, or per team
// of four warps where they all fit at once); a warp takes units from
// one global counter, so uneven step counts and uneven t_final balance out.
static tl_status run_batch(tl_batch_item* items, int n, cudaStream_t st) {
    const auto t0 = std::chrono::steady_clock::now();
    if (!items || n < 1) {
        set_last_error("empty batch");
        return TL_ERR_INVALID_ARGUMENT;
    }
    std::vector<Job> jobs((size_t)n);
    int device = -1, pop = 0;
    for (int i = 0; i < n; ++i) {
        Job& J = jobs[(size_t)i];
        J.m = items[i].model;
        J.cfg = items[i].cfg;
        J.res = items[i].result;
        J.grad = items[i].grad;
        tl_status ps = job_prepare(J);
        if (ps != TL_OK) return ps;
        if (J.plain) {
            set_last_error("the plain form cannot be batched");
            return TL_ERR_UNSUPPORTED;
        }
        if (device < 0) {
            device = J.m->d.device;
            pop = J.m->h.pop_bits;
        } else if (device != J.m->d.device || pop != J.m->h.pop_bits) {
            set_last_error("batched models must share device and population width");
            return TL_ERR_INVALID_ARGUMENT;
        }
    }
    TLC(cudaSetDevice(device));
    const int smax = max_smem_optin() - 2048;
    // unit kind per item; the warp slot is the largest need
    std::vector<int> lane(n);
    size_t wslot = 0;
    int bmode = kModeFast;  // the build every item can run on
    long long lane_total = 0;
    bool small_only = true;  // every item runs as lane units
    int lane_size = 1;  // channels or species of the largest thread-group item
    for (int i = 0; i < n; ++i) {
        Job& J = jobs[(size_t)i];
        const tl_model* m = J.m;
        bmode = std::max(bmode, J.mode);
        if (!m->d.fast_ok || m->d.chan8 || m->d.ent_wide) bmode = kModeGeneral;
        lane[(size_t)i] = (m->h.M <= 16 && m->h.N <= 16) ? 1 : 0;
        small_only &= lane[(size_t)i] != 0;
        if (lane[(size_t)i]) {
            lane_total += J.total;
            lane_size = std::max(lane_size, std::max(m->h.M, m->h.N));
        }
    }
    const size_t spb = al16(sizeof(SimParams));
    int thin = 1, unit_lanes = 32;
    for (;;) {
        thin = 1;
        unit_lanes = 32;
        if (bmode != kModeGeneral) thin_plan(lane_size <= 4 ? 4 : 16, lane_total, sm_count(),
                                             thin_most_warps_batch(lane_size, small_only, bmode == kModeScores), thin, unit_lanes);
        wslot = 0;
        for (int i = 0; i < n; ++i) {
            Job& J = jobs[(size_t)i];
            Plan& pl = J.pl;
            pl.variant = lane[(size_t)i] ? TL_VARIANT_THREAD : TL_VARIANT_WARP;
            pl.mode = bmode;
            pl.batch = true;
            pl.lanes = unit_lanes;
            pl.thin = thin;
            pl.slot = slot_layout(J.m, J.sens, bmode, lane[(size_t)i] ? 1 : 32, 32);
            const size_t unit = !lane[(size_t)i] ? pl.slot.bytes : thin == 1 ? (size_t)unit_lanes * pl.slot.bytes : 0;
            wslot = std::max(wslot, unit);
        }
        wslot = al16(wslot);
        // the general build's slot is smaller for wide models
        if (wslot + spb <= (size_t)smax || bmode == kModeGeneral) break;
        bmode = kModeGeneral;
    }
    const auto tables = [&](const tl_model* m) { return bmode == kModeGeneral ? m->d.blob : m->d.fblob; };
    const auto table_bytes = [&](const tl_model* m) {
        return bmode == kModeGeneral ? m->d.stage_bytes : m->d.f_stage_bytes;
    };
    // stage every model's tables when they fit next to 4 warps' slots
    std::vector<tl_model*> uniq;
    for (auto& J : jobs)
        if (std::find(uniq.begin(), uniq.end(), J.m) == uniq.end()) uniq.push_back(J.m);
    size_t stage = 0;
    std::vector<size_t> stage_off(uniq.size());
    for (size_t u = 0; u < uniq.size(); ++u) {
        stage_off[u] = stage;
        stage += (size_t)table_bytes(uniq[u]);
    }
    bool staged = true;
    for (auto& J : jobs) staged &= !J.compat_stoich;
    if (stage + 4 * (wslot + spb) > (size_t)smax) staged = false;
    if (!staged) stage = 0;
    int warps = 8;
    while (warps > 1 && stage + (size_t)warps * (wslot + spb) > (size_t)smax) --warps;
    if (stage + (size_t)warps * (wslot + spb) > (size_t)smax) {
        set_last_error("a batched model is too large for a warp unit; run it with tl_simulate");
        return TL_ERR_UNSUPPORTED;
    }
    // four-warp teams where all larger items' realizations run at once on them
    bool team = bmode != kModeGeneral && staged && thin > 1;
    for (auto& J : jobs) team &= J.cfg->seed == jobs[0].cfg->seed;
    long long big_total = 0;
    bool wide_item = false;
    size_t tslot = 0;
    for (int i = 0; i < n; ++i)
        if (!lane[(size_t)i]) {
            const Job& J = jobs[(size_t)i];
            big_total += J.total;
            wide_item |= team_pays(J.m, J.total, sm_count());
            tslot = std::max(tslot, slot_layout(J.m, J.sens, bmode, 0, 128).bytes);
        }
    tslot = al16(tslot);
    const size_t team_smem = stage + 2 * (tslot + spb);
    int team_bps = 0;
    if (team && wide_item && team_smem <= (size_t)smax) {
        const BatchParams none{};
        const cudaError_t oe = pop == 64 ? launch_batch_team<long long>(none, bmode, thin, 0, team_smem, st, &team_bps)
                                         : launch_batch_team<int>(none, bmode, thin, 0, team_smem, st, &team_bps);
        if (oe != cudaSuccess) return cuda_fail(oe, "batch occupancy");
    }
    team = big_total > 0 && big_total <= 2LL * team_bps * sm_count();
    if (team) {
        warps = 8;
        wslot = tslot;
        for (int i = 0; i < n; ++i)
            if (!lane[(size_t)i]) jobs[(size_t)i].pl.slot = slot_layout(jobs[(size_t)i].m, jobs[(size_t)i].sens, bmode, 0, 128);
    }
    // scratch: every job's buffers, the item table, the staged tables, a counter
    Carver c;
    for (auto& J : jobs) job_layout(J, c);
    const size_t o_items = c.take(sizeof(BatchItem) * (size_t)n);
    const size_t o_stage = c.take(std::max<size_t>(stage, 16));
    const size_t o_wctr = c.take(16);
    tl_model* owner = jobs[0].m;
    void* base = nullptr;
    tl_status ps = scratch_get(owner, c.off, &base);
    if (ps != TL_OK) return ps;
    unsigned char* B = reinterpret_cast<unsigned char*>(base);
    for (auto& J : jobs) {
        ps = job_bind(J, B, st);
        if (ps != TL_OK) return ps;
    }
    if (staged)
        for (size_t u = 0; u < uniq.size(); ++u)
            TLC(cudaMemcpyAsync(B + o_stage + stage_off[u], tables(uniq[u]), (size_t)table_bytes(uniq[u]),
                                cudaMemcpyDeviceToDevice, st));
    // unit table: warp-unit items first (longer realizations), then lane units
    std::vector<int> order;
    for (int i = 0; i < n; ++i)
        if (!lane[(size_t)i]) order.push_back(i);
    for (int i = 0; i < n; ++i)
        if (lane[(size_t)i]) order.push_back(i);
    std::vector<BatchItem> hb((size_t)n);
    const int per_unit = unit_lanes / thin * (team ? 4 : 1);
    long long units = 0;
    for (int k = 0; k < n; ++k) {
        const int i = order[(size_t)k];
        Job& J = jobs[(size_t)i];
        BatchItem& b = hb[(size_t)k];
        b.p = J.p;
        b.p.stage_bytes = 0;
        b.lane_mode = lane[(size_t)i];
        b.unit_begin = units;
        b.units = lane[(size_t)i] ? (J.total + per_unit - 1) / per_unit : J.total;
        units += b.units;
        b.stage_off = -1;
        if (staged) {
            const size_t u = (size_t)(std::find(uniq.begin(), uniq.end(), J.m) - uniq.begin());
            b.stage_off = (int)stage_off[u];
        }
        J.pl.block = 32 * warps;
    }
    TLC(cudaMemcpyAsync(B + o_items, hb.data(), sizeof(BatchItem) * (size_t)n, cudaMemcpyHostToDevice, st));
    TLC(cudaMemsetAsync(B + o_wctr, 0, 16, st));
    BatchParams bp{};
    bp.items = reinterpret_cast<const BatchItem*>(B + o_items);
    bp.n_items = n;
    bp.total_units = units;
    bp.stage_src = B + o_stage;
    bp.stage_bytes = (int)stage;
    bp.warp_slot_bytes = (int)wslot;
    bp.params_bytes = (int)spb;
    bp.wctr = reinterpret_cast<unsigned long long*>(B + o_wctr);
    round_keys(jobs[0].p.k0, jobs[0].p.k1, bp.rk);
    const int minb = batch_minb(units, warps, sm_count(), small_only && thin == 1 && staged && bmode != kModeGeneral);
    const size_t smem = team ? team_smem : stage + (size_t)warps * (wslot + spb);
    int bps = team_bps;
    cudaError_t le = team ? cudaSuccess : pop == 64 ? batch_occupancy<long long>(bmode, staged, minb, thin, 32 * warps, smem, &bps)
                               : batch_occupancy<int>(bmode, staged, minb, thin, 32 * warps, smem, &bps);
    if (le != cudaSuccess) return cuda_fail(le, "batch occupancy");
    const int grid = (int)std::min<long long>((long long)sm_count() * std::max(bps, 1),
                                              team ? (units + 1) / 2 : (units + warps - 1) / warps);
    for (auto& J : jobs) J.pl.grid = grid;
    cudaEvent_t e0, e1;
    ps = timing_events(owner, &e0, &e1);
    if (ps != TL_OK) return ps;
    le = cudaEventRecord(e0, st);
    if (le == cudaSuccess)
        le = team ? (pop == 64 ? launch_batch_team<long long>(bp, bmode, thin, grid, smem, st, nullptr)
                               : launch_batch_team<int>(bp, bmode, thin, grid, smem, st, nullptr))
             : pop == 64 ? launch_batch<long long>(bp, bmode, minb, thin, 32 * warps, grid, smem, st)
                       : launch_batch<int>(bp, bmode, minb, thin, 32 * warps, grid, smem, st);
    if (le == cudaSuccess) le = cudaEventRecord(e1, st);
    if (le != cudaSuccess) return cuda_fail(le, "batch launch");
    for (auto& J : jobs) {
        ps = job_reduce(J, st);
        if (ps != TL_OK) return ps;
    }
    TLC(cudaStreamSynchronize(st));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    tl_status worst = TL_OK;
    for (auto& J : jobs) {
        const tl_status s2 = job_finish(J, ms, 1, ms_since(t0));
        if (s2 != TL_OK && (worst == TL_OK || worst == TL_ERR_STEP_CAP)) worst = s2;
    }
    return worst;
}

}  // namespace tl

using namespace tl;

extern "C" {

const char* tl_status_str(tl_status s) {
    switch (s) {
    case TL_OK: return "ok";
    case TL_ERR_INVALID_ARGUMENT: return "invalid argument";
    case TL_ERR_INVALID_MODEL: return "invalid model";
    case TL_ERR_UNSUPPORTED: return "unsupported";
    case TL_ERR_OVERFLOW: return "population overflow";
    case TL_ERR_STEP_CAP: return "step cap reached";
    case TL_ERR_CUDA: return "CUDA error";
    case TL_ERR_WAIT_TIMEOUT: return "device wait timeout";
    case TL_ERR_NO_DEVICE: return "no CUDA device";
    case TL_ERR_OUT_OF_MEMORY: return "out of memory";
    case TL_ERR_IO: return "I/O error";
    case TL_ERR_PARSE: return "parse error";
    case TL_ERR_NUMERIC: return "numeric error";
    }
    return "unknown status";
}

const char* tl_last_error(void) { return g_last_error.c_str(); }
int32_t tl_abi_version(void) { return TL_ABI_VERSION; }

tl_status tl_set_device(int32_t device) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceCount");
    if (device < 0 || device >= n) {
        set_last_error("device index out of range");
        return TL_ERR_INVALID_ARGUMENT;
    }
    g_device = device;
    TLC(cudaSetDevice(device));
    return TL_OK;
}

tl_status tl_model_create(const tl_model_desc* d, tl_model** out) {
    if (!d || !out || !d->x0 || !d->rate || !d->col_ptr || (d->nnz > 0 && (!d->row_ind || !d->stoich)) ||
        d->n_species <= 0 || d->n_channels <= 0 || d->nnz < 0) {
        set_last_error("incomplete model description");
        return TL_ERR_INVALID_ARGUMENT;
    }
    *out = nullptr;
    tl_model* m = new tl_model();
    HostModel& h = m->h;
    h.N = d->n_species;
    h.M = d->n_channels;
    h.pop_bits = d->pop_bits;
    h.x0.assign(d->x0, d->x0 + h.N);
    h.rate.assign(d->rate, d->rate + h.M);
    h.col_ptr.assign(d->col_ptr, d->col_ptr + h.M + 1);
    if (h.col_ptr[(size_t)h.M] != d->nnz) {
        set_last_error("col_ptr[M] != nnz");
        delete m;
        return TL_ERR_INVALID_MODEL;
    }
    h.row_ind.assign(d->row_ind, d->row_ind + d->nnz);
    h.stoich.assign(d->stoich, d->stoich + d->nnz);
    return finish_model(m, out);
}

tl_status tl_model_from_stochkit(const char* path, int32_t pop_bits, tl_model** out) {
    if (!path || !out) {
        set_last_error("null path");
        return TL_ERR_INVALID_ARGUMENT;
    }
    *out = nullptr;
    tl_model* m = new tl_model();
    std::string err;
    tl_status s = parse_stochkit_file(path, m->h, m->channels, err);
    if (s != TL_OK) {
        set_last_error(err);
        delete m;
        return s;
    }
    m->h.pop_bits = pop_bits;
    return finish_model(m, out);
}

void tl_gen_params_init(tl_gen_params* g, int32_t family) {
    if (!g) return;
    memset(g, 0, sizeof *g);
    g->family = family;
    switch (family) {
    case TL_GEN_DIMER:  // dimerisation decay with S1 = 100000
        g->n_species = 3;
        g->n_channels = 4;
        g->x0_min = g->x0_max = 100000;
        g->seed = 1;
        break;
    case TL_GEN_TOY:  // 128 species, 256 channels, x0 U[0,10000], c logU[1e-3,1]
        g->n_species = 128;
        g->n_channels = 256;
        g->x0_min = 0;
        g->x0_max = 10000;
        g->rate_min = 1e-3;
        g->rate_max = 1.0;
        g->seed = 7;
        break;
    case TL_GEN_CHAIN:  // 1024 species, rate 1, x0 U[1000,2000]
        g->n_species = 1024;
        g->n_channels = 1024;
        g->x0_min = 1000;
        g->x0_max = 2000;
        g->rate_min = g->rate_max = 1.0;
        g->seed = 11;
        break;
    case TL_GEN_COLLOID:  // 250 species, 31250 channels, x0 U[1000,2000], int64
        g->n_species = 250;
        g->n_channels = 31250;
        g->x0_min = 1000;
        g->x0_max = 2000;
        g->rate_assoc = 1e-4;
        g->rate_dissoc = 0.1;
        g->pop_bits = 64;
        g->seed = 13;
        break;
    default:
        break;
    }
}

tl_status tl_model_generate(const tl_gen_params* g, tl_model** out) {
    if (!g || !out) {
        set_last_error("null argument");
        return TL_ERR_INVALID_ARGUMENT;
    }
    *out = nullptr;
    tl_model* m = new tl_model();
    std::string err;
    tl_status s = generate_model(*g, m->h, m->channels, err);
    if (s != TL_OK) {
        set_last_error(err);
        delete m;
        return s;
    }
    return finish_model(m, out);
}

void tl_model_destroy(tl_model* m) {
    if (!m) return;
    if (m->d.blob || m->d.x0 || m->d.rate || m->scratch) {
        int cur = 0;
        cudaGetDevice(&cur);
        cudaSetDevice(m->d.device);
        if (m->d.blob) cudaFree(m->d.blob);
        if (m->d.x0) cudaFree(m->d.x0);
        if (m->d.rate) cudaFree(m->d.rate);
        if (m->scratch) cudaFree(m->scratch);
        for (void* e : m->ev)
            if (e) cudaEventDestroy((cudaEvent_t)e);
        cudaSetDevice(cur);
    }
    delete m;
}

tl_status tl_model_get_info(const tl_model* m, tl_model_info* info) {
    if (!m || !info) return TL_ERR_INVALID_ARGUMENT;
    info->n_species = m->h.N;
    info->n_channels = m->h.M;
    info->nnz_raw = (int32_t)m->h.raw_vc.size();
    info->nnz_net = (int32_t)m->h.net_vc.size();
    info->pop_bits = m->h.pop_bits;
    info->max_order = m->h.max_order;
    return TL_OK;
}

const char* tl_model_species_name(const tl_model* m, int32_t i) {
    if (!m || i < 0 || i >= m->h.N) return nullptr;
    return m->h.names[(size_t)i].c_str();
}

int32_t tl_model_species_index(const tl_model* m, const char* name) {
    if (!m || !name) return -1;
    for (int i = 0; i < m->h.N; ++i)
        if (m->h.names[(size_t)i] == name) return i;
    return -1;
}

tl_status tl_model_get_desc(const tl_model* m, int64_t* x0, double* rate, int32_t* col_ptr, int32_t* row_ind,
                            int8_t* stoich) {
    if (!m) return TL_ERR_INVALID_ARGUMENT;
    const HostModel& h = m->h;
    if (x0) std::copy(h.x0.begin(), h.x0.end(), x0);
    if (rate) std::copy(h.rate.begin(), h.rate.end(), rate);
    if (col_ptr) std::copy(h.col_ptr.begin(), h.col_ptr.end(), col_ptr);
    if (row_ind) std::copy(h.row_ind.begin(), h.row_ind.end(), row_ind);
    if (stoich) std::copy(h.stoich.begin(), h.stoich.end(), stoich);
    return TL_OK;
}

tl_status tl_model_get_tables(const tl_model* m, int8_t* order, int32_t* s0, int32_t* s1, int32_t* rp,
                              int32_t* vc) {
    if (!m) return TL_ERR_INVALID_ARGUMENT;
    const HostModel& h = m->h;
    if (order) std::copy(h.order.begin(), h.order.end(), order);
    if (s0) std::copy(h.s0.begin(), h.s0.end(), s0);
    if (s1) std::copy(h.s1.begin(), h.s1.end(), s1);
    if (rp) std::copy(h.raw_rp.begin(), h.raw_rp.end(), rp);
    if (vc) std::copy(h.raw_vc.begin(), h.raw_vc.end(), vc);
    return TL_OK;
}

tl_status tl_model_write_stochkit(const tl_model* m, const char* path) {
    if (!m || !path) return TL_ERR_INVALID_ARGUMENT;
    std::vector<Channel> ch = m->channels;
    if (ch.empty()) {
        // models built from a descriptor: rebuild channels from the raw entries
        const HostModel& h = m->h;
        ch.resize((size_t)h.M);
        for (int j = 0; j < h.M; ++j) {
            ch[(size_t)j].rate = h.rate[(size_t)j];
            for (int q = h.col_ptr[(size_t)j]; q < h.col_ptr[(size_t)j + 1]; ++q) {
                const int v = h.stoich[(size_t)q];
                if (v < 0) ch[(size_t)j].reactants.push_back({h.row_ind[(size_t)q], -v});
                else if (v > 0) ch[(size_t)j].products.push_back({h.row_ind[(size_t)q], v});
            }
        }
    }
    std::string err;
    tl_status s = write_stochkit_file(path, m->h, ch, "generated by tau_leaping_gb300", err);
    if (s != TL_OK) set_last_error(err);
    return s;
}

void tl_run_cfg_init(tl_run_cfg* cfg) {
    if (!cfg) return;
    memset(cfg, 0, sizeof *cfg);
    cfg->t_final = 1.0;
    cfg->eps = 0.03;  // cl_parser.cpp:22
    cfg->n_realizations = 1;
    cfg->seed = 1;
    cfg->n_intervals = 1;
    cfg->variant = TL_VARIANT_AUTO;
}

tl_status tl_simulate(tl_model* m, const tl_run_cfg* cfg, tl_result* res) { return run(m, cfg, res, nullptr); }

tl_status tl_simulate_batch(tl_batch_item* items, int32_t n_items, void* stream) {
    return run_batch(items, n_items, (cudaStream_t)stream);
}

tl_status tl_sensitivity(tl_model* m, const tl_run_cfg* cfg, tl_result* res, tl_grad_result* grad) {
    if (!grad) {
        set_last_error("grad result is NULL");
        return TL_ERR_INVALID_ARGUMENT;
    }
    return run(m, cfg, res, grad);
}

tl_status tl_eval_leap(tl_model* m, const int64_t* x, int32_t n, double eps, uint32_t flags, int32_t nc, float* a,
                       uint8_t* crit, float* mu, float* sigma2, float* tau1, double* a0) {
    if (!m || !x || n <= 0) {
        set_last_error("bad arguments to tl_eval_leap");
        return TL_ERR_INVALID_ARGUMENT;
    }
    const HostModel& h = m->h;
    const int N = h.N, M = h.M;
    {
        tl_status ds = ensure_device(m);
        if (ds == TL_OK) ds = ensure_tables(m, true, false, 0);
        if (ds != TL_OK) return ds;
    }
    TLC(cudaSetDevice(m->d.device));
    const size_t smem = slot_bytes(m);
    if (smem > (size_t)max_smem_optin()) {
        set_last_error("model too large for tl_eval_leap");
        return TL_ERR_UNSUPPORTED;
    }
    Carver c;
    const size_t ox = c.take((size_t)n * N * 8), oa = c.take((size_t)n * M * 4), oc = c.take((size_t)n * M),
                 om = c.take((size_t)n * N * 4), os = c.take((size_t)n * N * 4), ot = c.take((size_t)n * 4),
                 o0 = c.take((size_t)n * 8);
    void* base = nullptr;
    tl_status s = scratch_get(m, c.off, &base);
    if (s != TL_OK) return s;
    unsigned char* B = reinterpret_cast<unsigned char*>(base);
    TLC(cudaMemcpy(B + ox, x, (size_t)n * N * 8, cudaMemcpyHostToDevice));
    SimParams p{};
    p.N = N;
    p.M = M;
    p.g = global_view(m, (flags & TL_FLAG_COMPAT_STOICH) != 0, false);
    p.rates = m->d.rate;
    p.eps = (float)eps;
    p.nc = nc > 0 ? nc : 5;
    p.flags = flags;
    cudaError_t e = h.pop_bits == 64
                        ? launch_eval<long long>(p, reinterpret_cast<long long*>(B + ox), n,
                                                 reinterpret_cast<float*>(B + oa), B + oc, reinterpret_cast<float*>(B + om),
                                                 reinterpret_cast<float*>(B + os), reinterpret_cast<float*>(B + ot),
                                                 reinterpret_cast<double*>(B + o0), smem, 0)
                        : launch_eval<int>(p, reinterpret_cast<long long*>(B + ox), n, reinterpret_cast<float*>(B + oa),
                                           B + oc, reinterpret_cast<float*>(B + om), reinterpret_cast<float*>(B + os),
                                           reinterpret_cast<float*>(B + ot), reinterpret_cast<double*>(B + o0), smem, 0);
    if (e != cudaSuccess) return cuda_fail(e, "eval launch");
    if (a) TLC(cudaMemcpy(a, B + oa, (size_t)n * M * 4, cudaMemcpyDeviceToHost));
    if (crit) TLC(cudaMemcpy(crit, B + oc, (size_t)n * M, cudaMemcpyDeviceToHost));
    if (mu) TLC(cudaMemcpy(mu, B + om, (size_t)n * N * 4, cudaMemcpyDeviceToHost));
    if (sigma2) TLC(cudaMemcpy(sigma2, B + os, (size_t)n * N * 4, cudaMemcpyDeviceToHost));
    if (tau1) TLC(cudaMemcpy(tau1, B + ot, (size_t)n * 4, cudaMemcpyDeviceToHost));
    if (a0) TLC(cudaMemcpy(a0, B + o0, (size_t)n * 8, cudaMemcpyDeviceToHost));
    return TL_OK;
}

tl_status tl_replay(tl_model* m, const int64_t* x0, const int32_t* k, int32_t n_leaps, int32_t raw, int64_t* x_out) {
    if (!m || !x0 || !k || n_leaps <= 0 || !x_out) {
        set_last_error("bad arguments to tl_replay");
        return TL_ERR_INVALID_ARGUMENT;
    }
    const HostModel& h = m->h;
    const int N = h.N, M = h.M;
    for (int i = 0; i < N; ++i)
        if (h.pop_bits == 32 && (x0[i] > 2147483647LL || x0[i] < -2147483647LL)) {
            set_last_error("x0 exceeds int32 for a 32-bit model");
            return TL_ERR_OVERFLOW;
        }
    {
        tl_status ds = ensure_device(m);
        if (ds == TL_OK) ds = ensure_tables(m, true, false, 0);
        if (ds != TL_OK) return ds;
    }
    TLC(cudaSetDevice(m->d.device));
    const size_t w = h.pop_bits == 64 ? 8 : 4;
    const size_t smem = al16((size_t)N * w) * 2 + 16;
    if (smem > (size_t)max_smem_optin()) {
        set_last_error("model too large for tl_replay");
        return TL_ERR_UNSUPPORTED;
    }
    Carver c;
    const size_t ox = c.take((size_t)N * 8), ok = c.take((size_t)n_leaps * M * 4),
                 oo = c.take((size_t)n_leaps * N * 8), ost = c.take(16);
    void* base = nullptr;
    tl_status s = scratch_get(m, c.off, &base);
    if (s != TL_OK) return s;
    unsigned char* B = reinterpret_cast<unsigned char*>(base);
    TLC(cudaMemcpy(B + ox, x0, (size_t)N * 8, cudaMemcpyHostToDevice));
    TLC(cudaMemcpy(B + ok, k, (size_t)n_leaps * M * 4, cudaMemcpyHostToDevice));
    TLC(cudaMemset(B + ost, 0, 16));
    SimParams p{};
    p.N = N;
    p.M = M;
    p.g = global_view(m, false, raw != 0);
    cudaError_t e = w == 8 ? launch_replay<long long>(p, reinterpret_cast<long long*>(B + ox),
                                                      reinterpret_cast<int*>(B + ok), n_leaps,
                                                      reinterpret_cast<long long*>(B + oo), reinterpret_cast<int*>(B + ost),
                                                      smem, 0)
                           : launch_replay<int>(p, reinterpret_cast<long long*>(B + ox), reinterpret_cast<int*>(B + ok),
                                                n_leaps, reinterpret_cast<long long*>(B + oo),
                                                reinterpret_cast<int*>(B + ost), smem, 0);
    if (e != cudaSuccess) return cuda_fail(e, "replay launch");
    TLC(cudaDeviceSynchronize());
    int stt = 0;
    TLC(cudaMemcpy(&stt, B + ost, 4, cudaMemcpyDeviceToHost));
    TLC(cudaMemcpy(x_out, B + oo, (size_t)n_leaps * N * 8, cudaMemcpyDeviceToHost));
    if (stt) {
        set_last_error("replay left the int32 range");
        return TL_ERR_OVERFLOW;
    }
    return TL_OK;
}

tl_status tl_philox(const uint32_t* ctr, const uint32_t* key, int32_t n, uint32_t* out) {
    if (!ctr || !key || !out || n <= 0) return TL_ERR_INVALID_ARGUMENT;
    TLC(cudaSetDevice(g_device));
    void *dc = nullptr, *dk = nullptr, *dout = nullptr;
    TLC(cudaMalloc(&dc, (size_t)n * 16));
    TLC(cudaMalloc(&dk, (size_t)n * 8));
    TLC(cudaMalloc(&dout, (size_t)n * 16));
    cudaMemcpy(dc, ctr, (size_t)n * 16, cudaMemcpyHostToDevice);
    cudaMemcpy(dk, key, (size_t)n * 8, cudaMemcpyHostToDevice);
    cudaError_t e = launch_philox(dc, dk, n, dout, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, (size_t)n * 16, cudaMemcpyDeviceToHost);
    cudaFree(dc);
    cudaFree(dk);
    cudaFree(dout);
    if (e != cudaSuccess) return cuda_fail(e, "philox");
    return TL_OK;
}

tl_status tl_poisson(const float* mean, int32_t n, uint64_t seed, uint32_t step, int32_t compat, int32_t* out) {
    if (!mean || !out || n <= 0) return TL_ERR_INVALID_ARGUMENT;
    for (int i = 0; i < n; ++i)
        if (!(mean[i] >= 0.f) || mean[i] > 1e9f) {
            set_last_error("Poisson means must be in [0, 1e9]");
            return TL_ERR_INVALID_ARGUMENT;
        }
    TLC(cudaSetDevice(g_device));
    float* dm = nullptr;
    int* dout = nullptr;
    TLC(cudaMalloc(&dm, (size_t)n * 4));
    TLC(cudaMalloc(&dout, (size_t)n * 4));
    cudaMemcpy(dm, mean, (size_t)n * 4, cudaMemcpyHostToDevice);
    cudaError_t e = launch_poisson(dm, n, (unsigned)(seed & 0xFFFFFFFFu), (unsigned)(seed >> 32), step, compat, dout, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, (size_t)n * 4, cudaMemcpyDeviceToHost);
    cudaFree(dm);
    cudaFree(dout);
    if (e != cudaSuccess) return cuda_fail(e, "poisson");
    return TL_OK;
}

tl_status tl_merge_moments(int32_t n_parts, int32_t L, const int64_t* counts, const double* means,
                           const double* stddevs, int64_t* count_out, double* mean_out, double* stddev_out) {
    if (n_parts < 1 || L < 1 || !counts || !means || !stddevs || !count_out || !mean_out || !stddev_out) {
        set_last_error("bad arguments to tl_merge_moments");
        return TL_ERR_INVALID_ARGUMENT;
    }
    for (int l = 0; l < L; ++l) {
        double n = 0.0, mean = 0.0, m2 = 0.0;
        for (int p = 0; p < n_parts; ++p) {
            const double nb = (double)counts[p];
            if (nb <= 0) continue;
            const double mb = means[(size_t)p * L + l];
            const double sb = stddevs[(size_t)p * L + l];
            const double m2b = nb > 1 ? sb * sb * (nb - 1.0) : 0.0;
            const double nn = n + nb;
            const double d = mb - mean;
            mean += d * nb / nn;
            m2 += m2b + d * d * n * nb / nn;
            n = nn;
        }
        mean_out[l] = mean;
        stddev_out[l] = n > 1 ? sqrt(m2 / (n - 1.0)) : 0.0;
    }
    int64_t tot = 0;
    for (int p = 0; p < n_parts; ++p) tot += counts[p] > 0 ? counts[p] : 0;
    *count_out = tot;
    return TL_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// tl_simulate_static: tl_simulate's run with its device scratch in one
// file-scope array instead of cudaMalloc'ed memory (see include/tl.h for
// who needs this and the limits).
// ---------------------------------------------------------------------------
namespace tl {

// Held by every GPU that loads the library, until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[TL_STATIC_SCRATCH_BYTES];

// Device address of g_static_scratch per device ordinal.  In host code the
// array's name is only a host-side stand-in, never a device address: the
// address is looked up once per device, with that device current, and kept
// for the life of the process (so the library must not be used across a
// cudaDeviceReset, which would unmap it).
static std::mutex g_static_mu;
static void* g_static_addr[256];

static tl_status static_scratch_address(int device, void** out) {
    if (device < 0 || device >= 256) {
        set_last_error("device ordinal out of range for the static scratch table");
        return TL_ERR_INVALID_ARGUMENT;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_addr[device]) {
        void* ptr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(static scratch)");
        g_static_addr[device] = ptr;
    }
    *out = g_static_addr[device];
    return TL_OK;
}

}  // namespace tl

extern "C" tl_status tl_simulate_static(tl_model* m, const tl_run_cfg* cfg, tl_result* res) {
    const auto t0 = std::chrono::steady_clock::now();
    if (!m || !cfg) {
        set_last_error("null model or config");
        return TL_ERR_INVALID_ARGUMENT;
    }
    if (!m->d.blob) {
        set_last_error("the model's tables are not on the device yet; tl_simulate_static never allocates, so run "
                       "tl_simulate (or tl_eval_leap / tl_replay) on this model once first");
        return TL_ERR_INVALID_ARGUMENT;
    }
    if (cfg->variant == TL_VARIANT_PLAIN) {
        set_last_error("tl_simulate_static runs the fused variants only");
        return TL_ERR_UNSUPPORTED;
    }
    Job J;
    J.m = m;
    J.cfg = cfg;
    J.res = res;
    J.fixed_scratch = true;
    tl_status ps = job_prepare(J);  // the tables are resident: no upload happens
    if (ps != TL_OK) return ps;
    TLC(cudaSetDevice(m->d.device));
    cudaStream_t st = (cudaStream_t)cfg->stream;
    ps = make_plan(m, cfg->variant, cfg->block_threads, J.mode, J.sens, J.compat_stoich,
                   (cfg->flags & TL_FLAG_NO_STAGE) != 0, J.total, J.scale, J.pl, (cfg->flags & TL_FLAG_GLOBAL_SLOTS) != 0);
    if (ps != TL_OK) return ps;
    Carver c;
    job_layout(J, c);
    if (c.off > (size_t)TL_STATIC_SCRATCH_BYTES && J.pl.gslot && J.pl.mode != kModeGeneral) {
        // the general build's slots are smaller and may fit shared memory
        ps = make_plan(m, cfg->variant, cfg->block_threads, kModeGeneral, J.sens, J.compat_stoich,
                       (cfg->flags & TL_FLAG_NO_STAGE) != 0, J.total, J.scale, J.pl, (cfg->flags & TL_FLAG_GLOBAL_SLOTS) != 0);
        if (ps != TL_OK) return ps;
        c = Carver{};
        job_layout(J, c);
    }
    if (c.off > (size_t)TL_STATIC_SCRATCH_BYTES) {
        set_last_error("this run needs " + std::to_string(c.off) + " bytes of device scratch; tl_simulate_static has " +
                       std::to_string((size_t)TL_STATIC_SCRATCH_BYTES) +
                       " (fewer realizations, tracked species or grid points, or use tl_simulate)");
        return TL_ERR_INVALID_ARGUMENT;
    }
    void* base = nullptr;
    ps = static_scratch_address(m->d.device, &base);
    if (ps != TL_OK) return ps;
    ps = job_bind(J, reinterpret_cast<unsigned char*>(base), st);  // clears the counters
    if (ps != TL_OK) return ps;
    const auto tk = std::chrono::steady_clock::now();
    cudaError_t le = J.w == 8 ? launch_fused<long long>(J.p, launch_kind(J.pl), J.pl.mode, J.pl.stage > 0, J.pl.block, J.pl.grid, J.pl.smem, st)
                              : launch_fused<int>(J.p, launch_kind(J.pl), J.pl.mode, J.pl.stage > 0, J.pl.block, J.pl.grid, J.pl.smem, st);
    if (le != cudaSuccess) return cuda_fail(le, "simulation launch");
    ps = job_reduce(J, st);
    if (ps != TL_OK) return ps;
    TLC(cudaStreamSynchronize(st));
    return job_finish(J, ms_since(tk), 1, ms_since(t0));
}
