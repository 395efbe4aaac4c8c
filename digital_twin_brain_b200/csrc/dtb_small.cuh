// Small-network step loop (sm_100a): n time steps of a network of up to kSmallMaxNeurons neurons in
// one launch of one thread-block cluster, everything a step writes kept in (distributed) shared memory.
//
// Such a network is bound by latency: the per-step kernels spend 10-40 us a step on two launches,
// dependent L2 round trips and a handful of busy warps.  Here a CTA owns up to kSmallTiles 128-neuron
// tiles for the whole launch (V, t_last, J, push-row bounds), and a step is
//   phase A: update of the CTA's neurons (models/block.py:133-142), one warp per 32-neuron word; the
//            contributions of the previous step's firing rows are added first, in pull-row order, from
//            the neuron's slots in shared memory (bit-identical to the row gather);
//   barrier; phase B: the CTA's firing rows, dealt out over its warps in quarters: every synapse claims
//            a slot of its target with a shared-memory atomic, in another CTA of the cluster through
//            distributed shared memory; the statistics of the step before are folded beside it; barrier.
// The only memory a step waits for is one read of the firing rows' synapses.  The barrier is the
// hardware cluster barrier (__syncthreads for one CTA): nothing spins.
// Both propagation modes run this way: the ordered sums are a valid order for push.
// Runs whose neurons get more contributions a step than their slots hold stay with the per-step
// kernels (small_pays).
// Measured (single block of 2,000 neurons, K = 100, p = 0.01): a step of a closed loop 39.9 -> 5.9 us,
// one step per call with its statistics on the host 87 -> 36 us.  The same loop on a grid of all SMs
// (counts, slots and J in L2, a barrier in memory) was no faster than two launches a step from
// 30,000 neurons on, so kSmallMaxNeurons is what one cluster's shared memory holds.
#pragma once

#include "dtb_kernels.cuh"

namespace dtb {

constexpr int kSmallWarps = 15;                          // warps that update and scatter; one more folds statistics
constexpr int kSmallThreads = (kSmallWarps + 1) * 32;
constexpr int kSmallTiles = 12;                          // tiles per CTA
constexpr int kSmallTilesFew = 3;                        // tiles per CTA while the cluster can still grow (2,000 neurons:
                                                         // 2 / 3 / 4 / 6 tiles 5.8 / 5.9 / 6.9 / 7.4 us a step; 300: 5.0 / 4.0 / 4.0 / 4.1)
constexpr int kSmallClusterMax = 8;                      // portable cluster size
constexpr int64_t kSmallMaxNeurons = (int64_t)kSmallTiles * kSmallClusterMax * kWarpNeurons;
constexpr int kSmallMaxWords = (int)(kSmallMaxNeurons / 32);
// per neuron: V, t_last, two J pairs, slot count, row offset and length, list entry; and 12 bytes a slot record
constexpr int kSmallCell = 4 + 4 + 16 + 4 + 4 + 4 + 2;
constexpr int kSmallCapMin = 8, kSmallCapMax = 24;       // slot records per neuron: what shared memory holds
constexpr int kSmallBits = 2 * kSmallMaxWords * 4;       // the whole network's firing bits, two steps
constexpr int kSmallUnits = 8;                           // quarter rows a warp scatters together
constexpr uint32_t kSmallSteps = 256;                    // steps per launch

constexpr int kSmallSmemMax = 224 * 1024;

inline size_t small_smem(int tiles, int cap) { return (size_t)tiles * kWarpNeurons * (kSmallCell + 12 * cap) + kSmallBits; }
inline int small_cap(int tiles)
{
    int cap = kSmallCapMax;
    while (cap > kSmallCapMin && small_smem(tiles, cap) > (size_t)kSmallSmemMax) --cap;
    return cap;
}
static_assert((long long)kSmallTiles * kWarpNeurons * (kSmallCell + 12 * kSmallCapMin) + kSmallBits <= kSmallSmemMax, "shared memory");

// tile / tiles_per_cta as a product and a shift, for every tile of the largest network
constexpr uint32_t small_magic(int tiles_per_cta) { return (65536u + (uint32_t)tiles_per_cta - 1u) / (uint32_t)tiles_per_cta; }
constexpr bool small_magic_exact()
{
    for (uint32_t c = 1; c <= (uint32_t)kSmallTiles; ++c)
        for (uint32_t t = 0; t < (uint32_t)(kSmallTiles * kSmallClusterMax); ++t)
            if ((t * small_magic((int)c)) >> 16 != t / c) return false;
    return true;
}
static_assert(small_magic_exact(), "tile division");

struct SmallArgs {
    int n_steps;
    int tiles_per_cta;
    uint32_t tile_magic;     // tile / tiles_per_cta == (tile * tile_magic) >> 16 for every tile
    int isolated;
    float noise_rate;
    int write_v;             // V to global memory every step (sampled neurons read it)
    uint32_t cap;            // slot records per neuron
    uint32_t* host_nact;     // (nullable, pinned host memory) the steps' propagated counts, then Ctl::err
    // per-subblock accumulators by step parity (the first are also the step kernels'); selected, not
    // indexed: an index into a kernel parameter would copy it to local memory
    uint32_t *spk0, *spk1;
    uint32_t *nact0, *nact1;
    double *vsum0, *vsum1;
    uint32_t *unmapped0, *unmapped1;
};

__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t cta)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}

// All threads of the cluster; their shared and global writes before it are visible after it.
__device__ __forceinline__ void small_barrier()
{
    __syncwarp();
    if (gridDim.x == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// gather_row with the firing bits in shared memory.
__device__ __forceinline__ float4 small_gather_row(const DevState& s, const uint32_t* bits, int64_t n, int lane)
{
    const int64_t e0 = __ldg(s.prow + n), e1 = __ldg(s.prow + n + 1);
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
    for (int64_t e = e0; e < e1; e += 32) {
        const int64_t idx = e + lane;
        const uint32_t c = idx < e1 ? __ldg(s.pcol + idx) : 0u;
        const uint32_t p = c & kIndexMask;
        const bool act = idx < e1 && ((bits[p >> 5] >> (p & 31)) & 1u);
        unsigned m = __ballot_sync(0xffffffffu, act);
        float2 w = make_float2(0.0f, 0.0f);
        if (act) w = __ldg(s.pw + idx);
        while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            const float wx = __shfl_sync(0xffffffffu, w.x, l), wy = __shfl_sync(0xffffffffu, w.y, l);
            const uint32_t cl = __shfl_sync(0xffffffffu, c, l);
            if (cl & kKindBit) { a2 = __fadd_rn(a2, wx); a3 = __fadd_rn(a3, wy); }
            else { a0 = __fadd_rn(a0, wx); a1 = __fadd_rn(a1, wy); }
        }
    }
    return make_float4(a0, a1, a2, a3);
}

// The statistics of one finished step: group g's subblocks into the per-step row and the window
// totals, its region's BOLD step (k_stats' work, without a launch of its own).
__device__ __forceinline__ void small_stats(const DevState& s, const SmallArgs& a, int par, int64_t row, int g)
{
    uint32_t* const a_spk = par ? a.spk1 : a.spk0;
    uint32_t* const a_nact = par ? a.nact1 : a.nact0;
    double* const a_vsum = par ? a.vsum1 : a.vsum0;
    uint32_t nact_sum = 0;
    double spk_sum = 0.0;
    const int k1 = __ldg(s.grp_ptr + g + 1);   // (the barriers' acquire empties L1, not the read-only path)
    for (int k = __ldg(s.grp_ptr + g); k < k1; ++k) {
        const int i = __ldg(s.grp_sub + k);
        const uint32_t spk = __ldcg(a_spk + i), nact = __ldcg(a_nact + i);
        const double vsum = __ldcg(a_vsum + i);
        a_spk[i] = 0u;
        a_nact[i] = 0u;
        a_vsum[i] = 0.0;
        const uint32_t cnt = __ldg(s.sub_count + i);
        if (s.win_spk) s.win_spk[i] += spk;
        s.st_spk[row * s.n_sub + i] = (float)spk;
        s.st_mean[row * s.n_sub + i] = cnt ? (float)(vsum / (double)cnt) : __int_as_float(0x7fc00000);
        nact_sum += nact;
        spk_sum += (double)spk;
    }
    const int r = __ldg(s.grp_region + g);
    if (r >= 0 && s.bold.n_regions > 0) {
        const BoldDev& b = s.bold;
        const double rn = __ldg(b.region_n + r);
        const double act = rn > 0.0 ? spk_sum / rn : 0.0;
        b.act[r] = act;
        bold_region_step(b, r, act > 1e-5 ? act : 1e-5);
    }
    if (nact_sum) atomicAdd(s.st_nact + row, nact_sum);
}

__global__ void __launch_bounds__(kSmallThreads, 1) k_small(DevState s, SmallArgs a)
{
    extern __shared__ __align__(16) unsigned char small_sm[];
    __shared__ int sh_sub[kSmallWarps];
    __shared__ uint32_t sh_spk[kSmallWarps];
    __shared__ uint32_t sh_nact[kSmallWarps];
    __shared__ double sh_vsum[kSmallWarps];
    __shared__ uint32_t sh_rows[2];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int C = a.tiles_per_cta * kWarpNeurons;              // cells of a CTA
    float2* sJ0 = reinterpret_cast<float2*>(small_sm);
    float2* sJ1 = sJ0 + C;
    const uint32_t cap = a.cap;
    float2* sSW = sJ1 + C;                                     // slot weights [cap][C]
    uint32_t* sSP = reinterpret_cast<uint32_t*>(sSW + (size_t)cap * C);   // slot positions | kind [cap][C]
    uint32_t* sCnt = sSP + (size_t)cap * C;
    float* sV = reinterpret_cast<float*>(sCnt + C);
    float* sT = sV + C;
    uint32_t* sE0 = reinterpret_cast<uint32_t*>(sT + C);
    uint32_t* sLen = sE0 + C;
    uint32_t* sBits = sLen + C;                                // [2][kSmallMaxWords] firing bits of the network
    uint16_t* sList = reinterpret_cast<uint16_t*>(sBits + 2 * kSmallMaxWords);

    const int64_t n0 = (int64_t)blockIdx.x * C;
    const int cells = (int)(n0 >= s.N ? 0 : (s.N - n0 < C ? s.N - n0 : C));
    const int nw = (cells + 31) / 32;                          // words of this CTA
    // the warp's run of words
    const int w_b = wid < kSmallWarps ? nw * wid / kSmallWarps : 0, w_e = wid < kSmallWarps ? nw * (wid + 1) / kSmallWarps : 0;
    const unsigned long long step0 = s.ctl->steps_done;
    float t = s.ctl->t;
    const float noise_rate = a.noise_rate;
    const int isolated = a.isolated;
    for (int i = threadIdx.x; i < cells; i += kSmallThreads) {
        sV[i] = __ldcg(s.V + n0 + i);
        sT[i] = __ldcg(s.tlast + n0 + i);
        sJ0[i] = __ldcg(s.J2 + n0 + i);
        sJ1[i] = __ldcg(s.J2 + s.j_ps + n0 + i);
        const int64_t e0 = __ldg(s.qrow + n0 + i);
        sE0[i] = (uint32_t)e0;
        sLen[i] = (uint32_t)(__ldg(s.qrow + n0 + i + 1) - e0);
        sCnt[i] = 0u;
    }
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < a.n_steps; i += kSmallThreads) s.st_nact[i] = 0u;
    if (threadIdx.x < 2) sh_rows[threadIdx.x] = 0u;
    // noise threshold: u01(x) < rate exactly when (x >> 8) < ceil(rate 2^24)
    const uint32_t noise_thr = noise_rate >= 0.0f ? (uint32_t)fminf(ceilf(noise_rate * 16777216.0f), 16777216.0f) : 0u;
    const uint32_t cnt_addr = smem_u32(sCnt), sp_addr = smem_u32(sSP), sw_addr = smem_u32(sSW), bits_addr = smem_u32(sBits);
    small_barrier();   // every CTA of the cluster has started and cleared its counts

    // J of the lane's neuron (cell i) with its slots added, which are emptied
    auto fold = [&](int i, int64_t n, bool valid, const uint32_t* gbits) -> float4 {
        float4 J = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t c = 0u;
        if (valid) {
            const float2 x = sJ0[i], y = sJ1[i];
            J = make_float4(x.x, x.y, y.x, y.y);
            c = sCnt[i];
            if (c) sCnt[i] = 0u;
        }
        float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        auto rec = [&](uint32_t k) -> uint4 {
            const float2 w = sSW[k * C + i];
            return make_uint4(sSP[k * C + i], 0u, __float_as_uint(w.x), __float_as_uint(w.y));
        };
        if (c && c <= 2u) {   // one or two terms added to +0: the same float in either order
            slot_add(rec(0), a0, a1, a2, a3);
            if (c == 2u) slot_add(rec(1), a0, a1, a2, a3);
        } else if (c && c <= 8u) {
            uint4 v[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
                v[k] = make_uint4(kIndexMask, 0u, 0u, 0u);
                if (k < c) v[k] = rec(k);
            }
            // odd-even merge network: the first four keys, then (more than four records) all eight
            slot_order(v[0], v[1]); slot_order(v[2], v[3]); slot_order(v[0], v[2]); slot_order(v[1], v[3]);
            slot_order(v[1], v[2]);
            if (c > 4u) {
                slot_order(v[4], v[5]); slot_order(v[6], v[7]); slot_order(v[4], v[6]); slot_order(v[5], v[7]);
                slot_order(v[5], v[6]);
                slot_order(v[0], v[4]); slot_order(v[1], v[5]); slot_order(v[2], v[6]); slot_order(v[3], v[7]);
                slot_order(v[2], v[4]); slot_order(v[3], v[5]);
                slot_order(v[1], v[2]); slot_order(v[3], v[4]); slot_order(v[5], v[6]);
            }
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
                if (k < c) slot_add(v[k], a0, a1, a2, a3);
        } else if (c && c <= cap) {   // more: the next position found by scanning
            uint32_t last = 0u;
            for (uint32_t q = 0; q < c; ++q) {
                uint32_t bp = 0xffffffffu, bk = 0u;
                for (uint32_t k = 0; k < c; ++k) {
                    const uint32_t pk = sSP[k * C + i] & kIndexMask;
                    if ((q == 0u || pk > last) && pk < bp) { bp = pk; bk = k; }
                }
                slot_add(rec(bk), a0, a1, a2, a3);
                last = bp;
            }
        }
        float4 sum = make_float4(a0, a1, a2, a3);
        unsigned m = __ballot_sync(0xffffffffu, c > cap);   // overflowed: the whole row, in order
        while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            const float4 g = small_gather_row(s, gbits, n - lane + l, lane);
            if (lane == l) sum = g;
        }
        return add4(J, sum);
    };

    unsigned long long events = 0;
    const bool worker = wid < kSmallWarps;
    // statistics groups: the lanes of the CTAs' last warps (a group stays with its thread)
    const int g0 = (int)blockIdx.x + (int)gridDim.x * lane, gstride = (int)gridDim.x * 32;
    auto fold_stats = [&](int par, int64_t row) {
        for (int g = g0; g < s.n_groups; g += gstride) small_stats(s, a, par, row, g);
        if (blockIdx.x == 0 && lane == 0) {
            uint32_t* const unm = par ? a.unmapped1 : a.unmapped0;
            const uint32_t un = __ldcg(unm);
            if (un) { *unm = 0u; atomicAdd(s.st_nact + row, un); }
        }
    };
    for (int k = 0; k < a.n_steps; ++k) {
        const unsigned long long step = step0 + (unsigned long long)k;
        const int par = k & 1;
        uint32_t* const a_spk = par ? a.spk1 : a.spk0;
        uint32_t* const a_nact = par ? a.nact1 : a.nact0;
        double* const a_vsum = par ? a.vsum1 : a.vsum0;
        uint32_t* const a_unm = par ? a.unmapped1 : a.unmapped0;
        const uint32_t* const gbits = sBits + (par ^ 1) * kSmallMaxWords;
        t = __fadd_rn(t, s.dt);
        // statistics of the current run of one-class words: per lane, reduced when the subblock changes
        int cur_sub = -1;
        uint32_t acc_spk = 0, acc_nact = 0;
        double acc_v = 0.0;
        uint32_t cur_cls = kMixedTile;   // class held in p
        ParamClass p;
        int64_t q_off = 0;               // the member's first tile and noise stream
        uint32_t q_stream = s.stream_id;
        U4 rnd = {0u, 0u, 0u, 0u};

        // ---- phase A: update
#pragma unroll 1
        for (int w = w_b; w < w_e; ++w) {
            const int64_t base = n0 + w * 32;
            const int64_t n = base + lane;
            const int64_t tile = base / kWarpNeurons;
            const int i = w * 32 + lane;
            const bool whole = base + 32 <= s.N;
            const uint32_t tcls = __ldg(s.tile_cls + tile);
            const bool mixed = tcls == kMixedTile;
            const uint32_t c0 = mixed ? __ldg(s.cls + tile * kWarpNeurons) : tcls;
            if (c0 != cur_cls) {
                cur_cls = c0;
                p = load_class(s.pc, c0);
                q_off = 0;
                q_stream = s.stream_id;
                if (s.member_start && p.member >= 0) {   // noise words as in k_step: member-local inside an ensemble
                    q_off = __ldg(s.member_start + p.member) / kWarpNeurons;
                    q_stream += (uint32_t)p.member;
                }
            }
            if (w == w_b || (w & 3) == 0)
                rnd = philox4x32_10(U4{(uint32_t)((uint64_t)(tile - q_off) * 32 + lane), q_stream, (uint32_t)step,
                                       (uint32_t)(step >> 32)},
                                    (uint32_t)s.seed, (uint32_t)(s.seed >> 32));
            const uint32_t word = (w & 2) ? ((w & 1) ? rnd.w : rnd.z) : ((w & 1) ? rnd.y : rnd.x);
            float4 J;
            if (k > 0) {
                J = fold(i, n, n < s.N, gbits);
            } else {   // the previous launch left J complete
                const float2 x = n < s.N ? sJ0[i] : make_float2(0.f, 0.f), y = n < s.N ? sJ1[i] : make_float2(0.f, 0.f);
                J = make_float4(x.x, x.y, y.x, y.y);
            }
            // V after the step (models/block.py:89-111) before the minimum with V_th
            auto membrane = [&](const ParamClass& q) -> float {
                const float v = sV[i];
                const float isyn = isyn_of(q, v, J);
                const float mainp = __fmul_rn(-q.gL, __fsub_rn(v, q.VL));
                const float cd = __fadd_rn(__fadd_rn(mainp, isyn), q.Iext);
                const float vn = __fadd_rn(v, __fmul_rn(q.rCdt, cd));
                return t >= __fadd_rn(sT[i], q.Tref) ? vn : q.Vreset;
            };
            auto store_state = [&](float v, float4 d, bool act) {
                sV[i] = v;
                if (a.write_v) __stcg(s.V + n, v);
                sJ0[i] = make_float2(d.x, d.y);
                sJ1[i] = make_float2(d.z, d.w);
                if (act) sT[i] = t;
            };
            uint32_t ma, mn;
            if (whole && !mixed && p.sub >= 0 && p.sub < s.n_sub && !isnan(p.Vth)) {
                // one class: the firing masks are ballots of the predicates, the minimum with V_th is
                // the threshold test's select (a NaN stays NaN, as in torch.minimum)
                if (p.sub != cur_sub) {
                    if (cur_sub >= 0) {
                        const uint32_t cs = __reduce_add_sync(0xffffffffu, acc_spk), cn = __reduce_add_sync(0xffffffffu, acc_nact);
                        double vw = acc_v;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) vw += __shfl_xor_sync(0xffffffffu, vw, o);
                        if (lane == 0) {
                            atomicAdd(a_spk + cur_sub, cs);
                            atomicAdd(a_nact + cur_sub, cn);
                            atomicAdd(a_vsum + cur_sub, vw);
                        }
                    }
                    cur_sub = p.sub; acc_spk = 0; acc_nact = 0; acc_v = 0.0;
                }
                const float vs = membrane(p);
                const bool act = vs >= p.Vth;
                const float v = act ? p.Vth : vs;
                const bool nz = noise_rate >= 0.0f ? (word >> 8) < noise_thr : u01(word) < p.noise;
                const bool na = nz || (act && !isolated);
                store_state(v, mul4(J, p.decay), act);
                ma = __ballot_sync(0xffffffffu, act);
                mn = __ballot_sync(0xffffffffu, na);
                if (act) ++acc_spk;
                if (na) ++acc_nact;
                acc_v += (double)v;
            } else {
                // a partial word, a tile of several classes, or neurons outside the subblocks
                const bool valid = n < s.N;
                bool act = false, na = false;
                int sub = -1;
                float v = 0.0f;
                if (valid) {
                    const ParamClass q = load_class(s.pc, mixed ? __ldg(s.cls + n) : tcls);
                    const float vs = membrane(q);
                    act = vs >= q.Vth;
                    v = (vs < q.Vth || isnan(vs)) ? vs : q.Vth;
                    const bool nz = noise_rate >= 0.0f ? (word >> 8) < noise_thr : u01(word) < q.noise;
                    na = isolated ? nz : (nz || act);
                    sub = q.sub;
                    store_state(v, mul4(J, q.decay), act);
                }
                ma = __ballot_sync(0xffffffffu, act);
                mn = __ballot_sync(0xffffffffu, na);
                unsigned rem = __ballot_sync(0xffffffffu, valid);
                while (rem) {   // one reduction per subblock
                    const int sb = __shfl_sync(0xffffffffu, sub, __ffs(rem) - 1);
                    const bool mine = valid && sub == sb;
                    const unsigned m = __ballot_sync(0xffffffffu, mine);
                    rem &= ~m;
                    double vw = mine ? (double)v : 0.0;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) vw += __shfl_xor_sync(0xffffffffu, vw, o);
                    if (lane == 0) {
                        if (sb >= 0 && sb < s.n_sub) {
                            if (ma & m) atomicAdd(a_spk + sb, (uint32_t)__popc(ma & m));
                            if (mn & m) atomicAdd(a_nact + sb, (uint32_t)__popc(mn & m));
                            atomicAdd(a_vsum + sb, vw);
                        } else if (mn & m) {
                            atomicAdd(a_unm, (uint32_t)__popc(mn & m));
                        }
                    }
                }
            }
            const int64_t gw = base >> 5;   // the word's place in the network's bitmasks
            if (lane < (int)gridDim.x) {    // the firing bits to every CTA of the cluster
                const uint32_t dst = mapa_u32(bits_addr + (uint32_t)((par * kSmallMaxWords + (int)gw) * 4), (uint32_t)lane);
                asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(dst), "r"(mn) : "memory");
            }
            if (lane == 0 && (s.n_samples > 0 || k + 1 == a.n_steps)) {
                s.abits[gw] = ma;
                ((step & 1ull) ? s.bits[1] : s.bits[0])[gw] = mn;
            }
            if (mn) {   // the word's firing rows into the CTA's list
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&sh_rows[par], (uint32_t)__popc(mn));
                at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(mn & ((1u << lane) - 1u));
                if ((mn >> lane) & 1u) sList[at] = (uint16_t)i;
            }
        }
        acc_spk = __reduce_add_sync(0xffffffffu, acc_spk);
        acc_nact = __reduce_add_sync(0xffffffffu, acc_nact);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc_v += __shfl_xor_sync(0xffffffffu, acc_v, o);
        if (lane == 0 && worker) { sh_sub[wid] = cur_sub; sh_spk[wid] = acc_spk; sh_nact[wid] = acc_nact; sh_vsum[wid] = acc_v; }
        small_barrier();

        // ---- phase B: the last warp adds this step's subblock sums and folds the previous step's statistics, ...
        if (!worker) {
            if (lane == 0) sh_rows[par ^ 1] = 0u;
            const int l = lane < kSmallWarps ? lane : kSmallWarps - 1;
            const int sb = lane < kSmallWarps ? sh_sub[l] : -1;
            const int sf = __shfl_sync(0xffffffffu, sb, 0);
            double v = sb >= 0 ? sh_vsum[l] : 0.0;
            uint32_t cs = sb >= 0 ? sh_spk[l] : 0u, cn = sb >= 0 ? sh_nact[l] : 0u;
            const bool one = __all_sync(0xffffffffu, sb < 0 || sb == sf);
            if (one) {                                    // one subblock in the CTA: one set of atomics
                cs = __reduce_add_sync(0xffffffffu, cs);
                cn = __reduce_add_sync(0xffffffffu, cn);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (sb >= 0 && (!one || lane == 0)) {
                if (cs) atomicAdd(a_spk + sb, cs);
                if (cn) atomicAdd(a_nact + sb, cn);
                atomicAdd(a_vsum + sb, v);
            }
        }
        if (!worker && k > 0) fold_stats(par ^ 1, k - 1);
        // ... the others scatter the CTA's firing rows, quarter by quarter (entries 32 h + lane, + 128, ...)
        const int units = (int)sh_rows[par] * 4;
        for (int u0 = worker ? wid : units; u0 < units; u0 += kSmallWarps * kSmallUnits) {
            uint32_t e[kSmallUnits];
            int left[kSmallUnits];
            int most = 0;
#pragma unroll
            for (int u = 0; u < kSmallUnits; ++u) {
                const int q = u0 + u * kSmallWarps;
                e[u] = 0u;
                left[u] = 0;
                if (q < units) {
                    const int i = sList[q >> 2];
                    const int off = (q & 3) * 32 + lane;
                    e[u] = sE0[i] + (uint32_t)off;
                    left[u] = (int)sLen[i] - off;
                    if ((q & 3) == 0 && lane == 0) events += (unsigned long long)sLen[i];
                }
                most = left[u] + lane > most ? left[u] + lane : most;   // warp-uniform: lane 0's
            }
            most = __reduce_max_sync(0xffffffffu, (unsigned)most);
            for (int o = 0; o < most; o += 128) {
                uint32_t c[kSmallUnits], pp[kSmallUnits];
                float2 wt[kSmallUnits];
#pragma unroll
                for (int u = 0; u < kSmallUnits; ++u) {
                    c[u] = 0xffffffffu;
                    if (o < left[u]) {
                        c[u] = __ldg(s.qcol + e[u] + o);
                        wt[u] = __ldg(s.qw + e[u] + o);
                        pp[u] = __ldg(s.qpos + e[u] + o);
                    }
                }
                uint32_t at[kSmallUnits], cta[kSmallUnits], cell[kSmallUnits];
#pragma unroll
                for (int u = 0; u < kSmallUnits; ++u) {
                    at[u] = cap;
                    if (c[u] != 0xffffffffu) {
                        const uint32_t post = c[u] & kIndexMask;
                        cta[u] = ((post >> 7) * a.tile_magic) >> 16;
                        cell[u] = post - cta[u] * (uint32_t)C;
                        const uint32_t dst = mapa_u32(cnt_addr + cell[u] * 4u, cta[u]);
                        asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(at[u]) : "r"(dst) : "memory");
                    }
                }
#pragma unroll
                for (int u = 0; u < kSmallUnits; ++u) {
                    if (at[u] < cap) {
                        const uint32_t idx = at[u] * (uint32_t)C + cell[u];
                        const uint32_t dp = mapa_u32(sp_addr + idx * 4u, cta[u]), dw = mapa_u32(sw_addr + idx * 8u, cta[u]);
                        asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(dp), "r"(pp[u] | (c[u] & kKindBit)) : "memory");
                        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" :: "r"(dw), "f"(wt[u].x), "f"(wt[u].y) : "memory");
                    }
                }
            }
        }
        if (s.n_samples > 0) {
            const int64_t ring = (int64_t)(step % (unsigned long long)s.samp_cap);
            for (int i = (int)blockIdx.x * kSmallThreads + (int)threadIdx.x; i < s.n_samples; i += (int)gridDim.x * kSmallThreads) {
                const uint32_t n = s.samples[i];
                s.samp_spk[ring * s.n_samples + i] = (uint8_t)((__ldcg(s.abits + (n >> 5)) >> (n & 31)) & 1u);
                s.samp_v[ring * s.n_samples + i] = __ldcg(s.V + n);
            }
        }
        small_barrier();
    }
    if (a.n_steps > 0) {
        const int k = a.n_steps;   // the last step's statistics
        const int par = (k - 1) & 1;
        if (!worker) fold_stats(par, k - 1);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s.ctl->t = t;
            s.ctl->steps_done = step0 + (unsigned long long)k;
            s.ctl->run_base = step0 + (unsigned long long)k;
        }
        // the last step's slots into J, which a run leaves complete; the state back to global memory
        for (int w = w_b; w < w_e; ++w) {
            const int i = w * 32 + lane;
            const int64_t n = n0 + i;
            const float4 J = fold(i, n, n < s.N, sBits + par * kSmallMaxWords);
            if (n < s.N) {
                __stcg(s.J2 + n, make_float2(J.x, J.y));
                __stcg(s.J2 + s.j_ps + n, make_float2(J.z, J.w));
                __stcg(s.V + n, sV[i]);
                __stcg(s.tlast + n, sT[i]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) events += __shfl_xor_sync(0xffffffffu, events, o);
        if (lane == 0 && worker) add_events(s, events, blockIdx.x * kSmallWarps + wid);
        if (a.host_nact) {   // the counts straight to the caller's host buffer, once every CTA has added its own
            small_barrier();
            if (blockIdx.x == 0) {
                for (int i = threadIdx.x; i < k; i += kSmallThreads) a.host_nact[i] = __ldcg(s.st_nact + i);
                if (threadIdx.x == 0) a.host_nact[k] = __ldcg(&s.ctl->err);
            }
        }
    }
}

}  // namespace dtb
