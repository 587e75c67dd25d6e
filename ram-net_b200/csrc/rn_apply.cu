// Prefill apply kernel: reads and updates over the event lists of rn_lists.cuh.
//
// One CTA per (b,h, group of CS channels, owner): the rows [rows][CS] of the owner's slots stay in shared memory for the
// whole sequence (128 KB at 4096 slots, 32 channels, 4 owners).  A step is two sweeps with a barrier behind each:
//     gather   token-major: y_t = sum coef * row over the read entries of token t, rows of the state and of x alike
//     update   slot-major: s += gain * (x - s) for the writes of a slot, in time order
// Rows of 128 bytes are read without bank conflicts whatever slots a warp's units touch, where 32-byte rows (one CTA
// holding all slots of eight channels) cost 1.6 to 2 times the conflict-free count, and an entry is decoded once per 32
// channels instead of once per 8.
//
// Sixteen compute warps do the two sweeps and nothing else; four service warps keep the lists (bulk copies) and the x rows
// of the steps two deep and finish y.  The owners of a channel group are a cluster: each sums the reads of its own slots,
// and the partial rows of y travel to the CTA that finishes the token (token / (L / N)) by stores through distributed
// shared memory (st.async, one barrier update per 16 bytes, was slower by a fifth).  Barriers, all with two buffers by parity of the step:
//     full    lists and x rows of a step are there          (bulk copy + one arrival per service warp)
//     free    the compute warps are done with a step         (one arrival)
//     yfull   the parts of y of a step are there             (one arrival per CTA of the cluster)
//     yfree   every CTA of the cluster has finished the y of a step: its buffers may be sent to again  (one arrival each)
// No float atomics; owners are summed in order: results do not vary from run to run.  Every wait is bounded (about a
// second); one that runs out is reported through the status word and ends the kernel.
#include "rn_lists.cuh"

constexpr int RN_AP_COMPUTE = 512, RN_AP_SERVICE = 128, RN_AP_THREADS = RN_AP_COMPUTE + RN_AP_SERVICE;

// shared-memory accesses by 32-bit address
__device__ __forceinline__ uint32_t rn_lds_u8(uint32_t a) { uint32_t v; asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t rn_lds_u16(uint32_t a) { uint32_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 rn_lds_u2(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 rn_lds_u4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 rn_lds_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void rn_sts_f4(uint32_t a, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void rn_st_cluster4(uint32_t addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void rn_mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void rn_mbar_arrive_remote(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <bool CLUSTER>
__device__ __forceinline__ bool rn_mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (CLUSTER)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
template <bool CLUSTER>
__device__ __noinline__ bool rn_mbar_wait_slow(uint32_t bar, uint32_t parity) {
    const long long start = clock64();
    while (!rn_mbar_try<CLUSTER>(bar, parity))
        if (clock64() - start > (1ll << 31)) return false;
    return true;
}
template <bool CLUSTER>
__device__ __forceinline__ bool rn_mbar_wait(uint32_t bar, uint32_t parity) {  // bounded: about a second
    return rn_mbar_try<CLUSTER>(bar, parity) || rn_mbar_wait_slow<CLUSTER>(bar, parity);
}
// barrier ID of THREADS threads; the answer is whether any of them brought `bad`
template <int ID, int THREADS>
__device__ __forceinline__ bool rn_bar_or(bool bad) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(uint32_t(bad)), "n"(ID), "n"(THREADS) : "memory");
    return any != 0;
}
__device__ __forceinline__ bool rn_compute_sync(bool bad) { return rn_bar_or<1, RN_AP_COMPUTE>(bad); }
__device__ __forceinline__ float rn_dot4(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }
// the same whichever half a unit holds first: which unit has a row varies from run to run
__device__ __forceinline__ float rn_dot8(float4 a0, float4 b0, float4 a1, float4 b1) { return rn_dot4(a0, b0) + rn_dot4(a1, b1); }
__device__ __forceinline__ void rn_stg_f4(float *p, float4 v) { __stcs(reinterpret_cast<float4 *>(p), v); }

// MODE: RN_FORWARD, or RN_REPLAY, the first sweep of the backward pass, over lists of its own (rn_bwd_lists.cu): it runs the state
// again, the gather takes <row, d_y> of every read instead of sums (no y, hence no cluster), the update stores x - row of every
// write for the reverse sweep.  The reads of an owner are dealt evenly to the units, since nothing is summed over a token.
template <typename T, int CS, int MODE>
__global__ void __launch_bounds__(RN_AP_THREADS, 1) rn_apply_kernel(const RnListParams p) {
    constexpr int LPU = CS / 4;                    // lanes of a row (state and x transfers, y)
    constexpr bool Y = MODE != RN_REPLAY;          // rows of y (d_x) are finished
    constexpr int ROW = CS * 4;                    // bytes of a row
    constexpr int XT = RN_LST_LMAX * LPU / RN_AP_SERVICE;  // x pieces per service thread
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) uint64_t bars[8];      // full, free, yfull, yfree
    __shared__ volatile int stop;

    const int lg = p.lg, N = 1 << lg, L = p.L, C = p.C, rows = 1 << p.lr;
    const int own = blockIdx.x & (N - 1);
    const int grp = int(blockIdx.x >> lg) % p.ngroups;
    const int bh = int(blockIdx.x >> lg) / p.ngroups;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x;
    const int Lq = L >> lg;                        // tokens this CTA finishes per step
    const unsigned char *recs = p.recs + int64_t(bh) * p.nblocks * p.blk_bytes;
    const uint4 *first = p.first + ((int64_t(bh) << lg) + own) * p.nblocks;
    const uint32_t data_at = rn_list_data_at(L, lg);

    unsigned char *S = dyn;                        // [rows][CS] f32
    unsigned char *xt = S + (size_t(ROW) << p.lr); // [2][L][CS]; read entries count its rows on from those of S
    unsigned char *yb = xt + size_t(2 * L) * ROW;  // [2][N sources][Lq][CS] (N > 1); RN_REPLAY: d_y, as xt
    unsigned char *lists = yb + (N > 1 || !Y ? size_t(2 * L) * ROW : 0);
    const uint32_t bar0 = rn_smem_u32(bars);
    auto FULL = [&](int s) { return bar0 + (s & 1) * 8u; };
    auto FREE = [&](int s) { return bar0 + 16u + (s & 1) * 8u; };
    auto YFULL = [&](int s) { return bar0 + 32u + (s & 1) * 8u; };
    auto YFREE = [&](int s) { return bar0 + 48u + (s & 1) * 8u; };
    auto phase = [](int s) { return uint32_t(s >> 1) & 1u; };

    if (tid == 0) {
        stop = 0;
        for (int i = 0; i < 2; ++i) {
            rn_mbar_init(&bars[i], 1 + RN_AP_SERVICE / 32);
            rn_mbar_init(&bars[2 + i], 1);
            rn_mbar_init(&bars[4 + i], N);
            rn_mbar_init(&bars[6 + i], N);
        }
        rn_mbar_fence_init();
    }
    // ---- the rows of this CTA's slots (a = row * N + owner XOR the row's folded digits) -------------------------------
    auto slot_of = [&](int r) {
        const int f = lg == 0 ? 0 : lg == 1 ? rn_fold<1>(r) : lg == 2 ? rn_fold<2>(r) : rn_fold<3>(r);
        return (r << lg) | (own ^ f);
    };
    const int words = rn_touch_words(p.lr);
    const uint32_t *touch = p.touch ? p.touch + ((int64_t(bh) << lg) + own) * 2 * words : nullptr;
    __syncthreads();
    if (Y && N > 1) rn_cluster_sync();  // every CTA's barriers are set up before the first remote arrival

    bool failed = false;
    if (tid >= RN_AP_COMPUTE) {
        // ================================ service warps ================================================================
        const int sid = tid - RN_AP_COMPUTE, lane = tid & 31;
        const int ul = sid % LPU, st0 = sid / LPU;         // this thread's lane of a row and first token
        constexpr int TSTEP = RN_AP_SERVICE / LPU;
        const int ch = grp * CS + ul * 4;
        const bool chan_ok = ch < C;
        const T *x = static_cast<const T *>(p.x) + b * p.xb + h * p.xh + ch;
        T *y = static_cast<T *>(p.y) + b * p.yb + h * p.yh + ch;
        uint32_t peer_free = 0;
        if (sid < N) peer_free = rn_mapa(bar0 + 48u, uint32_t(sid));

        rn_wait_for_front();                               // the lists are there

        // x of the block that comes next: requested a block ahead, kept as loaded until it is put into shared memory
        RnRaw4<T> xr[XT], dr[Y ? 1 : XT];
        const T *dy = Y ? nullptr : static_cast<const T *>(p.dy) + b * p.dyb + h * p.dyh + ch;
        int ptok[2] = {0, 0}, plen[2] = {0, 0};            // tokens of the two steps before, by parity
        auto request = [&](int bk) {
            const int len = chan_ok ? p.T - bk * L - st0 : 0;
            const T *src = x + int64_t(bk * L + st0) * p.xt, *dsrc = Y ? nullptr : dy + int64_t(bk * L + st0) * p.dyt;
#pragma unroll
            for (int i = 0; i < XT; ++i) {
                xr[i] = rn_zero_raw4<T>();
                if (i * TSTEP < len && st0 + i * TSTEP < L) xr[i] = rn_load_raw4<T>(src);
                src += int64_t(TSTEP) * p.xt;
                if constexpr (!Y) {
                    dr[i] = rn_zero_raw4<T>();
                    if (i * TSTEP < len && st0 + i * TSTEP < L) dr[i] = rn_load_raw4<T>(dsrc);
                    dsrc += int64_t(TSTEP) * p.dyt;
                }
            }
        };
        // The table is read two steps ahead, x a block; the copy of a list starts as soon as its buffer is free.  Turn -1 only
        // requests the first x, the last two turns only finish y: every part of the loop stands here once, which keeps
        // the kernel's code small (instruction fetch is what a longer one would wait for).  Failure is collective: one warp
        // that gives up takes the others along at the barrier of the turn.
        int blk = 0, st = 0, cur_blk = -1, cur_st = 0;
        uint4 cur = make_uint4(0, 0, 0, 0), nxt = rn_step_entry(p, first, recs, 0, 0, own);
        int last = 1 << 30;
#pragma unroll 1
        for (int step = -1; step < last + 2; ++step) {
            const bool more = st + 1 < rn_steps_of(nxt);
            const int nblk = more ? blk : blk + 1, nst = more ? st + 1 : 0;   // (blk, st): the step after this one
            uint4 nn = make_uint4(0, 0, 0, 0);
            if (rn_steps_of(nxt) != 0) nn = rn_step_entry(p, first, recs, nblk, nst, own);
            if (step >= 0 && step < last) {
                if (step >= 2 && !rn_mbar_wait<false>(FREE(step), phase(step - 2))) failed = true;
                if (sid == 0) {
                    const uint32_t bytes = (cur.x >> 16) << 4;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(FULL(step)), "r"(bytes) : "memory");
                    rn_bulk_g2s(lists + size_t(step & 1) * p.list_max, recs + cur_blk * p.blk_bytes + data_at + (size_t(cur.x & 0xffffu) << 4),
                                bytes, &bars[step & 1]);
                }
                if (cur_st == 0) {
                    const size_t at = (size_t(cur_blk & 1) * L + st0) * ROW + ul * 16;
#pragma unroll
                    for (int i = 0; i < XT; ++i) {
                        rn_pin(xr[i]);
                        if constexpr (!Y) rn_pin(dr[i]);
                    }
#pragma unroll
                    for (int i = 0; i < XT; ++i)
                        if (st0 + i * TSTEP < L) {
                            *reinterpret_cast<float4 *>(xt + at + i * TSTEP * ROW) = rn_cvt_raw4(xr[i]);
                            if constexpr (!Y) *reinterpret_cast<float4 *>(yb + at + i * TSTEP * ROW) = rn_cvt_raw4(dr[i]);
                        }
                }
                __syncwarp();
                if (lane == 0) rn_mbar_arrive(FULL(step));
            }
            if (step < last && cur_st == 0) {
                if (cur_blk + 1 < p.nblocks) request(cur_blk + 1);
            }
            if (rn_steps_of(nxt) == 0 && step + 1 < last) last = step + 1;
            if (Y && N > 1) {
                bool arrive = false;
                if (step >= 2) {                           // y of the step before the last, from the parts of all owners
                    const int s = step - 2, mine = max(0, min(Lq, plen[s & 1] - own * Lq));
                    if (!rn_mbar_wait<true>(YFULL(s), phase(s))) failed = true;
                    const unsigned char *src = yb + (size_t(s & 1) * L + st0) * ROW + ul * 16;
                    T *dst = y + int64_t(ptok[s & 1] + own * Lq + st0) * p.yt;
#pragma unroll 1
                    for (int t = st0; t < mine && !failed; t += TSTEP) {
                        float4 a = *reinterpret_cast<const float4 *>(src);
#pragma unroll 1
                        for (int o = 1; o < N; ++o) {
                            const float4 v = *reinterpret_cast<const float4 *>(src + size_t(o) * Lq * ROW);
                            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
                        }
                        if (chan_ok) rn_store4<T>(dst, a);
                        src += TSTEP * ROW;
                        dst += int64_t(TSTEP) * p.yt;
                    }
                    arrive = true;
                }
                // all service warps are done with the buffer before the cluster hears of it
                failed = rn_bar_or<2, RN_AP_SERVICE>(failed || stop);
                if (failed) break;
                if (arrive && sid < N) rn_mbar_arrive_remote(peer_free + (step & 1) * 8u);
                if (step >= 0 && step < last) {
                    ptok[step & 1] = cur_blk * L + int(cur.y & 0xffffu);
                    plen[step & 1] = int(cur.y >> 16);
                }
            } else {
                failed = rn_bar_or<2, RN_AP_SERVICE>(failed || stop);
                if (failed || step >= last) break;
            }
            cur = nxt;
            cur_blk = blk;
            cur_st = st;
            nxt = nn;
            blk = nblk;
            st = nst;
        }
        if (failed) stop = 1;
    } else {
        // ================================ compute warps ================================================================
        // A unit of CS / 8 lanes has a row in two 16-byte pieces per lane, one in each half of the row; odd units take the
        // halves the other way round, so that the eight lanes of a shared-memory access cover all banks.
        constexpr int LPU = CS / 8, NU = RN_AP_COMPUTE / LPU, HALF = ROW / 2;
        const int u = tid / LPU, ul = tid % LPU;
        const int upt = min(NU / L, 32 / LPU);             // units of a token: consecutive ones in one warp
        const int tu = u / upt, part = u - tu * upt;       // place among the tokens, place among the token's units
        const uint32_t lane_off = ul * 16 + (u & 1) * HALF;
        const uint32_t sl = rn_smem_u32(S) + lane_off, xl = rn_smem_u32(xt) + lane_off, yl = rn_smem_u32(yb) + uint32_t(own * Lq * ROW) + lane_off;
        const int ch0 = grp * CS + int(lane_off) / 4, ch1 = grp * CS + int(lane_off ^ HALF) / 4;
        T *y = static_cast<T *>(p.y) + b * p.yb + h * p.yh;
        const uint32_t dy_tile = rn_smem_u32(yb) + lane_off;                                             // RN_REPLAY
        // RN_REPLAY: this lane's channels of token 0, write 0 in the workspace of the reverse sweep, in slices of its width
        auto delta_at = [&](int ch) {
            return MODE == RN_REPLAY ? p.delta + (int64_t(bh) * ((C + p.dcs - 1) / p.dcs) + ch / p.dcs) * p.T * p.Kw * p.dcs + ch % p.dcs : nullptr;
        };
        float *const delta0 = delta_at(ch0), *const delta1 = delta_at(ch1);
        const int lq = 31 - __clz(Lq);
        {   // the rows into shared memory, eight requests of a thread at a time; the service warps fetch the first step meanwhile
            constexpr int LD = CS / 4, STEP = RN_AP_COMPUTE / LD;
            if (touch != nullptr) rn_wait_for_front();     // the touched rows are the gains kernel's
            const int sub = tid % LD, ch = grp * CS + sub * 4;
            const float *src = p.slot_in && ch < C ? p.slot_in + int64_t(bh) * p.A * C + ch : nullptr;
#pragma unroll 1
            for (int r0 = tid / LD; r0 < rows; r0 += 8 * STEP) {
                float4 v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = r0 + i * STEP, a = slot_of(r);
                    const bool on = r < rows && src != nullptr && a < p.A && (touch == nullptr || (touch[r >> 5] >> (r & 31) & 1u) != 0);
                    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (on) v[i] = *reinterpret_cast<const float4 *>(src + int64_t(a) * C);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (r0 + i * STEP < rows) *reinterpret_cast<float4 *>(S + size_t(r0 + i * STEP) * ROW + sub * 16) = v[i];
            }
            if (rn_compute_sync(false)) failed = true;
        }
        int blk = -1;
#pragma unroll 1
        for (int step = 0;; ++step) {
            if (!rn_mbar_wait<false>(FULL(step), phase(step))) failed = true;
            const uint32_t lst = rn_smem_u32(lists) + uint32_t(step & 1) * p.list_max;
            const RnListHdr hd = *reinterpret_cast<const RnListHdr *>(lists + uint32_t(step & 1) * p.list_max);
            const int len = hd.len & 0xff, t0 = (hd.len >> 8) & 0x7f;
            const uint32_t tok = lst + 16, Wl = lst + (uint32_t(hd.atW) << 4);
            blk += t0 == 0;

            // ---- the units' shares ------------------------------------------------------------------------------------
            const uint32_t tile = uint32_t(blk & 1) * uint32_t(L * ROW);
            constexpr int LU = CS == 32 ? 7 : 8;               // log2 of NU
            static_assert((1 << LU) == NU, "units");
            [[maybe_unused]] auto share = [&](uint32_t table, uint32_t n, uint32_t &from, uint32_t &to) {  // run of unit u (rn_lists.cuh)
                const uint32_t q = (n + NU - 1) >> LU;
                from = to = n;
                if (u * q < n) {
                    from = rn_lds_u16(table + u * 2);
                    if ((u + 1) * q < n && u + 1 < NU) to = rn_lds_u16(table + u * 2 + 2);
                }
            };
            // ---- gather -------------------------------------------------------------------------------------------------
            int tk = -1;
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if constexpr (MODE == RN_REPLAY) {
                // <row, d_y> of every read: entries {coef, row of S or x | token << 12 | k << 19 | last of its read << 31} two at
                // a time.  All units of a warp go round together (they shuffle); one that is through goes on with zeros.
                float *out = p.part + ((int64_t(bh) * p.ngroups + grp) * p.T + blk * L) * p.Kr;
                uint32_t q, end;
                share(tok, hd.nR, q, end);
                const uint32_t rl = lst + (uint32_t(hd.atR) << 4);
                q = rl + q * 8u;
                end = rl + end * 8u;
                const uint2 none = make_uint2(0, 0);
                uint2 ea = none, eb = none;
                if (q < end) ea = rn_lds_u2(q);
                if (q + 8u < end) eb = rn_lds_u2(q + 8u);
                uint32_t have = ~0u;                           // the token whose d_y is in d0, d1
                float4 d0 = make_float4(0.f, 0.f, 0.f, 0.f), d1 = d0;
                float run = 0.f;                               // per lane; summed over the lanes at the end of a read
                auto dot = [&](uint32_t m, const float4 &r0, const float4 &r1) {
                    const uint32_t t = m >> 12 & 0x7fu;
                    if (t != have) {
                        d0 = rn_lds_f4(dy_tile + tile + t * ROW);
                        d1 = rn_lds_f4((dy_tile + tile + t * ROW) ^ HALF);
                        have = t;
                    }
                    return rn_dot8(r0, d0, r1, d1);
                };
#pragma unroll 1
                while (__any_sync(RN_FULL, q < end)) {
                    const uint2 ca = ea, cb = eb;
                    const uint32_t r0 = sl + (ca.y & 0xfffu) * ROW, r1 = sl + (cb.y & 0xfffu) * ROW;
                    const float4 a0 = rn_lds_f4(r0), b0 = rn_lds_f4(r0 ^ HALF), a1 = rn_lds_f4(r1), b1 = rn_lds_f4(r1 ^ HALF);
                    q += 16u;
                    ea = eb = none;
                    if (q < end) ea = rn_lds_u2(q);
                    if (q + 8u < end) eb = rn_lds_u2(q + 8u);
                    const float va = fmaf(__uint_as_float(ca.x), dot(ca.y, a0, b0), run);
                    run = int(ca.y) < 0 ? 0.f : va;
                    const float vb = fmaf(__uint_as_float(cb.x), dot(cb.y, a1, b1), run);
                    run = int(cb.y) < 0 ? 0.f : vb;
                    // even lanes add up the first entry, odd lanes the second
                    float v = (ul & 1) ? vb : va;
                    v += __shfl_xor_sync(RN_FULL, (ul & 1) ? va : vb, 1);
#pragma unroll
                    for (int o = 2; o < LPU; o <<= 1) v += __shfl_xor_sync(RN_FULL, v, o);
                    const uint32_t m = (ul & 1) ? cb.y : ca.y;
                    if (ul < 2 && int(m) < 0) out[int(m >> 12 & 0x7fu) * p.Kr + int(m >> 19 & 0x7fu)] = v;
                }
            } else {
                // two entries at a time, the next two requested before they are used
                uint32_t q = 0, end = 0;
                uint4 e = make_uint4(0, 0, 0, 0);
                if (tu < len) {
                    tk = rn_lds_u8(Wl - ((len + 15) & ~15) + tu);
                    const uint32_t rl = lst + (uint32_t(hd.atR) << 4);
                    q = rl + rn_lds_u16(tok + tk * 2) * 8u + part * 16u;
                    end = rl + rn_lds_u16(tok + tk * 2 + 2) * 8u;
                    if (q < end) e = rn_lds_u4(q);
                }
#pragma unroll 1
                while (q < end) {
                    const uint32_t r0 = sl + e.y, r1 = sl + e.w;
                    const float c0 = __uint_as_float(e.x), c1 = __uint_as_float(e.z);
                    const float4 a0 = rn_lds_f4(r0), b0 = rn_lds_f4(r0 ^ HALF), a1 = rn_lds_f4(r1), b1 = rn_lds_f4(r1 ^ HALF);
                    q += upt * 16u;
                    if (q < end) e = rn_lds_u4(q);
                    acc[0] = fmaf(c0, a0.x, acc[0]); acc[1] = fmaf(c0, a0.y, acc[1]); acc[2] = fmaf(c0, a0.z, acc[2]); acc[3] = fmaf(c0, a0.w, acc[3]);
                    acc[4] = fmaf(c0, b0.x, acc[4]); acc[5] = fmaf(c0, b0.y, acc[5]); acc[6] = fmaf(c0, b0.z, acc[6]); acc[7] = fmaf(c0, b0.w, acc[7]);
                    acc[0] = fmaf(c1, a1.x, acc[0]); acc[1] = fmaf(c1, a1.y, acc[1]); acc[2] = fmaf(c1, a1.z, acc[2]); acc[3] = fmaf(c1, a1.w, acc[3]);
                    acc[4] = fmaf(c1, b1.x, acc[4]); acc[5] = fmaf(c1, b1.y, acc[5]); acc[6] = fmaf(c1, b1.z, acc[6]); acc[7] = fmaf(c1, b1.w, acc[7]);
                }
            }
            if (Y && upt > 1) {
                // units of a token take the halves in turns: first bring both to the even unit's order
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float lo = (u & 1) ? acc[4 + i] : acc[i], hi = (u & 1) ? acc[i] : acc[4 + i];
                    acc[i] = lo;
                    acc[4 + i] = hi;
                }
#pragma unroll 1
                for (int o = LPU; o < LPU * upt; o <<= 1) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(RN_FULL, acc[i], o);
                }
            }
            // the y buffers of this parity are free again in every CTA of the cluster
            if (Y && N > 1 && tid == 0 && step >= 2 && !rn_mbar_wait<true>(YFREE(step), phase(step - 2))) failed = true;
            if (rn_compute_sync(failed || stop)) {
                failed = true;
                break;
            }
            if (Y && part == 0 && tk >= 0) {  // (an even unit where upt > 1)
                if (N > 1) {  // to the CTA that finishes the token, at this owner's place
                    const uint32_t q = uint32_t(tk) >> lq;
                    const uint32_t at = rn_mapa(yl + (uint32_t(step & 1) * uint32_t(L) + (uint32_t(tk) & uint32_t(Lq - 1))) * ROW, q);
                    rn_st_cluster4(at, make_float4(acc[0], acc[1], acc[2], acc[3]));
                    rn_st_cluster4(at ^ HALF, make_float4(acc[4], acc[5], acc[6], acc[7]));
                } else {
                    T *dst = y + int64_t(blk * L + t0 + tk) * p.yt;
                    if (ch0 < C) rn_store4<T>(dst + ch0, make_float4(acc[0], acc[1], acc[2], acc[3]));
                    if (ch1 < C) rn_store4<T>(dst + ch1, make_float4(acc[4], acc[5], acc[6], acc[7]));
                }
            }
            // ---- update ------------------------------------------------------------------------------------------
            const uint32_t xs = xl + tile, starts = MODE == RN_REPLAY ? tok + min(int(hd.nR), NU) * 2 : tok + (len + 1) * 2;
            const int64_t block_row = int64_t(blk * L) * p.Kw * p.dcs;
            // x - row of a write, for the reverse sweep
            auto keep = [&](uint32_t m, const float4 &s0, const float4 &s1, const float4 &x0, const float4 &x1) {
                if constexpr (MODE == RN_REPLAY) {
                    const int64_t at = block_row + (int(m >> 11 & 0x7fu) * p.Kw + int(m >> 18 & 0x7fu)) * p.dcs;
                    if (ch0 < C) rn_stg_f4(delta0 + at, make_float4(x0.x - s0.x, x0.y - s0.y, x0.z - s0.z, x0.w - s0.w));
                    if (ch1 < C) rn_stg_f4(delta1 + at, make_float4(x1.x - s1.x, x1.y - s1.y, x1.z - s1.z, x1.w - s1.w));
                }
            };
            auto apply = [&](float4 &s, const float4 &xv, float g) {
                s.x = fmaf(g, xv.x - s.x, s.x);
                s.y = fmaf(g, xv.y - s.y, s.y);
                s.z = fmaf(g, xv.z - s.z, s.z);
                s.w = fmaf(g, xv.w - s.w, s.w);
            };
            // slots written more than once: the row stays in registers along the slot's writes
#pragma unroll 1
            for (int i = u; i < hd.nM; i += NU) {
                uint32_t q = Wl + rn_lds_u16(starts + i * 2) * 8u;
                uint2 e = rn_lds_u2(q), e1 = rn_lds_u2(q + 8u);
                const uint32_t cell = sl + (e.y & 0x7ffu) * ROW;
                float4 s0 = rn_lds_f4(cell), s1 = rn_lds_f4(cell ^ HALF);
                uint32_t xa = xs + ((e.y >> 11) & 0x7fu) * ROW;
                float4 x0 = rn_lds_f4(xa), x1 = rn_lds_f4(xa ^ HALF);
                for (;;) {  // the next write and its x are requested before this one is applied
                    xa = xs + ((e1.y >> 11) & 0x7fu) * ROW;
                    const float4 n0 = rn_lds_f4(xa), n1 = rn_lds_f4(xa ^ HALF);
                    keep(e.y, s0, s1, x0, x1);
                    apply(s0, x0, __uint_as_float(e.x));
                    apply(s1, x1, __uint_as_float(e.x));
                    x0 = n0;
                    x1 = n1;
                    e = e1;
                    if (int(e.y) < 0) break;
                    q += 8u;
                    e1 = rn_lds_u2(q + 8u);
                }
                keep(e.y, s0, s1, x0, x1);
                apply(s0, x0, __uint_as_float(e.x));
                apply(s1, x1, __uint_as_float(e.x));
                rn_sts_f4(cell, s0);
                rn_sts_f4(cell ^ HALF, s1);
            }
            // slots written once
            int i = u - (hd.nM & (NU - 1));  // units with a slot of the former kind more start behind the others
            if (i < 0) i += NU;
            uint2 e = make_uint2(0, 0);
            if (i < hd.nS) e = rn_lds_u2(Wl + i * 8u);
#pragma unroll 1
            while (i < hd.nS) {
                const uint32_t cell = sl + (e.y & 0x7ffu) * ROW, xa = xs + ((e.y >> 11) & 0x7fu) * ROW;
                const uint32_t m = e.y;
                const float g = __uint_as_float(e.x);
                float4 s0 = rn_lds_f4(cell), s1 = rn_lds_f4(cell ^ HALF);
                const float4 x0 = rn_lds_f4(xa), x1 = rn_lds_f4(xa ^ HALF);
                i += NU;
                if (i < hd.nS) e = rn_lds_u2(Wl + i * 8u);
                keep(m, s0, s1, x0, x1);
                apply(s0, x0, g);
                apply(s1, x1, g);
                rn_sts_f4(cell, s0);
                rn_sts_f4(cell ^ HALF, s1);
            }
            if (rn_compute_sync(false)) break;
            if (tid == 0) rn_mbar_arrive(FREE(step));
            if (Y && N > 1 && tid < N) rn_mbar_arrive_remote(rn_mapa(YFULL(step), uint32_t(tid)));
            if ((hd.len & 0x8000) != 0) break;
        }
    }
    if (failed) {
        stop = 1;
        atomicMax(p.status, RN_STATUS_WAIT_TIMEOUT);
    }
    __syncthreads();
    if (!stop && p.slot_out != nullptr) {
        const int ul = tid % LPU, ch = grp * CS + ul * 4;
        float *dst = p.slot_out + int64_t(bh) * p.A * C + ch;
#pragma unroll 1
        for (int r = tid / LPU; r < rows; r += RN_AP_THREADS / LPU) {
            const int a = slot_of(r);
            const bool on = touch == nullptr || (touch[words + (r >> 5)] >> (r & 31) & 1u) != 0;
            if (on && ch < C && a < p.A) *reinterpret_cast<float4 *>(dst + int64_t(a) * C) = *reinterpret_cast<const float4 *>(S + size_t(r) * ROW + ul * 16);
        }
    }
    if (Y && N > 1) rn_cluster_sync();  // nobody's shared memory goes away while a store or arrival to it may be under way
}

template <typename T, int CS, int MODE>
static int rn_launch_apply_t(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    RN_CUDA(cudaFuncSetAttribute(rn_apply_kernel<T, CS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pl.smem_apply)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(p.B) * unsigned(p.H) * unsigned(pl.ngroups) * unsigned(pl.N));
    cfg.blockDim = dim3(RN_AP_THREADS);
    cfg.dynamicSmemBytes = pl.smem_apply;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = unsigned(pl.N);
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = MODE != RN_REPLAY && pl.N > 1 ? 2 : 1;
    RN_CUDA(cudaLaunchKernelEx(&cfg, rn_apply_kernel<T, CS, MODE>, p));
    return 0;
}

template <typename T>
static int rn_launch_mode(const RnListParams &p, const RnListPlan &pl, int mode, cudaStream_t stream) {
    if (mode == RN_FORWARD) return pl.cs == 32 ? rn_launch_apply_t<T, 32, RN_FORWARD>(p, pl, stream) : rn_launch_apply_t<T, 16, RN_FORWARD>(p, pl, stream);
    return pl.cs == 32 ? rn_launch_apply_t<T, 32, RN_REPLAY>(p, pl, stream) : rn_launch_apply_t<T, 16, RN_REPLAY>(p, pl, stream);
}

static int rn_launch_dtype(const RnListParams &p, const RnListPlan &pl, int mode, int dtype, cudaStream_t stream) {
    if (dtype == RN_F32) return rn_launch_mode<float>(p, pl, mode, stream);
    if (dtype == RN_F16) return rn_launch_mode<__half>(p, pl, mode, stream);
    return rn_launch_mode<__nv_bfloat16>(p, pl, mode, stream);
}

int rn_launch_apply(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream) {
    return rn_launch_dtype(p, pl, RN_FORWARD, dtype, stream);
}

int rn_launch_replay(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream) {
    return rn_launch_dtype(p, pl, RN_REPLAY, dtype, stream);
}
