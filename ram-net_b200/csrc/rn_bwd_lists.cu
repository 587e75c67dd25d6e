// Event lists of the replay of the backward pass (see rn_lists.cuh for the idea, rn_apply.cu for the sweep).
//
// The gains of all writes are known from the schedule kernel, so one kernel makes the finished lists, all blocks at once.  A
// read's entries carry no weight (its gradient is <row at the read, d_y>): {Π(1-g), row}, then {g_j Π(1-g), x(tau_j)} for the
// writes g_j before it in its step.  List of a step and owner (parts on 16-byte boundaries):
//   header RnListHdr
//   u16 run[]            first read entry of every unit (rn_runs);  u16 start[nM]  first write of every slot written more than once
//   {f32 gain, u32 row | token of the block << 11 | k << 18 | last of its slot << 31}[nW]   as in rn_lists.cuh
//   {f32 coef, u32 row of the state or of x | token of the block << 12 | k << 19 | last entry of its read << 31}[nR]
// Same phases as rn_lists_kernel; what bounds it is instruction issue and the latency of its barriers.
#include "rn_lists.cuh"

template <int LG, int KP>
__global__ void __launch_bounds__(RN_LISTS_THREADS, 1) rn_replay_lists_kernel(const RnListParams p) {
    constexpr int NT = RN_LISTS_THREADS, N = 1 << LG;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint32_t nsingle[N], nmulti[N];  // slots written once; writes of the others | such slots << 16
    __shared__ uint32_t own_reads[N];
    __shared__ uint32_t at_hdr[N + 1], at_W[N], at_R[N];  // in 16 bytes from the step's first list
    __shared__ int s_fail;

    const int bh = blockIdx.x / p.nblocks, blk = blockIdx.x % p.nblocks;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Kw = p.Kw, Kr = p.Kr, KT = Kw + Kr, L = p.L, lr = p.lr, A = p.A;
    const int slots = N << lr, row_mask = (1 << lr) - 1;
    unsigned char *img = dyn;
    uint32_t *tab = reinterpret_cast<uint32_t *>(img + p.step_max);  // first event of a slot << 16 | events (counting: events)
    uint16_t *order = reinterpret_cast<uint16_t *>(tab + slots);     // [N][capW] event ids
    uint16_t *tok = order + N * p.capW;
    const int tb = blk * L, Lb = min(L, p.T - tb);
    unsigned char *rec = p.recs + (int64_t(bh) * p.nblocks + blk) * p.blk_bytes;
    uint4 *table = reinterpret_cast<uint4 *>(rec);
    uint4 *first = p.first + (int64_t(bh) << LG) * p.nblocks + blk;
    unsigned char *data = rec + rn_list_data_at(L, LG);
    const uint32_t xbase = (uint32_t(1) << lr) + uint32_t(blk & 1) * uint32_t(L);  // row of token 0 in the tile

    const int P = min(NT / L, 32);
    const int t = tid / P, part = tid & (P - 1);
    const int kw = (Kw + P - 1) / P, kr = (Kr + P - 1) / P;
    uint32_t ws[KP], rs[KP];
    float wc[KP];                          // gains
    {
        const int at = tb + t;
        const bool tok_live = t < Lb && (p.mask == nullptr || p.mask[b * p.mb + at * p.mt] != 0);
        const int64_t base = b * p.ib + h * p.ih + int64_t(at) * p.it;
        const int32_t *idx = p.idx + base;
        const float *val = p.val + base;
        const unsigned char *srec = p.sched + int64_t(bh) * ((p.T + p.sched_L - 1) / p.sched_L) * p.sched_bytes + int64_t(at / p.sched_L) * p.sched_bytes;
        const float *coef = reinterpret_cast<const float *>(srec + RN_GSU_HDR_BYTES + size_t(p.sched_NEp) * 4) + (at % p.sched_L) * KT;
        int wi[KP], ri[KP];
        float wv[KP], rv[KP];
#pragma unroll
        for (int j = 0; j < KP; ++j) { wi[j] = ri[j] = 0; wv[j] = rv[j] = wc[j] = 0.f; }
        if (tok_live) {
            const int ik = int(p.ik), k0 = part * kw, q0 = part * kr;
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                if (j < kw && k0 + j < Kw) { wi[j] = idx[(k0 + j) * ik]; wv[j] = val[(k0 + j) * ik]; wc[j] = coef[k0 + j]; }
                if (j < kr && q0 + j < Kr) { ri[j] = idx[(Kw + q0 + j) * ik]; rv[j] = val[(Kw + q0 + j) * ik]; }
            }
        }
        auto modulo = [&](int raw) {
            uint32_t r = uint32_t(raw) - __umulhi(uint32_t(raw), p.a_magic) * uint32_t(A);
            r = min(r, r - uint32_t(A));
            return int(min(r, r - uint32_t(A)));
        };
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            wi[j] = modulo(wi[j]);
            ri[j] = modulo(ri[j]);
            ws[j] = wv[j] != 0.f ? uint32_t((rn_owner_of<LG>(wi[j]) << lr) | (wi[j] >> LG)) : ~0u;
            rs[j] = rv[j] != 0.f ? uint32_t((rn_owner_of<LG>(ri[j]) << lr) | (ri[j] >> LG)) : ~0u;
        }
    }
    int nsteps = 0, t0 = 0, len = Lb;
    uint32_t step_at = 0;
    while (t0 < Lb) {
        len = min(len, Lb - t0);
        const bool mine = t >= t0 && t < t0 + len;
#pragma unroll 1
        for (int i = tid; i < slots / 4; i += NT) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) s_fail = 0;
        if (tid < N) nsingle[tid] = nmulti[tid] = 0;
        __syncthreads();
        uint32_t rank[KP], cnt[KP], pos[KP];
#pragma unroll
        for (int j = 0; j < KP; ++j) rank[j] = mine && ws[j] != ~0u ? atomicAdd(&tab[ws[j]], 1u) : 0u;
        __syncthreads();
        bool many = false;
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            cnt[j] = mine && ws[j] != ~0u ? tab[ws[j]] : 0u;
            many |= cnt[j] > 255u;
        }
        // places of the slots with one event: counted per owner by ballots
        {
            uint32_t tot = 0;
#pragma unroll
            for (int o = 0; o < N; ++o) {
                uint32_t run = 0;
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    const bool one = cnt[j] == 1u && (ws[j] >> lr) == uint32_t(o);
                    const unsigned m = __ballot_sync(RN_FULL, one);
                    if (one) pos[j] = run + __popc(m & ((1u << lane) - 1u));
                    run += __popc(m);
                }
                if (lane == o) tot = run;
            }
            uint32_t base = 0;
            if (lane < N) base = atomicAdd(&nsingle[lane], tot);
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                const uint32_t bj = __shfl_sync(RN_FULL, base, cnt[j] != 0 ? int(ws[j] >> lr) : 0);
                if (cnt[j] == 1u) pos[j] += bj;
                else if (cnt[j] > 1u && rank[j] == 0u) pos[j] = atomicAdd(&nmulti[ws[j] >> lr], cnt[j] | 0x10000u);
            }
        }
        many = __syncthreads_or(many);
#pragma unroll
        for (int o = 0; o < N; ++o) many |= nsingle[o] + (nmulti[o] & 0xffffu) > uint32_t(p.capW);
        if (many && len > 1) {
            len = (len + 1) >> 1;
            __syncthreads();
            continue;
        }
        uint32_t spoke = 0;
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            if (cnt[j] == 0u || (cnt[j] > 1u && rank[j] != 0u)) continue;
            const uint32_t s = ws[j], o = s >> lr;
            const uint32_t q = cnt[j] > 1u ? nsingle[o] + (pos[j] & 0xffffu) : pos[j];
            if (cnt[j] > 1u) spoke |= 1u << j;
            tab[s] = (q << 16) | cnt[j];
            if (cnt[j] == 1u) order[o * p.capW + q] = uint16_t(t * Kw + part * kw + j);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < KP; ++j)
            if (cnt[j] > 1u) order[(ws[j] >> lr) * p.capW + (tab[ws[j]] >> 16) + rank[j]] = uint16_t(t * Kw + part * kw + j);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            rank[j] = 0;
            if (cnt[j] <= 1u) continue;
            const uint32_t e = uint32_t(t * Kw + part * kw + j), a0 = (ws[j] >> lr) * p.capW + (tab[ws[j]] >> 16);
            uint32_t n = 0;
#pragma unroll 1
            for (uint32_t i = 0; i < cnt[j]; ++i) n += order[a0 + i] < e;
            rank[j] = n;
        }
        // the reads' entries: rn writes before it on its slot in the step; offset among the token's entries of the owner
        uint32_t rn[KP], roff[KP];
        {
            constexpr int HW = (N + 3) / 4;
            uint64_t have[HW] = {};
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                rn[j] = roff[j] = 0;
                if (!mine || rs[j] == ~0u) continue;
                const uint32_t v = tab[rs[j]], c = v & 0xffffu, o = rs[j] >> lr;
                uint32_t n = 0;
                if (c != 0u) {
                    const uint32_t a0 = o * p.capW + (v >> 16), lim = uint32_t(t + 1) * Kw;
#pragma unroll 1
                    for (uint32_t i = 0; i < c; ++i) n += order[a0 + i] < lim;
                }
                rn[j] = n;
                if (len == 1) n = min(n, 1u);  // writes of one token to one slot: one row of x
#pragma unroll
                for (int w = 0; w < HW; ++w)
                    if (HW == 1 || (o >> 2) == uint32_t(w)) {
                        roff[j] = uint32_t(have[w] >> ((o & 3u) * 16u)) & 0xffffu;
                        have[w] += uint64_t(n + 1u) << ((o & 3u) * 16u);
                    }
            }
            uint64_t pre[HW];
#pragma unroll
            for (int w = 0; w < HW; ++w) {
                pre[w] = have[w];
#pragma unroll 1
                for (int o = 1; o < P; o <<= 1) {
                    const uint64_t x = __shfl_up_sync(RN_FULL, pre[w], o, P);
                    if ((lane & (P - 1)) >= o) pre[w] += x;
                }
                have[w] = pre[w] - have[w];
            }
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                const uint32_t o = rs[j] >> lr;
#pragma unroll
                for (int w = 0; w < HW; ++w)
                    if (HW == 1 || (o >> 2) == uint32_t(w)) roff[j] += uint32_t(have[w] >> ((o & 3u) * 16u)) & 0xffffu;
            }
            if (mine && (lane & (P - 1)) == P - 1) {
#pragma unroll
                for (int o = 0; o < N; ++o) tok[o * (L + 1) + t - t0] = uint16_t(pre[o >> 2] >> ((o & 3) * 16));
            }
        }
        __syncthreads();
        if (warp < N) {
            uint16_t *tk = tok + warp * (L + 1);
            uint32_t n[4], tot = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t x = lane * 4 + i < len ? tk[lane * 4 + i] : 0u;
                n[i] = tot;
                tot += x;
            }
            uint32_t pre = tot;
#pragma unroll
            for (int q = 1; q < 32; q <<= 1) {
                const uint32_t x = __shfl_up_sync(RN_FULL, pre, q);
                if (lane >= q) pre += x;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (lane * 4 + i <= len) tk[lane * 4 + i] = uint16_t(min(pre - tot + n[i], 0xffffu));
            if (lane == 31) {
                if (len == 128) tk[len] = uint16_t(min(pre, 0xffffu));
                own_reads[warp] = pre;
                if (len > 1 && pre > uint32_t(p.capR)) s_fail = 1;
            }
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t at = 0, reads = 0;
#pragma unroll 1
            for (int o = 0; o < N; ++o) {
                const uint32_t nw = nsingle[o] + (nmulti[o] & 0xffffu), nr = own_reads[o];
                at_hdr[o] = at;
                at += 1u + ((rn_runs(nr, p.rs) + (nmulti[o] >> 16) + 7u) >> 3);
                at_W[o] = at;
                at += (nw + 1u) >> 1;
                at_R[o] = at;
                at += (nr + 1u) >> 1;
                reads += own_reads[o];
            }
            at_hdr[N] = at;
            if (len > 1 && reads > 2u * uint32_t(len) * uint32_t(Kr)) s_fail = 1;
            if (nsteps > 0) rn_bulk_wait_read();
        }
        __syncthreads();
        if (s_fail) {
            len = (len + 1) >> 1;
            __syncthreads();
            continue;
        }
        // ---- the lists: update events first, the readers' products run over them ----------------------------------------
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            if (cnt[j] == 0u) continue;
            const uint32_t s = ws[j], o = s >> lr, q = (tab[s] >> 16) + rank[j];
            reinterpret_cast<uint2 *>(img + (at_W[o] << 4))[q] =
                make_uint2(__float_as_uint(wc[j]), (s & uint32_t(row_mask)) | (uint32_t(t) << 11) | (uint32_t(part * kw + j) << 18) |
                                                       (rank[j] + 1u == cnt[j] ? 1u << 31 : 0u));
            if (spoke & (1u << j))
                reinterpret_cast<uint16_t *>(img + (at_hdr[o] << 4) + 16)[rn_runs(own_reads[o], p.rs) + (pos[j] >> 16)] = uint16_t(tab[s] >> 16);
        }
        __syncthreads();
        if (mine) {
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                const uint32_t s = rs[j];
                if (s == ~0u) continue;
                const uint32_t o = s >> lr, tag = uint32_t(t) << 12 | uint32_t(part * kr + j) << 19;
                uint2 *r = reinterpret_cast<uint2 *>(img + (at_R[o] << 4)) + uint32_t(tok[o * (L + 1) + t - t0]) + roff[j];
                const uint2 *W = reinterpret_cast<const uint2 *>(img + (at_W[o] << 4)) + (tab[s] >> 16);
                float c = 1.f, one = 0.f;
#pragma unroll 1
                for (int i = int(rn[j]); i > 0; --i) {
                    const uint2 ev = W[i - 1];
                    const float g = __uint_as_float(ev.x), f = c * g;
                    one += f;                              // one-token step: a single row of x for all writes
                    const int at = len == 1 ? 1 : i;
                    r[at] = make_uint2(__float_as_uint(len == 1 ? one : f),
                                       (xbase + ((ev.y >> 11) & 0x7fu)) | tag | (len == 1 || i == int(rn[j]) ? 1u << 31 : 0u));
                    c *= 1.f - g;
                }
                r[0] = make_uint2(__float_as_uint(c), (s & uint32_t(row_mask)) | tag | (rn[j] == 0u ? 1u << 31 : 0u));
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < N << rn_units_log2(p.rs); i += NT) {
            const uint32_t o = uint32_t(i) >> rn_units_log2(p.rs), u = uint32_t(i) & ((1u << rn_units_log2(p.rs)) - 1u), n = own_reads[o];
            if (u < rn_runs(n, p.rs)) {
                const uint2 *R = reinterpret_cast<const uint2 *>(img + (at_R[o] << 4));
                uint32_t at = u * ((n + (1u << rn_units_log2(p.rs)) - 1u) >> rn_units_log2(p.rs));
                while (at > 0u && at < n && int(R[at - 1].y) >= 0) ++at;
                reinterpret_cast<uint16_t *>(img + (at_hdr[o] << 4) + 16)[u] = uint16_t(min(at, n));
            }
        }
        if (tid < N) {
            RnListHdr hd;
            hd.len = uint16_t(len | (t0 << 8) | (tb + t0 + len >= p.T ? 0x8000 : 0));
            hd.nS = uint16_t(nsingle[tid]);
            hd.nM = uint16_t(nmulti[tid] >> 16);
            hd.nW = uint16_t(nsingle[tid] + (nmulti[tid] & 0xffffu));
            hd.nR = uint16_t(own_reads[tid]);
            hd.nF = 0;
            hd.atW = uint16_t(at_W[tid] - at_hdr[tid]);
            hd.atR = uint16_t(at_R[tid] - at_hdr[tid]);
            *reinterpret_cast<RnListHdr *>(img + (at_hdr[tid] << 4)) = hd;
            const uint32_t size = at_hdr[tid + 1] - at_hdr[tid];
            (nsteps == 0 ? first[tid * p.nblocks] : table[nsteps * N + tid]) =
                make_uint4((step_at + at_hdr[tid]) | (size << 16), uint32_t(t0) | (uint32_t(len) << 16), size << 16, 0u);
        }
        rn_fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            rn_bulk_s2g(data + (size_t(step_at) << 4), img, at_hdr[N] << 4);
            rn_bulk_commit();
        }
        step_at += at_hdr[N];
        t0 += len;
        ++nsteps;
        __syncthreads();
    }
#pragma unroll 1
    for (int i = tid; i < nsteps * N; i += NT) (i < N ? first[i * p.nblocks] : table[i]).z |= uint32_t(nsteps);
    rn_let_next_start();  // not earlier: the next kernel's blocks would crowd on the SMs that are done first
    if (tid == 0) rn_bulk_wait_read();
}

bool rn_replay_plan(int64_t B, int64_t H, int64_t T, int64_t A, int64_t C, int64_t Kw, int64_t Kr, RnListPlan *pl) {
    if (C % 4 != 0 || A > 16384 || Kw > 128 || Kr > 128) return false;
    constexpr int64_t STATE = 128 * 1024;
    pl->cs = C > 16 && A * 32 * 4 <= STATE * RN_LST_OWNERS ? 32 : 16;
    pl->ngroups = int((C + pl->cs - 1) / pl->cs);
    const int rs = pl->cs == 32 ? 7 : 6;
    const int64_t K = Kw > Kr ? Kw : Kr;
    auto fits = [&](int lg, int L) {
        const int N = 1 << lg;
        pl->lr = 2;
        while ((int64_t(1) << pl->lr << lg) < A) ++pl->lr;
        if ((1 << pl->lr) > RN_LST_ROWS || (int64_t(pl->cs) * 4 << pl->lr) > STATE) return false;
        pl->lg = lg;
        pl->N = N;
        pl->L = L;
        pl->nblocks = int((T + L - 1) / L);
        pl->capW = int(N == 1 ? L * Kw : L * Kw * 5 / (4 * N));
        pl->capR = int(N == 1 ? 2 * L * Kr : L * Kr * 7 / (4 * N));
        if (pl->capW < Kw) pl->capW = int(Kw);
        if (pl->capR < 2 * Kr + 2) pl->capR = int(2 * Kr + 2);
        pl->list_max = uint32_t(rn_align(size_t(16 + 8 * (pl->capW + pl->capR) + 64) + 2 * rn_runs(pl->capR, rs) + pl->capW, 128));
        pl->whole_max = 0;
        // at most 9 bytes a write, 20 a read, and 5 roundings of 16 bytes per owner
        const int64_t events = int64_t(L) * (9 * Kw + 20 * Kr);
        pl->step_max = uint32_t(rn_align(size_t(N) * (16 + 80) + events, 128));
        pl->blk_bytes = int64_t(rn_align(rn_list_data_at(L, lg) + size_t(N) * L * 96 + events, 128));
        pl->smem_lists = size_t(pl->step_max) + (size_t(N) << pl->lr) * 4 + size_t(N) * pl->capW * 2 + size_t(N) * (L + 1) * 2;
        pl->smem_gains = 0;
        // state rows, the tiles of x and d_y twice, the lists twice
        pl->smem_apply = (size_t(pl->cs) * 4 << pl->lr) + size_t(L) * pl->cs * 4 * 4 + 2 * size_t(pl->list_max);
        return pl->smem_lists <= 220 * 1024 && pl->smem_apply <= 226 * 1024 && (pl->blk_bytes >> 4) <= 0xffff;
    };
    bool found = false;
    int L0 = RN_LST_LMAX;
    while (L0 * K > RN_LST_EVENTS) L0 >>= 1;
    for (int L = L0; L >= 16 && !found; L >>= 1)
        for (int lg = 0; (1 << lg) <= RN_LST_OWNERS && !found; ++lg) found = fits(lg, L);
    if (!found) return false;
    pl->off_first = size_t(B * H) * pl->nblocks * pl->blk_bytes;
    pl->off_touch = 0;
    pl->total = rn_align(pl->off_first + (size_t(B * H) * pl->nblocks << pl->lg) * 16, 256);
    return true;
}

template <int LG, int KP>
static int rn_launch_replay_lists_t(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    RN_CUDA(cudaFuncSetAttribute(rn_replay_lists_kernel<LG, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pl.smem_lists)));
    rn_replay_lists_kernel<LG, KP><<<unsigned(p.B) * unsigned(p.H) * unsigned(pl.nblocks), RN_LISTS_THREADS, pl.smem_lists, stream>>>(p);
    RN_CUDA(cudaGetLastError());
    return 0;
}

int rn_launch_replay_lists(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    // addresses of a thread: min(1024 / L, 32) threads a token
    const int per = RN_LISTS_THREADS / pl.L < 32 ? RN_LISTS_THREADS / pl.L : 32;
    const int K = p.Kw > p.Kr ? p.Kw : p.Kr, kp = (K + per - 1) / per <= 2 ? 2 : 4;
#define RN_CASE(G, Q) \
    if (pl.lg == G && kp == Q) return rn_launch_replay_lists_t<G, Q>(p, pl, stream);
    RN_CASE(0, 2) RN_CASE(1, 2) RN_CASE(2, 2) RN_CASE(3, 2) RN_CASE(0, 4) RN_CASE(1, 4) RN_CASE(2, 4) RN_CASE(3, 4)
#undef RN_CASE
    rn_set_error("no replay lists kernel for 2^%d owners", pl.lg);
    return 1;
}
