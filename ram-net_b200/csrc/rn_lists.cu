// Lists and gains kernels of the prefill path (see rn_lists.cuh).
#include "rn_lists.cuh"

// ------------------------------------------------------------------------------------------
// lists kernel
// ------------------------------------------------------------------------------------------
// Bound by instruction issue (~20 instructions per event and phase) with a dozen barriers in between: blocks are
// independent and fill every SM.  1024 / L threads per token with KP writes and KP reads each (KP = 2 up to K = 64, else
// 4), which stay in registers through all phases; the step's lists are put together in shared memory and leave it in one
// bulk copy.  Inner loops stay rolled and KP small for the sake of the code's size: every CTA runs through it once, and a
// version of 82 KB (KP = 4) spent most of its time on instruction fetch.
template <typename T, int LG, int KP>
__global__ void __launch_bounds__(RN_LISTS_THREADS, 1) rn_lists_kernel(const RnListParams p) {
    constexpr int NT = RN_LISTS_THREADS, N = 1 << LG;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint32_t nsingle[N], nmulti[N];   // slots written once; writes of the others | such slots << 16
    __shared__ uint32_t own_reads[N], nfix[N];
    __shared__ uint32_t at_hdr[N + 1], at_W[N], at_R[N], at_AW[N], at_F[N];  // in 16 bytes from the step's first list
    __shared__ uint32_t bins[N][64];
    __shared__ int s_fail;

    const int bh = blockIdx.x / p.nblocks, blk = blockIdx.x % p.nblocks;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Kw = p.Kw, Kr = p.Kr, L = p.L, lr = p.lr, A = p.A;
    const int slots = N << lr, row_mask = (1 << lr) - 1;
    // dynamic smem: image of the step's lists | tab [N << lr]: first write of the slot in its owner's list << 16 | writes << 8
    // (while counting: writes) | order [N][capW]: event of a write (those of one slot in any order) | tok [N][L + 1]
    unsigned char *img = dyn;
    uint32_t *tab = reinterpret_cast<uint32_t *>(img + p.step_max);
    uint16_t *order = reinterpret_cast<uint16_t *>(tab + slots);
    uint16_t *tok = order + N * p.capW;
    uint8_t *perm = reinterpret_cast<uint8_t *>(tok + N * (L + 1));
    const int tb = blk * L, Lb = min(L, p.T - tb);  // tokens of this block
    unsigned char *rec = p.recs + (int64_t(bh) * p.nblocks + blk) * p.blk_bytes;
    uint4 *table = reinterpret_cast<uint4 *>(rec);                                    // steps behind the first
    uint4 *first = p.first + (int64_t(bh) << LG) * p.nblocks + blk;                   // [owner][blocks]
    unsigned char *data = rec + rn_list_data_at(L, LG);

    // ---- this thread's events ----------------------------------------------------------------------------------------
    const int P = min(NT / L, 32);         // threads of a token, a power of two, in one warp
    const int t = tid / P, part = tid & (P - 1);
    const int kw = (Kw + P - 1) / P, kr = (Kr + P - 1) / P;  // <= KP
    uint32_t ws[KP], rs[KP];               // owner << lr | row, or ~0
    float wv[KP], rv[KP];
    float gate, eg;                        // forget gate of the token and exp(-|gate|)
    {
        const bool tok_live = t < Lb && (p.mask == nullptr || p.mask[b * p.mb + (tb + t) * p.mt] != 0);
        const int64_t base = b * p.ib + h * p.ih + int64_t(tb + t) * p.it;
        const int32_t *idx = p.idx + base;
        const float *val = p.val + base;
        int wi[KP], ri[KP];
#pragma unroll
        for (int j = 0; j < KP; ++j) { wi[j] = ri[j] = 0; wv[j] = rv[j] = 0.f; }
        if (tok_live) {
            const int ik = int(p.ik), k0 = part * kw, q0 = part * kr;
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                if (j < kw && k0 + j < Kw) { wi[j] = idx[(k0 + j) * ik]; wv[j] = val[(k0 + j) * ik]; }
                if (j < kr && q0 + j < Kr) { ri[j] = idx[(Kw + q0 + j) * ik]; rv[j] = val[(Kw + q0 + j) * ik]; }
            }
        }
        gate = tok_live ? rn_to_float<T>(static_cast<const T *>(p.gamma)[b * p.gb + h * p.gh + int64_t(tb + t) * p.gt]) : 0.f;
        eg = expf(-fabsf(gate));
        // index modulo A, the batch and head offset taken off: quotient by multiplication, at most two too small
        auto modulo = [&](int raw) {
            uint32_t r = uint32_t(raw) - __umulhi(uint32_t(raw), p.a_magic) * uint32_t(A);
            r = min(r, r - uint32_t(A));
            return int(min(r, r - uint32_t(A)));
        };
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            wi[j] = modulo(wi[j]);
            ri[j] = modulo(ri[j]);
            wv[j] = fabsf(wv[j]);
            rv[j] = fabsf(rv[j]);
            ws[j] = wv[j] != 0.f ? uint32_t((rn_owner_of<LG>(wi[j]) << lr) | (wi[j] >> LG)) : ~0u;
            rs[j] = rv[j] != 0.f ? uint32_t((rn_owner_of<LG>(ri[j]) << lr) | (ri[j] >> LG)) : ~0u;
        }
    }

    int nsteps = 0, t0 = 0, len = Lb;
    uint32_t step_at = 0;  // in 16 bytes from data
    while (t0 < Lb) {
        len = min(len, Lb - t0);
        const bool mine = t >= t0 && t < t0 + len;
#pragma unroll 1
        for (int i = tid; i < slots / 4; i += NT) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) s_fail = 0;
        if (tid < N) nfix[tid] = nsingle[tid] = nmulti[tid] = 0;
        __syncthreads();
        // ---- writes per slot; the first to come speaks for the slot -----------------------------------------------------
        uint32_t rank[KP], cnt[KP];
#pragma unroll
        for (int j = 0; j < KP; ++j) rank[j] = mine && ws[j] != ~0u ? atomicAdd(&tab[ws[j]], 1u) : 0u;
        __syncthreads();
        // ---- places in the owners' write lists: slots written once, then the others.  In any order: a slot's writes stay
        // together and in time order, and nothing else depends on where they stand
        uint32_t pos[KP];
        {
            uint32_t tot = 0;
#pragma unroll
            for (int j = 0; j < KP; ++j) cnt[j] = mine && ws[j] != ~0u ? tab[ws[j]] : 0u;
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
        {
            // counts have eight bits below; a token names a slot at most 128 times
            bool many = false;
#pragma unroll
            for (int j = 0; j < KP; ++j) many |= cnt[j] > 255u;
            many = __syncthreads_or(many);
#pragma unroll
            for (int o = 0; o < N; ++o) many |= nsingle[o] + (nmulti[o] & 0xffffu) > uint32_t(p.capW);
            if (many && len > 1) {  // the same answer in every thread
                len = (len + 1) >> 1;
                __syncthreads();
                continue;
            }
        }
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            if (cnt[j] == 0u || (cnt[j] > 1u && rank[j] != 0u)) continue;
            const uint32_t o = ws[j] >> lr;
            const uint32_t q = cnt[j] == 1u ? pos[j] : nsingle[o] + (pos[j] & 0xffffu);
            tab[ws[j]] = (q << 16) | (cnt[j] << 8);
            if (cnt[j] == 1u) order[o * p.capW + q] = uint16_t(t * Kw + part * kw + j);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < KP; ++j)
            if (cnt[j] > 1u) order[(ws[j] >> lr) * p.capW + (tab[ws[j]] >> 16) + rank[j]] = uint16_t(t * Kw + part * kw + j);
        __syncthreads();
        uint32_t spoke = 0;
#pragma unroll
        for (int j = 0; j < KP; ++j)
            if (rank[j] == 0u) spoke |= 1u << j;
        // ---- a write's place in time among those of its slot; earlier writes of every read; read entries per (owner, token)
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            if (cnt[j] <= 1u) {
                rank[j] = 0;
                continue;
            }
            const uint32_t e = uint32_t(t * Kw + part * kw + j), a0 = (ws[j] >> lr) * p.capW + (tab[ws[j]] >> 16);
            uint32_t n = 0;
#pragma unroll 1
            for (uint32_t i = 0; i < cnt[j]; ++i) n += order[a0 + i] < e;
            rank[j] = n;
        }
        uint32_t rn[KP], roff[KP], fx[KP];  // n; offset among the token's entries of the owner; place in the fix list
        {
            constexpr int HW = (N + 3) / 4;   // entries of this thread's reads so far, 16 bits per owner
            uint64_t have[HW] = {};
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                rn[j] = roff[j] = fx[j] = 0;
                if (!mine || rs[j] == ~0u) continue;
                const uint32_t v = tab[rs[j]], c = (v >> 8) & 0xffu, o = rs[j] >> lr;
                uint32_t n = 0;
                if (c != 0) {
                    const uint32_t a0 = o * p.capW + (v >> 16), lim = uint32_t(t + 1) * Kw;
#pragma unroll 1
                    for (uint32_t i = 0; i < c; ++i) n += order[a0 + i] < lim;
                    if (n != 0) fx[j] = atomicAdd(&nfix[o], 1u);
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
                for (int o = 0; o < N; ++o) tok[o * (L + 1) + t - t0] = uint16_t((uint32_t(pre[o >> 2] >> ((o & 3) * 16)) & 0xffffu) + 1u & ~1u);
            }
        }
        __syncthreads();
        // ---- per owner: where its tokens start, how much it has, whether that fits -----------------------------------------
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
            // the tokens by number of entries, largest first (any order among equals): the apply kernel pairs them up
            bins[warp][lane] = bins[warp][lane + 32] = 0;
            __syncwarp();
            uint32_t bin[4], place[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bin[i] = 63u - min((i < 3 ? n[i + 1 < 4 ? i + 1 : 3] : tot) - n[i], 63u);
                place[i] = lane * 4 + i < len ? atomicAdd(&bins[warp][bin[i]], 1u) : 0u;
            }
            __syncwarp();
            {
                const uint32_t b0 = bins[warp][lane * 2], b1 = bins[warp][lane * 2 + 1];
                uint32_t s = b0 + b1;
#pragma unroll
                for (int q = 1; q < 32; q <<= 1) {
                    const uint32_t x = __shfl_up_sync(RN_FULL, s, q);
                    if (lane >= q) s += x;
                }
                bins[warp][lane * 2] = s - b0 - b1;
                bins[warp][lane * 2 + 1] = s - b1;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (lane * 4 + i < len) perm[warp * L + bins[warp][bin[i]] + place[i]] = uint8_t(lane * 4 + i);
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
                const RnListAt a = rn_list_at(len, nmulti[o] >> 16, nsingle[o] + (nmulti[o] & 0xffffu), own_reads[o], nfix[o]);
                at_hdr[o] = at;
                at_W[o] = at + a.W;
                at_R[o] = at + a.R;
                at_AW[o] = at + a.AW;
                at_F[o] = at + a.F;
                at += a.end;
                reads += own_reads[o];
            }
            at_hdr[N] = at;
            if (len > 1 && reads > 2u * uint32_t(len) * uint32_t(Kr) + uint32_t(N * len)) s_fail = 1;
            if (nsteps > 0) rn_bulk_wait_read();  // the image may be written to again
        }
        __syncthreads();
        if (s_fail) {  // hot slots: shorter steps
            len = (len + 1) >> 1;
            __syncthreads();
            continue;
        }
        // ---- the lists ------------------------------------------------------------------------------------------------
        if (tid < N) {
            RnListHdr hd;
            hd.len = uint16_t(len | (t0 << 8) | (tb + t0 + len >= p.T ? 0x8000 : 0));
            hd.nS = uint16_t(nsingle[tid]);
            hd.nM = uint16_t(nmulti[tid] >> 16);
            hd.nW = uint16_t(nsingle[tid] + (nmulti[tid] & 0xffffu));
            hd.nR = uint16_t(own_reads[tid]);
            hd.nF = uint16_t(nfix[tid]);
            hd.atW = uint16_t(at_W[tid] - at_hdr[tid]);
            hd.atR = uint16_t(at_R[tid] - at_hdr[tid]);
            *reinterpret_cast<RnListHdr *>(img + (at_hdr[tid] << 4)) = hd;
            (nsteps == 0 ? first[tid * p.nblocks] : table[nsteps * N + tid]) = make_uint4((step_at + at_hdr[tid]) | ((at_AW[tid] - at_hdr[tid]) << 16), uint32_t(t0) | (uint32_t(len) << 16),
                                                 (at_hdr[tid + 1] - at_hdr[tid]) << 16, 0u);
        }
#pragma unroll
        for (int o = 0; o < N; ++o)
#pragma unroll 1
            for (int i = tid; i <= len; i += NT) {
                reinterpret_cast<uint16_t *>(img + (at_hdr[o] << 4) + 16)[i] = tok[o * (L + 1) + i];
                if (i < len) (img + (at_W[o] << 4) - ((len + 15) & ~15))[i] = perm[o * L + i];
            }
#pragma unroll
        for (int j = 0; j < KP; ++j) {
            if (cnt[j] == 0u) continue;
            const uint32_t o = ws[j] >> lr, q = (tab[ws[j]] >> 16) + rank[j];
            reinterpret_cast<uint2 *>(img + (at_W[o] << 4))[q] =
                make_uint2(0u, (ws[j] & uint32_t(row_mask)) | (uint32_t(t) << 11) | (rank[j] + 1u == cnt[j] ? 1u << 31 : 0u));
            // rn_alpha() with the exponential taken once per token
            const float cw = 1.f - wv[j];
            const float alpha = (gate >= 0.f ? cw * eg : cw) / (gate >= 0.f ? wv[j] + eg * cw : cw + eg * wv[j]);
            reinterpret_cast<float2 *>(img + (at_AW[o] << 4))[q] = make_float2(alpha, wv[j]);
            // pos of the slot's speaker still holds its place among the slots written more than once
            if (cnt[j] > 1u && (spoke & (1u << j))) reinterpret_cast<uint16_t *>(img + (at_hdr[o] << 4) + 16)[len + 1 + (pos[j] >> 16)] = uint16_t(q - rank[j]);
        }
        if (mine) {
            if (part < N) {  // the entry that makes a token's number even; overwritten where the number is even by itself
                const uint32_t end = tok[part * (L + 1) + t - t0 + 1];
                if (end != uint32_t(tok[part * (L + 1) + t - t0])) reinterpret_cast<uint2 *>(img + (at_R[part] << 4))[end - 1] = make_uint2(0u, 0u);
            }
            __syncwarp(__activemask());
#pragma unroll
            for (int j = 0; j < KP; ++j) {
                if (rs[j] == ~0u) continue;
                const uint32_t o = rs[j] >> lr, row = rs[j] & uint32_t(row_mask), n = rn[j];
                const uint32_t i = uint32_t(tok[o * (L + 1) + t - t0]) + roff[j];
                uint2 *r = reinterpret_cast<uint2 *>(img + (at_R[o] << 4)) + i;
                uint32_t m = row << p.rs;
                if (n != 0 || p.mass_aware) {
                    m = row | (n << 22) | (1u << 31);
                    if (n != 0) {
                        m |= (tab[rs[j]] >> 16) << 11;
                        reinterpret_cast<uint16_t *>(img + (at_F[o] << 4))[fx[j]] = uint16_t(i);
                    }
                }
                r[0] = make_uint2(__float_as_uint(rv[j]), m);
#pragma unroll 1
                for (uint32_t q = 1; q <= (len == 1 ? min(n, 1u) : n); ++q) r[q] = make_uint2(0u, 0u);
            }
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
        __syncthreads();  // the offsets are written again in the next step
    }
#pragma unroll 1
    for (int i = tid; i < nsteps * N; i += NT) (i < N ? first[i * p.nblocks] : table[i]).z |= uint32_t(nsteps);
    rn_let_next_start();  // not earlier: the next kernel's blocks would crowd on the SMs that are done first
    if (tid == 0) rn_bulk_wait_read();
}

// ------------------------------------------------------------------------------------------
// gains kernel: one CTA per (b,h, owner), steps in order
// ------------------------------------------------------------------------------------------
// Latency bound (per step: wait for the list, written slots, barrier, reads): the owners of a head are independent, so
// four CTAs share an SM.  The mass of the owner's slots stays in shared memory; a step's list arrives by one bulk copy, a
// step ahead.  Mass-aware reads are the exception: their scale sums over all addresses of a token, so the owners are a
// cluster there and exchange their sums through distributed shared memory, one cluster barrier per step.
template <int LG, bool MA>
__global__ void __launch_bounds__(RN_GAINS_THREADS) rn_gains_kernel(const RnListParams p) {
    constexpr int NT = RN_GAINS_THREADS, N = 1 << LG;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t touched[2][RN_LST_ROWS / 32];
    const int own = blockIdx.x & (N - 1), bh = blockIdx.x >> LG, tid = threadIdx.x;
    const int A = p.A, rows = 1 << p.lr;

    unsigned char *buf = dyn;                                                // [2][whole_max]
    float *mass = reinterpret_cast<float *>(dyn + 2 * size_t(p.whole_max));  // [rows]
    // mass-aware reads: [2][2][L] sums of the tokens' weights by parity of the step, [capR] weight times mass of the entries
    float *part = mass + rows, *um = part + 4 * p.L;
    if (tid == 0) {
        rn_mbar_init(&mbar[0], 1);
        rn_mbar_init(&mbar[1], 1);
        rn_mbar_fence_init();
    }
    __syncthreads();
    unsigned char *recs = p.recs + int64_t(bh) * p.nblocks * p.blk_bytes;
    const uint4 *first = p.first + ((int64_t(bh) << LG) + own) * p.nblocks;
    const uint32_t data_at = rn_list_data_at(p.L, LG);
    auto fetch = [&](int step, int blk, const uint4 &e) {
        const uint32_t bytes = (e.z >> 16) << 4;
        rn_mbar_expect_tx(&mbar[step & 1], bytes);
        rn_bulk_g2s(buf + size_t(step & 1) * p.whole_max, recs + blk * p.blk_bytes + data_at + (size_t(e.x & 0xffffu) << 4), bytes, &mbar[step & 1]);
    };
    if (!MA) rn_let_next_start();  // a cluster that exchanges sums every step is slowed by early neighbours
    const float *mass_in = p.mass_in ? p.mass_in + int64_t(bh) * A : nullptr;
    if (p.touch != nullptr)
        for (int i = tid; i < 2 * RN_LST_ROWS / 32; i += NT) touched[0][i] = 0;  // both rows of the array
    auto touch = [&](int set, uint32_t r) {
        if (!(touched[set][r >> 5] & (1u << (r & 31)))) atomicOr(&touched[set][r >> 5], 1u << (r & 31));
    };
#pragma unroll 1
    for (int r = tid; r < rows; r += NT) {
        const int a = rn_slot_of<LG>(own, r);
        mass[r] = mass_in == nullptr ? p.mass_init : a < A ? mass_in[a] : 0.f;
    }

    rn_wait_for_front();
    int blk = 0, st = 0;
    uint4 cur = rn_step_entry(p, first, recs, 0, 0, own);
    if (tid == 0) fetch(0, 0, cur);
    int nblk = rn_steps_of(cur) > 1 ? 0 : 1, nst = rn_steps_of(cur) > 1 ? 1 : 0;
    uint4 nxt = rn_step_entry(p, first, recs, nblk, nst, own);

    bool failed = false;
    for (int step = 0; blk < p.nblocks; ++step) {
        // thread 0 keeps the copies a step ahead; entries are read two steps ahead
        if (tid == 0 && rn_steps_of(nxt) != 0) fetch(step + 1, nblk, nxt);  // that buffer was last used before the barrier that ended the step before
        const bool more = nst + 1 < rn_steps_of(nxt);
        const int nnblk = more ? nblk : nblk + 1, nnst = more ? nst + 1 : 0;
        const uint4 nn = rn_step_entry(p, first, recs, nnblk, nnst, own);
        if (tid == 0) failed = failed || !rn_mbar_wait_bounded(&mbar[step & 1], uint32_t(step >> 1) & 1u);
        failed = __syncthreads_or(failed);
        if (failed && !MA) break;
        unsigned char *lst = buf + size_t(step & 1) * p.whole_max;
        unsigned char *glst = recs + blk * p.blk_bytes + data_at + (size_t(cur.x & 0xffffu) << 4);
        RnListHdr hd = *reinterpret_cast<const RnListHdr *>(lst);
        if (failed) hd.len = hd.nS = hd.nM = hd.nW = hd.nR = hd.nF = 0;  // stays in step with the cluster and does nothing else
        uint2 *W = reinterpret_cast<uint2 *>(lst + (uint32_t(hd.atW) << 4)), *R = reinterpret_cast<uint2 *>(lst + (uint32_t(hd.atR) << 4));
        uint2 *gW = reinterpret_cast<uint2 *>(glst + (uint32_t(hd.atW) << 4)), *gR = reinterpret_cast<uint2 *>(glst + (uint32_t(hd.atR) << 4));
        float2 *aw = reinterpret_cast<float2 *>(R + ((hd.nR + 1) & ~1));
        const int len = hd.len & 0xff;
        const uint16_t *tok = reinterpret_cast<const uint16_t *>(lst + 16), *start = tok + len + 1;
        const uint16_t *fix = reinterpret_cast<const uint16_t *>(aw + ((hd.nW + 1) & ~1));

        if (p.touch != nullptr) {
#pragma unroll 1
            for (int i = tid; i < hd.nR; i += NT) touch(0, (R[i].y >> 31) != 0 ? R[i].y & 0x7ffu : R[i].y >> p.rs);
#pragma unroll 1
            for (int q = tid; q < hd.nW; q += NT) touch(1, W[q].y & 0x7ffu);
        }
        if (MA) {  // weight times mass for the reads that no write of the step precedes
#pragma unroll 1
            for (int i = tid; i < hd.nR; i += NT) {
                const uint32_t m = R[i].y;
                if ((m >> 31) != 0 && ((m >> 22) & 0x1ffu) == 0) um[i] = __uint_as_float(R[i].x) * mass[m & 0x7ffu];
            }
            __syncthreads();
        }
        auto write = [&](int q, float m) {                    // rn_gate(): mass' = alpha * mass + w, gain = w / (mass' + eps)
            const float2 v = aw[q];
            m = fmaf(v.x, m, v.y);
            const uint32_t g = __float_as_uint(v.y / (m + p.eps));
            if (MA) aw[q].x = m;
            W[q].x = g;
            gW[q].x = g;
            return m;
        };
#pragma unroll 1
        for (int q = tid; q < hd.nS; q += NT) {
            float *cell = mass + (W[q].y & 0x7ffu);
            *cell = write(q, *cell);
        }
#pragma unroll 1
        for (int i = tid; i < hd.nM; i += NT) {
            int q = start[i];
            uint32_t meta = W[q].y;
            float *cell = mass + (meta & 0x7ffu);
            float m = *cell;
            for (;;) {
                m = write(q, m);
                if ((meta >> 31) != 0) break;
                meta = W[++q].y;
            }
            *cell = m;
        }
        __syncthreads();
        const uint32_t xrow = uint32_t(rows) + uint32_t(blk & 1) * uint32_t(p.L);
        auto settle = [&](int i, float c, uint32_t m) {       // coefficients of a read
            const int n = int((m >> 22) & 0x1ffu), q = int((m >> 11) & 0x7ffu);
            float one = 0.f;
#pragma unroll 1
            for (int j = n; j > 0; --j) {
                const uint2 w = W[q + j - 1];
                const float g = __uint_as_float(w.x), f = c * g;
                const int at = len == 1 ? i + 1 : i + j;
                one += f;                                     // one-token step: a single row of x for all n writes
                gR[at] = make_uint2(__float_as_uint(len == 1 ? one : f), (xrow + ((w.y >> 11) & 0x7fu)) << p.rs);
                c *= 1.f - g;
            }
            gR[i] = make_uint2(__float_as_uint(c), (m & 0x7ffu) << p.rs);
        };
        if (!MA) {
#pragma unroll 1
            for (int f = tid; f < hd.nF; f += NT) {
                const int i = fix[f];
                const uint2 e = R[i];
                settle(i, __uint_as_float(e.x), e.y);
            }
        } else {
            // y_t = sum_k (r m slot) * sum r / (sum r m + eps); a read behind a write of the step sees the mass it left
            float *mine = part + size_t(step & 1) * 2 * p.L;
#pragma unroll 1
            for (int t = tid; t < len; t += NT) {
                float sr = 0.f, srm = 0.f;
#pragma unroll 1
                for (int i = tok[t]; i < tok[t + 1]; ++i) {
                    const uint32_t m = R[i].y, n = (m >> 22) & 0x1ffu;
                    if ((m >> 31) == 0) continue;
                    if (n > 0) um[i] = __uint_as_float(R[i].x) * aw[((m >> 11) & 0x7ffu) + n - 1].x;
                    sr += __uint_as_float(R[i].x);
                    srm += um[i];
                }
                mine[t] = sr;
                mine[p.L + t] = srm;
            }
            __syncthreads();
            if (N > 1) rn_cluster_sync();
#pragma unroll 1
            for (int t = tid; t < len; t += NT) {
                float sr = 0.f, srm = 0.f;
#pragma unroll
                for (int o = 0; o < N; ++o) {
                    float a, c;
                    const uint32_t at = rn_mapa(rn_smem_u32(mine + t), uint32_t(o));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(a) : "r"(at));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(c) : "r"(at + uint32_t(p.L) * 4u));
                    sr += a;
                    srm += c;
                }
                const float scale = sr / (srm + p.eps);
#pragma unroll 1
                for (int i = tok[t]; i < tok[t + 1]; ++i)
                    if ((R[i].y >> 31) != 0) settle(i, um[i] * scale, R[i].y);
            }
        }
        rn_fence_proxy_async();  // this buffer was written to and is the target of the next copy but one
        __syncthreads();
        blk = nblk;
        st = nst;
        cur = nxt;
        nblk = nnblk;
        nst = nnst;
        nxt = nn;
    }
    if (failed && tid == 0) atomicMax(p.status, RN_STATUS_WAIT_TIMEOUT);
    float *mass_out = p.mass_out + int64_t(bh) * A;
#pragma unroll 1
    for (int r = tid; r < rows && !failed; r += NT) {
        const int a = rn_slot_of<LG>(own, r);
        if (a < A) mass_out[a] = mass[r];
    }
    if (p.touch != nullptr) {  // the loop ended with a barrier
        const int words = rn_touch_words(p.lr);
        for (int i = tid; i < words; i += NT) {
            uint32_t *out = p.touch + blockIdx.x * 2 * words + i;
            out[0] = touched[0][i] | touched[1][i];
            out[words] = touched[1][i];
        }
    }
    if (MA && N > 1) rn_cluster_sync();  // the sums may still be read from another CTA
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
bool rn_list_plan(int64_t B, int64_t H, int64_t T, int64_t A, int64_t C, int64_t Kw, int64_t Kr, int mass_aware, RnListPlan *pl) {
    if (C % 4 != 0 || A > 16384 || Kw > 128 || Kr > 128) return false;
    // channels of a CTA: rows of 32 channels (128 bytes) are read without bank conflicts; 16 where few channels exist or
    // where the rows of an owner would not fit
    constexpr int64_t STATE = 128 * 1024;
    pl->cs = C > 16 && A * 32 * 4 <= STATE * RN_LST_OWNERS ? 32 : 16;
    pl->ngroups = int((C + pl->cs - 1) / pl->cs);
    const int K = int(Kw > Kr ? Kw : Kr);
    auto fits = [&](int lg, int L) {
        const int N = 1 << lg;
        pl->lr = 2;
        while ((int64_t(1) << pl->lr << lg) < A) ++pl->lr;
        if ((1 << pl->lr) > RN_LST_ROWS || (int64_t(pl->cs) * 4 << pl->lr) > STATE) return false;
        pl->lg = lg;
        pl->N = N;
        pl->L = L;
        pl->nblocks = int((T + L - 1) / L);
        // an even share of the writes and half of it more; of the reads, as much again for the corrections.  A step of one
        // token always fits.
        pl->capW = N == 1 ? L * int(Kw) : L * int(Kw) * 3 / (2 * N);
        pl->capR = 2 * L * int(Kr) / N;
        if (pl->capW < Kw) pl->capW = int(Kw);
        if (pl->capR < 2 * Kr + 2) pl->capR = int(2 * Kr + 2);
        const RnListAt most = rn_list_at(L, pl->capW / 2, pl->capW, pl->capR, pl->capR / 2);
        pl->list_max = uint32_t(rn_align(size_t(most.AW) * 16, 128));
        pl->whole_max = uint32_t(rn_align(size_t(most.end) * 16, 128));
        // all parts of all owners: at most 3 bytes a token, 17 a write, 16 + 2 a read (8 more per token and owner), and 6
        // roundings of 16 bytes
        const int64_t events = int64_t(L) * (17 * Kw + 18 * Kr + 8 * N);
        pl->step_max = uint32_t(rn_align(size_t(N) * (16 + 3 * (L + 1) + 96) + events, 128));
        pl->blk_bytes = int64_t(rn_align(rn_list_data_at(L, lg) + size_t(N) * L * 118 + events, 128));
        pl->smem_lists = size_t(pl->step_max) + (size_t(N) << pl->lr) * 4 + size_t(N) * pl->capW * 2 + size_t(N) * (L + 1) * 2 + size_t(N) * L;
        pl->smem_gains = 2 * size_t(pl->whole_max) + (size_t(4) << pl->lr) + (mass_aware ? size_t(4) * L * 4 + size_t(pl->capR) * 4 : 0);
        pl->smem_apply = (size_t(pl->cs) * 4 << pl->lr) + size_t(L) * pl->cs * 4 * (N > 1 ? 4 : 2) + 2 * size_t(pl->list_max);
        return pl->smem_lists <= 220 * 1024 && pl->smem_gains <= 225 * 1024 && pl->smem_apply <= 226 * 1024 && (pl->blk_bytes >> 4) <= 0xffff;
    };
    // the longest block that fits, with as few owners as hold the state; the threads of a token share a warp in the lists
    // kernel, so a block has at least 16 tokens
    bool found = false;
    int L0 = RN_LST_LMAX;
    while (L0 * K > RN_LST_EVENTS) L0 >>= 1;
    for (int L = L0; L >= 16 && !found; L >>= 1)
        for (int lg = 0; (1 << lg) <= RN_LST_OWNERS && !found; ++lg) found = fits(lg, L);
    if (!found) return false;
    pl->off_first = size_t(B * H) * pl->nblocks * pl->blk_bytes;
    pl->off_touch = pl->off_first + (size_t(B * H) * pl->nblocks << pl->lg) * 16;
    pl->total = rn_align(pl->off_touch + (size_t(B * H) << pl->lg) * 8 * rn_touch_words(pl->lr), 256);
    return true;
}

template <int LG, bool MA>
static int rn_launch_gains(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    RN_CUDA(cudaFuncSetAttribute(rn_gains_kernel<LG, MA>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pl.smem_gains)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned(p.B) * unsigned(p.H)) << LG);
    cfg.blockDim = dim3(RN_GAINS_THREADS);
    cfg.dynamicSmemBytes = pl.smem_gains;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1u << LG;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = MA && LG > 0 ? 2 : 1;
    RN_CUDA(cudaLaunchKernelEx(&cfg, rn_gains_kernel<LG, MA>, p));
    return 0;
}

template <typename T, int LG, int KP>
static int rn_launch_lists_k(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    RN_CUDA(cudaFuncSetAttribute(rn_lists_kernel<T, LG, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pl.smem_lists)));
    rn_lists_kernel<T, LG, KP><<<unsigned(p.B * p.H) * unsigned(pl.nblocks), RN_LISTS_THREADS, pl.smem_lists, stream>>>(p);
    return 0;
}

template <typename T, int LG>
static int rn_launch_lists_t(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream) {
    const int per_token = pl.L < 32 ? 32 : RN_LISTS_THREADS / pl.L;
    const bool two = 2 * per_token >= p.Kw && 2 * per_token >= p.Kr;
    if (int rc = two ? rn_launch_lists_k<T, LG, 2>(p, pl, stream) : rn_launch_lists_k<T, LG, 4>(p, pl, stream)) return rc;
    RN_CUDA(cudaGetLastError());
    rn_prof_mark(stream);
    if (int rc = p.mass_aware ? rn_launch_gains<LG, true>(p, pl, stream) : rn_launch_gains<LG, false>(p, pl, stream)) return rc;
    RN_CUDA(cudaGetLastError());
    rn_prof_mark(stream);
    return 0;
}

int rn_launch_lists(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream) {
#define RN_CASE(G)                                                                                                  \
    if (pl.lg == G)                                                                                                 \
        return dtype == RN_F32 ? rn_launch_lists_t<float, G>(p, pl, stream)                                         \
               : dtype == RN_F16 ? rn_launch_lists_t<__half, G>(p, pl, stream) : rn_launch_lists_t<__nv_bfloat16, G>(p, pl, stream);
    RN_CASE(0) RN_CASE(1) RN_CASE(2) RN_CASE(3)
#undef RN_CASE
    rn_set_error("no lists kernel for %d owners", pl.N);
    return 1;
}
