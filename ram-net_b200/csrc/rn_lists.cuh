// Event lists of the prefill path: what the update / read kernels of rn_apply.cu walk.
//
// The sequence is cut into blocks of L tokens.  Inside a block all reads are taken against the state at the START of the
// block: a read (t, k) of slot a with weight r, after the block's writes g_1 .. g_n (tokens <= t, same slot), is
//     r * S_t(a) = r (1-g_1)..(1-g_n) * S_0(a)  +  sum_j  r g_j (1-g_{j+1})..(1-g_n) * x(tau_j)
// i.e. one row of the state plus n rows of x ("corrections", n = 0 for most reads), with scalar coefficients that do not
// depend on the channel.  So a block is two sweeps with one barrier between them: all reads (token-major), then all
// writes (slot-major, the writes of one slot in time order by one thread group), and no read ever waits for a write
// of its own block.
//
// The slots of a (b,h) are dealt to N owners (a power of two), row r of owner o is slot rn_slot_of(o, r); an owner is one
// CTA of a cluster (rn_apply.cu), and each owner gets lists of its own.  Two kernels make them:
//     lists  one CTA per block, all blocks at once: groups the block's events by slot (count, scan, place) and lays out
//            the lists; everything but what needs the mass
//     gains  one CTA per (b,h), blocks in order: the mass recurrence, the gain of every write, the coefficients of the
//            reads that follow a write of their block
//
// A step is what one pass of the apply kernel handles: normally the whole block; a block whose lists would not fit (hot
// slots: n grows with the square of the tokens) is cut into shorter steps, down to one token (n <= 1 there).
//
// Block record (fixed size per call), byte offsets:
//     0           uint4 table[L][N], steps behind the first (the first steps' entries are in an array of their own,
//                 [bh][owner][block], so that walking the blocks reads consecutive memory): entry = {offset of the owner's list | size for the apply kernel << 16,
//                 first token | tokens << 16, steps of the block | whole size << 16, -}, offsets (from off_data) and
//                 sizes in 16 bytes
//     off_data    the steps' lists, contiguous; per step and owner (every part on a 16-byte boundary)
//                   header RnListHdr
//                   u16 tok[len + 1]     read entries of token i: tok[i] .. tok[i+1] (an even number: the last may be a
//                                        zero);  u16 start[nM]  first write of
//                                        every slot that is written more than once
//                   u8 perm[len]         the tokens, those with most read entries first
//                   {f32 gain, u32 row | token of the block << 11 | last of its slot << 31}[nW]   the nS slots that are
//                                        written once, then the others, slot by slot in time order
//                   {f32 coef, u32 ref}[nR]   ref: byte offset from the owner's first row, of a row of the state or of x
//                                        (which follow them: x(token of the block) is row rows + parity of the block * L + token)
//                   -- up to here copied by the apply kernel --
//                   {f32 alpha, f32 weight}[nW]
//                   u16 fix[nF]          read entries that follow a write
//     In the read list the lists kernel leaves {weight, row | first write << 11 | n << 22} at a read with n > 0 (for
//     mass-aware reads, at every read, bit 31 set) and {0, 0} at the n entries that follow it; the gains kernel turns
//     these into coefficients.
#pragma once

#include "rn_prefill.cuh"

constexpr int RN_LST_LMAX = 128;       // longest block
constexpr int RN_LST_EVENTS = 2048;    // most writes (and most reads) of a block
constexpr int RN_LST_ROWS = 2048;      // most rows of an owner
constexpr int RN_LST_OWNERS = 8;
constexpr int RN_LISTS_THREADS = 1024;
constexpr int RN_GAINS_THREADS = 256;

// digits (base N) of row XOR-ed together: the low bits of a slot are its owner XOR this, so slots whose addresses share
// digits (the combinations of a few best digits that a token selects) spread over the owners
template <int LG>
__host__ __device__ __forceinline__ int rn_fold(int row) {
    if (LG == 0) return 0;
    int x = row;
    if (LG == 1) { x ^= x >> 8; x ^= x >> 4; x ^= x >> 2; x ^= x >> 1; }
    if (LG == 2) { x ^= x >> 8; x ^= x >> 4; x ^= x >> 2; }
    if (LG == 3) { x ^= (x >> 3) ^ (x >> 6) ^ (x >> 9); }
    return x & ((1 << LG) - 1);
}
template <int LG> __host__ __device__ __forceinline__ int rn_owner_of(int a) { return (a & ((1 << LG) - 1)) ^ rn_fold<LG>(a >> LG); }
template <int LG> __host__ __device__ __forceinline__ int rn_slot_of(int owner, int row) { return (row << LG) | (owner ^ rn_fold<LG>(row)); }

struct __align__(16) RnListHdr {
    uint16_t len;  // tokens | first token of the step in its block << 8 | 0x8000 in the last step of the sequence
    uint16_t nS, nM, nW, nR, nF;
    uint16_t atW, atR;  // in 16 bytes from the header
};
static_assert(sizeof(RnListHdr) == 16, "list header");
// Shares of the replay.  The read entries of an owner are dealt to the 2^lu thread groups of the apply kernel that have a row
// each (512 threads, 32 bytes of a row each): unit u gets the reads whose first entry lies in [u q, (u + 1) q), q = ceil(n / 2^lu),
// a read whole.  run[u] (u q < n) is its first entry.
__host__ __device__ __forceinline__ int rn_units_log2(int rs) { return 14 - rs; }
__host__ __device__ __forceinline__ uint32_t rn_runs(uint32_t n, int rs) {  // entries kept for n
    const uint32_t units = 1u << rn_units_log2(rs);
    return n < units ? n : units;
}
struct RnListAt {  // parts of a list, in 16 bytes from its header
    uint32_t W, R, AW, F, end;
};
__host__ __device__ __forceinline__ RnListAt rn_list_at(uint32_t len, uint32_t nM, uint32_t nW, uint32_t nR, uint32_t nF) {
    RnListAt a;
    a.W = 1u + ((len + 1u + nM + 7u) >> 3) + ((len + 15u) >> 4);
    a.R = a.W + ((nW + 1u) >> 1);
    a.AW = a.R + ((nR + 1u) >> 1);
    a.F = a.AW + ((nW + 1u) >> 1);
    a.end = a.F + ((nF + 7u) >> 3);
    return a;
}

struct RnListPlan {
    int L, nblocks, lg, N, lr;    // lr: log2 of the rows of an owner, rounded up
    int cs, ngroups;              // channels of a CTA, channel groups
    int capR, capW;               // most entries of an owner's lists in one step
    int64_t blk_bytes;
    uint32_t list_max;            // largest list of an owner and step (the part the apply kernel copies)
    uint32_t whole_max;           // likewise, the whole list
    uint32_t step_max;            // largest step (all owners)
    size_t smem_lists, smem_gains, smem_apply;
    size_t off_first, off_touch, total;  // workspace: first-step table, touched rows, bytes
};
__host__ __device__ __forceinline__ uint32_t rn_list_data_at(int L, int lg) { return (uint32_t(L) << lg) * 16u; }

struct RnListParams {
    const int32_t *idx;
    const float *val;
    int64_t ib, ih, ik, it;
    const void *gamma;
    int64_t gb, gh, gt;
    const uint8_t *mask;
    int64_t mb, mt;
    const void *x;
    int64_t xb, xh, xt;
    void *y;
    int64_t yb, yh, yt;
    const float *slot_in;  // null: zeros
    float *slot_out;
    const float *mass_in;  // null: mass_init everywhere
    float *mass_out;
    float mass_init;
    int B, H, T, A, C, Kw, Kr;
    int L, nblocks, lg, lr, ngroups, capR, capW;
    int64_t blk_bytes;
    uint32_t list_max, whole_max, step_max;
    uint32_t a_magic;      // 2^32 / A, rounded down
    int rs;                // log2 of the bytes of a row
    int mass_aware;
    float eps;
    int *status;
    unsigned char *recs;
    uint4 *first;
    // optional, for a short sequence on a state that is updated in place: [bh][owner][2][rn_touch_words] bits of the rows that
    // the call reads or writes and of those that it writes; the others stay in global memory
    uint32_t *touch;
    // replay of the backward pass (rn_apply.cu)
    const void *dy;            // upstream gradient of y
    int64_t dyb, dyh, dyt;
    float *delta;              // [bh][slice][t][Kw][dcs]: x - row at every write, slices of dcs channels
    int dcs;
    float *part;               // [bh][group][t][Kr]: partial dot products, d_r
    const unsigned char *sched;  // chunk records of the schedule kernel: coefficients of all events
    int64_t sched_bytes;
    int sched_L, sched_NEp;
};

enum { RN_FORWARD = 0, RN_REPLAY = 1 };

// walks the steps of a (b,h): the entry of an owner in step st of block blk; all zero behind the last block
// (first: this owner's first steps)
__device__ __forceinline__ uint4 rn_step_entry(const RnListParams &p, const uint4 *first, const unsigned char *recs, int blk, int st,
                                               int owner) {
    if (blk >= p.nblocks) return make_uint4(0u, 0u, 0u, 0u);
    if (st == 0) return first[blk];
    return *(reinterpret_cast<const uint4 *>(recs + blk * p.blk_bytes) + (st << p.lg) + owner);
}

__device__ __forceinline__ int rn_steps_of(const uint4 &e) { return int(e.z & 0xffffu); }

// The gains and the apply kernel are launched while the kernel in front still runs (programmatic dependent launch): they set up
// their barriers, masses and rows, which that kernel does not write, and wait before they touch its lists.
__device__ __forceinline__ void rn_wait_for_front() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void rn_let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- cluster primitives -----------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rn_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void rn_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__host__ __device__ __forceinline__ int rn_touch_words(int lr) { return lr < 5 ? 1 : 1 << (lr - 5); }

// false: not a shape of these kernels
bool rn_list_plan(int64_t B, int64_t H, int64_t T, int64_t A, int64_t C, int64_t Kw, int64_t Kr, int mass_aware, RnListPlan *pl);
int rn_launch_lists(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream);
int rn_launch_apply(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream);
// the same for the replay of the backward pass (rn_bwd_lists.cu)
bool rn_replay_plan(int64_t B, int64_t H, int64_t T, int64_t A, int64_t C, int64_t Kw, int64_t Kr, RnListPlan *pl);
int rn_launch_replay_lists(const RnListParams &p, const RnListPlan &pl, cudaStream_t stream);
int rn_launch_replay(const RnListParams &p, const RnListPlan &pl, int dtype, cudaStream_t stream);
