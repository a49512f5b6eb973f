// elp_rank.cu -- chains rebuilt from the site words by list ranking, with the
// integrity check of the whole lattice beside it.
//
// The chains of a melt are linked lists through the site words: a run's
// b_out leads to the next run's site.  walk_kernel (elp_walk.cu) follows
// each chain run by run, several hundred dependent loads per ring of a
// relaxed melt, so its time is one ring's latency (330 us at L = 128, 1.4 ms
// at L = 256).  Here the lists are cut in front of every labelled run (the
// run holding monomer 0) and again at the sites of a sublattice that holds a
// quarter or an eighth of them (nodes):
//   segments  every node walks to the next node of its chain, or to the
//             chain's last run, and adds up the monomers on the way;
//   rounds    the nodes jump along their chains by strides that grow eightfold
//             (Wyllie's list ranking, there by doubling), ceil(log8 N) rounds
//             over the nodes alone: each learns the monomers from its run to
//             the chain's last one and which run that is;
//   chains    each labelled run checks its chain's length and its last run;
//   bonds     every node walks its segment again and writes the bonds.
// A few hops of every chain at once instead of a pass over all sites per
// round (ranking every site took 10 rounds of 10.5 us at L = 128 and 13 of
// 110 at L = 256, where its 16 bytes a site leave L2).  The walks and rounds
// are chains of L2 latencies, and what a launch waits for the one before it
// costs as much as a small box's round: hence few rounds (by doubling, a
// checked fetch at L = 64 took 111 us, by eights 91) and launches that are
// set up while the kernel before them runs (83).  L = 128: 127 us a check by
// doubling in plain launches, now 88; L = 256: 303, now 247.  Boxes up to 20^3
// do all of it in one kernel on a cluster of CTAs.
//
// The output is the TUV content of cpupol/efpol_io.c:70-77 (start site of
// monomer 0, N bond codes), the same bytes as walk_kernel writes, and a chain
// that walk_kernel would reject (a bond that is not a lattice bond, a run
// leading to an empty site or into another chain, a wrong monomer count) gets
// status 4 here too.  A pass over all site words adds up their monomers: runs
// joined to a chain from outside, or off every chain, leave that sum and the
// chains' apart.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "elp_common.h"
#include "elp_internal.h"

namespace elp {
namespace {

namespace cg = cooperative_groups;

// Per-node state {link, sum}.  link < FIN: a later node of the same chain,
// sum the monomers from this node's run up to that node's run (exclusive).
// link with FIN set: finished, the low bits name the site of the chain's last
// run (its tail) and sum counts the monomers from this node's run to the tail
// (inclusive).  EMPTY: no node.
constexpr uint32_t FIN = 0x80000000u;
constexpr uint32_t EMPTY = 0xFFFFFFFFu;

struct RankArgs {
    const uint32_t* lat;
    const uint32_t* rec;
    int L, N, P, linear;
    int q, row;                 // sublattice: one site in q of a row, row = ceil(L / q) nodes a row
    uint32_t heads;             // nodes of the sublattice; node heads + p is chain p's labelled run
    uint2* x[2];                // double-buffered node state
    uint32_t* chain_of;         // per site: chain whose tail it is, where tail[chain] agrees (never cleared)
    uint32_t* tail;             // per chain
    elp_chain_head* head;       // zeroed before
    int32_t* start;             // [P][3] or null
    uint8_t* bonds;             // [P][N], zeroed before
    int32_t* status;            // [P]
    const uint32_t* flags;      // device error flags to hand back, or null
};

struct Site {
    int t, u, v;
    __device__ __forceinline__ void step(uint32_t b, int L)
    {
        t += elp_bt(b); u += elp_bu(b); v += elp_bv(b);
        t += t < 0 ? L : 0; t -= t >= L ? L : 0;
        u += u < 0 ? L : 0; u -= u >= L ? L : 0;
        v += v < 0 ? L : 0; v -= v >= L ? L : 0;
    }
    __device__ __forceinline__ uint32_t index(int L) const
    {
        return (uint32_t)t + (uint32_t)L * ((uint32_t)u + (uint32_t)L * (uint32_t)v);
    }
    // node of the sublattice t + 2 u + 3 v = 0 (mod q), q a power of two
    __device__ __forceinline__ bool is_node(int q) const { return ((t + 2 * u + 3 * v) & (q - 1)) == 0; }
    __device__ __forceinline__ uint32_t node(const RankArgs& a) const
    {
        return (uint32_t)(t / a.q) + (uint32_t)a.row * ((uint32_t)u + (uint32_t)a.L * (uint32_t)v);
    }
};
__device__ __forceinline__ Site site_of(uint32_t s, int L)
{
    const uint32_t uL = (uint32_t)L;
    return Site{(int)(s % uL), (int)((s / uL) % uL), (int)(s / (uL * uL))};
}

// First run of a node: its site, word and monomers.  A labelled run counts
// from monomer 0 (those ahead of it close the ring).  False: no such run (a
// chain whose record is no good gets its status from the chain check).
__device__ __forceinline__ bool node_run(const RankArgs& a, uint32_t i, Site& s, uint32_t& w, uint32_t& mono)
{
    if (i < a.heads) {
        const uint32_t k = i % (uint32_t)a.row, uv = i / (uint32_t)a.row;
        s.u = (int)(uv % (uint32_t)a.L);
        s.v = (int)(uv / (uint32_t)a.L);
        s.t = (int)k * a.q + ((-(2 * s.u + 3 * s.v)) & (a.q - 1));
        if (s.t >= a.L) return false;
        w = a.lat[s.index(a.L)];
        mono = w >> ELP_CSHIFT;
        return w != 0 && !(w & ELP_LBIT);
    }
    const uint32_t p = i - a.heads;
    const uint4 r = *reinterpret_cast<const uint4*>(a.rec + ELP_REC_WORDS * (size_t)p);
    if (r.x >= (uint32_t)a.L * a.L * a.L || r.z >= r.y || (a.linear && r.z != 0)) return false;
    s = site_of(r.x, a.L);
    w = a.lat[r.x];
    mono = r.y - r.z;
    return (w & ELP_LBIT) && (w >> 5) == p;
}

// Threads of the whole grid or of one cluster.
struct Span {
    uint32_t first, count;
};

__device__ __forceinline__ void segments(const RankArgs& a, Span sp)
{
    for (uint32_t i = sp.first; i < a.heads + (uint32_t)a.P; i += sp.count) {
        Site s;
        uint32_t w, mono;
        uint2 e = make_uint2(EMPTY, 0u);
        if (node_run(a, i, s, w, mono)) {
            e.y = mono;
            for (int hop = 0;; hop++) {
                // a run is its chain's last unless a plain (unlabelled) run
                // follows; a path of more than N runs is no chain
                e.x = FIN | s.index(a.L);
                const uint32_t b = w & 15;
                if (!elp_valid_bond(b) || hop > a.N) break;
                Site n = s;
                n.step(b, a.L);
                const uint32_t wn = a.lat[n.index(a.L)];
                if (!wn || (wn & ELP_LBIT)) break;
                s = n;
                w = wn;
                if (s.is_node(a.q)) {
                    e.x = s.node(a);
                    break;
                }
                e.y += w >> ELP_CSHIFT;
            }
        }
        a.x[0][i] = e;
    }
}

// One round: every unfinished node takes up to STRIDE - 1 jumps along the links
// of the round before, each adding that node's sum and taking its link.  (Four
// at L = 64: 95 us a checked fetch, eight 91, sixteen 91; at L = 256 302, 257
// and 259 us a check.)
constexpr int STRIDE = 8;
__device__ __forceinline__ void round_of(const RankArgs& a, Span sp, int r)
{
    const uint2* in = a.x[r & 1];
    uint2* out = a.x[(r & 1) ^ 1];
    for (uint32_t i = sp.first; i < a.heads + (uint32_t)a.P; i += sp.count) {
        uint2 e = __ldcg(in + i);
        for (int hop = 1; hop < STRIDE && !(e.x & FIN); hop++) {
            const uint2 f = __ldcg(in + e.x);
            e = make_uint2(f.x, e.y + f.y);
        }
        out[i] = e;
    }
}

// Per chain: its labelled run must have reached the chain's tail with the
// chain's monomer count, and the tail must close the ring on the labelled
// run (a linear chain: end in the marker 0xf).
__device__ __forceinline__ void chain_checks(const RankArgs& a, Span sp, int fin)
{
    for (uint32_t p = sp.first; p < (uint32_t)a.P; p += sp.count) {
        const uint2 e = __ldcg(a.x[fin] + a.heads + p);
        const uint4 r = *reinterpret_cast<const uint4*>(a.rec + ELP_REC_WORDS * (size_t)p);
        bool bad = e.x == EMPTY || !(e.x & FIN) || e.y != (a.linear ? (uint32_t)a.N : (uint32_t)a.N - r.z);
        const uint32_t tail = e.x & ~FIN;
        if (!bad) {
            const uint32_t b = a.lat[tail] & 15;
            Site s = site_of(tail, a.L);
            s.step(b, a.L);
            bad = a.linear ? b != 15 : (!elp_valid_bond(b) || s.index(a.L) != r.x);
        }
        a.tail[p] = bad ? EMPTY : tail;
        if (!bad) {
            a.chain_of[tail] = p;
            if (a.start) {
                const Site s = site_of(r.x, a.L);
                a.start[3 * p] = s.t;
                a.start[3 * p + 1] = s.u;
                a.start[3 * p + 2] = s.v;
            }
            atomicAdd(&a.head->chain_monomers, (unsigned long long)((uint32_t)a.N - (a.linear ? 0u : r.z)));
        }
        a.status[p] = bad ? 4 : 0;
        if (bad) atomicMax(&a.head->bad, (uint32_t)a.P - p);
    }
}

__device__ __forceinline__ void chain_bad(const RankArgs& a, uint32_t p)
{
    atomicExch(&a.status[p], 4);
    atomicMax(&a.head->bad, (uint32_t)a.P - p);
}

// Per run of a good chain: the bond of its last monomer, at that monomer's
// place in the chain (the other monomers of a run are stored: bond 0).
__device__ __forceinline__ void write_bonds(const RankArgs& a, Span sp, int fin)
{
    for (uint32_t i = sp.first; i < a.heads + (uint32_t)a.P; i += sp.count) {
        const uint2 e = __ldcg(a.x[fin] + i);
        if (e.x == EMPTY || !(e.x & FIN)) continue;
        const uint32_t tail = e.x & ~FIN;
        const uint32_t p = __ldcg(a.chain_of + tail);
        if (p >= (uint32_t)a.P || __ldcg(a.tail + p) != tail) {
            // no good chain ends there; two (linear) chains with one tail are no chains
            if (i >= a.heads && __ldcg(a.tail + (i - a.heads)) == tail) chain_bad(a, i - a.heads);
            continue;
        }
        if (i >= a.heads && p != i - a.heads) {
            if (__ldcg(a.tail + (i - a.heads)) == tail) {
                chain_bad(a, i - a.heads);
                chain_bad(a, p);
            }
            continue;
        }
        Site s;
        uint32_t w, mono;
        if (!node_run(a, i, s, w, mono)) continue;
        const uint32_t off = a.linear ? 0u : a.rec[ELP_REC_WORDS * (size_t)p + 2];
        long at = (long)a.N - (long)off - (long)e.y;   // place of the run's first monomer
        uint8_t* out = a.bonds ? a.bonds + (size_t)p * a.N : nullptr;
        for (int hop = 0;; hop++) {
            if (mono == 0 || at < 0 || at + (long)mono > (long)a.N) {
                chain_bad(a, p);
                break;
            }
            const uint32_t b = w & 15;
            at += mono;
            if (out) out[at - 1] = (uint8_t)b;
            if (!elp_valid_bond(b) || hop > a.N) break;
            s.step(b, a.L);
            w = a.lat[s.index(a.L)];
            if (!w || (w & ELP_LBIT) || s.is_node(a.q)) break;
            mono = w >> ELP_CSHIFT;
        }
    }
}

// All site words: monomers (labelled runs from monomer 0), monomers in full
// and words that break a rule by themselves (scan_kernel's conditions).
__device__ __forceinline__ void scan_words(const RankArgs& a, Span sp)
{
    const uint32_t S = (uint32_t)a.L * a.L * a.L;
    unsigned long long after = 0, mono = 0;
    uint32_t bad = 0;
    for (uint32_t i = sp.first; i < S; i += sp.count) {
        const uint32_t w = a.lat[i];
        if (!w) continue;
        uint32_t c = w >> ELP_CSHIFT, off = 0;
        if (w & ELP_LBIT) {
            const uint32_t ch = w >> 5;
            uint4 r = make_uint4(EMPTY, 0, 0, 0);
            if (ch < (uint32_t)a.P) r = *reinterpret_cast<const uint4*>(a.rec + ELP_REC_WORDS * (size_t)ch);
            if (r.x != i) {
                bad++;
                continue;
            }
            c = r.y;
            off = a.linear ? 0u : (r.z < r.y ? r.z : r.y);
        } else if (w & 0xFFE0u) {
            bad++;
        }
        if (!(elp_valid_bond(w & 15) || (a.linear && (w & 15) == 15)) || c == 0) bad++;
        mono += c;
        after += c - off;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mono += __shfl_xor_sync(0xffffffffu, mono, o);
        after += __shfl_xor_sync(0xffffffffu, after, o);
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (mono) atomicAdd(&a.head->monomers, mono);
        if (after) atomicAdd(&a.head->site_monomers, after);
        if (bad) atomicAdd(&a.head->bad_words, (unsigned long long)bad);
    }
}

__device__ __forceinline__ Span grid_span()
{
    return Span{blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x};
}
// Zero the head and the bonds (`clear` bytes) for the kernels behind.
__device__ __forceinline__ void clear_out(const RankArgs& a, Span sp, size_t clear)
{
    uint4* zero = reinterpret_cast<uint4*>(a.head);
    for (size_t i = sp.first; i < clear / 16; i += sp.count) zero[i] = make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void all_chain_checks(const RankArgs& a, Span sp, int fin)
{
    chain_checks(a, sp, fin);
    if (sp.first == 0 && a.flags) a.head->flags = *a.flags;
}
// First statement of every kernel here: let the next launch be set up, then
// wait until the one before has ended and its results are there.  The
// pointers go through the wait, so that no load moves ahead of it; loads that
// assume read-only memory (ld.global.nc) have no place in kernels that start
// before their inputs are written.
__device__ __forceinline__ void in_turn(RankArgs& a)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;"
                 : "+l"(a.lat), "+l"(a.rec), "+l"(a.x[0]), "+l"(a.x[1]), "+l"(a.chain_of), "+l"(a.tail), "+l"(a.head),
                   "+l"(a.start), "+l"(a.bonds), "+l"(a.status), "+l"(a.flags) :: "memory");
}
__global__ void __launch_bounds__(256) rank_segments(RankArgs a, size_t clear)
{
    in_turn(a);
    clear_out(a, grid_span(), clear);
    segments(a, grid_span());
}
__global__ void __launch_bounds__(256) rank_round(RankArgs a, int r) { in_turn(a); round_of(a, grid_span(), r); }
__global__ void __launch_bounds__(256) rank_chains(RankArgs a, int fin) { in_turn(a); all_chain_checks(a, grid_span(), fin); }
__global__ void __launch_bounds__(256) rank_bonds(RankArgs a, int fin)
{
    in_turn(a);
    write_bonds(a, grid_span(), fin);
    scan_words(a, grid_span());
}

// All phases in one launch of one cluster: they hand their results over through
// global memory, and each ends in a cluster barrier, which releases and
// acquires them; loads that cross it bypass L1.
__global__ void __launch_bounds__(1024) rank_cluster(RankArgs a, int rounds, size_t clear)
{
    in_turn(a);
    cg::cluster_group cl = cg::this_cluster();
    const Span sp = grid_span();
    clear_out(a, sp, clear);
    segments(a, sp);
    for (int r = 0; r < rounds; r++) {
        cl.sync();
        round_of(a, sp, r);
    }
    cl.sync();
    all_chain_checks(a, sp, rounds & 1);
    cl.sync();
    write_bonds(a, sp, rounds & 1);
    scan_words(a, sp);
}

// Only when the sums disagree or a word breaks a rule: monomers of all runs that
// reach each chain's tail, one run per thread, and the chains with more than
// their own.  A word of no monomers (an empty run, a label of no chain) that
// reaches a tail makes its chain bad by itself.
__global__ void __launch_bounds__(256) rank_joined(RankArgs a, uint32_t* total)
{
    const uint32_t S = (uint32_t)a.L * a.L * a.L;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x) {
        uint32_t w = a.lat[i];
        if (!w) continue;
        uint32_t mono = w >> ELP_CSHIFT;
        if (w & ELP_LBIT) {
            const uint32_t ch = w >> 5;
            const uint32_t* r = a.rec + ELP_REC_WORDS * (size_t)ch;
            mono = ch < (uint32_t)a.P && r[2] < r[1] ? r[1] - r[2] : 0u;
        }
        Site s = site_of(i, a.L);
        uint32_t tail = i;
        for (int hop = 0; hop <= a.N; hop++) {
            if (!elp_valid_bond(w & 15)) break;
            s.step(w & 15, a.L);
            w = a.lat[s.index(a.L)];
            if (!w || (w & ELP_LBIT)) break;
            tail = s.index(a.L);
        }
        const uint32_t p = a.chain_of[tail];
        if (p >= (uint32_t)a.P || a.tail[p] != tail) continue;
        if (mono) atomicAdd(&total[p], mono);
        else chain_bad(a, p);
    }
}
__global__ void rank_totals(RankArgs a, const uint32_t* total)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.P || a.status[p]) return;
    const uint32_t off = a.linear ? 0u : a.rec[ELP_REC_WORDS * (size_t)p + 2];
    if (total[p] != (uint32_t)a.N - off) chain_bad(a, (uint32_t)p);
}

// Boxes up to this many sites (20^3) are ranked by one cluster, whose barriers
// cost less than launches while its eight SMs are enough: a checked fetch at
// L = 16 takes 45.7 us (N = 50) and 47 (N = 800), 46.3 and 54 by launches; at
// L = 32 62 us, 55 by launches.
constexpr size_t CLUSTER_SITES = (size_t)1 << 13;
constexpr int CLUSTER = 8;   // CTAs (portable cluster size)

RankArgs rank_args(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear, elp_walk_bufs* b)
{
    RankArgs a;
    a.lat = lat; a.rec = rec; a.L = L; a.N = N; a.P = P; a.linear = linear;
    // a quarter of the sites as nodes: short walks; an eighth where the node
    // state would leave L2 otherwise
    a.q = (size_t)L * L * L <= ((size_t)1 << 22) ? 4 : 8;
    a.row = (L + a.q - 1) / a.q;
    a.heads = (uint32_t)a.row * L * L;
    const size_t nodes = (size_t)a.heads + P;
    a.x[0] = reinterpret_cast<uint2*>(b->d_rank);
    a.x[1] = a.x[0] + nodes;
    a.chain_of = reinterpret_cast<uint32_t*>(a.x[1] + nodes);
    a.tail = a.chain_of + (size_t)L * L * L;
    a.head = b->head();
    a.start = b->d_start();
    a.bonds = b->d_bonds();
    a.status = b->d_status;
    a.flags = nullptr;
    return a;
}
}  // namespace
}  // namespace elp

cudaError_t elp_rank_chains(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear, bool want_bonds,
                            const uint32_t* flags, elp_walk_bufs* b, cudaStream_t s)
{
    using namespace elp;
    const size_t S = (size_t)L * L * L;
    if (S > ELP_RANK_MAX_SITES || P <= 0) return cudaErrorNotSupported;
    const int q = S <= ((size_t)1 << 22) ? 4 : 8;
    const size_t nodes = (size_t)((L + q - 1) / q) * L * L + P;
    cudaError_t e = elp_scratch_grow(b, &b->d_rank, &b->cap_rank, nodes * 16 + S * 4 + (size_t)P * 4);
    if (e != cudaSuccess) return e;
    RankArgs a = rank_args(lat, rec, L, N, P, linear, b);
    a.flags = flags;
    if (!want_bonds) {
        a.bonds = nullptr;
        a.start = nullptr;
    }
    // a chain has at most N runs, so at most N nodes: STRIDE^R >= N jumps reach its tail from any of them
    int R = 0;
    for (long reach = 1; reach < (long)N; reach *= STRIDE) R++;
    const size_t clear = want_bonds ? b->clear_bytes() : sizeof(elp_chain_head);
    const unsigned blocks = (unsigned)((nodes + 255) / 256 < 148 * 8 ? (nodes + 255) / 256 : 148 * 8);
    const int fin = R & 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (S <= CLUSTER_SITES) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = CLUSTER;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
        cfg.gridDim = dim3(CLUSTER);
        cfg.blockDim = dim3(1024);
        return cudaLaunchKernelEx(&cfg, rank_cluster, a, R, clear);
    }
    if ((e = cudaLaunchKernelEx(&cfg, rank_segments, a, clear)) != cudaSuccess) return e;
    for (int r = 0; r < R; r++)
        if ((e = cudaLaunchKernelEx(&cfg, rank_round, a, r)) != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)((P + 255) / 256));
    if ((e = cudaLaunchKernelEx(&cfg, rank_chains, a, fin)) != cudaSuccess) return e;
    cfg.gridDim = dim3(blocks);
    return cudaLaunchKernelEx(&cfg, rank_bonds, a, fin);
}

cudaError_t elp_rank_joined(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear, elp_walk_bufs* b,
                            cudaStream_t s)
{
    using namespace elp;
    const RankArgs a = rank_args(lat, rec, L, N, P, linear, b);
    uint32_t* total = reinterpret_cast<uint32_t*>(a.x[0]);   // the node state has served
    cudaError_t e = cudaMemsetAsync(total, 0, (size_t)P * 4, s);
    if (e != cudaSuccess) return e;
    rank_joined<<<148 * 8, 256, 0, s>>>(a, total);
    rank_totals<<<(P + 255) / 256, 256, 0, s>>>(a, total);
    return cudaGetLastError();
}
