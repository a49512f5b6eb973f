// elp_sweep2.cu -- specialised sweep kernels for the common domain shapes.
//
// Same schedule and results as the generic sweep_kernel (elp_sweep.cu); what
// changes is how the work is fed to the SM:
//   * tile edges and shared-memory strides are compile-time constants;
//   * the K anchors a thread owns in a substep are processed stage by stage
//     (all first loads, then all second loads, ...), so the dependent
//     shared-memory loads of independent moves overlap;
//   * monomer 0's runs are handled inline: while a domain is on chip each
//     labelled word carries its run length (bits 16-31) and the number of a
//     slot of a small shared-memory table {chain, offset of monomer 0}; the
//     chain records in global memory are read when the domain is loaded and
//     written back when it is stored, so no move waits on global memory.  A
//     ring tile that holds more monomer-0 runs than the table (short rings
//     crowded together, as CreatePolymers leaves them) runs its substeps with
//     the general move of elp_device.cuh instead, which keeps that
//     bookkeeping in the chain records: slower, the same bits;
//   * a tile's rows move in 16-byte words.  The origin shift makes a row
//     start anywhere, so each row fetch takes the 16-byte aligned span around
//     the row (TX + 4 words) and the tile sits sh = x0 mod 4 words into it;
//     the words of the span outside the tile become halo words.  Rows are
//     16-byte aligned in shared memory, and the threads of a warp take
//     anchors from an 8 x 4 block of rows so that their first loads hit 32
//     different banks;
//   * the grid is persistent over the tiles, and a launch of several steps
//     over a tiled box is cooperative, with a grid barrier between steps;
//   * whole boxes of rings have kernels of their own (sweep_slabs), in slabs
//     on the CTAs of a cluster where one SM would be the bound.
#include <cuda_runtime.h>
#include <math.h>

#include <atomic>

#include "elp_device.cuh"
#include "elp_kernels.h"

namespace elp {

__device__ __forceinline__ void cp_async16(uint32_t* sdst, const uint32_t* gsrc)
{
    uint32_t s = (uint32_t)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Polls of the grid barrier before a wait gives up (about a second with the
// back-off below); a launch can ask for fewer (BatchLaunch.wait_polls).
constexpr uint32_t WAIT_POLLS = 1u << 24;

// Barrier over all CTAs of a cooperative launch, in two halves: each CTA adds
// one to bar[0] (its stores before that are visible to every CTA's loads
// after the wait: tiles and records are loaded with ld.global.cg, through L2)
// and later waits (bounded) until the count reaches `target`.
__device__ __forceinline__ void grid_arrive(uint32_t* bar)
{
    __threadfence();
    atomicAdd(bar, 1u);
}
// Returns false, in every thread of the CTA, when the wait gave up.
__device__ __forceinline__ bool grid_wait(uint32_t* bar, uint32_t target, uint32_t polls)
{
    bool ok = true;
    if (threadIdx.x == 0) {
        for (uint32_t n = 0; ld_acquire_gpu(bar) < target; n++) {
            if (n >= polls) { ok = false; break; }
            __nanosleep(32);
        }
    }
    return __syncthreads_or(!ok) == 0;
}
// Last act of every CTA of a cooperative launch: the last one to leave
// zeroes the barrier counts for the next launch on the stream.
__device__ __forceinline__ void grid_exit(uint32_t* bar)
{
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
        atomicExch(bar, 0u);
        atomicExch(bar + 1, 0u);
    }
}

template <int TX, int TY, int TZ, bool PER, int NC, int SX, int SXY, int CAP, int K, int MINB>
struct Shape {
    static constexpr int R = TY * TZ;
    static constexpr int A = R * (TX / NC);   // anchors per substep
    static constexpr int G = A / 4;           // Philox counters per substep group
    static constexpr int AT = A / K;          // threads that own anchors
    static constexpr bool TILED = !PER;
    static constexpr int THREADS = (AT + 31) / 32 * 32;
    static constexpr bool TAIL = AT != THREADS;   // threads without anchors fill the last warp
    // Tiled domains: row y of plane z starts at OX + SX y + SXY z (16-byte
    // aligned) and holds the copied span of TX + 4 words, the tile at offset
    // sh in it; rows y = -1, TY and planes z = -1, TZ are halo, as is the
    // word before each row (the previous row's padding).
    static constexpr int SPAN = TX + 4;
    static constexpr int OX = PER ? 0 : SX + SXY + 4;
    static constexpr int WORDS = PER ? (SXY * TZ + 3) & ~3 : ((OX + SX * TY + SXY * TZ + SPAN + 3) & ~3);
    // A tile moves in NP passes: thread tid < AT takes word quad tid % CB of
    // row tid / CB, ZS planes further on each pass; the quad at the row's end
    // (held words if sh > 0) is one more pass over the rows.
    static constexpr int CB = TX / 4;
    static constexpr int NP = R * CB / AT;
    static constexpr int ZS = TZ / NP > 0 ? TZ / NP : 1;
    // threads of a warp take anchors from an 8 x 4 block of (y, z) rows
    static constexpr bool PERM = !PER && TY % 8 == 0 && TZ % 4 == 0 && AT % R == 0;
    // neighbour offsets: 27 boundary classes of a periodic box, one class in a tile
    static constexpr int NOFF = PER ? 27 * 16 : 16;
    // a labelled on-chip word holds its slot number + 1 above bit LSH (a
    // tile's bit 4 marks walls, a whole box has none)
    static constexpr int LSH = PER ? 4 : 5;
    static constexpr uint32_t LMASK = 0xFFFFu & ~((1u << LSH) - 1u);
    static constexpr int SLOTS = CAP < (int)(LMASK >> LSH) ? CAP : (int)(LMASK >> LSH);
    // shared-memory word offsets: lattice, move table, neighbour
    // offsets (tiles: plain word offsets too, for the general move), colours,
    // slot table (chain, offset of monomer 0 in its run), head-move rows,
    // random bytes
    static constexpr int TABW = WORDS;
    static constexpr int OFFW = TABW + ELP_MOVE_ENTRIES;
    static constexpr int WOFFW = OFFW + NOFF;
    static constexpr int TABS = WOFFW + (PER ? 0 : 16) - TABW;   // words of these tables
    static constexpr int COLW = (WOFFW + (PER ? 0 : 16) + 3) & ~3;
    static constexpr int NSLW = COLW + 4 * ((2 * NC + 3) / 4);   // slot count
    static constexpr int TILEW = (NSLW + 4) & ~3;                // the tile at hand and the next (Tile)
    static constexpr int SCHW = TILEW + 2 * 20;
    static constexpr int SLOW = SCHW + CAP;
    static constexpr int HTABW = SLOW + CAP;  // table rows (0xf, x): moves of a linear chain's monomer 0
    static constexpr int RNDW = (HTABW + 64 + 3) & ~3;
    static constexpr int NSUB = 2 * NC;              // substeps per step
    static constexpr int NG = (NSUB + 3) / 4;        // groups of four substeps
    // Random bytes, one word (four substeps) per anchor and group.  With one
    // anchor a thread, and where MINB CTAs still fit on an SM (228 KB, 1 KB
    // reserved per CTA), all NG groups of the step, drawn before its substeps
    // (PRE): no warp is late at a barrier for drawing (us per step: linear chains
    // of L = 16 13.3 -> 12.9, tiles of 16^3 at L = 64 12.7 -> 12.0, 32x16x16 at
    // L = 128 18.6 -> 17.4, 24^3 at L = 72 23.4 -> 22.5).  Else one group's, read
    // into registers as the group starts and overwritten with the next group's
    // after its first barrier: with two anchors a thread it makes no difference
    // where they fit (L = 32 28.9 both ways).
    static constexpr bool PRE = K == 1 && (size_t)MINB * ((size_t)(RNDW + NG * A) * 4 + 1024) <= 233472;
    static constexpr int TOTW = RNDW + (PRE ? NG : 1) * A;
    static constexpr size_t BYTES = (size_t)TOTW * 4;
    // neighbour offsets in words fit 16 signed bits (else they are taken
    // modulo 2^16, the reach of a shared-memory word index)
    static constexpr bool SOFF = !PER || (TX - 1) * (1 + SX + SXY) <= 32767;
    static_assert(A % 4 == 0 && A % K == 0 && THREADS <= 1024 && G <= THREADS, "anchors and draws per thread");
    static_assert(K == 1 || K == 2, "anchors per thread");
    static_assert(CAP <= 2048, "slot numbers");
    static_assert(PER || (SX % 4 == 0 && SXY % 4 == 0 && SX >= SPAN + 1 && SXY >= SX * (TY + 2)),
                  "tiled rows: 16-byte aligned, room for the span and the halo word before it");
    static_assert(PER || (NP * AT == R * CB && AT % (CB * TY) == 0 && TZ % NP == 0 && R <= AT && TX % 4 == 0),
                  "a pass of the tile copy takes whole planes");
    static_assert(WORDS < 65536, "slot sites are 16-bit word indices");
    static_assert(BYTES <= 232448, "dynamic shared memory of one CTA");
};

// Halo word of tiled domains: bit 4 (no other on-chip word has it), run
// length 1, b_out 3 (not a bond).  A slot-1 move whose next run lies in the
// halo looks up row (b_out(P), 3) of the move table, which is empty; a target
// in the halo meets the entry's test bits (bit 4 among them for moves onto a
// site or a run).
constexpr uint32_t HWALL = ELP_CUNIT | 0x10u | 3u;

extern __shared__ __align__(16) uint32_t g_smem[];

// Shared-memory word at byte offset b (offsets are kept in bytes so that a
// load or store needs no index scaling).
__device__ __forceinline__ uint32_t& SW(int b) { return *reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(g_smem) + b); }

// A labelled word (global form: chain id in bits 5-31) has come into shared
// memory at word idx: claim a slot for its chain.  Past the table's capacity
// it is only counted.
template <class SH>
__device__ __forceinline__ void claim_slot(uint32_t wv, int idx)
{
    const uint32_t slot = atomicAdd(g_smem + SH::NSLW, 1u);
    if (slot >= (uint32_t)SH::SLOTS) return;
    g_smem[SH::SCHW + slot] = wv >> 5;
    g_smem[SH::SLOW + slot] = (uint32_t)idx;   // until the record is fetched
}
// A labelled word on its way out, from box site `site`: write the chain's
// record and return the word's global form.
template <class SH>
__device__ __forceinline__ uint32_t leave_slot(uint32_t wv, uint32_t site, uint32_t* rec)
{
    const uint32_t slot = ((wv & SH::LMASK) >> SH::LSH) - 1u;
    const uint32_t chain = g_smem[SH::SCHW + slot];
    *reinterpret_cast<uint4*>(rec + ELP_REC_WORDS * (size_t)chain) =
        make_uint4(site, wv >> ELP_CSHIFT, g_smem[SH::SLOW + slot], 0u);
    return (wv & 15) | ELP_LBIT | (chain << 5);
}

// Monomer 0 sits in one of the runs an accepted move touched, whose new words
// are stored (each with the label bits its old word had): bring its slot
// number and offset to the run that holds it now.  Rarely needed, so it works
// from what the move has in registers anyway and stores through volatile
// accesses: otherwise the compiler computes its operands on every move, or
// folds its stores into the move's own as selects (8 to 13 of 60 instructions
// of every substep; now 3).
template <class SH, bool PER>
__device__ __forceinline__ void follow_label(int p, int pB, int pY, uint32_t wP, uint32_t wB, uint32_t wY, uint32_t R,
                                             uint32_t E)
{
    constexpr uint32_t LMASK = SH::LMASK;
    volatile uint32_t* const slot_off = g_smem + SH::SLOW - 1;
    volatile char* const S = reinterpret_cast<volatile char*>(g_smem);
    auto put = [&](int b, uint32_t w) { *reinterpret_cast<volatile uint32_t*>(S + b) = w; };
    const bool s = (R & 0x8000u) != 0, d1 = PER ? (E >> 28) != 0 : ((int)E >> 18) != 0, join = (E & (15u << 9)) == 0;
    const uint32_t nP = *reinterpret_cast<volatile uint32_t*>(S + p), nY = wY + ELP_CUNIT + ((E >> 9) & 15u);
    if (wP & LMASK) {
        // the anchor's run: monomer 0 leaves it as its last monomer only
        const uint32_t lb = wP & LMASK;
        if (!s && slot_off[lb >> SH::LSH] == (wP >> ELP_CSHIFT) - 1) {
            put(p, nP & ~LMASK);
            put(pY, nY | lb);
            slot_off[lb >> SH::LSH] = 0;
        }
    } else if (s && (wB & LMASK)) {
        // the next run, whose first monomer moves: monomer 0 stays (one place
        // nearer the front) unless it is that monomer
        const uint32_t lb = wB & LMASK, off0 = slot_off[lb >> SH::LSH];
        if (off0 > 0) {
            slot_off[lb >> SH::LSH] = off0 - 1;
        } else {
            put(pB, wB >= 2u * ELP_CUNIT ? (wB - ELP_CUNIT) & ~LMASK : 0u);
            if (d1) put(pY, nY | lb);   // to the target, or to the end of P's run
            else put(p, nP | lb);
            slot_off[lb >> SH::LSH] = d1 ? 0u : (nP >> ELP_CSHIFT) - 1;
        }
    } else if (join && (wY & LMASK)) {
        const uint32_t sl = (wY & LMASK) >> SH::LSH;   // a monomer joins its front
        slot_off[sl] = slot_off[sl] + 1;
    }
}

// The tile at hand, in shared memory: what its load and store need, which
// would otherwise hold registers through the substeps.
struct Tile {
    uint32_t* lat;
    uint32_t* rec;
    uint2 key;
    uint32_t t;         // absolute step
    int d, L;           // domain, box edge
    int x0, y0, z0;     // box site of the tile's first word
    unsigned long long* acc;
};
static_assert(sizeof(Tile) <= 80, "20 words of shared memory");
// The tile at hand and the next one are slots par and par ^ 1.
template <class SH>
__device__ __forceinline__ Tile& tile(int par) { return *reinterpret_cast<Tile*>(g_smem + SH::TILEW + 20 * par); }

// Random bytes of one substep group: byte q of words 0-3 of Philox counter
// {t, d, group, gq} serves anchor gq + q G in the group's four substeps: bit
// 0 the slot s, bits 1-4 the table option.  Kept as one word per anchor, a
// byte per substep, with s in bit 7 and the option in bits 2-5: the slot then
// spreads over a byte by sign replication and the option is a word offset.
// (One 32-bit load per anchor and group; four words per counter took a
// 128-bit load, 2 % more per step.)
template <class SH>
__device__ __forceinline__ void draw_bytes(uint32_t* r, uint32_t t, int d, int group, int gq, uint2 key)
{
    uint4 v = philox(make_uint4(t, (uint32_t)d, (uint32_t)group, (uint32_t)gq), key);
    v.x = ((v.x << 7) & 0x80808080u) | ((v.x << 1) & 0x3C3C3C3Cu);
    v.y = ((v.y << 7) & 0x80808080u) | ((v.y << 1) & 0x3C3C3C3Cu);
    v.z = ((v.z << 7) & 0x80808080u) | ((v.z << 1) & 0x3C3C3C3Cu);
    v.w = ((v.w << 7) & 0x80808080u) | ((v.w << 1) & 0x3C3C3C3Cu);
    const uint32_t xy01 = __byte_perm(v.x, v.y, 0x5140), zw01 = __byte_perm(v.z, v.w, 0x5140);
    const uint32_t xy23 = __byte_perm(v.x, v.y, 0x7362), zw23 = __byte_perm(v.z, v.w, 0x7362);
    r[gq] = __byte_perm(xy01, zw01, 0x5410);
    r[gq + SH::G] = __byte_perm(xy01, zw01, 0x7632);
    r[gq + 2 * SH::G] = __byte_perm(xy23, zw23, 0x5410);
    r[gq + 3 * SH::G] = __byte_perm(xy23, zw23, 0x7632);
}
// Group g's words (one buffer unless PRE).
template <class SH>
__device__ __forceinline__ uint32_t* random_words(int g) { return g_smem + SH::RNDW + (SH::PRE ? g * SH::A : 0); }

// All groups of a step (PRE), in two parts.
template <class SH, int PART>
__device__ __forceinline__ void draw_step(uint32_t t, int d, uint2 key)
{
    constexpr int N = SH::NG * SH::G, H = (N / SH::THREADS + 1) / 2 * SH::THREADS;
    for (int i = threadIdx.x + (PART ? H : 0); i < (PART ? N : (H < N ? H : N)); i += SH::THREADS)
        draw_bytes<SH>(random_words<SH>(i / SH::G), t, d, i / SH::G, i % SH::G, key);
}

// Byte kk of a random word as the low byte, its top bit spread over the next
// byte, zeros above.
template <int KK>
__device__ __forceinline__ uint32_t spread_byte(uint32_t w)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"(0x4400 | (8 | KK) << 4 | KK));
    return r;
}

// The step's colours, in bytes of x offset, drawn by one warp of the CTA;
// lane 31 returns the words of the step's domain shift.
template <class SH, int NC>
__device__ __forceinline__ uint4 draw_schedule(uint32_t t, int d, uint2 key)
{
    const uint32_t lane = threadIdx.x & 31;
    const bool shift = lane == 31;
    const uint4 w = philox(make_uint4(t, shift ? 0u : (uint32_t)d, shift ? ELP_STREAM_SHIFT : (lane | ELP_STREAM_COLOUR), 0u), key);
    if (lane < SH::NG)
        reinterpret_cast<uint4*>(g_smem + SH::COLW)[lane] =
            make_uint4(4 * bounded(w.x, NC), 4 * bounded(w.y, NC), 4 * bounded(w.z, NC), 4 * bounded(w.w, NC));
    return w;
}

// Set up a tile (one warp): domain item.y of melt J at `step`.
template <class SH, int TX, int TY, int TZ, int NC>
__device__ __forceinline__ void set_tile(const BatchJob& J, int d, uint32_t step, int par)
{
    const int ntx = J.ntx, nty = J.nty;
    const uint32_t t = J.step0 + step;
    const uint2 key = make_uint2(J.seed, J.salt);
    const uint4 w = draw_schedule<SH, NC>(t, d, key);
    if ((threadIdx.x & 31) == 31) {
        Tile& T = tile<SH>(par);
        T.lat = J.lat;
        T.rec = J.rec;
        T.key = key;
        T.t = t;
        T.d = d;
        T.L = J.L;
        T.x0 = (int)bounded(w.x, TX) + (d % ntx) * TX;
        T.y0 = (int)bounded(w.y, TY) + ((d / ntx) % nty) * TY;
        T.z0 = (int)bounded(w.z, TZ) + (d / ntx / nty) * TZ;
        T.acc = J.acc;
        g_smem[SH::NSLW] = 0;
    }
}

// Fetch the chain record of each claimed slot: the word gets the slot number
// and the run length, the slot monomer 0's offset.  A tile's other random
// bytes (PRE) are drawn while the records are on their way.
template <class SH>
__device__ __forceinline__ void fill_slots(const Tile& T, uint32_t ns)
{
    const uint32_t tid = threadIdx.x;
    uint4 rr = make_uint4(0, 0, 0, 0);
    if (tid < ns) rr = __ldcg(reinterpret_cast<const uint4*>(T.rec + ELP_REC_WORDS * (size_t)g_smem[SH::SCHW + tid]));
    if (SH::PRE && SH::TILED) draw_step<SH, 1>(T.t, T.d, T.key);
    for (uint32_t sl = tid; sl < ns; sl += SH::THREADS) {
        if (sl != tid) rr = __ldcg(reinterpret_cast<const uint4*>(T.rec + ELP_REC_WORDS * (size_t)g_smem[SH::SCHW + sl]));
        const uint32_t idx = g_smem[SH::SLOW + sl];
        g_smem[idx] = (g_smem[idx] & 15) | ((sl + 1) << SH::LSH) | (rr.y << ELP_CSHIFT);
        g_smem[SH::SLOW + sl] = rr.z;
    }
}

// threadIdx.x as the compiler cannot know it: what is computed from it here
// is not kept in registers from one tile to the next.
__device__ __forceinline__ int fresh_tid()
{
    int v;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(v));
    return v;
}

// This thread's anchors of a substep.  Byte offsets: anchor base + 4 xr; the
// x offset of colour 0 in the anchor's row (rot); whole box: address of the
// boundary class's offsets inside the box along x (cls) and the colour
// offsets at which the anchor's x is 0 or L - 1.
template <int K>
struct Anchors {
    int base[K], rot[K], cls[K], xlo[K], xhi[K], an[K];
};
// Anchor an = g + q G of a substep takes byte q of Philox counter g.  Thread
// tid owns anchors an = tid + q AT, or with PERM the anchors of the same x
// group whose row is the tid-th of the 8 x 4 row blocks.
template <class SH, int TX, int TY, int TZ, bool PER, int NC, int SX, int SXY, int K>
__device__ __forceinline__ void set_anchors(Anchors<K>& o)
{
    const int tid = SH::TAIL && (int)threadIdx.x >= SH::AT ? 0 : (int)threadIdx.x;
    int tperm = tid;
    if (SH::PERM) {
        const int r = tid % SH::R, lane = r & 31, w = r >> 5;
        const int y = (lane & 7) + 8 * (w % (TY / 8)), z = (lane >> 3) + 4 * (w / (TY / 8));
        tperm = tid - r + y + TY * z;
    }
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int an = tperm + q * SH::AT;
        o.an[q] = an;
        const int j = an / SH::R, row = an % SH::R;
        const int y = row % TY, z = row / TY;
        const int m = (2 * y + 3 * z) % NC;
        o.rot[q] = 4 * (m ? NC - m : 0);
        o.base[q] = 4 * (SH::OX + SX * y + SXY * z + NC * j);
        const int cy = y == 0 ? 0 : (y == TY - 1 ? 2 : 1);
        const int cz = z == 0 ? 0 : (z == TZ - 1 ? 2 : 1);
        o.cls[q] = PER ? 4 * SH::OFFW + 64 * (1 + 3 * cy + 9 * cz) : 0;
        o.xlo[q] = j == 0 ? 0 : -1;
        o.xhi[q] = j == TX / NC - 1 ? 4 * (NC - 1) : -1;
    }
}

// Colour offset of an anchor: (c4 + rot) mod 4 NC.
template <int NC>
__device__ __forceinline__ int colour_x(int c4, int rot)
{
    int xr4 = c4 + rot;
    if ((NC & (NC - 1)) == 0) xr4 &= 4 * (NC - 1);
    else xr4 -= xr4 >= 4 * NC ? 4 * NC : 0;
    return xr4;
}

// All substeps of a ring tile whose monomer-0 runs outnumber the slots, with
// the general move (op: words in their global form, monomer 0's bookkeeping
// in the chain records, halo words ELP_WALL).  Not inlined: it runs rarely,
// and its registers stay out of the main substep loop.  Same anchors, random
// words and order as the main loop.  Returns this thread's accepted moves.
// The anchors are passed by value so that the caller's copies stay in
// registers.
template <class SH, int K, int NC, int SX, int SXY>
__device__ __noinline__ uint32_t general_substeps(const Anchors<K> an, const uint8_t* table, int par)
{
    const int* woffs = reinterpret_cast<const int*>(g_smem + SH::WOFFW);
    const Tile T = tile<SH>(par);
    const int sh4 = 4 * (T.x0 & 3);
    Dom D;
    D.S = g_smem; D.tab = table; D.rec = T.rec;
    D.ox = SH::OX + (T.x0 & 3); D.sx = SX; D.sxy = SXY; D.L = T.L;
    D.x0 = T.x0; D.y0 = T.y0; D.z0 = T.z0;
    uint32_t acc = 0;
    for (int g = 0; g < SH::NG; g++) {
        uint32_t rw[K];
        for (int q = 0; q < K; q++) rw[q] = random_words<SH>(g)[an.an[q]];
        for (int kk = 0; kk < 4 && 4 * g + kk < SH::NSUB; kk++) {
            const int c4 = (int)g_smem[SH::COLW + 4 * g + kk];
            if (!SH::PRE && kk == 1 && (int)threadIdx.x < SH::G && g + 1 < SH::NG)
                draw_bytes<SH>(random_words<SH>(g + 1), T.t, T.d, g + 1, (int)threadIdx.x, T.key);
            for (int q = 0; q < K; q++) {
                const int xr4 = colour_x<NC>(c4, an.rot[q]);
                const uint32_t b = rw[q] >> (8 * kk);
                if (!SH::TAIL || (int)threadIdx.x < SH::AT)
                    acc += (uint32_t)op(D, (an.base[q] + sh4 + xr4) >> 2, woffs, ((b >> 7) & 1u) | ((b >> 1) & 0x1Eu));
            }
            __syncthreads();
        }
    }
    return acc;
}

// The K anchors of one thread, one substep, random bytes in byte KK of words
// rw.  Returns accepted moves.  c4 = 4 c, k the substep; LIN: the melt holds
// linear chains (head moves of monomer 0).
//
// The kernel is bound by instruction issue (the ALU pipe takes an instruction
// every other cycle) and by the chain of shared-memory loads, so the move is
// written for few instructions: 43 per warp and substep, 21 of them on the
// ALU pipe (the move of elp_device.cuh laid out the same way: 81 and 40).
// (A second table with each entry's change of the anchor's word takes four of
// them out, but its load costs as much: linear chains of L = 24 23.7 us per step
// with it, 23.1 without, L = 40 23.6 and 23.1, L = 32 in slabs 16.0 and 15.9.)
// One 32-bit entry of the move table carries everything the move's rows
// decide (target, test, the new words' parts), new words come from additions,
// and the target and next run are stored ahead of the anchor so that a move
// back into the anchor's run (target = anchor) needs no case of its own.
// L = 256: 145.8 -> 113.6 us per step together with the tile copy below (104.7
// with the label's branch as it is now).
// Loads predicated on the lanes that need them cut a tenth of the
// shared-memory wavefronts but were 3 % slower.
template <class SH, int K, bool PER, int NC, bool LIN, int KK>
__device__ __forceinline__ uint32_t substepK(const Anchors<K>& an, int sh4, const uint32_t (&rw)[K], uint32_t voff, int c4,
                                             uint32_t t, int d, int k, uint2 key)
{
    constexpr int TAB4 = 4 * SH::TABW;
    int p[K], tc[K];
    uint32_t wP[K], R[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int xr4 = colour_x<NC>(c4, an.rot[q]);
        p[q] = an.base[q] + sh4 + xr4;
        wP[q] = SW(p[q]);
        R[q] = spread_byte<KK>(rw[q]);
        if (SH::TAIL && (int)threadIdx.x >= SH::AT) wP[q] = R[q] = 0;   // slot 0 of an empty site: no move
        // whole box: the boundary class's offsets (64 bytes each)
        tc[q] = PER ? an.cls[q] + (xr4 == an.xlo[q] ? -64 : 0) + (xr4 == an.xhi[q] ? 64 : 0) : 0;
    }
    int pB[K];
    uint32_t wB[K], V[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        // {word offset of the step b_out << 16 | row of b_out << 10}: each
        // lane of a tile's warp holds one code's
        V[q] = PER ? SW(tc[q] + (int)((wP[q] & 15) << 2)) : __shfl_sync(0xffffffffu, voff, (int)wP[q]);
        pB[q] = SH::SOFF ? p[q] + ((int)V[q] >> 14) : (int)((uint32_t)(p[q] + (V[q] >> 14)) & 0x3FFFFu);
        // slot 0 looks at P's own run instead of the next one
        const uint32_t w1 = SW(pB[q]);
        wB[q] = (R[q] & 0x8000u) ? w1 : wP[q];
    }
    uint32_t E[K];
    bool c2[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        // row (s ? b_out : 0, src2): src2 is the next run's b_out if that run
        // holds one monomer (slot 1), P's own if it holds two or more (slot 0)
        const bool s = (R[q] & 0x8000u) != 0;
        c2[q] = wB[q] >= 2u * ELP_CUNIT;
        uint32_t ix = R[q] & (V[q] | 0x3Cu);
        if (c2[q] != s) ix += (wB[q] & 15) << 6;
        E[q] = SW(TAB4 + (int)ix);
    }
    int pY[K];
    uint32_t wY[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (PER) {
            const uint32_t V2 = SW(tc[q] + (int)(E[q] >> 26));
            pY[q] = SH::SOFF ? p[q] + ((int)V2 >> 14) : (int)((uint32_t)(p[q] + (V2 >> 14)) & 0x3FFFFu);
        } else {
            pY[q] = p[q] + ((int)E[q] >> 18);
        }
        wY[q] = SW(pY[q]);
    }
    uint32_t acc = 0;
#pragma unroll
    for (int q = 0; q < K; q++) {
        const bool s = (R[q] & 0x8000u) != 0;
        const bool ok = E[q] != 0 && (wY[q] & E[q] & (PER ? 0xFu : 0x1Fu)) == 0;
        const uint32_t nP = ((wP[q] & ~15u) | ((E[q] >> 5) & 15u)) + (E[q] & 0x30000u) - ELP_CUNIT;
        const uint32_t nB = c2[q] ? wB[q] - ELP_CUNIT : 0u;
        const uint32_t nY = wY[q] + ELP_CUNIT + ((E[q] >> 9) & 15u);
        if (ok) SW(pY[q]) = nY;
        if (ok && s) SW(pB[q]) = nB;
        if (ok) SW(p[q]) = nP;
        // (a labelled anchor matters to slot 0 only, where wB is its word)
        if (!LIN && ok && ((wB[q] | wY[q]) & SH::LMASK))
            follow_label<SH, PER>(p[q], pB[q], pY[q], wP[q], wB[q], wY[q], R[q], E[q]);
        // monomer 0 of a linear chain has no predecessor: no move but its own,
        // below, moves it or joins the front of its run (the branch cost
        // L = 64, N = 200 16.9 us per step, now 14.8; L = 192 63.8, now 58.4)
        if (LIN && ok) wP[q] = nP;
        acc += ok ? 1u : 0u;
    }
    // linear chains: monomer 0 has no predecessor and moves about monomer 1,
    // tried at the anchor holding it after that anchor's regular attempt:
    // with probability 1/2 (bit 0 of its own Philox word) one option of row
    // (0xf, run length > 1 ? 0 : b_out) -- it leaves to the empty site P - u
    // (its bond to monomer 1 becoming u), or, alone on P, joins the next run.
    // Monomer 0 of a linear chain is the first of its run: its offset stays 0.
    if (LIN) {
        const uint8_t* htab = reinterpret_cast<const uint8_t*>(g_smem + SH::HTABW);
#pragma unroll
        for (int q = 0; q < K; q++) {
            const uint32_t w0 = wP[q];
            if (!(w0 & SH::LMASK)) continue;
            const uint4 h = philox(make_uint4(t, (uint32_t)d, (uint32_t)k | ELP_STREAM_HEAD, (uint32_t)an.an[q]), key);
            if (!(h.x & 1)) continue;
            const uint32_t cP = w0 >> ELP_CSHIFT, bo = w0 & 15;
            const uint32_t e = htab[((cP >= 2 ? 0u : bo) << 4) | ((h.x >> 1) & 15)];
            if (!e) continue;
            const uint32_t d2 = e >> 4, code = cP >= 2 ? (~d2) & 15u : bo;
            const uint32_t Vh = SW((PER ? tc[q] : 4 * SH::OFFW) + (int)(code << 2));
            const int pH = SH::SOFF ? p[q] + ((int)Vh >> 14) : (int)((uint32_t)(p[q] + (Vh >> 14)) & 0x3FFFFu);
            const uint32_t wH = SW(pH);
            if (cP >= 2) {
                if (wH == 0) {
                    SW(pH) = d2 | (w0 & SH::LMASK) | ELP_CUNIT;
                    SW(p[q]) = (w0 & ~SH::LMASK) - ELP_CUNIT;
                    acc++;
                }
            } else if (wH != HWALL) {
                SW(pH) = (wH + ELP_CUNIT) | (w0 & SH::LMASK);
                SW(p[q]) = 0;
                acc++;
            }
        }
    }
    return acc;
}

// The substeps of one step of a domain.  Returns this thread's accepted moves.
template <class SH, int K, bool PER, int NC, bool LIN>
__device__ __forceinline__ uint32_t substeps(const Anchors<K>& an, int sh4, uint32_t voff, int par)
{
    uint32_t acc = 0;
    // what draws need in here (linear chains; groups drawn one at a time)
    uint32_t t = 0;
    int d = 0;
    uint2 key = make_uint2(0, 0);
    if (LIN || !SH::PRE) {
        t = tile<SH>(par).t;
        d = tile<SH>(par).d;
        key = tile<SH>(par).key;
    }
#pragma unroll 1
    for (int g = 0; g < SH::NG; g++) {
        const uint4 c4 = reinterpret_cast<const uint4*>(g_smem + SH::COLW)[g];
        uint32_t rw[K];
#pragma unroll
        for (int q = 0; q < K; q++) rw[q] = random_words<SH>(g)[an.an[q]];
        acc += substepK<SH, K, PER, NC, LIN, 0>(an, sh4, rw, voff, (int)c4.x, t, d, 4 * g, key);
        __syncthreads();
        // the next group's bytes: every thread has read this group's
        if (!SH::PRE && (int)threadIdx.x < SH::G && g + 1 < SH::NG)
            draw_bytes<SH>(random_words<SH>(g + 1), t, d, g + 1, (int)threadIdx.x, key);
        acc += substepK<SH, K, PER, NC, LIN, 1>(an, sh4, rw, voff, (int)c4.y, t, d, 4 * g + 1, key);
        __syncthreads();
        if (SH::NSUB % 4 && 4 * g + 2 >= SH::NSUB) break;
        acc += substepK<SH, K, PER, NC, LIN, 2>(an, sh4, rw, voff, (int)c4.z, t, d, 4 * g + 2, key);
        __syncthreads();
        acc += substepK<SH, K, PER, NC, LIN, 3>(an, sh4, rw, voff, (int)c4.w, t, d, 4 * g + 3, key);
        __syncthreads();
    }
    return acc;
}

// Add a thread's accepted moves to the melt's counter, one atomic per warp.
__device__ __forceinline__ void count_accepted(unsigned long long* acc, unsigned long long v)
{
    if (!acc) return;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, v);
}

// Tables of a launch into shared memory: moves, neighbour offsets (elp_move_table
// builds them in this order) and rows (0xf, x) of the transition table (moves of
// a linear chain's monomer 0).
template <class SH, bool PER>
__device__ __forceinline__ void load_tables(const BatchLaunch& a)
{
    static_assert(SH::TABS % 4 == 0 && SH::TABW % 4 == 0, "16-byte copies");
    for (int i = threadIdx.x; i < SH::TABS / 4; i += SH::THREADS) cp_async16(g_smem + SH::TABW + 4 * i, a.moves + 4 * i);
    for (int i = threadIdx.x; i < 64; i += SH::THREADS) g_smem[SH::HTABW + i] = a.table[960 + i];
}

// Words i < N of a whole box into shared memory, strided over the CTA: word i
// comes from src(i) and goes to word at(i); labelled(word, place) is called for
// the labelled ones, once a thread has copied all of its words.  (With a branch
// for them between the loads, and a record's latency behind it, a launch of one
// step took 18.8 us at L = 16 and 22.5 at L = 18, now 15.1 and 20.5.)
template <int N, int THREADS, class Src, class At, class Labelled>
__device__ __forceinline__ void load_words(Src src, At at, Labelled labelled)
{
    static_assert((N + THREADS - 1) / THREADS <= 32, "a bit for each of a thread's words");
    const int tid = threadIdx.x;
    uint32_t mask = 0;
#pragma unroll 8
    for (int k = 0; k < (N + THREADS - 1) / THREADS; k++) {
        const int i = tid + k * THREADS;
        const bool in = N % THREADS == 0 || i < N;
        const uint32_t wv = in ? __ldcg(src(i)) : 0u;
        if (in) g_smem[at(i)] = wv;
        mask |= wv & ELP_LBIT ? 1u << k : 0u;
    }
    for (; mask; mask &= mask - 1) {
        const int idx = at(tid + (__ffs(mask) - 1) * THREADS);
        labelled(g_smem[idx], idx);
    }
}

// Whole boxes of linear chains, and of rings where sweep_slabs below does not
// run: each CTA holds one melt for all steps of the launch.
//
// K anchors per thread: K = 2 where a domain has more than 1024 anchors per
// substep, else 1 (more warps hide latency better than more moves in flight
// per thread).  The random stream does not depend on K.
template <int TX, int NC, int SX, int SXY, int CAP, int K, bool LIN>
__global__ void __launch_bounds__(((TX * TX * (TX / NC) / K) + 31) / 32 * 32, 1) sweep_box(BatchLaunch a)
{
    using SH = Shape<TX, TX, TX, true, NC, SX, SXY, CAP, K, 1>;
    constexpr int SITES = TX * TX * TX;
    uint32_t* S = g_smem;
    const int tid = threadIdx.x;
    load_tables<SH, true>(a);
    Anchors<K> an;
    set_anchors<SH, TX, TX, TX, true, NC, SX, SXY, K>(an);
    const uint32_t step_dev = a.step_dev ? *a.step_dev : 0u;
    for (int it = blockIdx.x; it < a.nitems; it += gridDim.x) {
        const BatchJob& J = a.jobs[a.items[it].x];
        uint32_t* lat = J.lat;
        uint32_t* rec = J.rec;
        const uint2 key = make_uint2(J.seed, J.salt);
        const uint32_t t0 = J.step0 + a.step_base + step_dev;
        __syncthreads();   // the previous melt's words and slots have been read
        if (tid == 0) g_smem[SH::NSLW] = 0;
        __syncthreads();
        load_words<SITES, SH::THREADS>([&](int i) { return lat + i; },
                                       [](int i) { return i % TX + SX * (i / TX % TX) + SXY * (i / (TX * TX)); },
                                       [](uint32_t wv, int idx) { claim_slot<SH>(wv, idx); });
        cp_async_wait_all();
        __syncthreads();
        const uint32_t ns = g_smem[SH::NSLW];
        if (ns > (uint32_t)SH::SLOTS) {
            // more monomer-0 runs than slots: leave the box untouched, report
            if (tid == 0) atomicOr(a.error, 1u);
            continue;
        }
        if (tid == 0) tile<SH>(0).rec = rec;
        __syncthreads();
        fill_slots<SH>(tile<SH>(0), ns);
        unsigned long long accepted = 0;
        for (int st = 0; st < a.nsteps; st++) {
            const uint32_t t = t0 + (uint32_t)st;
            if (SH::PRE) {
                draw_step<SH, 0>(t, 0, key);
                draw_step<SH, 1>(t, 0, key);
            } else if (tid < SH::G) {
                draw_bytes<SH>(random_words<SH>(0), t, 0, 0, tid, key);
            }
            if (tid >= SH::THREADS - 32) draw_schedule<SH, NC>(t, 0, key);
            if (tid == 0) {
                tile<SH>(0).t = t;
                tile<SH>(0).d = 0;
                tile<SH>(0).key = key;
            }
            __syncthreads();
            accepted += substeps<SH, K, true, NC, LIN>(an, 0, 0u, 0);
        }
        for (int i = tid; i < SITES; i += SH::THREADS) {
            uint32_t wv = S[i % TX + SX * (i / TX % TX) + SXY * (i / (TX * TX))];
            if (wv & SH::LMASK) wv = leave_slot<SH>(wv, (uint32_t)i, rec);
            lat[i] = wv;
        }
        count_accepted(J.acc, accepted);
    }
}

// ---- whole boxes of rings, one anchor a thread -----------------------------------
//
// A box of 32^3 on one SM (sweep_box) is bound by that SM's issue slots and
// shared-memory wavefronts: 2048 anchors a substep, 29.5 us per step.  Here it
// lies in C slabs of whole planes on the CTAs of a cluster.  Each slab holds a
// copy of the plane below and of the plane above, so that a move, which
// touches the anchor's neighbours at most, reads this CTA's shared memory
// only; a new word that another slab holds too is sent there.  15.9 us per
// step with C = 8.
//
// What it took: words fetched from the neighbouring slab instead of kept as
// copies 26.5 us; a cluster barrier (release, acquire) per substep 20.9, as it
// waits for every store to be acknowledged (0.31 us in a loop of its own,
// against 0.13 for a barrier of arrivals that announce bytes); C = 4: 20.3.
// L = 30: 28.3 -> 18.0, L = 28: 24.0 -> 14.4.  L = 26 has slabs of 13 planes
// only: 20.1 -> 23.0, left alone.
//
// The boxes that fit the threads of one CTA (up to 24^3) run as one slab: they
// too are bound by latency, and gain from monomer 0's offsets kept by site
// (see slab_substep).  L = 16: 9.9 -> 8.9 us per step (N = 50; N = 20: 11.2
// -> 10.1), L = 18: 12.5 -> 11.1, L = 20: 14.4 -> 13.7, L = 22: 16.6 -> 16.0,
// L = 24: 18.8 -> 18.6.
__device__ __forceinline__ uint32_t cluster_address(uint32_t rank)   // of a CTA's g_smem
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(g_smem)), "r"(rank));
    return a;
}
// Barrier over the cluster, in two halves: stores before the arrival, to this
// CTA's shared memory or another's, are seen after the wait.
__device__ __forceinline__ void cluster_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Wait for the completion of a phase of an mbarrier; false when it gave up
// after `polls` tries of a microsecond at most.
constexpr uint32_t SLAB_POLLS = 1u << 20;
__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t parity, uint32_t polls)
{
    for (uint32_t n = 0; n < polls; n++) {
        uint32_t done;
        asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2, 1000;\n"
                     "selp.u32 %0, 1, 0, q;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// Slab of ZS planes of a box shared by C CTAs.  C > 1: on chip with a copy of
// the plane below and of the plane above (planes 0 and ZS + 1).
template <int TX, int NC, int SX, int SXY, int C>
struct Slab {
    static constexpr int ZS = TX / C, R = TX * TX, HALO = C > 1 ? 1 : 0, PLANES = ZS + 2 * HALO;
    static constexpr int A = R * (TX / NC), G = A / 4;      // anchors and counters of the whole box
    // one anchor a thread, WP x groups of each row; a warp's lanes take the
    // rows of one plane if there are other slabs
    static constexpr int WP = TX / NC, ROWS = C > 1 ? 32 : TX, THREADS = (ROWS * WP * ZS + 31) / 32 * 32;
    __device__ static bool idle()
    {
        return (ROWS != TX && (int)threadIdx.x % ROWS >= TX) || (ROWS * WP * ZS != THREADS && (int)threadIdx.x >= ROWS * WP * ZS);
    }
    static constexpr int NSUB = 2 * NC, NG = (NSUB + 3) / 4;
    // a labelled word holds its chain + 1 above bit LSH; monomer 0's offset
    // in the run at a site has a word of its own, copied as the site's is
    static constexpr int LSH = 4;
    static constexpr uint32_t LMASK = 0xFFF0u;
    static constexpr int MAXCHAINS = LMASK >> LSH;
    static constexpr int TABW = (SXY * PLANES + 3) & ~3;
    static constexpr int OFFW = TABW + ELP_MOVE_ENTRIES;
    static constexpr int TABS = ELP_MOVE_ENTRIES + 27 * 16;
    static constexpr int OFSW = TABW + TABS;                // offsets by site
    static constexpr int COLW = OFSW + TABW;                // colours of a step and the next
    static constexpr int BARW = COLW + 8 * NG;              // two mbarriers
    static constexpr size_t BYTES = (size_t)(BARW + 4) * 4;
    static_assert(TX % C == 0 && C <= 8 && THREADS <= 1024 && A % 4 == 0 && TABS % 4 == 0, "slabs of whole planes");
    static_assert(C == 1 || (TX <= 32 && ZS >= 4), "a warp's anchors lie in one plane and reach one other slab at most");
    static_assert((TX - 1) * (1 + SX + (C > 1 ? 0 : SXY)) + SXY <= 32767, "neighbour offsets in 16 signed bits");
    static_assert(BYTES <= 232448, "dynamic shared memory of one CTA");
};

// The words of anchor gq + q G for one substep group, as draw_bytes keeps them.
__device__ __forceinline__ uint32_t own_bytes(uint32_t t, int group, uint32_t gq, uint32_t sel, uint2 key)
{
    const uint4 v = philox(make_uint4(t, 0u, (uint32_t)group, gq), key);
    const uint32_t w = __byte_perm(__byte_perm(v.x, v.y, sel), __byte_perm(v.z, v.w, sel), 0x5410);
    return ((w << 7) & 0x80808080u) | ((w << 1) & 0x3C3C3C3Cu);
}

// Slabs: where a warp's new words go besides this CTA's copy.  Words of byte
// offsets from .. from + len - 1 are sent to the slab below or above (cluster
// address `to` plus the byte offset), announced at that slab's mbarrier.
struct Push {
    uint32_t to, bar, len;
    int from;
    uint32_t sent;      // bytes this thread has sent in the substep
};
// Word at byte offset b, belonging to the site at offset `site`.  Predicated:
// with branches around the sends L = 32 took 18.7 us per step, so 15.9.
__device__ __forceinline__ void push_word(Push& o, bool ok, int site, int b, uint32_t w)
{
    const uint32_t go = ok && (uint32_t)(site - o.from) < o.len ? 4u : 0u;
    asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %3, 0;\n"
                 "@q st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];\n}"
                 ::"r"(o.to + (uint32_t)b), "r"(w), "r"(o.bar), "r"(go) : "memory");
    o.sent += go;
}

// One substep of a slab: the move of substepK, one anchor a thread.  What
// bounds a slab is the chain of latencies from barrier to barrier (a warp or
// two per scheduler), so monomer 0's offsets at the runs that it may leave or
// be joined in are fetched along with the words, the new words are complete
// before they are stored, and each is sent once (words sent to one address
// would arrive in any order).
template <class SH, int NC, int KK>
__device__ __forceinline__ uint32_t slab_substep(const Anchors<1>& an, uint32_t rw, int c4, Push& push)
{
    const int xr4 = colour_x<NC>(c4, an.rot[0]);
    const int p = an.base[0] + xr4;
    const int tc = an.cls[0] + (xr4 == an.xlo[0] ? -64 : 0) + (xr4 == an.xhi[0] ? 64 : 0);
    uint32_t wP = SW(p), R = spread_byte<KK>(rw);
    if (SH::idle()) wP = R = 0;   // slot 0 of an empty site: no move
    const uint32_t V = SW(tc + (int)((wP & 15) << 2));
    const int pB = p + ((int)V >> 14);
    const bool s = (R & 0x8000u) != 0;
    const uint32_t w1 = SW(pB), wB = s ? w1 : wP;
    const int from = s ? pB : p;              // the run that the monomer leaves
    const uint32_t oB = SW(4 * SH::OFSW + from);
    const bool c2 = wB >= 2u * ELP_CUNIT;
    uint32_t ix = R & (V | 0x3Cu);
    if (c2 != s) ix += (wB & 15) << 6;
    const uint32_t E = SW(4 * SH::TABW + (int)ix);
    const uint32_t V2 = SW(tc + (int)(E >> 26));
    const int pY = p + ((int)V2 >> 14);
    const uint32_t wY = SW(pY), oY = SW(4 * SH::OFSW + pY);
    const bool ok = E != 0 && (wY & E & 0xFu) == 0, away = (E >> 28) != 0;   // away: not into the anchor's run
    uint32_t nP = ((wP & ~15u) | ((E >> 5) & 15u)) + (E & 0x30000u) - ELP_CUNIT;
    uint32_t nB = c2 ? wB - ELP_CUNIT : 0u, nY = wY + ELP_CUNIT + ((E >> 9) & 15u);
    int at = -1;                              // the run with monomer 0 whose offset changes
    uint32_t off = 0;
    if (ok && ((wB | wY) & SH::LMASK)) {
        const uint32_t lb = wB & SH::LMASK;
        if (lb) {
            off = oB;
            at = from;
            if (off == (s ? 0u : (wB >> ELP_CSHIFT) - 1)) {   // monomer 0 is the one that moves
                (s ? nB : nP) &= ~SH::LMASK;
                (away ? nY : nP) |= lb;
                off = away ? 0u : (nP >> ELP_CSHIFT) - 1;
                at = pY;
            } else if (s) {
                off--;
            }
        } else if (away) {                    // one joins the front of its run
            off = oY + 1;
            at = pY;
        }
    }
    if (ok && away) SW(pY) = nY;
    if (ok && s) SW(pB) = nB;
    if (ok) SW(p) = nP;
    if (at >= 0) SW(4 * SH::OFSW + at) = off;
    if (SH::HALO) {
        push_word(push, ok && away, pY, pY, nY);
        push_word(push, ok && s, pB, pB, nB);
        push_word(push, ok, p, p, nP);
        push_word(push, at >= 0, at, 4 * SH::OFSW + at, off);
    }
    return ok ? 1u : 0u;
}

template <int TX, int NC, int SX, int SXY, int C>
__global__ void __launch_bounds__(Slab<TX, NC, SX, SXY, C>::THREADS, 1) sweep_slabs(BatchLaunch a)
{
    using SH = Slab<TX, NC, SX, SXY, C>;
    uint32_t* S = g_smem;
    const int tid = threadIdx.x;
    uint32_t rank = 0;
    if (C > 1) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int row = tid / SH::ROWS, zl = row % SH::ZS, j = SH::idle() ? 0 : row / SH::ZS;
    // the two lowest planes' warps write words that the slab below holds too
    // (its planes ZS and ZS + 1), the two highest planes' the slab above
    Push push = {};
    const bool sends = C > 1 && (zl < 2 || zl >= SH::ZS - 2);   // the same for a warp
    if (sends) {
        const uint32_t at = cluster_address(zl < 2 ? (rank == 0 ? C - 1 : rank - 1) : (rank + 1 == C ? 0 : rank + 1));
        push.to = zl < 2 ? at + 4 * SXY * SH::ZS : at - 4 * SXY * SH::ZS;
        push.bar = at + 4 * SH::BARW;
        push.from = zl < 2 ? 0 : 4 * SXY * SH::ZS;
        push.len = 8 * SXY;
    }
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(S + SH::BARW);
    if (C > 1 && tid == 0) {
        // one arrival of each warp that sends here
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(4 * SH::WP) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8), "r"(4 * SH::WP) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < SH::TABS / 4; i += SH::THREADS) cp_async16(S + SH::TABW + 4 * i, a.moves + 4 * i);
    auto draw_colours = [&](uint32_t t, uint2 key) {   // of step t, by one warp
        const uint4 w = philox(make_uint4(t, 0u, (uint32_t)tid | ELP_STREAM_COLOUR, 0u), key);
        if (tid < SH::NG)
            reinterpret_cast<uint4*>(S + SH::COLW + 4 * SH::NG * (t & 1))[tid] =
                make_uint4(4 * bounded(w.x, NC), 4 * bounded(w.y, NC), 4 * bounded(w.z, NC), 4 * bounded(w.w, NC));
    };
    const BatchJob& J = a.jobs[a.items[blockIdx.x / C].x];
    uint32_t* lat = J.lat;
    uint32_t* rec = J.rec;
    const uint2 key = make_uint2(J.seed, J.salt);
    const uint32_t t0 = J.step0 + a.step_base + (a.step_dev ? *a.step_dev : 0u);
    load_words<SH::R * SH::PLANES, SH::THREADS>(
        [&](int i) {
            int z = SH::ZS * (int)rank + i / SH::R - SH::HALO;
            z += z < 0 ? TX : 0; z -= z >= TX ? TX : 0;
            return lat + i % SH::R + SH::R * z;
        },
        [](int i) { return i % TX + SX * (i / TX % TX) + SXY * (i / SH::R); },
        [&](uint32_t wv, int idx) {
            const uint32_t chain = wv >> 5;
            const uint4 rr = __ldcg(reinterpret_cast<const uint4*>(rec + ELP_REC_WORDS * (size_t)chain));
            S[idx] = (wv & 15) | ((chain + 1) << SH::LSH) | (rr.y << ELP_CSHIFT);
            S[SH::OFSW + idx] = rr.z;
        });
    Anchors<1> an;
    uint32_t gq, sel;
    {
        const int y = SH::idle() ? 0 : tid % SH::ROWS, z = zl + SH::ZS * (int)rank;
        const int n = y + TX * z + SH::R * j, m = (2 * y + 3 * z) % NC;
        an.an[0] = n;
        an.rot[0] = 4 * (m ? NC - m : 0);
        an.base[0] = 4 * (SX * y + SXY * (zl + SH::HALO) + NC * j);
        // boundary classes; z wraps only where there is one slab
        const int cy = y == 0 ? 0 : (y == TX - 1 ? 2 : 1), cz = C > 1 ? 1 : zl == 0 ? 0 : (zl == TX - 1 ? 2 : 1);
        an.cls[0] = 4 * SH::OFFW + 64 * (1 + 3 * cy + 9 * cz);
        an.xlo[0] = j == 0 ? 0 : -1;
        an.xhi[0] = j == TX / NC - 1 ? 4 * (NC - 1) : -1;
        gq = (uint32_t)(n % SH::G);
        sel = (uint32_t)(n / SH::G) * 0x11u + 0x40u;
    }
    if (tid < 32) draw_colours(t0, key);
    uint32_t rw = own_bytes(t0, 0, gq, sel, key);
    cp_async_wait_all();
    if (C > 1) {
        cluster_arrive();   // every slab is loaded, its mbarriers are set up: words may come
        cluster_wait();
    } else {
        __syncthreads();
    }

    const uint32_t polls = a.wait_polls ? a.wait_polls : SLAB_POLLS;
    uint32_t phase = 0;
    bool alive = true;
    // End of a substep, in two halves: a warp that sends tells the receiver
    // how many bytes (having read what it needed of the words that the
    // receiver may now change), then every thread waits for what this slab
    // receives and for the CTA.  One lane arrives for its warp, so __syncwarp
    // puts the other lanes' loads and stores of those words ahead of it (a
    // reduction orders no memory), and it releases them to the neighbour, whose
    // waits acquire at cluster scope.  The release covers this CTA's shared
    // memory only, where those words are: one that covers everything waits for
    // the words just sent (L = 32: 15.9 us per step, so 25.4; by a warp of its
    // own that sends nothing 20.3).  A thread whose wait gave up sends nothing
    // and announces nothing any more: unpaced by its neighbours it would arrive
    // at their mbarriers more often than a phase has room for.
    auto announce = [&]() {
        if (sends) {
            const uint32_t bytes = __reduce_add_sync(0xffffffffu, push.sent);
            __syncwarp();
            if ((tid & 31) == 0 && alive)
                asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n"
                             "mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(push.bar),
                             "r"(bytes) : "memory");
            push.sent = 0;
            push.bar ^= 8;
        }
    };
    auto settle = [&](int odd) {
        if (C > 1 && alive && !wait_parity(bar + 8 * odd, phase, polls)) {
            alive = false;
            push.len = 0;
        }
        phase ^= odd;
        __syncthreads();
    };
    unsigned long long accepted = 0;
    for (int st = 0; st < a.nsteps; st++) {
        const uint32_t t = t0 + (uint32_t)st;
        uint32_t acc = 0, next = 0;
        // a test may make one CTA leave after the first step
        if (C > 1 && st == 1 && (int)blockIdx.x + 1 == a.hold_cta1) {
            alive = false;
            break;
        }
#pragma unroll 1
        for (int g = 0; g < SH::NG; g++) {
            const uint4 c4 = reinterpret_cast<const uint4*>(S + SH::COLW + 4 * SH::NG * (t & 1))[g];
            acc += slab_substep<SH, NC, 0>(an, rw, (int)c4.x, push);
            announce();
            if (g == 0 && tid < 32) draw_colours(t + 1, key);
            settle(0);
            acc += slab_substep<SH, NC, 1>(an, rw, (int)c4.y, push);
            announce();
            // the next group's bytes while the words are on their way
            next = own_bytes(g + 1 < SH::NG ? t : t + 1, g + 1 < SH::NG ? g + 1 : 0, gq, sel, key);
            settle(1);
            if (!(SH::NSUB % 4 && 4 * g + 2 >= SH::NSUB)) {
                acc += slab_substep<SH, NC, 2>(an, rw, (int)c4.z, push);
                announce();
                settle(0);
                acc += slab_substep<SH, NC, 3>(an, rw, (int)c4.w, push);
                announce();
                settle(1);
            }
            rw = next;
        }
        accepted += acc;
        if (C > 1 && !(alive = __syncthreads_and(alive))) break;
    }
    if (alive) {
        for (int i = tid; i < SH::R * SH::ZS; i += SH::THREADS) {
            const int xy = i % SH::R, idx = xy % TX + SX * (xy / TX) + SXY * (i / SH::R + SH::HALO);
            const uint32_t site = (uint32_t)(i + SH::R * SH::ZS * (int)rank);
            uint32_t wv = S[idx];
            if (wv & SH::LMASK) {
                const uint32_t chain = ((wv & SH::LMASK) >> SH::LSH) - 1u;
                *reinterpret_cast<uint4*>(rec + ELP_REC_WORDS * (size_t)chain) =
                    make_uint4(site, wv >> ELP_CSHIFT, S[SH::OFSW + idx], 0u);
                wv = (wv & 15) | ELP_LBIT | (chain << 5);
            }
            lat[site] = wv;
        }
    } else if (tid == 0) {
        atomicOr(a.error, 4u);
    }
    count_accepted(J.acc, accepted);
    if (C > 1) {
        cluster_arrive();   // a slab that gave up may still be sent words
        cluster_wait();
    }
}

// Tiles: each CTA takes tile after tile of a step; a launch of several steps
// is cooperative, with a grid barrier between steps.
//
// At L = 128 (one tile per CTA and step) what surrounds the substeps took 10.7
// of a step's 23.2 us, mostly address arithmetic (1180 instructions per warp,
// now 790) and latencies in a row.  So a thread's quads differ by whole planes
// only, labelled words are found in registers on the way in and out, the
// step's random bytes are drawn while the quads and the chain records are on
// their way, the next tile is set up while this one is stored, and what a
// tile's load and store need sits in shared memory in between (held in
// registers it made the substep loop recompute its own).  18.4 us per step
// then, 23.4 before; 17.5 with the label's branch as it is now.
template <int TX, int TY, int TZ, int NC, int SX, int SXY, int CAP, int K, int MINB, bool LIN>
__global__ void __launch_bounds__(((TY * TZ * (TX / NC) / K) + 31) / 32 * 32, MINB) sweep_tiles(BatchLaunch a)
{
    using SH = Shape<TX, TY, TZ, false, NC, SX, SXY, CAP, K, MINB>;
    uint32_t* S = g_smem;
    const int tid = threadIdx.x;
    // launches of one step are set up while the one before them runs; what
    // comes before the wait reads the group's constant tables only
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    load_tables<SH, false>(a);
    for (int i = tid; i < SH::WORDS / 4; i += SH::THREADS)
        reinterpret_cast<uint4*>(S)[i] = make_uint4(HWALL, HWALL, HWALL, HWALL);
    cp_async_wait_all();
    __syncthreads();
    const uint32_t voff = g_smem[SH::OFFW + (tid & 15)];   // step of code lane & 15
    Anchors<K> an;
    set_anchors<SH, TX, TY, TZ, false, NC, SX, SXY, K>(an);
    const bool scheduler = tid >= SH::THREADS - 32;   // the warp that sets up the next tile
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t step0 = a.step_base + (a.step_dev ? *a.step_dev : 0u);

    unsigned long long accepted = 0;
    int par = 0;
    // one melt alone: its job stays in registers of the warp that needs it
    const bool alone = a.njobs == 1;
    BatchJob J;
    if (scheduler) {
        const uint2 item = alone ? make_uint2(0u, blockIdx.x) : a.items[blockIdx.x];
        J = a.jobs[item.x];
        set_tile<SH, TX, TY, TZ, NC>(J, (int)item.y, step0, 0);
    }
    __syncthreads();
    for (int so = 0, it = blockIdx.x;;) {
        // ---- load: quads of four words; a quad never straddles x = L (L and
        // xa are multiples of 4)
        {
            const Tile T = tile<SH>(par);
            const int ft = fresh_tid(), L = T.L;
            const bool mover = !SH::TAIL || ft < SH::AT, ender = SH::R == SH::THREADS || ft < SH::R;
            const uint32_t LL = (uint32_t)(L * L);
            const int xa = T.x0 & ~3, sh = T.x0 & 3;
            const int mc = ft % SH::CB, my = ft / SH::CB % TY, mz = ft / SH::CB / TY;
            const int ey = ft % TY, ez = ft / TY;   // the row whose end quad it moves
            uint4 ve = make_uint4(HWALL, HWALL, HWALL, HWALL);
            if (ender && sh) {
                int x = xa + TX; x -= x >= L ? L : 0;
                int y = T.y0 + ey; y -= y >= L ? L : 0;
                int z = T.z0 + ez; z -= z >= L ? L : 0;
                ve = __ldcg(reinterpret_cast<const uint4*>(T.lat + ((uint32_t)(x + L * y) + LL * (uint32_t)z)));
            }
            constexpr int NB = SH::NP <= 6 ? SH::NP : 4;   // quads in flight per thread
            static_assert(SH::NP % NB == 0, "passes per batch");
            int x = xa + 4 * mc; x -= x >= L ? L : 0;
            int y = T.y0 + my; y -= y >= L ? L : 0;
            int z = T.z0 + mz; z -= z >= L ? L : 0;
            const uint32_t* src = T.lat + (uint32_t)(x + L * y);
            const int at0 = SH::OX + SX * my + SXY * mz + 4 * mc;
#pragma unroll
            for (int i0 = 0; i0 < SH::NP; i0 += NB) {
                uint4 v[NB];
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    if (mover) v[i] = __ldcg(reinterpret_cast<const uint4*>(src + LL * (uint32_t)z));
                    z += SH::ZS; z -= z >= L ? L : 0;
                }
                // half of the step's random bytes while the quads are on their way
                if (SH::PRE && i0 == 0) draw_step<SH, 0>(T.t, T.d, T.key);
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    if (mc == 0) {   // words ahead of the tile
                        if (sh > 0) v[i].x = HWALL;
                        if (sh > 1) v[i].y = HWALL;
                        if (sh > 2) v[i].z = HWALL;
                    }
                    if (mover) {
                        const int at = at0 + (i0 + i) * SXY * SH::ZS;
                        *reinterpret_cast<uint4*>(S + at) = v[i];
                        if ((v[i].x | v[i].y | v[i].z | v[i].w) & ELP_LBIT) {
                            if ((v[i].x & ELP_LBIT) && v[i].x != HWALL) claim_slot<SH>(v[i].x, at);
                            if ((v[i].y & ELP_LBIT) && v[i].y != HWALL) claim_slot<SH>(v[i].y, at + 1);
                            if ((v[i].z & ELP_LBIT) && v[i].z != HWALL) claim_slot<SH>(v[i].z, at + 2);
                            if (v[i].w & ELP_LBIT) claim_slot<SH>(v[i].w, at + 3);
                        }
                    }
                }
            }
            if (ender) {   // words 0 .. sh-1 of the end quad are the tile's
                const int at = SH::OX + SX * ey + SXY * ez + TX;
                if (sh < 1) ve.x = HWALL; else if (ve.x & ELP_LBIT) claim_slot<SH>(ve.x, at);
                if (sh < 2) ve.y = HWALL; else if (ve.y & ELP_LBIT) claim_slot<SH>(ve.y, at + 1);
                if (sh < 3) ve.z = HWALL; else if (ve.z & ELP_LBIT) claim_slot<SH>(ve.z, at + 2);
                ve.w = HWALL;
                *reinterpret_cast<uint4*>(S + at) = ve;
            }
            if (!SH::PRE && tid < SH::G) draw_bytes<SH>(random_words<SH>(0), T.t, T.d, 0, tid, T.key);
        }
        __syncthreads();

        // ---- monomer-0 runs, substeps
        const uint32_t ns = g_smem[SH::NSLW];
        const bool crowded = ns > (uint32_t)SH::SLOTS;
        if (!crowded) {
            fill_slots<SH>(tile<SH>(par), ns);
            __syncthreads();
            accepted += substeps<SH, K, false, NC, LIN>(an, 4 * (tile<SH>(par).x0 & 3), voff, par);
        } else if (!LIN) {
            // a crowded ring tile: its words are still in their global form
            // and the records hold the runs' lengths and offsets; halo words
            // become the general move's walls
            for (int i = tid; i < SH::WORDS; i += SH::THREADS)
                if (S[i] == HWALL) S[i] = ELP_WALL;
            __syncthreads();
            if (SH::PRE) draw_step<SH, 1>(tile<SH>(par).t, tile<SH>(par).d, tile<SH>(par).key);
            __syncthreads();
            accepted += general_substeps<SH, K, NC, SX, SXY>(an, reinterpret_cast<const uint8_t*>(a.table), par);
            for (int i = tid; i < SH::WORDS; i += SH::THREADS)
                if (S[i] == ELP_WALL) S[i] = HWALL;
            __syncthreads();
        } else {
            // linear chains: the general move does not apply; leave the tile
            // untouched, report
            if (tid == 0) atomicOr(a.error, 1u);
            __syncthreads();   // every thread has read the count
        }

        // ---- store: quads inside the tile, single words at its ragged ends
        if (!crowded || !LIN) {
            const Tile T = tile<SH>(par);
            const int ft = fresh_tid(), L = T.L;
            const bool mover = !SH::TAIL || ft < SH::AT, ender = SH::R == SH::THREADS || ft < SH::R;
            const uint32_t LL = (uint32_t)(L * L), lmask = crowded ? 0u : SH::LMASK;
            const int xa = T.x0 & ~3, sh = T.x0 & 3;
            const int mc = ft % SH::CB, my = ft / SH::CB % TY, mz = ft / SH::CB / TY;
            int x = xa + 4 * mc; x -= x >= L ? L : 0;
            int y = T.y0 + my; y -= y >= L ? L : 0;
            int z = T.z0 + mz; z -= z >= L ? L : 0;
            const uint32_t xy = (uint32_t)(x + L * y);
            const int at0 = SH::OX + SX * my + SXY * mz + 4 * mc;
#pragma unroll
            for (int i = 0; i < SH::NP; i++) {
                const uint32_t site = xy + LL * (uint32_t)z;
                z += SH::ZS; z -= z >= L ? L : 0;
                if (!mover) continue;
                uint4 v = *reinterpret_cast<const uint4*>(S + at0 + i * SXY * SH::ZS);
                if ((v.x | v.y | v.z | v.w) & lmask) {
                    if (v.x & lmask) v.x = leave_slot<SH>(v.x, site, T.rec);
                    if (v.y & lmask) v.y = leave_slot<SH>(v.y, site + 1, T.rec);
                    if (v.z & lmask) v.z = leave_slot<SH>(v.z, site + 2, T.rec);
                    if (v.w & lmask) v.w = leave_slot<SH>(v.w, site + 3, T.rec);
                }
                if (mc != 0 || sh == 0) {
                    *reinterpret_cast<uint4*>(T.lat + site) = v;
                } else {
                    if (sh < 2) T.lat[site + 1] = v.y;
                    if (sh < 3) T.lat[site + 2] = v.z;
                    T.lat[site + 3] = v.w;
                }
            }
            if (ender && sh) {
                const int ey = ft % TY, ez = ft / TY;
                int x = xa + TX; x -= x >= L ? L : 0;
                int y = T.y0 + ey; y -= y >= L ? L : 0;
                int z = T.z0 + ez; z -= z >= L ? L : 0;
                const uint32_t es = (uint32_t)(x + L * y) + LL * (uint32_t)z;
                uint4 v = *reinterpret_cast<const uint4*>(S + SH::OX + SX * ey + SXY * ez + TX);
                if (v.x & lmask) v.x = leave_slot<SH>(v.x, es, T.rec);
                T.lat[es] = v.x;
                if (sh > 1) {
                    if (v.y & lmask) v.y = leave_slot<SH>(v.y, es + 1, T.rec);
                    T.lat[es + 1] = v.y;
                }
                if (sh > 2) {
                    if (v.z & lmask) v.z = leave_slot<SH>(v.z, es + 2, T.rec);
                    T.lat[es + 2] = v.z;
                }
            }
        }

        // ---- the next tile
        it += gridDim.x;
        const bool over = it >= a.nitems;   // the step's tiles are done
        if (over) {
            it = blockIdx.x;
            so++;
        }
        if (so >= a.nsteps) {
            count_accepted(tile<SH>(par).acc, accepted);
            break;
        }
        if (scheduler) {
            const uint2 item = alone ? make_uint2(0u, (uint32_t)it) : a.items[it];
            if (!alone) J = a.jobs[item.x];
            set_tile<SH, TX, TY, TZ, NC>(J, (int)item.y, step0 + (uint32_t)so, par ^ 1);
        }
        __syncthreads();   // the tile's words have been read, the next tile is set up
        unsigned long long* const acc = tile<SH>(par).acc;
        par ^= 1;
        if (acc != tile<SH>(par).acc) {
            count_accepted(acc, accepted);
            accepted = 0;
        }
        if (over) {
            // a test may keep one CTA from arriving at the first barrier
            if (tid == 0 && !(so == 1 && (int)blockIdx.x + 1 == a.hold_cta1)) grid_arrive(a.grid_bar);
            if (!grid_wait(a.grid_bar, gridDim.x * (uint32_t)so, a.wait_polls ? a.wait_polls : WAIT_POLLS)) {
                if (tid == 0) atomicOr(a.error, 4u);
                count_accepted(tile<SH>(par).acc, accepted);
                break;
            }
        }
    }
    if (a.nsteps > 1) grid_exit(a.grid_bar);
}

}  // namespace elp

// ---- dispatch ----------------------------------------------------------------
namespace {
// Resident CTAs per SM of one kernel, per device (a cooperative launch is
// sized by it); 0 until the group set-up on that device has asked.
constexpr int MAX_DEVICES = 64;
using Kernel = void (*)(BatchLaunch);

// Launch (or, with check_only, test) kernel k of shape SH.
template <class SH, bool PER, int CAP, int MINB>
cudaError_t launch2(const Sweep2Launch* l, Kernel k, std::atomic<int>* per_sm, cudaStream_t s)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    if (l->check_only) {
        // expected monomer-0 runs per domain must stay far inside the slot table
        const double m = l->max_runs_per_domain;
        if (!(PER ? m <= CAP : m + 8.0 * sqrt(m) + 16.0 <= CAP)) return cudaErrorNotSupported;
        // set the shared-memory limit and size the grid here, outside any
        // stream capture, once per device (groups are committed often in the
        // serving loop)
        if (per_sm[dev].load() < 1) {
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::BYTES);
            int n = 0;
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, SH::THREADS, SH::BYTES);
            if (e != cudaSuccess) return e;
            if (n < 1) return cudaErrorNotSupported;
            per_sm[dev].store(n);
        }
        const_cast<Sweep2Launch*>(l)->threads_out = SH::THREADS;
        const_cast<Sweep2Launch*>(l)->smem_out = SH::BYTES;
        return cudaSuccess;
    }
    int grid = l->args.nitems;
    if (PER || l->args.nsteps <= 1) {
        if (grid > l->nsm * MINB) grid = l->nsm * MINB;
        if (grid < 1) return cudaSuccess;
        if (PER) {
            k<<<grid, SH::THREADS, SH::BYTES, s>>>(l->args);
            return cudaGetLastError();
        }
    }
    // tiled, several steps: a cooperative launch (every CTA resident, or an
    // error) of at most as many CTAs as fit on the device at once
    const bool several = l->args.nsteps > 1;
    const int per = per_sm[dev].load();
    if (per < 1) return cudaErrorNotSupported;
    if (several && grid > l->nsm * per) grid = l->nsm * per;
    if (grid < 1) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(SH::THREADS);
    cfg.dynamicSmemBytes = SH::BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (several) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        // one step: tables and anchors ahead of the previous launch's end (50
        // steps at L = 128 22.4 -> 19.1 us each, L = 64 15.9 -> 13.5, L = 256
        // 108.9 -> 106.1), where two launches' CTAs fit side by side or fill
        // the SMs anyway: in between, the early ones share an SM with their
        // like later on (125 tiles at L = 80: 16.4 -> 19.0).  Not beside other
        // groups of a batch or a server, whose place they would take while they
        // wait.  Other contexts cannot be seen from here; several of them at
        // once (a thread each, 100 steps and a checked fetch in turn) still gain:
        // L = 64 twice 12.3 -> 10.8 ms for 600 steps, eight times 35.5 -> 22.4,
        // L = 128 four times 53.2 -> 37.5, against launches in plain order.
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = l->sole && (2 * grid <= l->nsm || grid > l->nsm);
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, l->args);
}

// Whole boxes of rings in C slabs.  Clusters only for the one group of a
// context or batch, and as many as are resident at once: a box on 8 SMs takes
// half the time of one on a single SM, so beside the other groups of a mix it
// would cost throughput.  Other contexts cannot be seen from here; many at once
// wait for the host more than for SMs (L = 32, a thread each, 600 steps and six
// checked fetches: 8 contexts 29 ms, 40 contexts 126, on the one-SM kernel of
// before 49 and 162).  cudaErrorNotSupported sends the caller to sweep_box.
template <int TX, int NC, int SX, int SXY, int C>
cudaError_t launch_slabs(const Sweep2Launch* l, cudaStream_t s)
{
    using SH = elp::Slab<TX, NC, SX, SXY, C>;
    static std::atomic<int> resident[MAX_DEVICES];   // clusters; 0: not asked yet
    const auto k = elp::sweep_slabs<TX, NC, SX, SXY, C>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    if (C > 1 && !l->sole) return cudaErrorNotSupported;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(l->args.nitems * C));
    cfg.blockDim = dim3(SH::THREADS);
    cfg.dynamicSmemBytes = SH::BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    if (l->check_only) {
        // chains are numbered in 12 bits; the bound is sweep_box's
        if (l->max_runs_per_domain > 2048) return cudaErrorNotSupported;
        static_assert(SH::MAXCHAINS > 2048, "chain numbers");
        // as in launch2: outside any capture, once per device
        if (resident[dev].load() < 1) {
            int n = 1;
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::BYTES);
            if (e == cudaSuccess && C > 1) e = cudaOccupancyMaxActiveClusters(&n, k, &cfg);
            if (e != cudaSuccess) return e;
            if (n < 1) return cudaErrorNotSupported;
            resident[dev].store(n);
        }
    }
    if (C > 1 && l->args.nitems > resident[dev].load()) return cudaErrorNotSupported;
    if (l->check_only) {
        const_cast<Sweep2Launch*>(l)->threads_out = SH::THREADS;
        const_cast<Sweep2Launch*>(l)->smem_out = SH::BYTES;
        return cudaSuccess;
    }
    if (l->args.nitems < 1) return cudaSuccess;
    return cudaLaunchKernelEx(&cfg, k, l->args);
}

template <int TX, int NC, int SX, int SXY, int CAP, int K, bool LIN>
cudaError_t launch_box(const Sweep2Launch* l, cudaStream_t s)
{
    static std::atomic<int> per_sm[MAX_DEVICES];   // zero-initialised (static storage)
    return launch2<elp::Shape<TX, TX, TX, true, NC, SX, SXY, CAP, K, 1>, true, CAP, 1>(
        l, elp::sweep_box<TX, NC, SX, SXY, CAP, K, LIN>, per_sm, s);
}

template <int TX, int TY, int TZ, int NC, int SX, int SXY, int CAP, int K, int MINB, bool LIN>
cudaError_t launch_tiles(const Sweep2Launch* l, cudaStream_t s)
{
    static std::atomic<int> per_sm[MAX_DEVICES];
    return launch2<elp::Shape<TX, TY, TZ, false, NC, SX, SXY, CAP, K, MINB>, false, CAP, MINB>(
        l, elp::sweep_tiles<TX, TY, TZ, NC, SX, SXY, CAP, K, MINB, LIN>, per_sm, s);
}
}  // namespace

// Launch (or, with check_only, test) the specialised kernel for a shape.
// Returns cudaErrorNotSupported when none fits (the caller then uses the
// generic kernel).
extern "C" cudaError_t elp_launch_sweep2(const Sweep2Launch* l, cudaStream_t s)
{
    const elp_geometry& g = l->geom;
// whole boxes of rings in slabs: edge, colour modulus, strides, slabs
#define SLABS(X_, NC_, SX_, SXY_, C_)                                                                              \
    if (g.L == X_ && g.periodic && g.ncol == NC_ && l->sx == SX_ && l->sxy == SXY_ && !l->linear) {                 \
        const cudaError_t e = launch_slabs<X_, NC_, SX_, SXY_, C_>(l, s);                                           \
        if (C_ == 1 || e != cudaErrorNotSupported) return e;                                                        \
    }
    SLABS(32, 16, 33, 1056, 8)
    SLABS(30, 15, 30, 900, 6)
    SLABS(28, 14, 30, 840, 7)
    SLABS(24, 24, 24, 576, 1)
    SLABS(22, 22, 22, 484, 1)
    SLABS(20, 20, 21, 422, 1)
    SLABS(18, 18, 20, 360, 1)
    SLABS(16, 16, 16, 256, 1)
#undef SLABS
    if (l->args.nsteps > 1 && !g.periodic && !l->args.grid_bar) return cudaErrorNotSupported;
// tiles: edges, colour modulus, shared-memory strides, slot capacity, anchors
// per thread, min blocks per SM
#define TILES(X_, Y_, Z_, NC_, SX_, SXY_, CAP_, K_, MINB_)                                                      \
    if (g.tx == X_ && g.ty == Y_ && g.tz == Z_ && !g.periodic && g.ncol == NC_ && l->sx == SX_ && l->sxy == SXY_) \
        return l->linear ? launch_tiles<X_, Y_, Z_, NC_, SX_, SXY_, CAP_, K_, MINB_, true>(l, s)                \
                         : launch_tiles<X_, Y_, Z_, NC_, SX_, SXY_, CAP_, K_, MINB_, false>(l, s);
// whole boxes: edge, colour modulus, strides, slot capacity, anchors per
// thread, linear chains
#define BOX(X_, NC_, SX_, SXY_, CAP_, K_, LIN_)                                                                 \
    if (g.L == X_ && g.periodic && g.ncol == NC_ && l->sx == SX_ && l->sxy == SXY_ && (l->linear != 0) == LIN_) \
        return launch_box<X_, NC_, SX_, SXY_, CAP_, K_, LIN_>(l, s);
    TILES(32, 32, 32, 16, 40, 1364, 1792, 2, 1)
    TILES(32, 32, 16, 16, 40, 1364, 1024, 1, 1)
    TILES(32, 16, 16, 16, 40, 724, 1024, 1, 2)
    // 16^3: three CTAs an SM leave the compiler registers for a faster kernel
    // (one box of L = 64: 12.0 us per step, 12.9 with four), but four take 512
    // tiles in one round (8 boxes of L = 64 22.8 against 31.1, L = 128 21.2
    // against 29.0).  A round's time is as the CTAs in it (16 and 21.4 us): four
    // where their rounds hold fewer slots in all (729 tiles, L = 144: 28.8 with
    // three, 39.5 with four; 2304 tiles: 92.1 and 85.2; 3072: 108 and 124).
    auto slots = [&](int per_sm) { return (l->args.nitems + l->nsm * per_sm - 1) / (l->nsm * per_sm) * per_sm; };
    if (slots(4) < slots(3)) {
        TILES(16, 16, 16, 16, 24, 444, 512, 1, 4)
    }
    TILES(16, 16, 16, 16, 24, 444, 512, 1, 3)
    TILES(48, 24, 24, 16, 56, 1456, 2048, 2, 1)
    BOX(16, 16, 16, 256, 2048, 1, true)
    BOX(32, 16, 33, 1056, 2048, 2, true)
    BOX(32, 16, 33, 1056, 2048, 2, false)
    BOX(24, 24, 24, 576, 2048, 1, true)
#undef TILES
// Shapes of rings only (linear chains of these boxes are refused): the even
// boxes between (18 to 22 as one slab, above), and the tiles that boxes of 40,
// 60, 72, 100, 120 ... take.  On the generic kernel a step took 171 us
// (L = 20), 175 (28), 238 (40) and 251 (72); here 13.7, 24.0 (14.4 in slabs),
// 23.1 and 22.4.
#define TILES(X_, Y_, Z_, NC_, SX_, SXY_, CAP_, K_, MINB_)                                                       \
    if (g.tx == X_ && g.ty == Y_ && g.tz == Z_ && !g.periodic && g.ncol == NC_ && l->sx == SX_ &&                \
        l->sxy == SXY_ && !l->linear)                                                                            \
        return launch_tiles<X_, Y_, Z_, NC_, SX_, SXY_, CAP_, K_, MINB_, false>(l, s);
    TILES(24, 24, 24, 24, 32, 832, 2048, 1, 1)
    TILES(40, 20, 20, 20, 48, 1056, 2048, 1, 1)
    TILES(20, 20, 20, 20, 28, 616, 1024, 1, 2)
    BOX(26, 13, 26, 676, 2048, 2, false)
    BOX(28, 14, 30, 840, 2048, 2, false)
    BOX(30, 15, 30, 900, 2048, 2, false)
#undef BOX
#undef TILES
    return cudaErrorNotSupported;
}
