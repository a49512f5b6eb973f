// elp_common.h -- pieces shared by the single-melt and batch C ABIs: error
// reporting, geometry choice, device-side ring reconstruction and checks,
// TUV text parsing.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/elp.h"
#include "elp_internal.h"

// Record a message for elp_last_error() and return `s`.
elp_status elp_fail(elp_status s, const char* fmt, ...);

#define ELP_CUDA_TRY(call)                                                                           \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ != cudaSuccess)                                                                       \
            return elp_fail(e_ == cudaErrorMemoryAllocation ? ELP_ERR_NOMEM : ELP_ERR_CUDA,          \
                            "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);    \
    } while (0)

// Rings and geometry of a job spec; returns ELP_OK or ELP_ERR_ARG.
elp_status elp_resolve_spec(const elp_job_spec* spec, int* P, elp_geometry* g);

// Device error flags written by kernels instead of trapping.
elp_status elp_device_errors(const uint32_t* d_flags, cudaStream_t s);

// The same from flags already on the host.
elp_status elp_flags_status(uint32_t flags);

// What a chain rebuild reports beside the chains.
struct elp_chain_head {
    unsigned long long chain_monomers;   // of the good chains, counted from monomer 0
    unsigned long long site_monomers;    // of all site words, the same way
    unsigned long long monomers;         // of all site words
    unsigned long long bad_words;        // site words that break a rule by themselves
    uint32_t bad;                        // P - (first broken chain), 0: none
    uint32_t flags;                      // the device error flags
    uint32_t pad[6];
};
static_assert(sizeof(elp_chain_head) == 64, "the bonds follow 16-byte aligned");
// The ranked chains hold every monomer of the melt and every site word is in
// order: integrity code 0.
inline bool elp_chains_good(const elp_chain_head& h, int N, int P)
{
    return !h.bad && !h.bad_words && h.chain_monomers == h.site_monomers && h.monomers == (unsigned long long)N * P;
}

// Scratch buffers for rebuilding chains on the device.
struct elp_walk_bufs {
    uint8_t* d_out = nullptr;              // head, bonds [P][N], start [P][3] of the melt at hand
    int P = 0, N = 0;                      // its layout (elp_walk_bufs_reserve)
    int32_t* d_status = nullptr;
    uint32_t* d_visit = nullptr;
    unsigned long long* d_cnt = nullptr;
    unsigned long long* d_obs = nullptr;   // observables: [P][6] ring sums + histogram
    int32_t* h_status = nullptr;           // pinned host copies of the ring statuses and counters
    unsigned long long* h_cnt = nullptr;
    uint8_t* h_out = nullptr;              // pinned host copy of the head and, of small melts, of all of d_out
    int unstaged = 0;                      // copies to pageable memory that it would have sped up
    void* d_rank = nullptr;                // list ranking (elp_rank.cu)
    size_t cap_out = 0, cap_status = 0, cap_visit = 0, cap_obs = 0, cap_rank = 0;   // device bytes
    size_t cap_h_rings = 0, cap_h_out = 0;
    size_t bytes = 0;                      // device bytes held
    size_t limit = 0;                      // test hook: no more than these (0: what the device has)
    cudaStream_t pooled = nullptr;         // set: device buffers from the device's memory pool, in this stream's order

    static size_t bond_bytes(int P, int N) { return ((size_t)P * N + 15) & ~(size_t)15; }
    elp_chain_head* head() const { return reinterpret_cast<elp_chain_head*>(d_out); }
    uint8_t* d_bonds() const { return d_out + sizeof(elp_chain_head); }
    int32_t* d_start() const { return reinterpret_cast<int32_t*>(d_bonds() + bond_bytes(P, N)); }
    size_t clear_bytes() const { return sizeof(elp_chain_head) + bond_bytes(P, N); }
    size_t out_bytes() const { return clear_bytes() + (size_t)P * 12; }
};
void elp_walk_bufs_free(elp_walk_bufs* b);
// Grow one of b's device buffers (*p, *cap bytes) to `need` bytes, by half at
// least where the device has room for that: a batch's members come in any
// order of size, and every growth synchronises the device.  The old contents
// are lost.  Where there is no room the ranking's scratch is given up first
// (its callers can walk); cudaErrorMemoryAllocation leaves the buffer empty.
cudaError_t elp_scratch_grow(elp_walk_bufs* b, void** p, size_t* cap, size_t need);
// Lay the scratch out for P chains of N (and grow it), with `sites` visit
// counters.
elp_status elp_walk_bufs_reserve(elp_walk_bufs* b, int P, int N, size_t sites);
// Build a melt's site words and chain records on the device from host chains
// (start[3*P], bonds[P*N]); ELP_ERR_INTEGRITY (codes 3/4) for invalid chains,
// which leave the lattice partly written.
elp_status elp_build_melt(uint32_t* lat, uint32_t* rec, int L, int N, int P, int linear, const int32_t* start,
                          const uint8_t* bonds, elp_walk_bufs* wb, cudaStream_t s);
// The reference initial melt (CreatePolymers) written on the device,
// stream-ordered: no transfer, no host wait.
elp_status elp_init_melt_device(uint32_t* lat, uint32_t* rec, int L, int N, int P, int linear, cudaStream_t s);

// Boxes up to this many sites (L = 512) rebuild their chains by list
// ranking; larger ones by the chain walk.
constexpr size_t ELP_RANK_MAX_SITES = (size_t)1 << 27;
// Chains of one melt into b's head, bonds, start and statuses by list ranking
// (elp_rank.cu), stream-ordered; without bonds the checks alone.  `flags`
// (or null): device error flags to put into the head.  cudaErrorNotSupported
// (nothing launched) above ELP_RANK_MAX_SITES sites, cudaErrorMemoryAllocation
// (nothing launched) if its scratch finds no room: the callers then walk.
cudaError_t elp_rank_chains(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear, bool want_bonds,
                            const uint32_t* flags, elp_walk_bufs* b, cudaStream_t s);
inline bool elp_must_walk(cudaError_t ranked)
{
    return ranked == cudaErrorNotSupported || ranked == cudaErrorMemoryAllocation;
}
// After it, where the head's sums disagree, a word breaks a rule or a chain is
// broken: also find the chains that other runs lead into.
cudaError_t elp_rank_joined(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear, elp_walk_bufs* b,
                            cudaStream_t s);
// Rebuild rings (start[3P], bonds[P*N]) of one melt into host buffers.  Error
// flags an earlier launch left in `flags` (may be null) take precedence.
elp_status elp_fetch_rings(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear,
                           const uint32_t* flags, elp_walk_bufs* b, int32_t* start, uint8_t* bonds, cudaStream_t s);
// Observables of one melt (elp_observe); any output may be null.
elp_status elp_observe_melt(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear,
                            const uint32_t* flags, elp_walk_bufs* b, double* cms_tuv, double* rg2, double* sl, uint64_t* run_hist, int nbins, cudaStream_t s);
// Rings of one melt into host buffers together with its integrity code (0, 3
// or 4).  A ring that cannot be walked gives code 4 with ELP_OK: the buffers
// are then unspecified.
elp_status elp_fetch_checked_melt(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear,
                                  const uint32_t* flags, elp_walk_bufs* b, int32_t* start, uint8_t* bonds, int32_t* code, cudaStream_t s);
// Integrity check of one melt (code 0, 3 or 4 as CheckIntegrity).
elp_status elp_check_melt(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear,
                          const uint32_t* flags, elp_walk_bufs* b, int32_t* code, cudaStream_t s);

// Parse TUV text for a melt of box L, P rings of N.  Returns ELP_OK or
// ELP_ERR_FORMAT (message set).
elp_status elp_parse_tuv(const char* text, const char* name, int L, int N, int P, int32_t* start, uint8_t* bonds);
elp_status elp_read_file(const char* path, char** text, size_t* len);
