// elp_observe.cu -- in-situ observables of a melt, computed on the device.
//
// The chains are rebuilt on the device (elp_rank.cu), and one warp per chain
// accumulates exact integer sums over its monomers, positions taken relative
// to monomer 0's site and unwrapped along the ring:
//   St, Su, Sv    sums of the lattice coordinates (t, u, v)
//   Sq            sum of x^2 + y^2 + z^2 with x = t+u-v, y = t-u, z = v
//   runs          occupied sites of the ring (zero bonds = N - runs; a
//                 linear chain ends in the run whose b_out is the marker 0xf)
// and a block-level histogram of run lengths (monomers per occupied site).
// Only these P x 48 bytes go to the host, where the centre of mass, the
// radius of gyration and the stored-length fraction are formed exactly as
// ComputeCMS / ComputeGyration / ComputeSL (analysis/mode_compute.c:145-217)
// form them from the PTL positions of LoadPTL (analysis/mode_io.c:509-606).
#include <cuda_runtime.h>
#include <string.h>

#include <vector>

#include "elp_common.h"
#include "elp_internal.h"
#include "elp_kernels.h"

namespace elp {

struct ObsArgs {
    const uint32_t* lat;
    const uint32_t* rec;
    int L, N, P, nbins, linear;
    unsigned long long* out;    // [P][6]: St, Su, Sv, Sq, runs | status << 32, site of monomer 0
    unsigned long long* hist;   // [nbins]
};

__global__ void observe_kernel(ObsArgs a)
{
    __shared__ unsigned long long hist[ELP_OBS_MAX_BINS];
    for (int i = threadIdx.x; i < a.nbins; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < a.P) {
        const int L = a.L, N = a.N;
        const size_t S = (size_t)L * L * L;
        const uint32_t site = a.rec[ELP_REC_WORDS * p], cnt = a.rec[ELP_REC_WORDS * p + 1],
                       off = a.rec[ELP_REC_WORDS * p + 2];
        int bad = (site >= S || off >= cnt || cnt == 0 || (a.linear && off != 0)) ? 1 : 0;
        if (!bad) {
            const uint32_t w = a.lat[site];
            if (!(w & ELP_LBIT) || (w >> 5) != (uint32_t)p) bad = 1;
        }
        long long st = 0, su = 0, sv = 0;
        unsigned long long sq = 0, runs = 0;
        int dt = 0, du = 0, dv = 0;    // position of the current run relative to monomer 0's site
        long mono = 0;
        uint32_t here = cnt - off, cur = site, len = cnt;
        // the current run's site in box coordinates, stepped without a division
        int t = (int)(site % (uint32_t)L), u = (int)((site / (uint32_t)L) % (uint32_t)L),
            v = (int)(site / ((uint32_t)L * L));
        while (!bad) {
            const uint32_t bo = a.lat[cur] & 15;
            const bool end = a.linear && bo == 15;   // last run of a linear chain
            if (!(elp_valid_bond(bo) || end) || mono + (long)here > (long)N) { bad = 1; break; }
            const long long x = dt + du - dv, y = dt - du, z = dv;
            st += (long long)here * dt;
            su += (long long)here * du;
            sv += (long long)here * dv;
            sq += (unsigned long long)here * (unsigned long long)(x * x + y * y + z * z);
            mono += here;
            runs++;
            atomicAdd(&hist[(len < (uint32_t)a.nbins ? len : (uint32_t)a.nbins) - 1], 1ull);
            if (end) break;
            // next run
            t += elp_bt(bo); u += elp_bu(bo); v += elp_bv(bo);
            dt += elp_bt(bo); du += elp_bu(bo); dv += elp_bv(bo);
            t += t < 0 ? L : 0; t -= t >= L ? L : 0;
            u += u < 0 ? L : 0; u -= u >= L ? L : 0;
            v += v < 0 ? L : 0; v -= v >= L ? L : 0;
            cur = (uint32_t)t + (uint32_t)L * ((uint32_t)u + (uint32_t)L * (uint32_t)v);
            const uint32_t wn = a.lat[cur];
            if (!wn) { bad = 1; break; }
            if (cur == site) break;
            if (wn & ELP_LBIT) { bad = 1; break; }
            here = len = wn >> ELP_CSHIFT;
            if (here == 0 || runs >= (unsigned long long)N) { bad = 1; break; }
        }
        if (!bad) {
            // monomers N-off .. N-1: the rest of monomer 0's run, reached again after the whole ring
            const long long x = dt + du - dv, y = dt - du, z = dv;
            st += (long long)off * dt;
            su += (long long)off * du;
            sv += (long long)off * dv;
            sq += (unsigned long long)off * (unsigned long long)(x * x + y * y + z * z);
            mono += off;
            if (mono != N) bad = 1;
        }
        unsigned long long* o = a.out + 6 * (size_t)p;
        o[0] = (unsigned long long)st;
        o[1] = (unsigned long long)su;
        o[2] = (unsigned long long)sv;
        o[3] = sq;
        o[4] = runs | ((unsigned long long)(bad ? 4 : 0) << 32);
        o[5] = site;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.nbins; i += blockDim.x)
        if (hist[i]) atomicAdd(&a.hist[i], hist[i]);
}

// The same sums from a chain's bonds (elp_rank.cu), one warp per chain: 128
// bonds at a time, four a lane, the lanes' displacements summed by a warp
// scan packed into one word.  The walk above follows a ring run by run (830
// dependent loads, 1.05 ms at L = 128, N = 1000); this reads the bonds once.
__global__ void observe_chains(ObsArgs a, const uint8_t* bonds, const int32_t* status)
{
    __shared__ unsigned int hist[ELP_OBS_MAX_BINS];
    for (int i = threadIdx.x; i < a.nbins; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    if (p < a.P) {
        const int N = a.N;
        const uint8_t* b = bonds + (size_t)p * N;
        const bool bad = status[p] != 0;
        long long st = 0, su = 0, sv = 0;
        unsigned long long sq = 0;
        uint32_t runs = 0;
        int ct = 0, cu = 0, cv = 0;    // position of the block's first monomer relative to monomer 0's site
        int prev = -1, first = -1;     // last run's end so far, the first run's end
        for (int m0 = 0; m0 < N && !bad; m0 += 128) {
            const int m = m0 + 4 * lane;
            uint32_t w = 0;
            for (int k = 0; k < 4; k++)
                if (m + k < N) w |= (uint32_t)b[m + k] << (8 * k);
            // displacement of the lane's four bonds, 10 bits a coordinate
            int dt = 0, du = 0, dv = 0;
            for (int k = 0; k < 4; k++) {
                const uint32_t bo = (w >> (8 * k)) & 15;
                dt += elp_bt(bo); du += elp_bu(bo); dv += elp_bv(bo);
            }
            int sum = dt + du * 1024 + dv * 1048576;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            const int all = __shfl_sync(0xffffffffu, sum, 31);
            int ex = sum - (dt + du * 1024 + dv * 1048576);
            // each coordinate of a block's sum is within +-128: unpack from the low end
            int t = (ex << 22) >> 22; ex = (ex - t) >> 10;
            int u = (ex << 22) >> 22;
            int v = (ex - u) >> 10;
            t += ct; u += cu; v += cv;
            // end of the last run ahead of this lane
            const uint32_t any = __ballot_sync(0xffffffffu, w != 0);
            const int mylast = w ? m + 3 - (__clz(w) >> 3) : -1;
            const uint32_t below = any & ((1u << lane) - 1u);
            int last = __shfl_sync(0xffffffffu, mylast, below ? 31 - __clz(below) : 0);
            if (!below) last = prev;
            for (int k = 0; k < 4; k++) {
                if (m + k < N) {
                    const long long x = t + u - v, y = t - u, z = v;
                    st += t; su += u; sv += v;
                    sq += (unsigned long long)(x * x + y * y + z * z);
                }
                const uint32_t bo = (w >> (8 * k)) & 15;
                if (bo) {
                    runs++;
                    if (last >= 0) atomicAdd(&hist[min(m + k - last, a.nbins) - 1], 1u);
                    last = m + k;
                    t += elp_bt(bo); u += elp_bu(bo); v += elp_bv(bo);
                }
            }
            if (first < 0 && any) {
                const int l = __ffs(any) - 1;
                const uint32_t wl = __shfl_sync(0xffffffffu, w, l);
                first = m0 + 4 * l + ((__ffs(wl) - 1) >> 3);
            }
            if (any) prev = __shfl_sync(0xffffffffu, mylast, 31 - __clz(any));
            int rest = all;
            int at = (rest << 22) >> 22; rest = (rest - at) >> 10;
            int au = (rest << 22) >> 22;
            ct += at; cu += au; cv += (rest - au) >> 10;
        }
        for (int o = 16; o > 0; o >>= 1) {
            st += __shfl_xor_sync(0xffffffffu, st, o);
            su += __shfl_xor_sync(0xffffffffu, su, o);
            sv += __shfl_xor_sync(0xffffffffu, sv, o);
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        runs = __reduce_add_sync(0xffffffffu, runs);
        if (lane == 0) {
            // monomer 0's run: to the first bond, and (rings) from the last one on
            if (!bad && first >= 0) atomicAdd(&hist[min(first + 1 + N - 1 - prev, a.nbins) - 1], 1u);
            unsigned long long* o = a.out + 6 * (size_t)p;
            o[0] = (unsigned long long)st;
            o[1] = (unsigned long long)su;
            o[2] = (unsigned long long)sv;
            o[3] = sq;
            o[4] = runs | ((unsigned long long)(bad ? 4 : 0) << 32);
            o[5] = a.rec[ELP_REC_WORDS * (size_t)p];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.nbins; i += blockDim.x)
        if (hist[i]) atomicAdd(&a.hist[i], (unsigned long long)hist[i]);
}

}  // namespace elp

elp_status elp_observe_melt(const uint32_t* lat, const uint32_t* rec, int L, int N, int P, int linear,
                            const uint32_t* flags, elp_walk_bufs* b, double* cms_tuv, double* rg2, double* sl,
                            uint64_t* run_hist, int nbins, cudaStream_t s)
{
    if (nbins < 0 || nbins > ELP_OBS_MAX_BINS)
        return elp_fail(ELP_ERR_ARG, "nbins must be in [0, %d]", ELP_OBS_MAX_BINS);
    if (run_hist && nbins < 1) return elp_fail(ELP_ERR_ARG, "run_hist needs nbins >= 1");
    const size_t words = (size_t)P * 6 + ELP_OBS_MAX_BINS;
    ELP_CUDA_TRY(elp_scratch_grow(b, (void**)&b->d_obs, &b->cap_obs, words * sizeof(unsigned long long)));
    elp::ObsArgs a;
    a.lat = lat; a.rec = rec; a.L = L; a.N = N; a.P = P; a.linear = linear;
    a.nbins = nbins > 0 ? nbins : 1;
    a.out = b->d_obs;
    a.hist = b->d_obs + (size_t)P * 6;
    ELP_CUDA_TRY(cudaMemsetAsync(a.hist, 0, ELP_OBS_MAX_BINS * sizeof(unsigned long long), s));
    std::vector<unsigned long long> o;
    // the chains by list ranking, then one pass over their bonds
    elp_status st = elp_walk_bufs_reserve(b, P, N, 0);
    if (st && st != ELP_ERR_NOMEM) return st;
    const cudaError_t re = st ? cudaErrorMemoryAllocation : elp_rank_chains(lat, rec, L, N, P, linear, true, flags, b, s);
    bool walk = elp_must_walk(re);
    if (!walk) {
        ELP_CUDA_TRY(re);
        elp::observe_chains<<<(unsigned)(((size_t)P * 32 + 127) / 128), 128, 0, s>>>(a, b->d_bonds(), b->d_status);
        ELP_CUDA_TRY(cudaGetLastError());
        o.resize(words);   // while the device works
        elp_chain_head h;
        ELP_CUDA_TRY(cudaMemcpyAsync(&h, b->d_out, sizeof(h), cudaMemcpyDeviceToHost, s));
        ELP_CUDA_TRY(cudaMemcpyAsync(o.data(), a.out, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        ELP_CUDA_TRY(cudaStreamSynchronize(s));
        if ((st = elp_flags_status(h.flags))) return st;
        // runs that lead into a chain from outside have written their bonds
        // into it too: nothing that was summed from them counts
        walk = !elp_chains_good(h, N, P);
    }
    // boxes above the ranking's size, no room for its scratch (the walk needs
    // none), melts it finds amiss: a walk along each ring from its label, which
    // sees the ring's own runs only
    if (walk) {
        o.resize(words);
        ELP_CUDA_TRY(cudaMemsetAsync(a.hist, 0, ELP_OBS_MAX_BINS * sizeof(unsigned long long), s));
        elp::observe_kernel<<<(P + 127) / 128, 128, 0, s>>>(a);
        ELP_CUDA_TRY(cudaGetLastError());
        ELP_CUDA_TRY(cudaMemcpyAsync(o.data(), a.out, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        ELP_CUDA_TRY(cudaStreamSynchronize(s));
        if (flags && (st = elp_device_errors(flags, s))) return st;
    }
    for (int p = 0; p < P; p++)
        if (o[6 * (size_t)p + 4] >> 32)
            return elp_fail(ELP_ERR_INTEGRITY, "ring %d cannot be walked", p);
    const double n = (double)N;
    for (int p = 0; p < P; p++) {
        const unsigned long long* r = &o[6 * (size_t)p];
        const long long st = (long long)r[0], su = (long long)r[1], sv = (long long)r[2];
        const uint32_t site = (uint32_t)r[5];
        if (cms_tuv) {
            cms_tuv[3 * (size_t)p + 0] = (double)(site % (uint32_t)L) + (double)st / n;
            cms_tuv[3 * (size_t)p + 1] = (double)((site / (uint32_t)L) % (uint32_t)L) + (double)su / n;
            cms_tuv[3 * (size_t)p + 2] = (double)(site / ((uint32_t)L * L)) + (double)sv / n;
        }
        if (rg2) {
            // Rg^2 = (N Sq - |S_xyz|^2) / (2 N^2), the numerator exact in 128 bits
            const __int128 sx = (__int128)st + su - sv, sy = (__int128)st - su, sz = sv;
            const __int128 num = (__int128)N * (__int128)r[3] - (sx * sx + sy * sy + sz * sz);
            rg2[p] = (double)num / (2.0 * n * n);
        }
        // zero bonds over the chain's bonds (a linear chain's end marker is none)
        if (sl) sl[p] = (double)((unsigned long long)N - (r[4] & 0xffffffffull)) / (linear ? n - 1.0 : n);
    }
    if (run_hist)
        for (int i = 0; i < nbins; i++) run_hist[i] = o[(size_t)P * 6 + (size_t)i];
    return ELP_OK;
}
