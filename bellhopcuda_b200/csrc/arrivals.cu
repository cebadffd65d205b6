// Arrivals and eigenray hits for the 2-D field modes (RunType 'A' / 'a' / 'E').
//
// The reference adds arrivals one contribution at a time (AddArr,
// src/arrivals.hpp:45-132): a contribution either merges into the receiver's
// last arrival (when its delay and phase are within 0.05 rad of it) or is
// appended / replaces the weakest one. The result depends on the order in
// which contributions reach a receiver, and the reference's single-threaded
// order (ray by ray in job order, step by step) is the one with merging
// enabled (src/mode/arr.hpp:78). Eigen hits (RecordEigenHit,
// src/eigenrays.hpp:24-40) are likewise listed in that order.
//
// On the GPU, with all rays traced concurrently, the order is rebuilt:
//   1. arr_gather_kernel (count pass): counts the contributions;
//   2. arr_gather_kernel (fill pass): writes one candidate per contribution
//      with a 64-bit key (receiver cell, ray, step) for arrivals or (field,
//      ray, step, column walk position, depth) for eigen hits;
//   3. a stable LSD radix sort of the keys (8-bit digits; per-tile histograms,
//      an exclusive scan per digit, warp-stable scatter);
//   4. arr_replay_kernel: one warp per receiver cell applies the AddArr rule
//      to its candidates in sorted order, then PostProcessArrivals' amplitude
//      scaling (src/mode/arr.cpp:24-74); eigen_emit_kernel writes the hits in
//      sorted order.
// The contribution math (InfluenceGeoCore, src/influence.hpp:897-1024) is FP64
// with the reference's operation order in both precisions of the tracer.
#include <cuda_runtime.h>

#include <utility>

#include "bhcb_internal.h"
#include "device_math.cuh"
#include "trace2d.cuh"
#include "influence2d.cuh"
#include "trace3d.cuh"

namespace bhcb {

namespace {

constexpr double RAD_DEG = 180.0 / BHCB_PI;
constexpr int SORT_TILE = 1024;   // keys per scatter tile (one warp)

__device__ __forceinline__ int group_of_cell(const GroupDev *groups, int ngroups, long long cell)
{
    int lo = 0, hi = ngroups - 1;
    while(lo < hi) {
        int m = (lo + hi + 1) >> 1;
        if(groups[m].field_base <= cell) lo = m; else hi = m - 1;
    }
    return lo;
}

// Walks every contribution of every segment; one thread per segment.
// COUNT: only counts (ctr->nevals). Otherwise writes candidate i with key /
// value (i) at i = atomicAdd(cursor).
template<typename R, bool GAUSS, bool COUNT>
__global__ void __launch_bounds__(128) arr_gather_kernel(
    const SegRec<R> *__restrict__ segs, unsigned long long cap, const GroupDev *__restrict__ groups,
    int ngroups, const double *__restrict__ freqs, ArrCand *cands, uint64_t *keys, uint32_t *vals,
    unsigned long long cand_cap, unsigned long long *cursor, RunCounters *ctr, ArrKeyBits kb)
{
    const unsigned long long nseg = min(__ldcg(&ctr->nseg), cap);
    unsigned long long count = 0;
    for(unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < nseg;
        k += (unsigned long long)gridDim.x * blockDim.x) {
        const SegRec<R> S = segs[k];
        if(S.job < 0) continue;
        const int gi = find_group(groups, ngroups, S.job);
        const GroupDev &G = groups[gi];
        const EnvDev &e = *G.env;
        const int local = (int)((long long)S.job - G.job_base);
        const int nal = e.isingle > 0 ? 1 : e.nalpha;
        const int isz = local / nal;
        const double freq = freqs[G.freq_base];
        // AdjustSigma (src/influence.hpp:91-100) and the depth window
        // (src/influence.hpp:1285-1292), as in the TL kernels
        R sig = S.sigma_seg, sigfloor = (R)0;
        if(GAUSS) {
            R lam = S.c0 / (R)freq;
            R fl = min((R)FLTD(0.2) * (R)freq * S.tau1r, (R)BHCB_PI * lam);
            sigfloor = fl;
            sig = max(sig, fl);
        }
        const double rmax = (GAUSS ? 4.0 : 1.0) * (double)sig;
        double zmin = -1.7976931348623157e308, zmax = 1.7976931348623157e308;
        if(fabs((double)S.tx) > FLTD(0.50001)) {
            zmin = (double)S.zlo - rmax;
            zmax = (double)S.zhi + rmax;
        }
        const bool irregular = e.irregular != 0;
        const int nrzp = e.nrz_per_range;
        int izlo = 0, izhi = 1;
        if(!irregular) {
            izlo = lower_f(e.rz, e.nrz, zmin);
            izhi = upper_f(e.rz, e.nrz, zmax);
        }
        const double tx = (double)S.tx, tz = (double)S.tz, rlen = (double)S.rlen;
        const double q0 = (double)S.q0, dq = (double)S.dq, rcpq = (double)S.rcp_q0;
        for(int ir = S.ir_lo; ir <= S.ir_hi; ++ir) {
            const double dr = e.rr[ir] - S.x0r;
            for(int iz = izlo; iz < izhi; ++iz) {
                const float zrf = irregular ? e.rz[ir] : e.rz[iz];
                if(irregular && ((double)zrf < zmin || (double)zrf > zmax)) continue;
                // InfluenceGeoCore (src/influence.hpp:897-1024), 2-D
                const double dz = (double)zrf - S.x0z;
                const double s = (dr * tx + dz * tz) / rlen;
                const double n1 = fabs(dz * tx - dr * tz);
                const double qF = q0 + s * dq;
                double sigma = fabs(qF * rcpq);
                const double sig0 = sigma;
                if(GAUSS) sigma = max(sigma, (double)sigfloor);
                if(n1 >= (GAUSS ? 4.0 : 1.0) * sigma) continue;
                if(COUNT) {
                    ++count;
                    continue;
                }
                const unsigned long long i = atomicAdd(cursor, 1ull);
                if(i >= cand_cap) continue;
                const int ialpha = e.isingle > 0 ? e.isingle - 1 : local % nal;
                uint64_t key;
                ArrCand c;
                if(kb.eigen) {
                    const int walk = S.tx > (R)0 ? ir : e.nrr - 1 - ir;
                    const int fidx = G.field_index;
                    key = ((uint64_t)fidx << kb.sh_cell) | ((uint64_t)local << kb.sh_job)
                          | ((uint64_t)S.is << kb.sh_is) | ((uint64_t)walk << kb.sh_walk) | (uint64_t)iz;
                    c.amp = 0.0;
                    c.phase = 0.0;
                    c.delay_re = 0.0;
                    c.delay_im = 0.0;
                    c.rcvr_decl = 0.f;
                    c.ntop = S.is;      // eigen: step index
                    c.nbot = ir;        // eigen: receiver range index
                    c.job = iz | (isz << 20);
                    c.aux = ialpha;
                } else {
                    const double cnst = (double)S.cnst_num / sqrt(fabs(qF));
                    double w;
                    if(GAUSS) w = exp(FLTD(-0.5) * (n1 / sigma) * (n1 / sigma)) * (sig0 / sigma);
                    else w = (sigma - n1) / sigma;
                    const bool caustic = (qF <= 0.0 && q0 > 0.0) || (qF >= 0.0 && q0 < 0.0);
                    const long long cell = G.field_base + ((long long)isz * nrzp + iz) * e.nrr + ir;
                    key = ((uint64_t)cell << kb.sh_cell) | ((uint64_t)local << kb.sh_job) | (uint64_t)S.is;
                    c.amp = cnst * w;
                    c.phase = (double)(caustic ? S.phase_b : S.phase_a);
                    c.delay_re = S.tau0r + s * (double)S.dtaur;
                    c.delay_im = (double)S.tau0i + s * (double)S.dtaui;
                    c.rcvr_decl = (float)S.rcvr_decl;
                    c.ntop = S.ntop;
                    c.nbot = S.nbot;
                    c.job = S.job;
                    c.aux = ialpha;
                }
                cands[i] = c;
                keys[i] = key;
                vals[i] = (uint32_t)i;
            }
        }
    }
    if(COUNT && count) atomicAdd(&ctr->nevals, count);
}

// ---------------------------------------------------------------- radix sort
// per-tile digit histogram, digit-major: hist[d * ntiles + tile]
__global__ void rs_hist_kernel(const uint64_t *__restrict__ keys, unsigned long long n, int shift,
                               uint32_t *hist, int ntiles)
{
    __shared__ uint32_t h[256];
    for(int d = threadIdx.x; d < 256; d += blockDim.x) h[d] = 0;
    __syncthreads();
    const int tile = blockIdx.x;
    const unsigned long long b = (unsigned long long)tile * SORT_TILE;
    const unsigned long long e = min(n, b + SORT_TILE);
    for(unsigned long long i = b + threadIdx.x; i < e; i += blockDim.x)
        atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    __syncthreads();
    for(int d = threadIdx.x; d < 256; d += blockDim.x) hist[(size_t)d * ntiles + tile] = h[d];
}

// One block per digit: exclusive scan of its ntiles counts; its total goes to
// hist[256 ntiles + digit], and the scatter adds the digits before it. One block
// of 1024 threads over all digits took 650 us for 6.4 M keys (1553 tiles of 4096),
// this 8 us for 6.0 M (5827 tiles of 1024).
__global__ void __launch_bounds__(256) rs_scan_kernel(uint32_t *hist, int ntiles)
{
    __shared__ uint32_t part[8];
    uint32_t *a = hist + (size_t)blockIdx.x * ntiles;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t carry = 0;
    for(int base = 0; base < ntiles; base += 1024) {
        const int i = base + 4 * (int)threadIdx.x;
        uint32_t v[4], sum = 0;
        for(int j = 0; j < 4; ++j) {
            v[j] = i + j < ntiles ? a[i + j] : 0u;
            sum += v[j];
        }
        uint32_t x = sum;
        for(int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += t;
        }
        if(lane == 31) part[w] = x;
        __syncthreads();
        uint32_t before = carry, all = 0;
        for(int j = 0; j < 8; ++j) {
            if(j < w) before += part[j];
            all += part[j];
        }
        before += x - sum;
        for(int j = 0; j < 4; ++j) {
            if(i + j < ntiles) a[i + j] = before;
            before += v[j];
        }
        carry += all;
        __syncthreads();
    }
    if(threadIdx.x == 0) hist[(size_t)256 * ntiles + blockIdx.x] = carry;
}

// stable scatter: one warp per tile, 32 keys at a time in order; lanes with the
// same digit are ranked by lane order (match_any), digit offsets in shared memory
__global__ void __launch_bounds__(32) rs_scatter_kernel(
    const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
    uint32_t *__restrict__ vout, unsigned long long n, int shift, const uint32_t *__restrict__ hist,
    int ntiles)
{
    __shared__ uint32_t off[256];
    const int tile = blockIdx.x, lane = threadIdx.x;
    {   // lane: digits 8 lane ... + 7
        const uint32_t *total = hist + (size_t)256 * ntiles + 8 * lane;
        uint32_t sum = 0, x;
        for(int j = 0; j < 8; ++j) sum += total[j];
        x = sum;
        for(int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += t;
        }
        x -= sum;
        for(int j = 0; j < 8; ++j) {
            off[8 * lane + j] = x + hist[(size_t)(8 * lane + j) * ntiles + tile];
            x += total[j];
        }
    }
    __syncwarp();
    const unsigned long long b = (unsigned long long)tile * SORT_TILE;
    const unsigned long long e = min(n, b + SORT_TILE);
    for(unsigned long long i0 = b; i0 < e; i0 += 32) {
        const unsigned long long i = i0 + lane;
        const bool have = i < e;
        uint64_t k = 0;
        uint32_t v = 0;
        uint32_t d = 256u + lane;   // distinct dummy digit for idle lanes
        if(have) {
            k = kin[i];
            v = vin[i];
            d = (uint32_t)((k >> shift) & 255u);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if(have) base = off[d];
        __syncwarp();
        if(have) {
            kout[base + rank] = k;
            vout[base + rank] = v;
            if(lane == leader) off[d] = base + __popc(peers);
        }
        __syncwarp();
    }
}

// -------------------------------------------------------------- replay
// AddArr (src/arrivals.hpp:45-132) over one receiver cell's candidates in
// (ray, step) order, then PostProcessArrivals (src/mode/arr.cpp:24-74).
// D3: 3-D run (source angles from the 3-D job, receiver azimuth from the
// candidate, no amplitude scaling); the replay continues from the counts
// already in narr_out, so job-ordered waves compose.
// One warp per cell: 32 candidates are loaded at once, and applied in order from
// there by all lanes together, the owner of each writing. The last arrival, which
// the next may merge with, stays in registers; the weakest of a full cell is
// found by all lanes and kept until an arrival changes. One thread per cell
// waited for memory at every candidate and at each of the max_narr amplitudes:
// 614k candidates of 4141 cells 1946 us, so 319; 6.36 M of 45000 (3-D) 2702 and 1138.
template<bool D3>
__global__ void __launch_bounds__(128) arr_replay_kernel(
    const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, const ArrCand *__restrict__ cands,
    unsigned long long n, const GroupDev *__restrict__ groups, int ngroups, const double *__restrict__ freqs,
    long long ncells, int sh_cell, int max_narr, int allow_merging, int32_t *narr_out, ArrivalRec *arr_out)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = (int)(threadIdx.x & 31);
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    for(long long cell = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); cell < ncells;
        cell += nwarps) {
        // candidate range of this cell in the sorted keys: even lanes its begin, odd its end
        const uint64_t want = (uint64_t)(cell + (lane & 1)) << sh_cell;
        unsigned long long lo = 0, hi = n;
        while(lo < hi) {
            unsigned long long m = (lo + hi) >> 1;
            if(keys[m] < want) lo = m + 1; else hi = m;
        }
        const unsigned long long begin = __shfl_sync(ALL, lo, 0), end = __shfl_sync(ALL, lo, 1);
        const GroupDev &G = groups[group_of_cell(groups, ngroups, cell)];
        const double omega = D3 ? 2.0 * BHCB_PI * G.env3->freq0 : 2.0 * BHCB_PI * freqs[G.freq_base];
        ArrivalRec *ba = arr_out + (size_t)cell * max_narr;
        int nt = D3 ? narr_out[cell] : 0;
        // of the last arrival
        float l_re = 0.f, l_im = 0.f, l_ph = 0.f;
        if(nt >= 1) {
            const ArrivalRec &L = ba[min(nt, max_narr) - 1];
            l_re = L.delay_re;
            l_im = L.delay_im;
            l_ph = L.Phase;
        }
        int weak_j = -1;         // weakest arrival of a full cell; -1: to be found
        float weak = 0.f;
        for(unsigned long long k0 = begin; k0 < end; k0 += 32) {
            const int cnt = (int)min((unsigned long long)32, end - k0);
            ArrCand c{};
            ArrivalRec A;
            if(lane < cnt) {
                c = cands[vals[k0 + lane]];
                double src_decl;
                if(D3) {
                    const Job3 J = job_indices3(*G.env3, (int)((long long)c.job - G.job_base));
                    src_decl = RAD_DEG * G.env3->alpha[J.ialpha];
                    A.SrcAzimAngle = (float)(RAD_DEG * G.env3->beta[J.ibeta]);
                    A.RcvrAzimAngle = c.rcvr_azim;
                } else {
                    src_decl = RAD_DEG * G.env->alpha[c.aux];
                    A.SrcAzimAngle = A.RcvrAzimAngle = __int_as_float(0x7fc00000);   // NaN: no azimuth in 2-D
                }
                A.a = (float)c.amp;
                A.Phase = (float)c.phase;
                A.delay_re = (float)c.delay_re;
                A.delay_im = (float)c.delay_im;
                A.SrcDeclAngle = (float)src_decl;
                A.RcvrDeclAngle = c.rcvr_decl;
                A.NTopBnc = c.ntop;
                A.NBotBnc = c.nbot;
            }
            if(!allow_merging) {
                if(lane < cnt && nt + lane < max_narr) ba[nt + lane] = A;
                nt = min(nt + cnt, max_narr);
                continue;
            }
            for(int i = 0; i < cnt; ++i) {
                const double phase = __shfl_sync(ALL, c.phase, i), dre = __shfl_sync(ALL, c.delay_re, i);
                const double dim = __shfl_sync(ALL, c.delay_im, i);
                bool second = false;
                const float PhaseTol = 0.05f;
                if(nt >= 1 && fabs((double)l_ph - phase) < (double)PhaseTol) {
                    const double ddr = dre - (double)l_re, ddi = dim - (double)l_im;
                    // hypot is at least the larger part, within its rounding
                    second = omega * fabs(ddr) < 1.0 && omega * hypot(ddr, ddi) < (double)PhaseTol;
                }
                if(!second) {
                    int slot = nt;
                    if(nt >= max_narr) {
                        if(weak_j < 0) {
                            __syncwarp();
                            weak = __int_as_float(0x7f800000);
                            weak_j = 0x7fffffff;
                            for(int j = lane; j < max_narr; j += 32)
                                if(ba[j].a < weak) {
                                    weak = ba[j].a;
                                    weak_j = j;
                                }
                            for(int o = 16; o > 0; o >>= 1) {
                                const float v = __shfl_xor_sync(ALL, weak, o);
                                const int j = __shfl_xor_sync(ALL, weak_j, o);
                                if(v < weak || (v == weak && j < weak_j)) {
                                    weak = v;
                                    weak_j = j;
                                }
                            }
                        }
                        if(!((double)weak < __shfl_sync(ALL, c.amp, i))) continue;
                        slot = weak_j;
                        weak_j = -1;
                    } else {
                        ++nt;
                    }
                    if(lane == i) ba[slot] = A;
                    if(slot == nt - 1) {
                        l_re = (float)dre;
                        l_im = (float)dim;
                        l_ph = (float)phase;
                    }
                } else {
                    __syncwarp();
                    if(lane == i) {
                        ArrivalRec &L = ba[nt - 1];
                        const float tot = __fadd_rn(L.a, A.a);
                        const float w1 = __fdiv_rn(L.a, tot), w2 = __fdiv_rn(A.a, tot);
                        l_re = __fadd_rn(__fmul_rn(w1, L.delay_re), __fmul_rn(w2, A.delay_re));
                        l_im = __fadd_rn(__fmul_rn(w1, L.delay_im), __fmul_rn(w2, A.delay_im));
                        L.delay_re = l_re;
                        L.delay_im = l_im;
                        L.a = tot;
                        L.SrcDeclAngle = __fadd_rn(__fmul_rn(w1, L.SrcDeclAngle), __fmul_rn(w2, A.SrcDeclAngle));
                        L.SrcAzimAngle = __fadd_rn(__fmul_rn(w1, L.SrcAzimAngle), __fmul_rn(w2, A.SrcAzimAngle));
                        L.RcvrDeclAngle = __fadd_rn(__fmul_rn(w1, L.RcvrDeclAngle), __fmul_rn(w2, A.RcvrDeclAngle));
                        L.RcvrAzimAngle = __fadd_rn(__fmul_rn(w1, L.RcvrAzimAngle), __fmul_rn(w2, A.RcvrAzimAngle));
                    }
                    l_re = __shfl_sync(ALL, l_re, i);
                    l_im = __shfl_sync(ALL, l_im, i);
                    weak_j = -1;
                }
            }
        }
        __syncwarp();
        // PostProcessArrivals (src/mode/arr.cpp:24-74): clamp the count; 2-D
        // and Nx2D scale the amplitudes (3-D factor 1)
        if(nt > max_narr) nt = max_narr;
        if(lane == 0) narr_out[cell] = nt;
        if(D3 && !G.env3->nx2d) continue;
        // 2-D rays (2-D and Nx2D): cylindrical spreading per receiver range,
        // the last index of both field layouts
        const double *rr = D3 ? G.env3->rr : G.env->rr;
        const int nrr = D3 ? G.env3->nrr : G.env->nrr;
        const int ir = (int)((cell - G.field_base) % nrr);
        float factor;
        if(!D3 && G.env->line_source) factor = (float)(FLTD(4.0) * sqrt(BHCB_PI));
        else if(fabs(rr[ir]) < DBL_EPS) factor = 1e5f;
        else factor = (float)(FLTD(1.0) / sqrt(rr[ir]));
        for(int j = lane; j < nt; j += 32) ba[j].a = __fmul_rn(ba[j].a, factor);
    }
}

// eigen hits in sorted order (RecordEigenHit layout, include/bhc/structs.hpp:353-361)
__global__ void eigen_emit_kernel(const uint32_t *__restrict__ vals, const ArrCand *__restrict__ cands,
                                  unsigned long long n, EigenHitRec *hits, int32_t *field_of_hit, int sh_cell,
                                  const uint64_t *__restrict__ keys)
{
    for(unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
        k += (unsigned long long)gridDim.x * blockDim.x) {
        const ArrCand &c = cands[vals[k]];
        EigenHitRec h;
        h.is = c.ntop;
        h.itheta = 0;
        h.ir = c.nbot;
        h.iz = c.job & 0xfffff;
        h.isx = 0;
        h.isy = 0;
        h.isz = c.job >> 20;
        h.ialpha = c.aux;
        h.ibeta = 0;
        hits[k] = h;
        field_of_hit[k] = (int32_t)(keys[k] >> sh_cell);
    }
}

} // namespace

template<typename R> cudaError_t launch_arr_gather(const void *segs, unsigned long long cap,
                                                   const GroupDev *groups, int ngroups, const double *freqs,
                                                   bool gauss, bool count, ArrCand *cands, uint64_t *keys,
                                                   uint32_t *vals, unsigned long long cand_cap,
                                                   unsigned long long *cursor, RunCounters *ctr, ArrKeyBits kb,
                                                   int grid, cudaStream_t st)
{
    const SegRec<R> *s = (const SegRec<R> *)segs;
    if(gauss && count)
        arr_gather_kernel<R, true, true><<<grid, 128, 0, st>>>(s, cap, groups, ngroups, freqs, cands, keys, vals,
                                                               cand_cap, cursor, ctr, kb);
    else if(gauss)
        arr_gather_kernel<R, true, false><<<grid, 128, 0, st>>>(s, cap, groups, ngroups, freqs, cands, keys, vals,
                                                                cand_cap, cursor, ctr, kb);
    else if(count)
        arr_gather_kernel<R, false, true><<<grid, 128, 0, st>>>(s, cap, groups, ngroups, freqs, cands, keys, vals,
                                                                cand_cap, cursor, ctr, kb);
    else
        arr_gather_kernel<R, false, false><<<grid, 128, 0, st>>>(s, cap, groups, ngroups, freqs, cands, keys,
                                                                 vals, cand_cap, cursor, ctr, kb);
    return cudaGetLastError();
}
template cudaError_t launch_arr_gather<float>(const void *, unsigned long long, const GroupDev *, int,
                                              const double *, bool, bool, ArrCand *, uint64_t *, uint32_t *,
                                              unsigned long long, unsigned long long *, RunCounters *, ArrKeyBits,
                                              int, cudaStream_t);
template cudaError_t launch_arr_gather<double>(const void *, unsigned long long, const GroupDev *, int,
                                               const double *, bool, bool, ArrCand *, uint64_t *, uint32_t *,
                                               unsigned long long, unsigned long long *, RunCounters *, ArrKeyBits,
                                               int, cudaStream_t);

size_t radix_sort_hist_entries(unsigned long long n)
{
    return (size_t)256 * (size_t)((n + SORT_TILE - 1) / SORT_TILE) + 256;
}

// Sorts (keys, vals) by the low `bits` bits of the keys; the result is in
// (k0, v0) when the number of passes is even, else in (k1, v1): returns which.
cudaError_t radix_sort_pairs(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, unsigned long long n,
                             int bits, uint32_t *hist, int *result_in_1, cudaStream_t st)
{
    *result_in_1 = 0;
    if(n == 0) return cudaSuccess;
    const int ntiles = (int)((n + SORT_TILE - 1) / SORT_TILE);
    uint64_t *ki = k0, *ko = k1;
    uint32_t *vi = v0, *vo = v1;
    int passes = 0;
    for(int shift = 0; shift < bits; shift += 8, ++passes) {
        rs_hist_kernel<<<ntiles, 256, 0, st>>>(ki, n, shift, hist, ntiles);
        rs_scan_kernel<<<256, 256, 0, st>>>(hist, ntiles);
        rs_scatter_kernel<<<ntiles, 32, 0, st>>>(ki, vi, ko, vo, n, shift, hist, ntiles);
        std::swap(ki, ko);
        std::swap(vi, vo);
    }
    *result_in_1 = passes & 1;
    return cudaGetLastError();
}

cudaError_t launch_arr_replay(const uint64_t *keys, const uint32_t *vals, const ArrCand *cands, unsigned long long n,
                              const GroupDev *groups, int ngroups, const double *freqs, long long ncells, int sh_cell,
                              int max_narr, int allow_merging, int32_t *narr, ArrivalRec *arr, int sm_count,
                              cudaStream_t st, bool d3)
{
    long long grid = (ncells + 3) / 4;
    if(grid > (long long)sm_count * 64) grid = (long long)sm_count * 64;
    if(grid < 1) grid = 1;
    if(d3)
        arr_replay_kernel<true><<<(int)grid, 128, 0, st>>>(keys, vals, cands, n, groups, ngroups, freqs, ncells,
                                                           sh_cell, max_narr, allow_merging, narr, arr);
    else
        arr_replay_kernel<false><<<(int)grid, 128, 0, st>>>(keys, vals, cands, n, groups, ngroups, freqs, ncells,
                                                            sh_cell, max_narr, allow_merging, narr, arr);
    return cudaGetLastError();
}

cudaError_t launch_eigen_emit(const uint32_t *vals, const ArrCand *cands, unsigned long long n, EigenHitRec *hits,
                              int32_t *field_of_hit, int sh_cell, const uint64_t *keys, int sm_count, cudaStream_t st)
{
    long long grid = (long long)((n + 255) / 256);
    if(grid > (long long)sm_count * 32) grid = (long long)sm_count * 32;
    if(grid < 1) grid = 1;
    eigen_emit_kernel<<<(int)grid, 256, 0, st>>>(vals, cands, n, hits, field_of_hit, sh_cell, keys);
    return cudaGetLastError();
}

} // namespace bhcb
