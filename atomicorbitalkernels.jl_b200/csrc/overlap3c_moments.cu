// overlap3c_moments.cu -- 3-center overlap of bases with f shells, host side: the set-up
// kernel, the panels and the moment buffer.  The kernels are in overlap3c_moments.cuh.
#include <algorithm>
#include <array>
#include <cstring>
#include <map>
#include <vector>

#include "overlap3c_moments.cuh"
#include "overlap3c_prep.cuh"

namespace aok {
namespace m3 {

// Moments or explicit E tables (k_overlap3c).  The recursions on moments cost the same for
// any number of primitive triples, the tables are rebuilt for each: moments are taken when a
// function of a block sums at least two triples on average.  Measured (whole calls, us,
// FP32C; tables / moments for 1, 33 and 400 elements of two species, 3 s, 2 p, d and f): s
// shells of 3, 1, 1 primitives and the rest of one (mean 1.3) 74/118, 113/175, 155/213; s of
// 6, 3, 1 and p of 3, 1 (mean 3.5) 155/124, 206/172, 268/215; two primitives in the f shell
// only (mean 2.7) 359/129, 548/179, 654/221; two in every shell (mean 8) 392/130, 598/185,
// 739/217.  FP64 the same (s of 3: 192/246 for 400, 6-3-1: 395/246).  The counts are on the
// device, so both paths are launched and the one not taken returns at once.
__device__ __forceinline__ void pick3(int* pick, const Item3* __restrict__ items, const int* pn, int n, int ns, int NZ) {
    __shared__ unsigned long long sums[2];
    if (threadIdx.x < 2) sums[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long f = 0, t = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const Item3 it = items[i];
        int na = 0, nb = 0, nc = 0;
        for (int g = 0; g < NZ; ++g) {
            na = max(na, pn[g * ns + it.sa]);
            nb = max(nb, pn[g * ns + it.sb]);
            nc = max(nc, pn[g * ns + it.sc]);
        }
        const unsigned long long comps = kClass3[it.cls].comps;
        f += comps;
        t += comps * (unsigned long long)((long long)na * nb * nc);
    }
    atomicAdd(&sums[0], f);
    atomicAdd(&sums[1], t);
    __syncthreads();
    if (threadIdx.x == 0) *pick = sums[1] >= 2 * sums[0];
}

// Per call, one CTA: the order of the moment kernel's items (blocks) and its cut into
// segments.  The items of one class are kept together, so that the warps in flight at any
// time run few distinct routines and the instruction cache holds them; classes by their
// heaviest item, heaviest first, and the items inside a class heaviest first, so the queue
// ends with cheap work.  Cost = primitive triples (the largest count over the species per
// shell) x (the exponential + a multiply-add per moment) + a fixed part.  Rank sort in
// shared memory.  The ordered list is then cut into segments of about total / G cost,
// G = target_units / tiles (a warp takes a whole segment of one tile per unit); an item
// that costs more than that is a segment alone.  More than kOrder3Max items keep the
// static order, one item per segment.
// segs: the nseg + 1 segment bounds, then nseg at [n + 1], H at [n + 2] and at [n + 3]
// whether this path is taken (see pick3).
__device__ __forceinline__ void order3c_body(Item3* __restrict__ order, int* __restrict__ segs,
                                             const Item3* __restrict__ items, const int* pn, int ntiles, int n,
                                             int ns, int NZ, int target_units) {
    __shared__ unsigned long long ikey[kOrder3Max], gkey[kOrder3Max];
    __shared__ int cst[kOrder3Max];
    __shared__ int gmax[20];
    __shared__ long long wtot[kOrder3Threads / 32];
    pick3(segs + n + 3, items, pn, n, ns, NZ);
    if (n > kOrder3Max) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            order[i] = items[i];
            segs[i] = i;
        }
        if (threadIdx.x == 0) {
            segs[n] = n;
            segs[n + 1] = n;
            segs[n + 2] = 0;
        }
        return;
    }
    for (int c = threadIdx.x; c < 20; c += blockDim.x) gmax[c] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const Item3 it = items[i];
        int na = 0, nb = 0, nc = 0;  // primitive counts, the largest over the species
        for (int g = 0; g < NZ; ++g) {
            na = max(na, pn[g * ns + it.sa]);
            nb = max(nb, pn[g * ns + it.sb]);
            nc = max(nc, pn[g * ns + it.sc]);
        }
        const long long cost = min((long long)na * nb * nc * (24 + kClass3[it.cls].D) + 300, (long long)0x7FFFFFFF);
        cst[i] = (int)cost;
        // ascending = heaviest first; equal costs by class, then by position
        ikey[i] = ((unsigned long long)(0x7FFFFFFF - cost) << 32) | ((unsigned)it.cls << 12) | (unsigned)i;
        atomicMax(&gmax[it.cls], (int)cost);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int ci = items[i].cls;
        gkey[i] = ((unsigned long long)(0x7FFFFFFF - gmax[ci]) << 32) | (unsigned)ci;
    }
    __syncthreads();
    int rank[kOrder3Per], rcost[kOrder3Per];
#pragma unroll
    for (int k = 0; k < kOrder3Per; ++k) {
        const int i = threadIdx.x + k * kOrder3Threads;
        rank[k] = -1;
        if (i >= n) continue;
        const unsigned long long gi = gkey[i], ki = ikey[i];
        int r = 0;
        for (int j = 0; j < n; ++j) {
            const unsigned long long gj = gkey[j];
            r += gj < gi || (gj == gi && ikey[j] < ki);
        }
        order[r] = items[i];
        rank[k] = r;
        rcost[k] = cst[i];
    }
    __syncthreads();
    // the costs in queue order
#pragma unroll
    for (int k = 0; k < kOrder3Per; ++k)
        if (rank[k] >= 0) cst[rank[k]] = rcost[k];
    __syncthreads();
    // exclusive cost prefix of this thread's kOrder3Per consecutive positions
    const int r0 = threadIdx.x * kOrder3Per;
    long long tsum = 0;
#pragma unroll
    for (int k = 0; k < kOrder3Per; ++k)
        if (r0 + k < n) tsum += cst[r0 + k];
    const long long incl = block_scan3(tsum, wtot);
    __shared__ long long total_s;
    if (threadIdx.x == kOrder3Threads - 1) total_s = incl;
    __syncthreads();
    const long long total = total_s;
    const long long G = max(1LL, min((long long)n, (long long)target_units / max(ntiles, 1)));
    const long long C = max(1LL, (total + G - 1) / G);
    // a segment starts at r when a multiple of C lies in (prefix(r - 1), prefix(r)], or next to an item of cost >= C
    long long P = incl - tsum;
    unsigned flags = 0u;
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < kOrder3Per; ++k) {
        const int r = r0 + k;
        if (r >= n) break;
        bool start = r == 0;
        if (!start) {
            const long long pc = cst[r - 1];
            start = (P / C) != ((P - pc) / C) || pc >= C || cst[r] >= C;
        }
        if (start) {
            flags |= 1u << k;
            ++cnt;
        }
        P += cst[r];
    }
    const long long pos_incl = block_scan3(cnt, wtot);
    int pos = (int)(pos_incl - cnt);
#pragma unroll
    for (int k = 0; k < kOrder3Per; ++k)
        if (flags & (1u << k)) segs[pos++] = r0 + k;
    if (threadIdx.x == kOrder3Threads - 1) {
        segs[pos_incl] = n;
        segs[n + 1] = (int)pos_incl;
    }
    // H: the leading items of cost >= 2C (each a segment alone), whose triples the CTA's
    // warps share for one tile per unit
    if (threadIdx.x == 0) {
        int h = 0;
        while (h < n && cst[h] >= 2 * C) ++h;
        segs[n + 2] = h;
    }
}

// One CTA per call, launched programmatically after k_prep3c, which leaves the primitive
// counts: the pick, the moment kernel's item order and segments, and zeroed work counters
// for the kernels of this call.  As there, order and segments are a function of (n, ntiles,
// target_units) and the counts alone, and key[] holds those of the last build.
__global__ void __launch_bounds__(kOrder3Threads) k_prepm3(const int* __restrict__ pn, Item3* __restrict__ order,
                                                           int* __restrict__ segs, int* __restrict__ key,
                                                           const Item3* __restrict__ items,
                                                           unsigned* __restrict__ counters, int ncounters, int ntiles,
                                                           int n, int ns, int NZ, int target_units) {
    __shared__ int spn[kMaxShells * 6];
    pdl_trigger();  // the kernels may launch now; they wait for this grid's end
    for (int i = threadIdx.x; i < ncounters; i += blockDim.x) counters[i] = 0;
    const int nc = ns * NZ;
    pdl_wait();
    for (int t = threadIdx.x; t < nc; t += blockDim.x) spn[t] = pn[t];
    __syncthreads();
    int same = threadIdx.x != 0 || (key[0] == n && key[1] == ntiles && key[2] == target_units && key[3] == nc);
    for (int t = threadIdx.x; t < nc; t += blockDim.x) same &= key[4 + t] == spn[t];
    if (__syncthreads_and(same)) return;
    order3c_body(order, segs, items, spn, ntiles, n, ns, NZ, target_units);
    for (int t = threadIdx.x; t < nc; t += blockDim.x) key[4 + t] = spn[t];
    if (threadIdx.x == 0) {
        key[0] = n;
        key[1] = ntiles;
        key[2] = target_units;
        key[3] = nc;
    }
}

// The output elements of a panel in (k, j, i) order, i over the whole run of A shells:
// which slab elements add up to each (the aliased layout lin = c1 + N1 c2 + N1 N2 c3) and
// where it goes.  Appends them to `table` when given; returns their number.
static int panel_table3(const aok_plan* p, const Panel3& pn, std::vector<Out3>* table) {
    const int lb = (int)p->ls[pn.sb], lc = (int)p->ls[pn.sc], NB = ncart(lb), NC = ncart(lc);
    const int i0 = (int)p->boff[pn.sa0], ni = (int)p->boff[pn.sa0 + pn.nsa] - i0;
    if (!table) return ni * NB * NC;
    const size_t first = table->size();
    const short none = (short)pn.comps;
    table->resize(first + (size_t)ni * NB * NC, Out3{{none, none, none, none}, 0, 0});
    int soff = 0;
    for (int t = 0; t < pn.nsa; ++t) {
        const int sa = pn.sa0 + t, la = (int)p->ls[sa], NA = ncart(la), N1 = 2 * la + 1, N2 = 2 * lb + 1;
        const int col = (int)p->boff[sa] - i0;
        for (int c3 = 0; c3 < NC; ++c3)
            for (int c2 = 0; c2 < NB; ++c2)
                for (int c1 = 0; c1 < NA; ++c1) {
                    const int lin = c1 + N1 * c2 + N1 * N2 * c3, i = lin % NA, j = (lin / NA) % NB, k = lin / (NA * NB);
                    Out3& o = (*table)[first + ((size_t)k * NB + j) * ni + col + i];
                    int w = 0;
                    while (o.o[w] != none) ++w;
                    o.o[w] = (short)(soff + c1 + NA * (c2 + NB * c3));
                }
        soff += NA * NB * NC;
    }
    for (int k = 0; k < NC; ++k)
        for (int j = 0; j < NB; ++j)
            for (int i = 0; i < ni; ++i)
                (*table)[first + ((size_t)k * NB + j) * ni + i].at = (int)(((int64_t)k * p->N + j) * p->N + i);
    return ni * NB * NC;
}

int setup_moments3(aok_plan* p) {
    if (p->d_mom3 || p->no_mom3) return AOK_OK;
    const int ns = (int)p->ns;
    const size_t fsz = p->prec == AOK_PREC_F64 ? sizeof(double) : sizeof(float);
    // Panels: per (B shell, C shell), runs of A shells whose blocks fit the CTA's slab; a
    // block too large for 32 elements is alone in its panel, which is taken once per group of
    // elements.  Panels of several blocks have as many elements in FP32 as in FP64, although
    // the slab would take twice as many: fewer panels leave SMs idle (33 elements of 25
    // functions, FP32: 235 -> 184 us; 777 of 32: 454 -> 428).
    const int room = fsz == 4 ? slab_room3<float>() : slab_room3<double>();
    auto fits = [&](int comps, int passes) { return ((comps + 1) | 1) * (32 / passes) <= room; };
    // the moment kernel's items: one per block, statically by class; slots of the moments
    std::vector<Item3> items;
    int slots = 0;
    for (int sc = 0; sc < ns; ++sc)
        for (int sb = 0; sb < ns; ++sb)
            for (int sa = 0; sa < ns; ++sa) {
                const int cls = canon3((int)p->ls[sa], (int)p->ls[sb], (int)p->ls[sc]).cls;
                items.push_back(Item3{(short)sa, (short)sb, (short)sc, (short)cls, slots});
                slots += kClass3Host[cls].D;
            }
    std::vector<Panel3> panels;
    std::vector<Out3> table;
    std::map<std::array<int, 4>, int> tables;  // (lb, lc, sa0, nsa) -> first entry
    for (int sc = 0; sc < ns; ++sc)
        for (int sb = 0; sb < ns; ++sb) {
            const int lb = (int)p->ls[sb], lc = (int)p->ls[sc];
            for (int sa = 0; sa < ns;) {
                Panel3 pn{(short)sa, 0, (short)sb, (short)sc, 0, 1, 0, 0, 0, items[(size_t)(sc * ns + sb) * ns + sa].moff};
                while (sa < ns && pn.nsa < kPanelItems3) {
                    const int la = (int)p->ls[sa], c = pn.comps + ncart(la) * ncart(lb) * ncart(lc);
                    if (pn.nsa && ((c + 1) | 1) * 32 > slab_room3<double>()) break;
                    while (!fits(c, pn.passes)) pn.passes *= 2;
                    pn.comps = c;
                    ++pn.nsa;
                    ++sa;
                    if (pn.passes > 1) break;
                }
                const auto at = tables.find({lb, lc, (int)pn.sa0, (int)pn.nsa});
                pn.tab = at != tables.end() ? at->second : (int)table.size();
                pn.nout = panel_table3(p, pn, at != tables.end() ? nullptr : &table);
                tables[{lb, lc, (int)pn.sa0, (int)pn.nsa}] = pn.tab;
                for (pn.pass = 0; pn.pass < pn.passes; ++pn.pass) panels.push_back(pn);
            }
        }
    // panels in claim order: the costliest transforms first, those of one kind together
    std::vector<std::pair<int64_t, int>> cost(panels.size());
    for (size_t i = 0; i < panels.size(); ++i) {
        const Panel3& pn = panels[i];
        int64_t c = 0;
        for (int t = 0; t < pn.nsa; ++t)
            c += kClass3Host[canon3((int)p->ls[pn.sa0 + t], (int)p->ls[pn.sb], (int)p->ls[pn.sc]).cls].ops;
        const int lb = (int)p->ls[pn.sb], lc = (int)p->ls[pn.sc];
        cost[i] = {-(((3 * c + pn.comps) / 64) * 16 + 4 * std::max(lb, lc) + std::min(lb, lc)), (int)i};
    }
    std::sort(cost.begin(), cost.end());
    std::vector<Panel3> ordered;
    for (const auto& c : cost) ordered.push_back(panels[(size_t)c.second]);
    panels.swap(ordered);
    std::stable_sort(items.begin(), items.end(), [](const Item3& a, const Item3& b) { return a.cls > b.cls; });
    p->nitemsm = (int)items.size();
    p->slots3 = slots;
    // moments are kept for at most kMoments3 bytes of tiles at a time; a larger batch goes
    // through in rounds.  One tile always fits: the panel schedule of the plan bounds N to
    // about 120 (64 shells of 83 functions: 70 MB).
    const int64_t most = (p->max_batch + 31) / 32 + bin_keys_max(p->NZ) + 1;
    const int64_t tile = (int64_t)slots * 32 * (int64_t)sizeof(double);
    p->round3 = (int)std::max<int64_t>(1, std::min(most, kMoments3 / tile));
    p->nrounds3 = (int)((most + p->round3 - 1) / p->round3);
    p->npanels3 = (int)panels.size();
    // one buffer: items, panels, output elements and the schedule key of k_prepm3 (all ones:
    // n = -1 matches no call, so the first builds), copied in one piece; then what the
    // kernels write
    size_t bytes = 0;
    auto place = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t nitems = sizeof(Item3) * items.size(), npanels = sizeof(Panel3) * panels.size(),
                 nout = sizeof(Out3) * table.size(), nkey = sizeof(int) * (size_t)(4 + ns * p->NZ);
    const size_t at_items = place(nitems), at_panels = place(npanels), at_out = place(nout), at_key = place(nkey);
    std::vector<char> host(bytes);
    memcpy(host.data() + at_items, items.data(), nitems);
    memcpy(host.data() + at_panels, panels.data(), npanels);
    memcpy(host.data() + at_out, table.data(), nout);
    memset(host.data() + at_key, 0xFF, nkey);
    const size_t at_order = place(nitems), at_segs = place(sizeof(int) * (items.size() + 4)),
                 at_cnt = place(sizeof(unsigned) * 2 * (size_t)p->nrounds3);
    // on a failure the plan has neither buffer; without memory it keeps to the explicit tables,
    // which need none of this (for good: a later call may be under stream capture, where
    // nothing can be allocated), after another failure the next call starts again
    void *sched = nullptr, *mom = nullptr;
    cudaError_t e = cudaMalloc(&sched, bytes);
    if (e == cudaSuccess) e = cudaMemcpy(sched, host.data(), host.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&mom, (size_t)(tile * p->round3));
    p->d_segsm = (int*)((char*)sched + at_segs);
    int st = AOK_OK;
    if (e == cudaSuccess)
        st = p->prec == AOK_PREC_F64 ? reserve_moments3_f64(p, &e) : reserve_moments3_f32(p, &e);
    if (e != cudaSuccess || st != AOK_OK) {
        if (sched) cudaFree(sched);
        if (mom) cudaFree(mom);
        p->d_segsm = nullptr;
        if (st == AOK_OK) st = cuda_status(e, "3C overlap: moments");
        p->no_mom3 = e == cudaErrorMemoryAllocation || e == cudaErrorLaunchOutOfResources;
        return p->no_mom3 ? AOK_OK : st;
    }
    char* base = (char*)sched;
    p->d_sched3 = sched;
    p->d_itemsm = base + at_items;
    p->d_panels3 = base + at_panels;
    p->d_out3 = base + at_out;
    p->d_keym = (int*)(base + at_key);
    p->d_orderm = base + at_order;
    p->d_cnt3 = (unsigned*)(base + at_cnt);
    p->d_mom3 = mom;
    return AOK_OK;
}

// The prep of the moment path on stream `side`, after k_prep3c (see k_prepm3).
int launch_prepm3(aok_plan* p, int64_t B, cudaStream_t side) {
    // about four (segment, tile) pairs per resident warp of the moment kernel
    const int target_units = p->num_sms * kMomCtas3 * kWarps3 * 4;
    const int ntiles = (int)std::min<int64_t>((B + 31) / 32, 1 << 30);
    const cudaError_t e = launch_pdl(k_prepm3, dim3(1), dim3(kOrder3Threads), 0, side, (const int*)p->d_npp3,
                                     (Item3*)p->d_orderm, p->d_segsm, p->d_keym, (const Item3*)p->d_itemsm, p->d_cnt3,
                                     2 * p->nrounds3, ntiles, p->nitemsm, (int)p->ns, (int)p->NZ, target_units);
    return cuda_status(e, "k_prepm3");
}

}  // namespace m3
}  // namespace aok
