// FP64 translations on the tensor cores (k_mma.cuh): one CTA per target and chunk of its sources, four sources per
// batch.  The direct operator (k_direct's launches and slabs) and the ML-FMM's passes over long lists.
#include <cmath>

#include "k_mma.cuh"

namespace foggy {

namespace {
using namespace mma;

// direction of a translation, rounded as in disp_vec (k_direct.cu): t = k (sign (c_s - c_t) + sh)
__device__ inline Dir pair_dir(const double* ct, const double* cs, double k, double sign, double sh0, double sh1,
                               double sh2) {
    const double d0 = __dmul_rn(k, __fma_rn(sign, __dsub_rn(cs[0], ct[0]), sh0));
    const double d1 = __dmul_rn(k, __fma_rn(sign, __dsub_rn(cs[1], ct[1]), sh1));
    const double d2 = __dmul_rn(k, __fma_rn(sign, __dsub_rn(cs[2], ct[2]), sh2));
    return direction(d0, d1, d2, sqrt(__fma_rn(d0, d0, __fma_rn(d1, d1, __dmul_rn(d2, d2)))));
}
// records are made once in eight batches: a call keeps their arithmetic out of the loop's code
__device__ __noinline__ Dir pair_dir_call(const double* ct, const double* cs, double k, double sign, double sh0,
                                          double sh1, double sh2) {
    return pair_dir(ct, cs, k, sign, sh0, sh1, sh2);
}

// The translations of one target of degree pj, `mine` batches of four units; unit(i, l, un, dir) fills the record of unit
// i of this CTA's batches, or leaves it empty.  The sums are in s.acc at the end, visible to every thread.
// Without tables (SUM) the coaxial coefficients are summed from g and the radial functions of selector z; zeta: shared
// memory for them (sum_smem_bytes).
template <int NI, int W, bool SUM, class UnitOf>
__device__ __forceinline__ void run_batches(const Shared& s, const MmaTabs& mt, int pp, int pj, int mine, const SGaunt& g,
                                            int z, double2* zeta, UnitOf unit) {
    constexpr int T = 32 * W, LD = phase_ld<NI>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Pj = pj * (pj + 2);
    // records of this CTA's batches 8g..8g+7, one unit per lane (one warp)
    auto records = [&](int g) {
        Dir d{1.0, 0.0, 1.0, 0.0, 1.0};
        Unit un{nullptr, nullptr, 0, -1, 1.0};
        unit(kRecs * g + lane, un, d);
        if (un.x) {
            un.rho = d.rho;
            un.km = d.rho == 0.0 ? -1 : min(pj, un.p);
        }
        s.dir[(g & 1) * kRecs + lane] = d;
        s.un[(g & 1) * kRecs + lane] = un;
    };
    auto slot = [](int i) { return ((i >> 3) & 1) * kRecs + (i & 7) * kUnits; };   // records of batch i
    // phase tables of batch i into half e; its coaxial rows are fetched into L2 meanwhile
    auto prep = [&](int i, int e) {
        const int at = slot(i);
#pragma unroll 1
        for (int t = tid; t < 2 * kUnits * LD; t += T) {
            const int half = t / (kUnits * LD), r = t - half * kUnits * LD;
            const int u = r / LD, m = r - u * LD;
            const Dir& g = s.dir[at + u];
            // e^{i m (phi + pi/2)}, or (-1)^s (2 cos s theta, 2 sin s theta) with (1, 0) at s = 0
            const cplx z = zpow(half ? mk(g.ct, g.st) : mk(-g.sp, g.cp), m);
            const double f = !half || m == 0 ? 1.0 : (m & 1) ? -2.0 : 2.0;
            (half ? s.eth : s.eps)[e * kUnits * LD + r] = make_double2(f * z.x, f * z.y);
        }
        if constexpr (SUM) {
            constexpr int ZL = zeta_ld<NI>();
            if (warp == i % W)
                radial(s.un + at, pj, z, zeta + e * kUnits * ZL, ZL, reinterpret_cast<double*>(zeta + 2 * kUnits * ZL), lane);
        } else if (warp == W - 1) {
#pragma unroll 1
            for (int u = 0; u < kUnits; ++u) {
                const Unit& un = s.un[at + u];
                const int M2 = max(pj, un.p) + 2;
                if (lane <= un.km) {
                    // the order's square block up to the last row of either reading: 16-byte entries, so aligned
                    const unsigned bytes = (unsigned)((pj + 1 - lane) * (M2 - lane) * sizeof(cplx));
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(un.s + block_offset(lane, M2)),
                                 "r"(bytes)
                                 : "memory");
                }
            }
        }
    };

    for (int t = tid; t < kPlanInts; t += T) s.blk[t] = mt.plan[kPlanInts * (pp + (SUM ? kMmaDegree + 1 : 0)) + t];
    if (tid < 4) s.zero[tid] = make_double2(0.0, 0.0);
    for (int t = tid; t < 2 * Pj; t += T) s.acc[t] = make_double2(0.0, 0.0);
    for (int t = tid; t < 8 * NI + 8; t += T) s.rn[t] = t ? 0.5 / (double)(t * (t + 1)) : 0.0;
    if (warp == W - 1) records(0);
    __syncthreads();
    prep(0, 0);
    const Lane<NI> L(s, pp, lane);
    __syncthreads();
    int cur = 0;
    for (int ib = 0; ib < mine; ++ib, cur ^= 1) {
        const Unit* un = s.un + slot(ib);
        const int pl4 = max(max(un[0].p, un[1].p), max(un[2].p, un[3].p));
        const Unit mine_u = un[L.u];   // this lane's unit in the rotations
        // one copy of the rotation's code for both directions
#pragma unroll 1
        for (int out = 0; out < 2; ++out) {
            rotate_all<NI>(s, L, mt.frag, warp, out ? pj : pl4, pj, mine_u, cur, out != 0);
            if (out) break;
            __syncthreads();
            if constexpr (SUM)
                coaxial_sum<NI>(s, un, 2 * (warp & 1), warp / 2, W / 2, pj, mt.wf, mt.ld, g,
                                zeta + cur * kUnits * zeta_ld<NI>(), zeta_ld<NI>(), lane);
            else
                coaxial<NI>(s, un[warp % kUnits], warp % kUnits, warp / kUnits, W / kUnits, pj, mt.wf, mt.ld, lane);
            if (ib + 1 < mine) {
                prep(ib + 1, cur ^ 1);
                // the next eight batches' records go where the last eight's were
                if ((ib & 7) == 5 && warp == (ib >> 3) % W) records((ib >> 3) + 1);
            }
            __syncthreads();
        }
        if (un[0].rho == 0.0 || un[1].rho == 0.0 || un[2].rho == 0.0 || un[3].rho == 0.0) {
            // coincident centres: the source is added unchanged, by the warp that owns the degree
            __syncwarp();
            for (int i = s.wfirst[warp]; i < s.wfirst[warp + 1]; ++i) {
                const int n = s.ord[i];
                for (int u = 0; u < kUnits; ++u)
                    if (un[u].rho == 0.0 && n <= min(pj, un[u].p))
                        for (int e = lane; e < 2 * (2 * n + 1); e += 32) {
                            const int part = e > 2 * n, m = e - part * (2 * n + 1);
                            const double2 v = un[u].x[part * un[u].p * (un[u].p + 2) + n * n - 1 + m];
                            double2* d = s.acc + part * Pj + n * n - 1 + m;
                            d->x += v.x;
                            d->y += v.y;
                        }
            }
            __syncwarp();
        }
    }
    __syncthreads();
}

// batches c, c + chunks, ... of a list of n units
__device__ __forceinline__ int batches_of(int n, int c, int chunks) {
    const int nb = (n + kUnits - 1) / kUnits;
    return c < nb ? (nb - c + chunks - 1) / chunks : 0;
}
}  // namespace

template <int NI, int W, int CTAS, bool SUM>
__global__ void __launch_bounds__(32 * W, CTAS) k_direct_mma(DirectArgs a, MmaTabs mt, const MmaWork* __restrict__ work,
                                                             int nw, int nrhs, int64_t ld, int per_rhs) {
    extern __shared__ __align__(16) double smem_d[];
    // the next class's CTAs may start once all of these have (they fill other slabs); each launch ends after the one before
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const SceneView& sc = a.sc;
    // right-hand side fastest: the CTAs that read one pair's coaxial block run together
    const int rhs = blockIdx.x % nrhs, unit = blockIdx.x / nrhs;
    // this CTA's share: the last one that starts no later (every warp looks, one load per lane and 32 shares)
    int at = -1;
    for (int b = 0; b < nw; b += 32) {
        const int i = b + (threadIdx.x & 31);
        at += __popc(__ballot_sync(0xffffffffu, i < nw && work[i].cta0 <= unit));
    }
    const MmaWork bk = work[at];
    const int tc = unit - bk.cta0, c = tc / bk.ntargets;
    const int j = bk.targets[tc % bk.ntargets];
    if (!sc.couple[j]) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    const cplx* const x = a.x + rhs * ld;
    const int pj = sc.p[j];
    // the summed variant's radial functions come first, so that the rest is laid out as ever
    double2* const zeta = reinterpret_cast<double2*>(smem_d);
    const Shared s = carve<NI>(SUM ? zeta + sum_smem_bytes<NI>() / 16 : zeta, bk.pp, bk.us);
    run_batches<NI, W, SUM>(s, mt, bk.pp, pj, batches_of(bk.nsources, c, bk.chunks), a.g, a.z, zeta,
                            [&](int r, Unit& un, Dir& d) {
        const int i = kUnits * (c + r / kUnits * bk.chunks) + r % kUnits;
        const int l = i < bk.nsources ? bk.sources[i] : j;
        if (l == j) return;
        un.x = reinterpret_cast<const double2*>(x + sc.off[l]);
        if (!SUM)
            un.s = reinterpret_cast<const double2*>(a.pt.stab + a.pt.pair_off[pair_index(min(j, l), max(j, l), sc.n)]);
        un.p = sc.p[l];
        d = pair_dir_call(sc.centres + 3 * (size_t)j, sc.centres + 3 * (size_t)l, sc.k, 1.0, 0.0, 0.0, 0.0);
    });
    cplx* out = a.partial + ((size_t)rhs * per_rhs + bk.slab + c) * a.n_unk + sc.off[j];
    for (int t = threadIdx.x; t < 2 * pj * (pj + 2); t += 32 * W) out[t] = mk(s.acc[t].x, s.acc[t].y);
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One ML-FMM pass over cached blocks (k_translate's arguments and results)
template <int NI, int W, int CTAS>
__global__ void __launch_bounds__(32 * W, CTAS) k_translate_mma(TransArgs a, MmaTabs mt, int pp, int us) {
    extern __shared__ __align__(16) double smem_d[];
    const int t = a.tbase + blockIdx.x, c = blockIdx.y, chunks = gridDim.y;
    const int pj = a.tgt.p[t];
    const int i0 = a.lptr[blockIdx.x], n = a.lptr[blockIdx.x + 1] - i0;
    const Shared s = carve<NI>(smem_d, pp, us);
    run_batches<NI, W, false>(s, mt, pp, pj, batches_of(n, c, chunks), SGaunt{}, 0, nullptr, [&](int r, Unit& un, Dir& d) {
        const int i = kUnits * (c + r / kUnits * chunks) + r % kUnits;
        if (i >= n) return;
        const int l = a.lidx[i0 + i];
        un.x = reinterpret_cast<const double2*>(a.x + a.src.off[l]);
        un.s = reinterpret_cast<const double2*>(a.tab + a.tab_off[i0 + i]);
        un.p = a.src.p[l];
        d = pair_dir_call(a.tgt.c + 3 * (size_t)t, a.src.c + 3 * (size_t)l, a.k, a.sign, a.sh[0], a.sh[1], a.sh[2]);
    });
    cplx* out = chunks == 1 ? a.out + a.tgt.off[t] : a.slab + ((size_t)c * gridDim.x + blockIdx.x) * a.slab_ld;
    const bool add = a.add && chunks == 1;
    for (int e = threadIdx.x; e < 2 * pj * (pj + 2); e += 32 * W) {
        const cplx v = mk(s.acc[e].x, s.acc[e].y);
        out[e] = add ? out[e] + v : v;
    }
}

int mma_ctas_per_sm(int pp, bool sum) { return pp <= 7 ? 4 : pp <= 15 ? (sum ? 2 : 3) : pp <= 19 ? 2 : pp <= 23 && !sum ? 2 : 1; }
int mma_class(int pp, bool sum) { return pp <= 7 ? 0 : pp <= 15 ? 1 : pp <= 19 && sum ? 2 : pp <= 23 ? 3 : 4; }
int mma_unit_size(int pp) { return mma::unit_size(pp); }

// f<NI, W, CTAS> of a launch of largest degree pp
template <bool SUM, class F>
static void by_degree(int pp, F f) {
    if (pp <= 7) f.template operator()<1, mma::warps_of(7, SUM), 4>();
    else if (pp <= 15) f.template operator()<2, mma::warps_of(15, SUM), SUM ? 2 : 3>();
    else if (pp <= 19) f.template operator()<3, mma::warps_of(19, SUM), 2>();
    else if (pp <= 23) f.template operator()<3, mma::warps_of(23, SUM), SUM ? 1 : 2>();
    else f.template operator()<4, mma::warps_of(31, SUM), 1>();
}

void launch_direct_mma(const DirectArgs& a, const MmaTabs& mt, const MmaWork* w, int nw, int ctas, int pp, int nrhs,
                       int64_t ld, int per_rhs, bool after_other, cudaStream_t s) {
    auto go = [&](auto* kernel, int warps, size_t smem) {
        raise_smem_ceiling(reinterpret_cast<const void*>(kernel), smem);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)ctas * nrhs);
        cfg.blockDim = dim3(32 * warps);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &at;
        cfg.numAttrs = after_other ? 1 : 0;
        cudaLaunchKernelEx(&cfg, kernel, a, mt, w, nw, nrhs, ld, per_rhs);
    };
    if (a.pt.stab)
        by_degree<false>(pp, [&]<int NI, int W, int CTAS>() { go(k_direct_mma<NI, W, CTAS, false>, W, mma::smem_bytes<NI>(pp)); });
    else
        by_degree<true>(pp, [&]<int NI, int W, int CTAS>() {
            go(k_direct_mma<NI, W, CTAS, true>, W, mma::smem_bytes<NI>(pp) + mma::sum_smem_bytes<NI>());
        });
}

void launch_translate_mma(const TransArgs& a, const MmaTabs& mt, int pp, int ntargets, int chunks, cudaStream_t s) {
    by_degree<false>(pp, [&]<int NI, int W, int CTAS>() {
        auto* kernel = k_translate_mma<NI, W, CTAS>;
        const size_t smem = mma::smem_bytes<NI>(pp);
        raise_smem_ceiling(reinterpret_cast<const void*>(kernel), smem);
        kernel<<<dim3(ntargets, chunks), 32 * W, smem, s>>>(a, mt, pp, mma::unit_size(pp));
    });
    if (chunks > 1) launch_translate_sum(a, ntargets, chunks, s);
}

// The host tables of the tensor-core operator for degrees <= pmax (k_mma.cuh).
void build_mma_tables(int pmax, const std::vector<double>& delta, std::vector<double>& frag, std::vector<double>& wf,
                      std::vector<int>& plan) {
    frag.clear();
    for (int n = 1; n <= pmax; ++n) {
        const double* Q = delta.data() + (size_t)n * (n + 1) * (2 * n + 1) / 6;
        const int K = mma::steps_of(n);
        for (int P = 0; P < 2; ++P)
            for (int t = 0; t < (K + 1) / 2; ++t)
                for (int r = 0; r < 2; ++r)
                    for (int j = 0; j < K; j += 2)
                        for (int lane = 0; lane < 32; ++lane)
                            for (int e = 0; e < (j + 1 < K ? 2 : 1); ++e) {
                                const int c = lane >> 2;   // column: output order 8t + 4 (c & 1) + c / 2
                                const int in = 2 * (4 * (j + e) + (lane & 3)) + r;
                                const int out = 2 * (8 * t + 4 * (c & 1) + (c >> 1)) + P;
                                frag.push_back(in <= n && out <= n ? Q[(size_t)in * (n + 1) + out] : 0.0);
                            }
    }
    // with tables, then without
    plan.assign((size_t)2 * mma::kPlanInts * (kMmaDegree + 1), 0);
    for (int sum = 0; sum < 2; ++sum)
        for (int pp = 1; pp <= kMmaDegree; ++pp)
            mma::make_plan(pp, mma::warps_of(pp, sum != 0),
                           plan.data() + (size_t)mma::kPlanInts * (pp + sum * (kMmaDegree + 1)));
    // rows padded: the coaxial step reads whole k-steps of 4
    const int ld = pmax + 8;
    wf.assign(2 * (size_t)(pmax + 1) * ld, 0.0);
    for (int k = 0; k <= pmax; ++k)
        for (int mu = k; mu < ld; ++mu) {
            double* f = wf.data() + 2 * ((size_t)k * ld + mu);
            f[0] = 2.0 * (mu - 1.0) * std::sqrt((double)mu * mu - (double)k * k);
            f[1] = 2.0 * (mu + 2.0) * std::sqrt((mu + 1.0) * (mu + 1.0) - (double)k * k);
        }
}

}  // namespace foggy
