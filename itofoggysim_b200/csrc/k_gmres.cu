// Krylov-space kernels of the device GMRES (replacing the CERFACS drive_zgmres loop the
// reference runs on the host, FoggySim/src/lib/mie_theory/lib_solver_GMRES.f90:116-316).
// All reductions are two-pass with a fixed order, so a solve is bit-reproducible.
#include <algorithm>

#include "foggy_kernels.cuh"

namespace foggy {

namespace {
constexpr int kT = 256;
constexpr int kMaxDots = 64;   // Krylov vectors handled per dots launch
}

__global__ void __launch_bounds__(kT) k_norm_partial(const cplx* w, int64_t n, double* part) {
    __shared__ double red[kT];
    int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    int64_t lo = (int64_t)blockIdx.x * chunk;
    int64_t hi = min(n, lo + chunk);
    double s = 0.0;
    for (int64_t t = lo + threadIdx.x; t < hi; t += blockDim.x) s += w[t].x * w[t].x + w[t].y * w[t].y;
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = kT / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(kT) k_norm_reduce(const double* part, double* out) {
    __shared__ double red[kT];
    double s = 0.0;
    for (int b = threadIdx.x; b < kRedBlocks; b += blockDim.x) s += part[b];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = kT / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sqrt(red[0]);
}

// v = w / nrm (v = 0 when nrm == 0)
__global__ void k_scale_copy(const cplx* w, const double* nrm, cplx* v, int64_t n) {
    double r = nrm[0];
    double inv = (r != 0.0) ? 1.0 / r : 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        v[t] = inv * w[t];
}

__global__ void k_sub(const cplx* b, const cplx* ax, cplx* r, int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        r[t] = b[t] - ax[t];
}

// g = (beta, 0, ...) at the start of a restart cycle
__global__ void k_init_cycle(cplx* g, int m1, const double* beta, int* flags) {
    for (int i = threadIdx.x; i < m1; i += blockDim.x) g[i] = mk(0, 0);
    __syncthreads();
    if (threadIdx.x == 0) {
        g[0] = mk(beta[0], 0.0);
        flags[0] = 0;
    }
}

// back substitution H[0:k,0:k] y = g[0:k], k <= 64, by one warp: lane l holds rows l and l + 32 and takes y_i times
// column i off them, the next column's entries loaded meanwhile.  A chain of k divisions, where one thread row by row was a
// chain of k^2 / 2 loads and products: 65 us for 26 columns, and with eight vectors of the update below in flight a solve of
// 32640 unknowns went from 4.30 to 4.09 ms, 32 of them as a block from 100 to 96 ms.
__device__ void trisolve(const cplx* H, int ldh, const cplx* g, int k, cplx* y) {
    const int lane = threadIdx.x & 31;
    const cplx zero = mk(0.0, 0.0);
    cplx s[2], c[2], d = zero;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = lane + 32 * e;
        s[e] = r < k ? g[r] : zero;
        c[e] = r < k ? H[(size_t)r * ldh + k - 1] : zero;   // column k - 1; rows up to k - 1
    }
    for (int i = k - 1; i >= 0; --i) {
        cplx nx[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = lane + 32 * e;
            nx[e] = r < i ? H[(size_t)r * ldh + i - 1] : zero;   // column i - 1; none when i = 0
        }
        const cplx yi = cdiv(i < 32 ? s[0] : s[1], i < 32 ? c[0] : c[1]);
        d = mk(__shfl_sync(0xffffffffu, yi.x, i & 31), __shfl_sync(0xffffffffu, yi.y, i & 31));
        if (lane == (i & 31)) y[i] = d;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (lane + 32 * e < i) s[e] = s[e] - c[e] * d;
            c[e] = nx[e];
        }
    }
}

__global__ void __launch_bounds__(32) k_trisolve(const cplx* H, int ldh, const cplx* g, int k, cplx* y) {
    trisolve(H, ldh, g, k, y);
}

// x += sum_{i<k} y_i V_i
__global__ void k_update_x(cplx* x, const cplx* V, int64_t ld, const cplx* y, int k, int64_t n) {
    __shared__ cplx ys[kMaxDots];
    for (int i = threadIdx.x; i < k; i += blockDim.x) ys[i] = y[i];
    __syncthreads();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        cplx acc = x[t];
#pragma unroll 8
        for (int i = 0; i < k; ++i) acc = acc + ys[i] * V[(size_t)i * ld + t];
        x[t] = acc;
    }
}


// ---- one Arnoldi step's orthogonalisation --------------------------------------------------------
// Classical Gram-Schmidt twice, the norm and the Givens rotation, for one Krylov space or one per slot
// (blockIdx.y), as three launches and a fourth that scales: dots | subtract, dots again | subtract, norm, Givens | next
// vector.  Each block owns a slice of w; the last block to finish (an atomic ticket, no waiting) adds the blocks' partial
// sums in block order, so a result does not depend on the order of arrival or on the other slots.
// Small problems are bound by launches (ten of them before), large ones by how much of the basis is in flight: a thread
// keeps its entries of w through subtraction and dots, so no barrier parts the two, and loads kGroup vectors' entries at
// once, zeros past the last; the dots' sums leave the registers once per group and slice.  50 steps, ten launches / four
// with a barrier per 256 entries between subtraction and dots / this, ms:  2800 unknowns 3.8 / 2.8 / 2.4, 32640 4.6 / 3.0 /
// 2.8, 349866 11.4 / 13.2 / 8.4, 1370820 41.4 / 43.6 / 25.7, 32 slots of 32640 31.2 / 28.3 / 23.9, 4 of 349866 30.3 /
// 33.7 / 27.6.
namespace {
// flags, and live / kend / tol of a slot (null for a single space), see GsArgs
__device__ void givens_column(const GsArgs& a, int b, const cplx* hs, double hk1, cplx* col, cplx* rot, double* rsn) {
    const int k = a.nv - 1, m = a.m, tid = threadIdx.x;
    cplx* H = a.H + (size_t)b * (m + 1) * m;
    cplx* cs = a.cs + (size_t)b * m;
    double* sn = a.sn + (size_t)b * m;
    cplx* g = a.g + (size_t)b * (m + 1);
    for (int i = tid; i <= k; i += kT) {
        col[i] = hs[i] + a.c[(size_t)b * (m + 1) + i];   // both passes
        if (i < k) {
            rot[i] = cs[i];
            rsn[i] = sn[i];
        }
    }
    __syncthreads();
    if (tid == 0) {
        for (int i = 0; i < k; ++i) {
            const cplx u = col[i], d = col[i + 1];
            col[i] = conjg(rot[i]) * u + rsn[i] * d;
            col[i + 1] = mk(-rsn[i], 0) * u + rot[i] * d;
        }
        const cplx u = col[k];
        const double den = sqrt(u.x * u.x + u.y * u.y + hk1 * hk1);
        if (den == 0.0) {   // breakdown
            a.flags[b] = 1;
            a.res[b] = 0.0;
            if (a.live) {
                a.live[b] = 0;
                a.kend[b] = k;
            }
        } else {
            const cplx c = mk(u.x / den, u.y / den);
            const double s = hk1 / den;
            cs[k] = c;
            sn[k] = s;
            col[k] = mk(den, 0);
            const cplx gk = g[k], gn = mk(-s, 0) * gk;
            g[k + 1] = gn;
            g[k] = conjg(c) * gk;
            const double re = sqrt(gn.x * gn.x + gn.y * gn.y);
            a.res[b] = re;
            if (!isfinite(re)) a.flags[b] = 2;
            if (a.live) {
                // a slot leaves the cycle when its estimate reaches its tolerance, at breakdown or when full
                a.kend[b] = k + 1;
                if (!isfinite(re) || re <= a.tol[b] || hk1 == 0.0 || k + 1 == m) a.live[b] = 0;
            }
        }
    }
    __syncthreads();
    for (int i = tid; i <= k; i += kT) H[(size_t)i * m + k] = col[i];
}
}  // namespace

constexpr int kGroup = 8;
// MODE 0: hh = V^H w.  1: w -= V hh, c = V^H w.  2: w -= V c, hn = |w|, Hessenberg column and Givens rotation.
template <int MODE>
__global__ void __launch_bounds__(kT) k_gs(GsArgs a) {
    __shared__ cplx hs[kMaxDots], col[kMaxDots], rot[kMaxDots];
    __shared__ double rsn[kMaxDots], red[kT / 32], sums[kT / 32][2 * kGroup];
    __shared__ bool last;
    // the next launch's blocks may take their places; this one's input is the launch before
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, q = tid >> 5, nv = a.nv, G = gridDim.x;
    if (a.live && !a.live[b]) return;
    const cplx* V = a.V + (size_t)b * a.ld;
    cplx* w = a.W + (size_t)b * a.ld;
    if (MODE > 0) {
        const cplx* h = (MODE == 1 ? a.hh : a.c) + (size_t)b * (a.m + 1);
        for (int i = tid; i < kMaxDots; i += kT) hs[i] = i < nv ? h[i] : mk(0.0, 0.0);
        __syncthreads();
    }
    const int64_t chunk = (a.n + G - 1) / G, lo = (int64_t)blockIdx.x * chunk, hi = min(a.n, lo + chunk);
    // kGroup vectors at a time, the ones past the last as zeros: so many loads are always in flight
    auto group = [&](int i0, int64_t t, cplx (&v)[kGroup]) {
#pragma unroll
        for (int e = 0; e < kGroup; ++e) v[e] = i0 + e < nv ? V[(size_t)(i0 + e) * a.ldi + t] : mk(0.0, 0.0);
    };
    if (MODE > 0) {
        double nrm = 0.0;
        for (int64_t t = lo + tid; t < hi; t += kT) {
            cplx acc = w[t];
            for (int i0 = 0; i0 < nv; i0 += kGroup) {
                cplx v[kGroup];
                group(i0, t, v);
#pragma unroll
                for (int e = 0; e < kGroup; ++e) acc = acc - hs[i0 + e] * v[e];
            }
            w[t] = acc;
            nrm += acc.x * acc.x + acc.y * acc.y;
        }
        if (MODE == 2) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
            if (lane == 0) red[q] = nrm;
            __syncthreads();
            if (tid == 0) {
                double v = 0.0;
                for (int e = 0; e < kT / 32; ++e) v += red[e];
                a.npart[(size_t)b * kRedBlocks + blockIdx.x] = v;
            }
        }
    }
    if (MODE < 2) {
        // a thread has the same entries as above
        for (int i0 = 0; i0 < nv; i0 += kGroup) {
            double s[2 * kGroup];
#pragma unroll
            for (int e = 0; e < 2 * kGroup; ++e) s[e] = 0.0;
            for (int64_t t = lo + tid; t < hi; t += kT) {
                cplx v[kGroup];
                group(i0, t, v);
                const cplx x = w[t];
#pragma unroll
                for (int e = 0; e < kGroup; ++e) {
                    s[2 * e] += v[e].x * x.x + v[e].y * x.y;
                    s[2 * e + 1] += v[e].x * x.y - v[e].y * x.x;
                }
            }
            // 16 sums over 32 lanes: each step halves the sums a lane carries; lane l ends with sum l / 2
#pragma unroll
            for (int o = 16, m = kGroup; o > 1; o >>= 1, m >>= 1)
#pragma unroll
                for (int e = 0; e < m; ++e) {
                    const bool up = (lane & o) != 0;
                    const double give = up ? s[e] : s[e + m], keep = up ? s[e + m] : s[e];
                    s[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
            __syncthreads();   // the sums of the group before have been read
            if (!(lane & 1)) sums[q][lane >> 1] = s[0];
            __syncthreads();
            if (tid < 2 * kGroup && i0 + tid / 2 < nv) {
                double v = 0.0;
#pragma unroll
                for (int e = 0; e < kT / 32; ++e) v += sums[e][tid];
                reinterpret_cast<double*>(a.part)[2 * (((size_t)b * nv + i0 + tid / 2) * kRedBlocks + blockIdx.x) + tid % 2] = v;
            }
        }
    }
    // the last block adds the partial sums
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(a.ticket + b, 1) == G - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (tid == 0) a.ticket[b] = 0;
    if (MODE == 2) {
        double v = 0.0;
        if (q == 0) {
            for (int e = lane; e < G; e += 32) v += __ldcg(a.npart + (size_t)b * kRedBlocks + e);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) {
                red[0] = sqrt(v);
                a.hn[b] = red[0];
            }
        }
        // the first pass's coefficients beside the second's
        __syncthreads();
        for (int i = tid; i < nv; i += kT) hs[i] = a.hh[(size_t)b * (a.m + 1) + i];
        __syncthreads();
        givens_column(a, b, hs, red[0], col, rot, rsn);
    } else {
        cplx* out = (MODE == 0 ? a.hh : a.c) + (size_t)b * (a.m + 1);
        for (int i = q; i < nv; i += kT / 32) {
            const double2* p = reinterpret_cast<const double2*>(a.part + ((size_t)b * nv + i) * kRedBlocks);
            double vx = 0.0, vy = 0.0;
#pragma unroll 4
            for (int e = lane; e < G; e += 32) {
                const double2 u = __ldcg(p + e);
                vx += u.x;
                vy += u.y;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                vx += __shfl_xor_sync(0xffffffffu, vx, o);
                vy += __shfl_xor_sync(0xffffffffu, vy, o);
            }
            if (lane == 0) out[i] = mk(vx, vy);
        }
    }
}

// v_b = w_b / hn[b] of the slots still in the cycle (v = 0 when hn = 0)
__global__ void __launch_bounds__(kT) k_gs_next(GsArgs a, cplx* Vn) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int b = blockIdx.y;
    if (a.live && !a.live[b]) return;
    const double r = a.hn[b], inv = (r != 0.0) ? 1.0 / r : 0.0;
    const cplx* w = a.W + (size_t)b * a.ld;
    cplx* v = Vn + (size_t)b * a.ld;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.n; t += (int64_t)gridDim.x * blockDim.x)
        v[t] = inv * w[t];
}

// Blocks by the vectors' length alone, so that a slot's sums do not depend on how many slots there are.
void launch_arnoldi_step(const GsArgs& a, int slots, cplx* Vnext, cudaStream_t s) {
    const int G = (int)std::min<int64_t>(kRedBlocks, (a.n + kT - 1) / kT);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(G, slots);
    cfg.blockDim = dim3(kT);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 0;   // the first waits for the operator's last launch as usual
    cudaLaunchKernelEx(&cfg, k_gs<0>, a);
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_gs<1>, a);
    cudaLaunchKernelEx(&cfg, k_gs<2>, a);
    cfg.gridDim = dim3((unsigned)std::min<int64_t>((a.n + kT - 1) / kT, 148 * 8), slots);
    cudaLaunchKernelEx(&cfg, k_gs_next, a, Vnext);
}

// ---- several right-hand sides ----------------------------------------------------------------
// One Krylov space per right-hand side, advanced in lock step so that the operator is applied to
// the whole block.  Slot b (blockIdx.y) owns basis vector i at V + i ldi + b ld; slots whose
// live[b] is 0 have left the current restart cycle and are skipped.  The same two-pass
// fixed-order reductions as above, so each slot's arithmetic does not depend on the others.

// nrm[b nstride] = ||w_b||; grid (kRedBlocks, slots) then (1, slots)
__global__ void __launch_bounds__(kT) k_norm_partial_b(const cplx* W, int64_t ld, int64_t n, const int* live,
                                                       double* part) {
    __shared__ double red[kT];
    const int b = blockIdx.y;
    if (live && !live[b]) return;
    const cplx* w = W + (size_t)b * ld;
    int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    int64_t lo = (int64_t)blockIdx.x * chunk;
    int64_t hi = min(n, lo + chunk);
    double s = 0.0;
    for (int64_t t = lo + threadIdx.x; t < hi; t += blockDim.x) s += w[t].x * w[t].x + w[t].y * w[t].y;
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = kT / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[(size_t)b * gridDim.x + blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(kT) k_norm_reduce_b(const double* part, const int* live, double* out,
                                                      int ostride) {
    __shared__ double red[kT];
    const int b = blockIdx.y;
    if (live && !live[b]) return;
    double s = 0.0;
    for (int q = threadIdx.x; q < kRedBlocks; q += blockDim.x) s += part[(size_t)b * kRedBlocks + q];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = kT / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[(size_t)b * ostride] = sqrt(red[0]);
}

// v_b = w_b / nrm[b nstride]
__global__ void k_scale_copy_b(const cplx* W, int64_t ldw, const double* nrm, int nstride, cplx* Vout, int64_t ldv,
                               int64_t n, const int* live) {
    const int b = blockIdx.y;
    if (live && !live[b]) return;
    const double r = nrm[(size_t)b * nstride];
    const double inv = (r != 0.0) ? 1.0 / r : 0.0;
    const cplx* w = W + (size_t)b * ldw;
    cplx* v = Vout + (size_t)b * ldv;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        v[t] = inv * w[t];
}

// r_b = b_b - (A x)_b
__global__ void k_sub_b(const cplx* Bv, const cplx* AX, cplx* Rv, int64_t ld, int64_t n) {
    const size_t o = (size_t)blockIdx.y * ld;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        Rv[o + t] = Bv[o + t] - AX[o + t];
}

// Start of a restart cycle for every slot: g = (beta, 0, ...), live = 1, kend = 0.
__global__ void k_init_cycle_b(cplx* g, int m1, const double* beta, int nslots, int* live, int* kend) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nslots) return;
    for (int i = 0; i < m1; ++i) g[(size_t)b * m1 + i] = mk(0, 0);
    g[(size_t)b * m1] = mk(beta[b], 0.0);
    live[b] = 1;
    kend[b] = 0;
}

// y_b = H_b^{-1} g_b over the slot's kend[b] columns (one warp per slot), then x_b += sum_i y_i V_i(b)
__global__ void __launch_bounds__(32) k_trisolve_b(const cplx* H, int m, const cplx* g, const int* kend, cplx* y) {
    const int b = blockIdx.x;
    trisolve(H + (size_t)b * (m + 1) * m, m, g + (size_t)b * (m + 1), kend[b], y + (size_t)b * (m + 1));
}

__global__ void k_update_x_b(cplx* X, int64_t ld, const cplx* V, int64_t ldi, const cplx* y, int ystride,
                             const int* kend, int64_t n) {
    __shared__ cplx ys[kMaxDots];
    const int b = blockIdx.y;
    const int k = kend[b];
    if (k == 0) return;
    for (int i = threadIdx.x; i < k; i += blockDim.x) ys[i] = y[(size_t)b * ystride + i];
    __syncthreads();
    cplx* x = X + (size_t)b * ld;
    const cplx* Vb = V + (size_t)b * ld;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        cplx acc = x[t];
#pragma unroll 8
        for (int i = 0; i < k; ++i) acc = acc + ys[i] * Vb[(size_t)i * ldi + t];
        x[t] = acc;
    }
}

}  // namespace foggy
