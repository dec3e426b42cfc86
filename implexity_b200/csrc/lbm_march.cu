// lbm_march.cu -- many steps of a small or middling grid in one launch.
//
// The staged kernels (lbm_forward.cu, lbm_adjoint.cu) run one step per launch.
// Below some 600 000 cells (a million in D3Q27) the step's own work is shorter
// than what a launch costs around it: the launch itself, the ring's set-up and
// first copies.  A 16-bit forward step gains at every size measured, up to 4.2M
// cells, for its ring costs more than direct loads.  Here one
// cooperative launch runs a whole run of passes: every thread owns its cells
// for the run, loads their streamed populations straight from L2 (19 or 27
// independent loads, the bounce-back slots selected by address, so that a
// wall costs no second trip), and a grid-wide barrier stands between passes.
// The mask, the resistance and, for one cell per thread, the running alpha
// cotangent stay in registers over the passes; the port maps stay in shared
// memory; the admission record of a pass is left as one partial per warp
// (written while the barrier fills) and combined by one kernel per run.
//
// What bounds it: the latency of one load-collide-store-barrier round on
// small grids, L2 bandwidth from some 10^5 cells on.
#include <algorithm>

#include "lbm_device.cuh"

// Compiled once per lattice and collision (LBM_PART) for the kernels, and once
// without it for the entry points.
namespace lbm {
cudaError_t march_forward_190(int storage, MarchFwdArgs& g, cudaStream_t s);
cudaError_t march_adjoint_190(int storage, MarchAdjArgs& g, cudaStream_t s);
cudaError_t march_forward_192(int storage, MarchFwdArgs& g, cudaStream_t s);
cudaError_t march_adjoint_192(int storage, MarchAdjArgs& g, cudaStream_t s);
cudaError_t march_forward_270(int storage, MarchFwdArgs& g, cudaStream_t s);
cudaError_t march_adjoint_270(int storage, MarchAdjArgs& g, cudaStream_t s);
cudaError_t march_forward_272(int storage, MarchFwdArgs& g, cudaStream_t s);
cudaError_t march_adjoint_272(int storage, MarchAdjArgs& g, cudaStream_t s);

#ifdef LBM_PART
namespace {

constexpr int MT = 256;  // threads per block (128 where a grid then still fits one block per SM)

// Neighbour offsets of one cell along each axis; a cell on a periodic face
// (MASK_WRAP) gets the wrapped ones.  Grids without periodic axes (WRAP = 0)
// have the same offsets in every cell: they stay in uniform registers.
struct Deltas {
    int32_t xm, xp, ym, yp, zm, zp;
};
template <int WRAP>
__device__ __forceinline__ Deltas deltas_of(const Geometry& G, uint32_t x, uint32_t m) {
    Deltas d{-(int32_t)G.sx, (int32_t)G.sx, -(int32_t)G.sy, (int32_t)G.sy, -1, 1};
    if (WRAP && (m & MASK_WRAP)) {
        const uint32_t ij = x / (uint32_t)G.nz, k = x - ij * (uint32_t)G.nz;
        const uint32_t i = ij / (uint32_t)G.ny, j = ij - i * (uint32_t)G.ny;
        if (i == 0) d.xm += (int32_t)G.n;
        if (i == (uint32_t)G.nx - 1) d.xp -= (int32_t)G.n;
        if (j == 0) d.ym += (int32_t)G.sx;
        if (j == (uint32_t)G.ny - 1) d.yp -= (int32_t)G.sx;
        if (k == 0) d.zm += (int32_t)G.sy;
        if (k == (uint32_t)G.nz - 1) d.zp -= (int32_t)G.sy;
    }
    return d;
}

// Slot the pull of direction q reads: pull_index (SIGN = -1) or
// pull_adj_index (SIGN = +1) without a branch.  A blocked link selects the
// own opposite slot, so the offsets of a closed face are never used.
template <int Q, int SIGN>
__device__ __forceinline__ uint32_t march_index(uint32_t n, uint32_t x, uint32_t m, const Deltas& d, int q) {
    using L = Lat<Q>;
    const int cx = SIGN * L::cx(q), cy = SIGN * L::cy(q), cz = SIGN * L::cz(q);
    int32_t o = 0;
    if (cx) o += cx > 0 ? d.xp : d.xm;
    if (cy) o += cy > 0 ? d.yp : d.ym;
    if (cz) o += cz > 0 ? d.zp : d.zm;
    const int link = SIGN < 0 ? q : opp<Q>(q);
    const uint32_t open = q * n + x + (uint32_t)o;
    return q && ((m >> link) & 1u) ? opp<Q>(q) * n + x : open;
}

// The slots are rewritten by other SMs during the launch: read at L2.
__device__ __forceinline__ float ldl2(const float* p) { return __ldcg(p); }
__device__ __forceinline__ __half ldl2(const __half* p) {
    return __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}
__device__ __forceinline__ __nv_bfloat16 ldl2(const __nv_bfloat16* p) {
    return __ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}

// Grid-wide barrier on a counter that is zero at the launch: every block adds
// one per pass, thread 0 waits until all blocks of pass `k` have.  The launch
// is cooperative, so every block is resident; the wait is bounded all the
// same, and a block that gives up leaves (the others then do too).
__device__ __forceinline__ void grid_arrive(unsigned* bar) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ __forceinline__ bool grid_wait(const unsigned* bar, unsigned target, int* err) {
    unsigned v;
    uint64_t t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if (v >= target) return true;
        if ((spin & 255u) == 255u) {
            const uint64_t t = global_ns();
            if (!t0) t0 = t;
            else if (t - t0 > kWaitNs) {
                atomicOr(err, 1);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void copy_ports(PortMap* to, const PortMap* from, int n) {
    const float* s = reinterpret_cast<const float*>(from);
    float* d = reinterpret_cast<float*>(to);
    for (int i = threadIdx.x; i < n * (int)(sizeof(PortMap) / 4); i += blockDim.x) d[i] = __ldg(s + i);
}

// ------------------------------------------------------------------ forward
template <int Q, int COLL, typename T, int RSP, int DP, int WRAP, int MB>
__global__ void __launch_bounds__(MT, MB) k_march_forward(const __grid_constant__ MarchFwdArgs g) {
    using L = Lat<Q>;
    constexpr int SC = Cvt<T>::scaled ? 1 : 0;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int go;
    PortMap* ports = reinterpret_cast<PortMap*>(smem);
    const FwdArgs& a = g.a;
    const uint32_t n = (uint32_t)a.G.n;
    const uint32_t stride = gridDim.x * blockDim.x, x0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool single = n <= stride;  // one cell per thread: its mask and alpha stay in registers
    const uint32_t warps = stride >> 5, warp = x0 >> 5;
    copy_ports(ports, a.ports, g.n_ports);
    __syncthreads();
    uint32_t m = 0;
    float alpha = 0.f;
    Deltas dl = deltas_of<0>(a.G, 0, 0);
    for (int pass = 0; pass < g.n_pass; ++pass) {
        const T* A = static_cast<const T*>(pass == 0 ? a.src : (pass & 1) ? a.dst : g.dst1);
        T* D = static_cast<T*>((pass & 1) ? g.dst1 : a.dst);
        const bool collide = !(g.inspect_last && pass == g.n_pass - 1);
        const bool apply = g.n_ports > 0 && (pass > 0 || a.apply_ports);
        float* const record = a.record ? a.record + (size_t)pass * g.record_stride : nullptr;
        DiagLocal acc;
        acc.init();
        double rsum[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (uint32_t x = x0; x < n; x += stride) {
            if (!single || pass == 0) {
                m = a.mask[x];
                alpha = a.alpha[x];
                if (WRAP) dl = deltas_of<WRAP>(a.G, x, m);
            }
            if (m & MASK_SOLID) {
                if constexpr (RSP) rsum[5] += (double)a.phi[x];
                continue;
            }
            T raw[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) raw[q] = ldl2(A + march_index<Q, -1>(n, x, m, dl, q));
            float v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] = sdec<T>(raw[q]);
            float exch = 0.f;
            if (apply && (m & MASK_PORT)) {
                if constexpr (SC) {  // the port maps act on g = f - w
#pragma unroll
                    for (int q = 0; q < Q; ++q) v[q] *= L::w(q);
                }
                const PortMap& pm = ports[((m >> MASK_PORT_SHIFT) & 7u) - 1];
                if (!pm.recon) {
                    exch = apply_port<Q>(pm, v);
                } else {  // regularized (an extrapolating port does not march)
                    float s0 = 0.f, s1 = 0.f;
#pragma unroll
                    for (int q = 0; q < Q; ++q) s0 += v[q];
                    regularized_apply<Q>(pm, v);
#pragma unroll
                    for (int q = 0; q < Q; ++q) s1 += v[q];
                    exch = s1 - s0;
                }
                if constexpr (SC) {
#pragma unroll
                    for (int q = 0; q < Q; ++q) v[q] *= (float)(1.0 / L::wd(q));
                }
            }
            const float mn = a.partial ? min_population<Q, SC>(v) : 0.f;
            float S[6];
            if (RSP || (record && a.record_s)) {
                float gg[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) gg[q] = SC ? L::w(q) * v[q] : v[q];
                second_moments<Q>(gg, S);
                if (record && a.record_s) {
#pragma unroll
                    for (int e = 0; e < 6; ++e) record[(size_t)(4 + e) * n + x] = S[e];
                }
            }
            float om = a.P.omega, omm = a.P.om;
            if (a.omega_cell) om = omm = a.omega_cell[x];
            Macro M;
            if constexpr (DP) M = collide_fused_dp<Q, COLL>(v, alpha, a.P, collide, om, omm);
            else M = collide_fused<Q, COLL, SC>(v, alpha, a.P, collide, om, omm);
            if (collide) store_own_pop<Q, T>(D, n, x, v, a.step + (uint32_t)pass);
            if constexpr (RSP) {
                float r6[6];
                response_cell<Q>(M.rp, M.u, S, alpha, a.sp, a.P, r6);
#pragma unroll
                for (int k = 0; k < 5; ++k) rsum[k] += (double)r6[k];
                rsum[5] += (double)a.phi[x];
                if (m & MASK_PORT) {
                    const float dpw = ports[((m >> MASK_PORT_SHIFT) & 7u) - 1].dp_weight;
                    rsum[6] += (double)(dpw * a.sp.dens * M.rp * a.sp.vel * a.sp.vel / 3.f);
                }
                rsum[7] += (double)r6[5];
            }
            if (a.partial) {
                acc.mass += M.rp;
                acc.exch += exch;
                acc.minf = fminf(acc.minf, mn);
                acc.maxu2 = fmaxf(acc.maxu2, M.u[0] * M.u[0] + M.u[1] * M.u[1] + M.u[2] * M.u[2]);
                if (!isfinite(M.rp)) acc.nf = 1;  // any non-finite population makes the density sum non-finite
            }
            if (record) {
                record[x] = M.rp;
                record[n + x] = M.u[0];
                record[2 * (size_t)n + x] = M.u[1];
                record[3 * (size_t)n + x] = M.u[2];
            }
        }
        const bool more = pass + 1 < g.n_pass;
        if (more) {
            __syncthreads();  // the block's stores are issued, its use of the port maps is over
            if (threadIdx.x == 0) grid_arrive(g.bar);
            if (g.port_stride) copy_ports(ports, a.ports + (size_t)(pass + 1) * g.port_stride, g.n_ports);
        }
        // the pass's record, while the barrier fills
        if (a.partial) store_partial(acc, a.partial + (size_t)pass * warps + warp);
        if constexpr (RSP) store_response_partial(rsum, a.rpartial + ((size_t)pass * warps + warp) * RESPONSE_PARTIAL);
        if (more) {
            if (threadIdx.x == 0) go = grid_wait(g.bar, (unsigned)(pass + 1) * gridDim.x, a.err);
            __syncthreads();
            if (!go) return;
        }
    }
}

// ------------------------------------------------------------------ adjoint
// A run of transposed steps (adj_one_cell of lbm_adjoint.cu, pass by pass):
// pass i is linearised at the record i slots before a.record.
template <int Q, int COLL, typename T, int STG, int WRAP, int MB>
__global__ void __launch_bounds__(MT, MB) k_march_adjoint(const __grid_constant__ MarchAdjArgs g) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int go;
    PortMap* ports = reinterpret_cast<PortMap*>(smem);
    const AdjArgs& a = g.a;
    const uint32_t n = (uint32_t)a.G.n;
    const uint32_t stride = gridDim.x * blockDim.x, x0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool single = n <= stride;
    copy_ports(ports, a.ports, g.n_ports);
    __syncthreads();
    double nsum = 0.0;
    uint32_t m = 0;
    float alpha = 0.f, ab_run = 0.f;
    Deltas dl = deltas_of<0>(a.G, 0, 0);
    for (int pass = 0; pass < g.n_pass; ++pass) {
        const T* B = static_cast<const T*>((pass & 1) ? a.dst : a.src);
        T* D = static_cast<T*>((pass & 1) ? const_cast<void*>(a.src) : a.dst);
        const float* rec = a.record - (size_t)pass * g.record_stride;
        const bool last = pass == g.n_pass - 1;
        const bool stage_on = STG && pass < g.stage_passes;
        const float in_inv = pass == 0 ? a.in_scale_inv : 1.f / a.out_scale;
        const float s_in = 1.f / in_inv, k_out = a.out_scale * in_inv;
        for (uint32_t x = x0; x < n; x += stride) {
            if (!single || pass == 0) {
                m = a.mask[x];
                alpha = a.alpha[x];
                if (WRAP) dl = deltas_of<WRAP>(a.G, x, m);
                ab_run = (m & MASK_SOLID) || (a.overwrite_abar && pass == 0) ? 0.f : a.abar[x];
            }
            if (m & MASK_SOLID) continue;
            T raw[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) raw[q] = ldl2(B + march_index<Q, 1>(n, x, m, dl, q));
            const float rp = rec[x];
            const float u[3] = {rec[n + x], rec[2 * (size_t)n + x], rec[3 * (size_t)n + x]};
            float v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] = Cvt<T>::to(raw[q]);
            float om = a.P.omega, omm = a.P.om;
            if (a.omega_cell) om = omm = a.omega_cell[x];
            const bool post = stage_on || (m & MASK_PORT);
            float ab = collide_vjp<Q, COLL, keeps_order<T>>(v, rp, u, alpha, a.P, om, omm, post ? 1.f : k_out) * in_inv;
            const PortMap* pm = (m & MASK_PORT) ? &ports[((m >> MASK_PORT_SHIFT) & 7u) - 1] : nullptr;
            if constexpr (STG) {
                if (stage_on) {
                    float Sm[6], fb[Q];
#pragma unroll
                    for (int e = 0; e < 6; ++e) Sm[e] = rec[(size_t)(4 + e) * n + x];
                    ab += response_vjp<Q, keeps_order<T>>(rp, u, Sm, alpha, pm ? pm->dp_weight : 0.f, pm != nullptr,
                                                          a.seed, a.P, fb);
#pragma unroll
                    for (int q = 0; q < Q; ++q) v[q] = fmaf(fb[q], s_in, v[q]);
                }
            }
            ab_run = fmaf(ab, a.abar_factor, ab_run);
            if (!single || last) a.abar[x] = ab_run;
            if (pm) {
                if (!pm->recon) {
                    port_transpose<Q>(*pm, v);
                } else {  // regularized, linearised at this cell's (rho, j / rho)
                    const float sc = 1.f + 0.5f * alpha;
                    const float um[3] = {u[0] * sc, u[1] * sc, u[2] * sc};
                    regularized_transpose<Q>(*pm, rp, um, v);
                }
            }
            if (post) {
#pragma unroll
                for (int q = 0; q < Q; ++q) v[q] *= k_out;
            }
            store_own_lam<Q, T>(D, n, x, v, 1.f);
            if (last && a.norm2) {
#pragma unroll
                for (int q = 0; q < Q; ++q) nsum += (double)v[q] * (double)v[q];
            }
        }
        if (!last) {
            __syncthreads();
            if (threadIdx.x == 0) grid_arrive(g.bar);
            if (g.port_stride) copy_ports(ports, a.ports - (size_t)(pass + 1) * g.port_stride, g.n_ports);
            if (threadIdx.x == 0) go = grid_wait(g.bar, (unsigned)(pass + 1) * gridDim.x, a.err);
            __syncthreads();
            if (!go) return;
        }
    }
    if (a.norm2) {
        Sums<1> sm;
        sm.init();
        sm.h[0] = nsum;
        finish_sums<1>(sm, a.norm2, a.red);
    }
}

// ------------------------------------------------------------------ launch
constexpr size_t PORT_SMEM = MAX_PORTS * sizeof(PortMap);

// Blocks per SM: two leave a thread 128 registers (no spills), three 80 (36 to
// 120 bytes spilled in D3Q19) but half as many threads again.  One round over
// the resident threads takes about 1.4 times as long with three, so they pay
// where they save enough rounds: us per FP32 forward step with two / three,
// 110 592 cells (2 rounds / 1) 5.8 / 5.3, 139 776 (2 / 2) 6.0 / 7.1, 262 144
// (4 / 3) 9.8 / 10.5, 614 400 (9 / 6) 24.2 / 21.5, 1 032 192 (14 / 10) 41.6 /
// 39.0; the adjoint alike.
inline bool three_blocks(int64_t n) {
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t two = (n + 2 * MT * sms - 1) / (2 * MT * sms), three = (n + 3 * MT * sms - 1) / (3 * MT * sms);
    return 7 * three < 5 * two;
}

struct MarchShape {
    int grid, threads;
};
// Threads: one cell each where the resident blocks allow it.  Up to one block
// of 128 per SM the smaller blocks spread a tiny grid over more SMs.
template <typename K>
MarchShape march_shape(K kernel, int64_t n) {
    const int one = persistent_grid((const void*)kernel, INT64_MAX / 2, PORT_SMEM, MT, MT);  // all resident blocks
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int threads = n <= (int64_t)sms * 128 ? 128 : MT;
    const int64_t blocks = (n + threads - 1) / threads;
    return {(int)(blocks < one ? blocks : one), threads};
}

template <typename K, typename A>
cudaError_t launch_cooperative(K kernel, const MarchShape& s, A& args, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(args.bar, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    void* p[] = {&args};
    e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(s.grid), dim3(s.threads), p, PORT_SMEM, st);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int Q, int COLL, typename T, int RSP, int DP>
cudaError_t run_march(MarchFwdArgs& g, cudaStream_t s) {
    void (*kernel)(const MarchFwdArgs) =
        g.a.G.periodic ? k_march_forward<Q, COLL, T, RSP, DP, 1, 2> : k_march_forward<Q, COLL, T, RSP, DP, 0, 2>;
    if constexpr (Q == 19 && !RSP && !DP)
        if (!g.a.G.periodic && three_blocks(g.a.G.n)) kernel = k_march_forward<Q, COLL, T, RSP, DP, 0, 3>;
    const MarchShape sh = march_shape(kernel, g.a.G.n);
    const uint32_t warps = (uint32_t)(sh.grid * sh.threads / 32);
    const int64_t per_pass = (int64_t)warps * ((g.diag ? sizeof(StepPartial) : 0) + (RSP ? RESPONSE_PARTIAL * sizeof(double) : 0));
    if (per_pass * g.n_pass > g.scratch_bytes) return cudaErrorInvalidValue;
    g.a.partial = g.diag ? static_cast<StepPartial*>(g.scratch) : nullptr;
    g.a.rpartial = RSP ? reinterpret_cast<double*>(static_cast<char*>(g.scratch) +
                                                   (g.diag ? (size_t)g.n_pass * warps * sizeof(StepPartial) : 0))
                       : nullptr;
    const cudaError_t e = launch_cooperative(kernel, sh, g, s);
    if (e != cudaSuccess || !per_pass) return e;
    return launch_reduce_partials(g.a.partial, g.a.rpartial, warps, warps, g.n_pass, g.diag, g.stage, s);
}

template <int Q, int COLL, typename T>
cudaError_t run_march_forward(MarchFwdArgs& g, cudaStream_t s) {
    if (g.a.dp_collision) {
        if constexpr (std::is_same<T, float>::value)
            return g.stage ? run_march<Q, COLL, T, 1, 1>(g, s) : run_march<Q, COLL, T, 0, 1>(g, s);
        else
            return cudaErrorInvalidValue;
    }
    return g.stage ? run_march<Q, COLL, T, 1, 0>(g, s) : run_march<Q, COLL, T, 0, 0>(g, s);
}

template <int Q, int COLL, typename T>
cudaError_t run_march_adjoint(MarchAdjArgs& g, cudaStream_t s) {
    void (*kernel)(const MarchAdjArgs) =
        g.a.rec_planes == 10
            ? (g.a.G.periodic ? k_march_adjoint<Q, COLL, T, 1, 1, 2> : k_march_adjoint<Q, COLL, T, 1, 0, 2>)
            : (g.a.G.periodic ? k_march_adjoint<Q, COLL, T, 0, 1, 2> : k_march_adjoint<Q, COLL, T, 0, 0, 2>);
    if constexpr (Q == 19)
        if (g.a.rec_planes != 10 && !g.a.G.periodic && three_blocks(g.a.G.n)) kernel = k_march_adjoint<Q, COLL, T, 0, 0, 3>;
    return launch_cooperative(kernel, march_shape(kernel, g.a.G.n), g, s);
}

}  // namespace

cudaError_t LBM_PART_NAME(march_forward)(int storage, MarchFwdArgs& g, cudaStream_t s) {
    LBM_STORAGE_DISPATCH(storage, T, return run_march_forward<LBM_PART / 10, LBM_PART % 10, T>(g, s))
    return cudaErrorInvalidValue;
}
cudaError_t LBM_PART_NAME(march_adjoint)(int storage, MarchAdjArgs& g, cudaStream_t s) {
    LBM_STORAGE_DISPATCH(storage, T, return run_march_adjoint<LBM_PART / 10, LBM_PART % 10, T>(g, s))
    return cudaErrorInvalidValue;
}
#else
namespace {
// One block per pass: the warps' partials combined in a fixed order.  Eight
// threads share a warp's response sums, one pair each: with a thread per warp
// and its eight sums one after the other, 64^3 runs spent 2.4 of 17.3 us a step
// here.
constexpr int REDUCE_THREADS = 512;
__global__ void __launch_bounds__(REDUCE_THREADS) k_reduce_partials(const StepPartial* part, const double* rpart,
                                                                    uint32_t warps, uint32_t stride, StepDiag* out,
                                                                    double* stage) {
    const size_t pass = blockIdx.x;
    if (out) {
        DiagAcc acc;
        acc.init();
        const double2* const p = reinterpret_cast<const double2*>(part + pass * stride);
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < warps; i += REDUCE_THREADS) {
            const double2 mass = p[3 * i], exch = p[3 * i + 1];
            const int4 rest = reinterpret_cast<const int4*>(p)[3 * i + 2];
            DiagAcc o;
            o.mh = mass.x;
            o.ml = mass.y;
            o.eh = exch.x;
            o.el = exch.y;
            o.minf = __int_as_float(rest.x);
            o.maxu2 = __int_as_float(rest.y);
            o.nf = rest.z;
            acc.merge(o);
        }
        acc = block_reduce(acc);
        if (threadIdx.x == 0) {
            StepDiag& d = out[pass];
            d.mass_hi = acc.mh;
            d.mass_lo = acc.ml;
            d.exch_hi = acc.eh;
            d.exch_lo = acc.el;
            d.min_f = acc.minf;
            d.max_u2 = acc.maxu2;
            d.nonfinite = acc.nf;
        }
    }
    if (stage) {
        __shared__ double2 sums[REDUCE_THREADS / 32][8];
        const uint32_t k = threadIdx.x & 7;
        const double2* p = reinterpret_cast<const double2*>(rpart + pass * stride * RESPONSE_PARTIAL);
        double h = 0.0, l = 0.0;
#pragma unroll 4
        for (uint32_t i = threadIdx.x >> 3; i < warps; i += REDUCE_THREADS / 8) {
            const double2 v = p[i * 8 + k];
            dd_add(h, l, v.x, v.y);
        }
#pragma unroll
        for (int off = 8; off < 32; off *= 2) {
            const double oh = __shfl_xor_sync(FULL, h, off), ol = __shfl_xor_sync(FULL, l, off);
            dd_add(h, l, oh, ol);
        }
        if ((threadIdx.x & 31) < 8) sums[threadIdx.x >> 5][k] = make_double2(h, l);
        __syncthreads();
        if (threadIdx.x < 8) {
            h = l = 0.0;
            for (int w = 0; w < REDUCE_THREADS / 32; ++w) dd_add(h, l, sums[w][k].x, sums[w][k].y);
            stage[pass * 16 + 2 * k] = h;
            stage[pass * 16 + 2 * k + 1] = l;
        }
    }
}

}  // namespace

int64_t pass_warps(int64_t n, int sms) {
    // eight (consumer) warps per 256 cells, at most 8 blocks per SM
    return std::min<int64_t>((n + 255) / 256 * 8, (int64_t)sms * 64);
}
int64_t march_scratch(int64_t n, int sms, bool stage) {
    return pass_warps(n, sms) * (int64_t)(sizeof(StepPartial) + (stage ? RESPONSE_PARTIAL * sizeof(double) : 0));
}

cudaError_t launch_reduce_partials(const StepPartial* part, const double* rpart, uint32_t warps, uint32_t stride,
                                   int passes, StepDiag* diag, double* stage, cudaStream_t s) {
    k_reduce_partials<<<passes, REDUCE_THREADS, 0, s>>>(part, rpart, warps, stride, diag, stage);
    return cudaGetLastError();
}

cudaError_t launch_march_forward(int Q, int coll, int storage, const MarchFwdArgs& g0, cudaStream_t s) {
    MarchFwdArgs g = g0;
    if (coll == CK_MRT || g.n_ports > MAX_PORTS || g.n_pass < 1) return cudaErrorInvalidValue;
    if (Q == 19) return coll == CK_MRT_BULK ? march_forward_192(storage, g, s) : march_forward_190(storage, g, s);
    return coll == CK_MRT_BULK ? march_forward_272(storage, g, s) : march_forward_270(storage, g, s);
}

cudaError_t launch_march_adjoint(int Q, int coll, int lstorage, const MarchAdjArgs& g0, cudaStream_t s) {
    MarchAdjArgs g = g0;
    if (coll == CK_MRT || g.n_ports > MAX_PORTS || g.n_pass < 1 || (g.a.rec_planes != 4 && g.a.rec_planes != 10))
        return cudaErrorInvalidValue;
    if (Q == 19) return coll == CK_MRT_BULK ? march_adjoint_192(lstorage, g, s) : march_adjoint_190(lstorage, g, s);
    return coll == CK_MRT_BULK ? march_adjoint_272(lstorage, g, s) : march_adjoint_270(lstorage, g, s);
}
#endif

}  // namespace lbm
