// nodes.cu -- the gradient of a Multipole's quintic tables carried back to its node tables.
//
// The table builder (prep_multipole.py) takes Phi_lm(r_i) and dPhi_lm/dr(r_i) to values f and
// log-r slopes m of each column (with log-scaling f_0 = log(inv - 1/Phi_0), f_c =
// Phi_c / Phi_0), solves a tridiagonal system A q = rhs(f, m) for the second derivatives, and
// forms six coefficients per interval.  Here the transpose of each step is applied in turn,
// a warp per column: lanes take intervals and nodes in parallel, the transposed solve is a
// forward and a backward sweep with the elimination factors (the same for all columns) formed
// once per block.  The work is small (a 91-column, 50-node table is 0.2 MB) and the launch is
// bound by latency, about two dependent passes over the nodes: 11 us, where the same chain as
// some 300 torch operations took 3.4 ms of host time.
#include <cuda_runtime.h>
#include "../../include/agb.h"
#include "agb_dev.cuh"
#include "launch.cuh"

#define NODE_WARPS 8
#define NODE_CONSTS AGB_MP_NCONST  // the builder's scalars, in the order of g_const
#define NODE_ENDS 6                // l=0 nodes they depend on: Phi_0 at 0, 1, n-2, n-1, then
                                   // dPhi_0/dr at 0, n-1

struct NodeArgs {
    int n, n_lm, log_scaling;
    double dlogr, inv;
    const double* poly;            // [n_lm][n-1][6] dL/d(coefficient)
    const double* r;               // [n] radial nodes
    const double* phi;             // [n][n_lm] node values
    const double* dphi;            // [n][n_lm] dPhi/dr
    const double* gconst;          // [8] or null
    double* gphi;                  // [n][n_lm] out; column 0 zeroed by the caller
    double* gdphi;
    double J[NODE_CONSTS][NODE_ENDS];
};

__device__ __forceinline__ double node_warp_sum(double v)
{
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// columns [c0, c1): the monopole's launch has c0 = 0, c1 = 1 and follows the others, which
// add their dependence on Phi_0 to column 0
__global__ void __launch_bounds__(32 * NODE_WARPS)
node_vjp_kernel(const __grid_constant__ NodeArgs a, int c0, int c1)
{
    extern __shared__ double sm[];
    const int n = a.n, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* ih = sm;               // 1 / (log r_{i+1} - log r_i)
    double* up = sm + n;           // A^T: elimination factors of the forward sweep
    double* piv = sm + 2 * n;      // and 1 / pivot
    double* gf = sm + 3 * n + wid * 3 * n;
    double* gm = gf + n;
    double* gq = gm + n;
    for (int i = threadIdx.x; i < n - 1; i += blockDim.x) ih[i] = 1.0 / (log(a.r[i + 1]) - log(a.r[i]));
    __syncthreads();
    // A^T[i][i-1] and A^T[i][i+1] (the end rows of A are one-sided)
    auto lower = [&](int i) { return i == 1 ? -2.0 * ih[0] : -ih[i - 1]; };
    auto upper = [&](int i) { return i == n - 2 ? -2.0 * ih[n - 2] : -ih[i]; };
    if (threadIdx.x == 0) {
        double w = 0.0;
        for (int i = 0; i < n; ++i) {
            double d = 3.0 * ((i > 0 ? ih[i - 1] : 0.0) + (i < n - 1 ? ih[i] : 0.0));
            if (i > 0) d -= lower(i) * w;
            piv[i] = 1.0 / d;
            w = i < n - 1 ? upper(i) * piv[i] : 0.0;
            up[i] = w;
        }
    }
    __syncthreads();
    const int c = c0 + blockIdx.x * NODE_WARPS + wid;
    if (c >= c1) return;
    const double h = a.dlogr, h2 = h * h;
    const double* G = a.poly + (long long)c * (n - 1) * 6;
    // the coefficients' transpose: node i from the intervals on both sides
    for (int i = lane; i < n; i += 32) {
        double f = 0.0, m = 0.0, q = 0.0;
        if (i < n - 1) {
            const double* g = G + 6 * i;
            f = g[0] - (10.0 * g[3] - 15.0 * g[4] + 6.0 * g[5]);
            m = h * (g[1] - 6.0 * g[3] + 8.0 * g[4] - 3.0 * g[5]);
            q = h2 * (0.5 * g[2] - 1.5 * g[3] + 1.5 * g[4] - 0.5 * g[5]);
        }
        if (i > 0) {
            const double* g = G + 6 * (i - 1);
            f += 10.0 * g[3] - 15.0 * g[4] + 6.0 * g[5];
            m += h * (-4.0 * g[3] + 7.0 * g[4] - 3.0 * g[5]);
            q += h2 * (0.5 * g[3] - g[4] + 0.5 * g[5]);
        }
        gf[i] = f;
        gm[i] = m;
        gq[i] = q;
    }
    __syncwarp();
    if (lane == 0) {               // A^T x = gq
        double v = 0.0;
        for (int i = 0; i < n; ++i) {
            v = (gq[i] - (i > 0 ? lower(i) * v : 0.0)) * piv[i];
            gq[i] = v;
        }
        for (int i = n - 2; i >= 0; --i) {
            v = gq[i] - up[i] * v;
            gq[i] = v;
        }
    }
    __syncwarp();
    // the right-hand side's transpose: row i of rhs has the terms of the intervals i-1 and i
    auto x = [&](int i) { return gq[i]; };
    double df[AGB_NODE_VJP_MAX / 32], dm[AGB_NODE_VJP_MAX / 32];
    #pragma unroll
    for (int t = 0; t < AGB_NODE_VJP_MAX / 32; ++t) {
        const int i = lane + 32 * t;
        df[t] = dm[t] = 0.0;
        if (i >= n) continue;
        // interval k = [k, k+1]: the weights of f_{k+1} - f_k, m_k and m_{k+1}
        auto terms = [&](int k, double& wf, double& wl, double& wr) {
            const double w = ih[k], w2 = w * w, w3 = w2 * w;
            wf = wl = wr = 0.0;
            if (k + 1 < n - 1) { wf -= 20.0 * w3 * x(k + 1); wr += 12.0 * w2 * x(k + 1); wl += 8.0 * w2 * x(k + 1); }
            else { wf -= 30.0 * w3 * x(k + 1); wl += 14.0 * w2 * x(k + 1); wr += 16.0 * w2 * x(k + 1); }
            if (k > 0) { wf += 20.0 * w3 * x(k); wl -= 12.0 * w2 * x(k); wr -= 8.0 * w2 * x(k); }
            else { wf += 30.0 * w3 * x(0); wr -= 14.0 * w2 * x(0); wl -= 16.0 * w2 * x(0); }
        };
        double wf, wl, wr;
        if (i < n - 1) {
            terms(i, wf, wl, wr);
            df[t] -= wf;
            dm[t] += wl;
        }
        if (i > 0) {
            terms(i - 1, wf, wl, wr);
            df[t] += wf;
            dm[t] += wr;
        }
    }
    double ginv = 0.0;
    #pragma unroll
    for (int t = 0; t < AGB_NODE_VJP_MAX / 32; ++t) {
        const int i = lane + 32 * t;
        if (i >= n) continue;
        const double F = gf[i] + df[t], M = gm[i] + dm[t], r = a.r[i];
        const long long at = (long long)i * a.n_lm + c, at0 = (long long)i * a.n_lm;
        if (!a.log_scaling) {
            a.gphi[at] = F;
            a.gdphi[at] = M * r;
            continue;
        }
        const double p0 = a.phi[at0], d0 = a.dphi[at0] * r;
        if (c > 0) {               // f = Phi / Phi_0, m = (Phi' - f Phi_0') / Phi_0
            const double ip = 1.0 / p0;
            const double f = a.phi[at] * ip, m = (a.dphi[at] * r - f * d0) * ip;
            a.gphi[at] = (F - M * d0 * ip) * ip;
            a.gdphi[at] = M * ip * r;
            atomicAdd(a.gphi + at0, (M * f * d0 * ip - F * f - M * m) * ip);
            atomicAdd(a.gdphi + at0, -M * f * ip * r);
        } else {                   // f = log(inv - 1/Phi_0), m = Phi_0' / (Phi_0 (inv Phi_0 - 1))
            // both differences cancel in a flat core: rounded as the builder rounds them
            const double e = __dadd_rn(a.inv, -(1.0 / p0));
            const double D = __dadd_rn(__dmul_rn(a.inv, p0), -1.0), q = __dmul_rn(p0, D);
            const double m = d0 / q, Mq = M / q;
            a.gphi[at] += F / (e * p0 * p0) - Mq * m * (D + p0 * a.inv);
            a.gdphi[at] += Mq * r;
            ginv += F / e - Mq * m * p0 * p0;
        }
    }
    if (c == 0 && a.gconst) {      // through the builder's scalars
        ginv = node_warp_sum(ginv);
        __syncwarp();
        if (lane < NODE_ENDS) {
            double g = 0.0;
            #pragma unroll
            for (int q = 0; q < NODE_CONSTS; ++q)
                g += a.J[q][lane] * (a.gconst[q] + (q == 0 && a.log_scaling ? ginv : 0.0));
            const int node = lane == 0 || lane == 4 ? 0 : lane == 1 ? 1 : lane == 2 ? n - 2 : n - 1;
            atomicAdd((lane < 4 ? a.gphi : a.gdphi) + (long long)node * a.n_lm, g);
        }
    }
}

extern "C" int agb_multipole_node_vjp(int n_nodes, int n_lm, int log_scaling, double dlogr,
                                      double inv, const double* g_poly, const double* r,
                                      const double* phi, const double* dphi,
                                      const double* g_const, const double* jacobian,
                                      double* g_phi, double* g_dphi, void* stream)
{
    if (n_nodes < 2 || n_nodes > AGB_NODE_VJP_MAX || n_lm < 1)
        return agb_set_error(AGB_ERR_ARG, "agb_multipole_node_vjp: 2 to 256 nodes and a column are needed");
    if (!g_poly || !r || !phi || !dphi || !g_phi || !g_dphi || (g_const && !jacobian))
        return agb_set_error(AGB_ERR_ARG, "agb_multipole_node_vjp: null argument");
    NodeArgs a;
    a.n = n_nodes; a.n_lm = n_lm; a.log_scaling = log_scaling;
    a.dlogr = dlogr; a.inv = inv;
    a.poly = g_poly; a.r = r; a.phi = phi; a.dphi = dphi; a.gconst = g_const;
    a.gphi = g_phi; a.gdphi = g_dphi;
    for (int q = 0; q < NODE_CONSTS; ++q)
        for (int e = 0; e < NODE_ENDS; ++e) a.J[q][e] = g_const ? jacobian[q * NODE_ENDS + e] : 0.0;
    cudaStream_t st = (cudaStream_t)stream;
    // at most 54 KB
    const size_t smem = sizeof(double) * 3 * (size_t)n_nodes * (1 + NODE_WARPS);
    static std::atomic<unsigned long long> set{0};      // one bit per device
    const unsigned long long bit = 1ull << current_device();
    if (!(set.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(node_vjp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(double) * 3 * AGB_NODE_VJP_MAX * (1 + NODE_WARPS));
        set.fetch_or(bit, std::memory_order_release);
    }
    if (n_lm > 1) {
        node_vjp_kernel<<<(n_lm - 1 + NODE_WARPS - 1) / NODE_WARPS, 32 * NODE_WARPS, smem, st>>>(a, 1, n_lm);
        const int rc = agb_check_launch("node_vjp_kernel");
        if (rc) return rc;
    }
    node_vjp_kernel<<<1, 32 * NODE_WARPS, smem, st>>>(a, 0, 1);
    return agb_check_launch("node_vjp_kernel");
}
