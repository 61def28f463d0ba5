// split.cu -- the kernel for calls too small to fill the GPU with one thread per point.
#include "eval_point.cuh"
#include "launch.cuh"
#include "mp_split.cuh"

// A few points per block, the harmonics split over its warps (mp_split.cuh): calls too small
// to fill the GPU with one thread per point.  Block b evaluates the tile of a.chunk <= 32
// points from b * a.chunk on.  Dynamic shared memory: two buffers of a.split_buf bytes with the
// |m| groups' shares of the sums [m][sum][point] (Hessians: their columns), then every leaf's
// results [leaf][value][point].
template <int MODE, typename R, bool DYN>
__global__ void __launch_bounds__(split_threads(MODE), 1)
agb_split_kernel(const __grid_constant__ EvalArgs a)
{
    constexpr bool VJP = MODE == AGB_MODE_VJP || MODE == AGB_MODE_VJPF;
    constexpr int CM = VJP ? AGB_MODE_HESS : MODE;
    constexpr int NO = split_out(CM);
    constexpr bool HESS = CM == AGB_MODE_HESS;
    extern __shared__ __align__(16) char split_smem[];
    __shared__ DevLeaf dyn_leaves[DYN ? AGB_MAX_LEAVES : 1];
    if (DYN) {
        for (int q = threadIdx.x; q < a.n_leaves; q += blockDim.x) dyn_leaves[q] = a.dleaves[q];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, S = blockDim.x >> 5;
    const int T = (int)a.chunk;
    const long long pos = (long long)blockIdx.x * T + lane;
    const bool live = lane < T && pos < a.n;
    double* res = reinterpret_cast<double*>(split_smem + 2 * a.split_buf);
    double x = 0.0, y = 0.0, z = 0.0;
    if (live) {
        if (a.soa) {
            x = a.x[pos]; y = a.y[pos]; z = a.z[pos];
        } else {
            x = a.xyz[3 * pos]; y = a.xyz[3 * pos + 1]; z = a.xyz[3 * pos + 2];
        }
    }
    int turn = 0, other = 0;            // leaves walked so far, other leaves so far
    for (int L = 0; L < a.n_leaves; ++L) {
        const DevLeaf& lf = DYN ? dyn_leaves[L] : a.leaves[L];
        if (lf.ampl == 0.0) continue;
        const DevComp& c = a.comps[lf.comp];
        const double lx = lf.sigma * x - lf.g0;
        const double ly = lf.sigma * y - lf.g1;
        const double lz = lf.sigma * z - lf.g2;
        const bool walked = c.kind == AGB_KIND_MULTIPOLE && c.structure != AGB_STRUCT_LIST;
        bool mine, grid = false;
        int k = 0;
        double s = 0.0, inv_r = 0.0, Rc = 0.0, cth = 1.0, sth = 0.0, cph = 1.0, sph = 0.0;
        char* buf = split_smem + (turn & 1) * a.split_buf;
        double* sums = reinterpret_cast<double*>(buf) + lane;
        R* cols = reinterpret_cast<R*>(buf) + lane;
        if (walked) {
            if (live) {
                const double r = sqrt(lx * lx + ly * ly + lz * lz);
                grid = mp_place(c, r, k, s);
                if (grid) {
                    Rc = sqrt(lx * lx + ly * ly);
                    inv_r = 1.0 / r;
                    cth = lz * inv_r;
                    sth = Rc * inv_r;
                    cph = (Rc > 1.0e-300) ? lx / Rc : 1.0;
                    sph = (Rc > 1.0e-300) ? ly / Rc : 0.0;
                    void* out = HESS ? (void*)cols : (void*)sums;
                    if (c.structure == AGB_STRUCT_EVEN)
                        mp_split_walk<CM, R, 2>(c, k, s, cth, sth, cph, sph, w, S, out, T);
                    else
                        mp_split_walk<CM, R, 1>(c, k, s, cth, sth, cph, sph, w, S, out, T);
                }
            }
            __syncthreads();
            mine = w == turn % S;
            ++turn;
        } else {
            mine = w == S - 1 - other % S;
            ++other;
        }
        if (!mine || !live) continue;
        PointOut o;
        o.phi = 0.0; o.rho = 0.0;
        o.g[0] = o.g[1] = o.g[2] = 0.0;
        #pragma unroll
        for (int q = 0; q < 6; ++q) o.h[q] = 0.0;
        if (grid) {
            MPSums t = {};
            if (HESS) {
                if (c.structure == AGB_STRUCT_EVEN)
                    mp_split_hess<R, 2>(c.lmax, cth, sth, cph, sph, cols, T, t);
                else
                    mp_split_hess<R, 1>(c.lmax, cth, sth, cph, sph, cols, T, t);
            } else {
                mp_split_total<CM>(c.lmax, sums, T, t);
            }
            mp_close<CM>(c, k, s, t, lx, ly, lz, inv_r, Rc, cth, sth, cph, sph, o);
        } else {
            eval_component<CM, R, VJP>(c, lx, ly, lz, o);
        }
        double* d = res + (long long)L * NO * T + lane;
        if (CM == AGB_MODE_DENS) {
            d[0] = o.rho;
        } else {
            d[0] = o.phi;
            if (CM != AGB_MODE_POT) { d[T] = o.g[0]; d[2 * T] = o.g[1]; d[3 * T] = o.g[2]; }
            if (CM == AGB_MODE_HESS) {
                #pragma unroll
                for (int q = 0; q < 6; ++q) d[(4 + q) * T] = o.h[q];
            }
        }
    }
    __syncthreads();
    if (w != 0 || !live) return;
    // the leaves in order, as agb_eval_kernel adds them
    double phi = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0, rho = 0.0;
    double h[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int L = 0; L < a.n_leaves; ++L) {
        const DevLeaf& lf = DYN ? dyn_leaves[L] : a.leaves[L];
        if (lf.ampl == 0.0) continue;
        const double* d = res + (long long)L * NO * T + lane;
        const double A = lf.ampl;
        if (CM == AGB_MODE_DENS) {
            rho += (A * lf.sigma * lf.sigma) * d[0];
            continue;
        }
        phi += A * d[0];
        if (CM != AGB_MODE_POT) {
            const double As = A * lf.sigma;
            g0 += As * d[T]; g1 += As * d[2 * T]; g2 += As * d[3 * T];
            if (CM == AGB_MODE_HESS) {
                const double As2 = As * lf.sigma;
                #pragma unroll
                for (int q = 0; q < 6; ++q) h[q] += As2 * d[(4 + q) * T];
            }
        }
    }
    eval_write<MODE>(a, pos, a.perm ? (long long)a.perm[pos] : pos, phi, g0, g1, g2, h, rho);
}

// dynamic shared memory of a block: lmax 32 with Hessians in FP64 needs 203 KB of columns, and
// 10 KB per four leaves of results (larger trees take one thread per point there)
#define AGB_SPLIT_SMEM (220 * 1024)

// Estimated time of an SM that evaluates `tiles` tiles with S warps each (S = 1: one thread
// per point), `cap` tiles at a time: per wave of resident warps the steps of a warp, each as
// long as the latency of one step (lat) or as the warps keep the pipe busy, and the tile's
// finish, in units of one warp's pipe time per step.
static long long split_cost(long long tiles, int S, long long cap, long long steps, int lat,
                            int finish)
{
    const long long full = tiles / cap, rest = tiles % cap;
    auto wave = [&](long long n) { return steps * std::max<long long>(lat, n * S) + finish; };
    return full * wave(cap) + (rest ? wave(rest) : 0);
}

// The split kernel's shape for this call: S warps per tile of T points; false where one
// thread per point is the better one (or the tree has no Multipole to split).
//
// T spreads the points over the SMs, at most 32 to a tile.  S comes from the estimate above:
// an SM holds 16 warps at 128 registers (8 at 255, the Hessian modes), a step's latency is
// about the pipe time of 11 warps (6), and finishing a leaf of a tile costs about 60 steps of
// one warp (twice that with Hessians).
// Measured (Multipole alone, FP64 force, one thread per point -> split): lmax 32 10k points
// 119 -> 45 us (S = 5), 20k 119 -> 73 (S = 3), 40k 167 -> 138 (S = 3), 100k 331 -> 290
// (S = 2), 300k 661 -> 768; lmax 16 40k 50 -> 46, 100k 96 -> 90; lmax 8 10k 15.5 -> 9.1,
// 20k 15.7 -> 11.5; lmax 4 40k 9.9 -> 12.4; the galaxy tree (lmax 16) with Hessians at 1000
// points 39 -> 11; the Milky Way tree (lmax 32) at 1000 points 187 -> 24.
template <int MODE, typename R>
static bool split_shape(EvalArgs& a, int& S, int& T, size_t& smem)
{
    constexpr int CM = (MODE == AGB_MODE_VJP || MODE == AGB_MODE_VJPF) ? AGB_MODE_HESS : MODE;
    constexpr int warps = split_threads(MODE) / 32;
    if (a.out_flags & AGB_OUT_SHAPE_BITS) return false;        // the caller's launch shape
    const long long sms = num_sms();
    if (a.n > sms * 32 * 22) return false;
    // the heaviest Multipole stands for the tree (device-time leaves may pick any of the
    // components)
    int lmax = 0;
    long long steps = 0;                // (l, |m|) pairs of its walk
    for (const DevComp& c : a.comps) {
        if (c.kind != AGB_KIND_MULTIPOLE || c.structure == AGB_STRUCT_LIST) continue;
        const long long h = c.lmax / 2 + 1, l1 = c.lmax + 1;
        lmax = std::max(lmax, c.lmax);
        steps = std::max(steps, c.structure == AGB_STRUCT_EVEN ? h * h : l1 * (l1 + 1) / 2);
    }
    if (lmax < 2) return false;
    T = (int)std::min<long long>(32, (a.n + sms - 1) / sms);
    const long long tiles = ((a.n + T - 1) / T + sms - 1) / sms;     // of an SM
    const int V = lmax / 2 + 1;
    a.split_buf = T * (lmax + 1) * (CM == AGB_MODE_HESS ? AGB_SPLIT_HESS_COLS * (int)sizeof(R)
                                                        : split_sums(CM) * (int)sizeof(double));
    a.split_buf = (a.split_buf + 15) & ~15;
    // tiles that fit an SM's shared memory, with the results of eight leaves
    const int fit = AGB_SPLIT_SMEM / (2 * a.split_buf + 8 * split_out(CM) * T * (int)sizeof(double));
    const int lat = warps == 16 ? 11 : 6;
    long long best = split_cost(tiles, S = 1, warps, steps, lat, 0);
    for (int s = 2; s <= std::min(warps, V); ++s) {
        const int cap = std::max(1, std::min(warps / s, fit));
        const long long t = split_cost(tiles, s, cap, steps * ((V + s - 1) / s) / V, lat,
                                       CM == AGB_MODE_HESS ? 120 : 60);
        if (t < best) {
            best = t;
            S = s;
        }
    }
    smem = 2 * (size_t)a.split_buf + sizeof(double) * T * (size_t)a.n_leaves * split_out(CM);
    return S >= 2 && smem <= AGB_SPLIT_SMEM;
}

template <int MODE, typename R, bool DYN>
static void launch_split(EvalArgs& a, int S, int T, size_t smem, cudaStream_t st)
{
    static std::atomic<unsigned long long> set{0};      // one bit per device
    const unsigned long long bit = 1ull << current_device();
    if (!(set.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(agb_split_kernel<MODE, R, DYN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             AGB_SPLIT_SMEM);
        set.fetch_or(bit, std::memory_order_release);
    }
    a.chunk = T;
    agb_split_kernel<MODE, R, DYN><<<(int)((a.n + T - 1) / T), 32 * S, smem, st>>>(a);
}

template <int MODE, typename R>
static bool try_split(EvalArgs& a, cudaStream_t st)
{
    int S, T;
    size_t smem;
    if (!split_shape<MODE, R>(a, S, T, smem)) return false;
    if constexpr (MODE != AGB_MODE_VJP && MODE != AGB_MODE_VJPF)
        if (a.dleaves) {
            launch_split<MODE, R, true>(a, S, T, smem, st);
            return true;
        }
    launch_split<MODE, R, false>(a, S, T, smem, st);
    return true;
}

bool agb_launch_split(int mode, bool mixed, EvalArgs& a, cudaStream_t st)
{
    switch (mode) {
    case AGB_MODE_POT:  return mixed ? try_split<AGB_MODE_POT, float>(a, st) : try_split<AGB_MODE_POT, double>(a, st);
    case AGB_MODE_GRAD: return mixed ? try_split<AGB_MODE_GRAD, float>(a, st) : try_split<AGB_MODE_GRAD, double>(a, st);
    case AGB_MODE_HESS: return mixed ? try_split<AGB_MODE_HESS, float>(a, st) : try_split<AGB_MODE_HESS, double>(a, st);
    case AGB_MODE_DENS: return mixed ? try_split<AGB_MODE_DENS, float>(a, st) : try_split<AGB_MODE_DENS, double>(a, st);
    case AGB_MODE_VJP:  return mixed ? try_split<AGB_MODE_VJP, float>(a, st) : try_split<AGB_MODE_VJP, double>(a, st);
    case AGB_MODE_VJPF: return mixed ? try_split<AGB_MODE_VJPF, float>(a, st) : try_split<AGB_MODE_VJPF, double>(a, st);
    default: return false;
    }
}
