// split.cu -- the kernel for calls too small to fill the GPU with one thread per point.
#include <cmath>
#include "eval_point.cuh"
#include "launch.cuh"
#include "mp_split.cuh"

// A few points per block, the harmonics split over its warps (mp_split.cuh): calls too small
// to fill the GPU with one thread per point.  Block b evaluates the tile of a.chunk <= 32
// points from b * a.chunk on.  Dynamic shared memory: every leaf's results [leaf][value][point],
// then a buffer of a.split_buf bytes with the |m| groups' shares of the sums [m][sum][point]
// (Hessians: their columns), and another one where several leaves are walked.
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
    double* res = reinterpret_cast<double*>(split_smem);
    char* bufs = split_smem + split_results(CM, T, a.n_leaves);
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
        char* buf = bufs + (turn & 1) * a.split_buf;
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

// dynamic shared memory of a block: two leaves of lmax 32 with Hessians in FP64 need 203 KB of
// columns, and 2.5 KB per leaf of results (larger trees take one thread per point there)
#define AGB_SPLIT_SMEM (220 * 1024)

// What a call's leaves cost a warp, in units of the latency of one (l, |m|) step.
struct SplitWork {
    double steps = 0.0;            // of the regular Multipoles, which the warps share
    int walked = 0;                // how many of them
    int groups = 0;                // and their |m| groups
    int lmax = 0;                  // most of any component, in use or (device-time leaves) not yet
    double columns = 0.0;          // of the other Multipoles,
    double harmonics = 0.0;        // of the CylSplines: one warp each
    int analytic = 0;
};

static SplitWork split_work(const EvalArgs& a)
{
    SplitWork t;
    for (const DevComp& c : a.comps)
        if (c.kind == AGB_KIND_MULTIPOLE && c.structure != AGB_STRUCT_LIST) t.lmax = std::max(t.lmax, c.lmax);
    for (int L = 0; L < a.n_leaves; ++L) {
        if (a.leaves[L].ampl == 0.0) continue;
        const DevComp& c = a.comps[a.leaves[L].comp];
        const int h = c.lmax / 2 + 1, l1 = c.lmax + 1;
        if (c.kind == AGB_KIND_CYLSPLINE) {
            t.harmonics += c.n_lm;
        } else if (c.kind != AGB_KIND_MULTIPOLE) {
            ++t.analytic;
        } else if (c.structure == AGB_STRUCT_LIST) {
            t.columns += c.n_lm;
        } else {
            ++t.walked;
            t.groups += l1;
            t.steps += c.structure == AGB_STRUCT_EVEN ? h * h : l1 * (l1 + 1) / 2;
        }
    }
    return t;
}

// Constants of the estimate below, in the same unit (0.25-0.35 us in FP64, 0.17-0.25 mixed).
struct SplitRates {
    double pipe, rows;             // a step's pipe time with broadcast records, and with a row per
                                   // lane (unsorted points, in proportion to the tile's lanes)
    double finish, group;          // finishing a walked leaf: its end and barrier, and per group
    double unsorted, mixed;        // factors of these: unsorted steps are longer, mixed ones shorter
    double analytic, analytic_pipe;
    double harmonic, harmonic_pipe;
    double margin;                 // a split has to be better by this
    double overlap;                // of the rounding up to whole waves, what tiles that end at
                                   // different times save
};

// Estimated time of an SM that evaluates `tiles` tiles of T points with S warps each (S = 1:
// one thread per point), `cap` tiles at a time: per wave of resident warps the steps of a warp,
// whose latency and whose share of the pipe's time add in quadrature, the finish of each leaf,
// and the other leaves, which the tile's warps take in turn.
static double split_time(const SplitWork& t, const SplitRates& r, long long tiles, int T, int S,
                         long long cap, bool sorted, bool mixed)
{
    const double pipe = sorted ? r.pipe : r.pipe + (r.rows - r.pipe) * T / 32;
    auto hypot2 = [](double a, double b) { return std::sqrt(a * a + b * b); };
    auto wave = [&](double k) {
        double x = t.steps / S * hypot2(1.0, k * S * pipe);
        if (S > 1)
            x += (t.walked * r.finish + t.groups * r.group) * (sorted ? 1.0 : r.unsorted) * (mixed ? r.mixed : 1.0);
        x += (double)t.analytic / S * hypot2(r.analytic, k * S * r.analytic_pipe);
        x += t.harmonics * hypot2(r.harmonic, k * r.harmonic_pipe);
        return x + t.columns * std::max(0.3, k * 0.06);
    };
    const long long full = tiles / cap, rest = tiles % cap;
    if (S == 1) return full * wave((double)cap) + (rest ? wave((double)rest) : 0.0);
    const double exact = std::max(1.0, (double)tiles / cap), whole = (double)(full + (rest ? 1 : 0));
    const double free = r.overlap * (1.0 - 1.0 / cap);
    return wave((double)std::min(tiles, cap)) * (exact * free + whole * (1.0 - free)) * r.margin;
}

// The split kernel's shape for this call: S warps per tile of T points; false where one
// thread per point is the better one (or the tree has no Multipole to split).
//
// T spreads the points over the SMs, at most 32 to a tile.  S comes from the estimate above,
// with the warps that an SM holds (16 at 128 registers, 8 at 255 with Hessians) and the tiles
// that fit its shared memory.  The rates are fitted to 26 trees (lmax 2 to 32, one to eight
// Multipoles, regular or not, with CylSplines and up to 20 analytic leaves), up to 26 sizes from
// 300 to 400003 points, four modes, both precisions, sorted and not, each with S = 1 to 16 (in
// steps of a third or less): over those 4768 calls the shape taken is 2 % (geometric mean) from
// the best one tried, and slower than one thread per point on points sorted from 16384 on by
// more than 5 % in 31 (up to 22 %: 20 analytic leaves with Hessians).  Forces, one thread per
// point -> split, us: lmax 8 FP64 1000 points 17 -> 9, 10007 17 -> 11, 24000 17 -> 15, 40009 20
// (not split); lmax 32 FP64 10007 89 -> 33, 40009 100 -> 78, mixed 58 -> 29, 69 -> 64; lmax 16
// with 20 analytic leaves, mixed, 100003 84 (not split; two warps a tile take 156).
template <int MODE, typename R>
static bool split_shape(EvalArgs& a, int& S, int& T, size_t& smem)
{
    constexpr int CM = (MODE == AGB_MODE_VJP || MODE == AGB_MODE_VJPF) ? AGB_MODE_HESS : MODE;
    constexpr bool HESS = CM == AGB_MODE_HESS;
    constexpr bool mixed = std::is_same<R, float>::value;
    constexpr int warps = split_threads(MODE) / 32;
    static constexpr SplitRates rates = HESS
        ? SplitRates{0.06, 0.23, 4.0, 0.7, 0.38, 1.4, 0.66, 2.8, 1.35, 0.32, 1.068, 0.3}
        : SplitRates{0.066, 0.1, 3.5, 0.35, 0.55, 1.5, 0.5, 1.2, 2.5, 0.36, 1.025, 0.5};
    if (a.out_flags & AGB_OUT_SHAPE_BITS) return false;        // the caller's launch shape
    const SplitWork work = split_work(a);
    if (work.lmax < 2 || !work.walked) return false;
    const long long sms = num_sms();
    T = (int)std::min<long long>(32, (a.n + sms - 1) / sms);
    a.split_buf = T * (work.lmax + 1) * (HESS ? AGB_SPLIT_HESS_COLS * (int)sizeof(R)
                                              : split_sums(CM) * (int)sizeof(double));
    a.split_buf = (a.split_buf + 15) & ~15;
    // leaves from the device may be walked or not, as their component at that time is
    const int buffers = work.walked > 1 || a.dleaves ? 2 : 1;
    smem = buffers * (size_t)a.split_buf + split_results(CM, T, a.n_leaves);
    if (smem > AGB_SPLIT_SMEM) return false;
    const int fit = std::max(1, 228 * 1024 / ((int)smem + 1024));
    auto per_sm = [&](long long tile) { return ((a.n + tile - 1) / tile + sms - 1) / sms; };
    const bool sorted = a.perm || a.stage;
    double best = split_time(work, rates, per_sm(32), 32, S = 1, warps, sorted, mixed);
    for (const int s : {2, 3, 4, 5, 6, 8, 11, 16}) {
        if (s > std::min(warps, work.lmax / 2 + 1)) break;
        const double t = split_time(work, rates, per_sm(T), T, s, std::max(1, std::min(warps / s, fit)),
                                    sorted, mixed);
        if (t < best) {
            best = t;
            S = s;
        }
    }
    return S >= 2;
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
