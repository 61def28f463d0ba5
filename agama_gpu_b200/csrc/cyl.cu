// cyl.cu -- evaluation of trees whose expansions are CylSplines (with any analytic leaves).
//
// Points of a disk are in no useful order, so a warp's lanes need records of up to 32 cells,
// and the record of a (cell, harmonic) is one 128-byte line.  A lane that loads its own record
// asks for 16 bytes of 32 different lines at a time: 256 L1 wavefronts per harmonic and warp,
// 194 of the 285 us of a 1M-point force call (7 harmonics).  Here the warp loads the 32 records
// together, consecutive lanes consecutive 16 bytes of a record, into shared memory, from where
// each lane reads its own: 32 + 32 + 32 wavefronts.  The next harmonic's loads are in flight while this one is
// evaluated.  Rows in shared memory are an odd number of 16-byte words apart, so that
// neither the writes (a record by consecutive lanes) nor the reads (one word of 32 rows)
// conflict.
#include "eval_point.cuh"
#include "launch.cuh"

// 128 threads, 12 warps an SM at 168 registers for forces (141 us at 1M points; 16 warps at 128
// registers spill 352 bytes, 148-152 us; 20 warps 196 us), 8 at 255 with second derivatives,
// one wave of blocks (two: 142 us and 187 against 182 us with Hessians).  Against a lane loading
// its own record: force 281 -> 141 us, Hessian 490 -> 182, potential 215 -> 112 at 1M points.
#define AGB_CYL_BLOCK 128
__host__ __device__ constexpr int cyl_min_blocks(int mode)
{
    return mode == AGB_MODE_POT ? 4 : mode == AGB_MODE_GRAD ? 3 : 2;
}

#define AGB_CYL_WORDS 8            // 16-byte words of a record
#define AGB_CYL_ROW 9              // and of its row in shared memory

// The records of a warp's 32 cells, harmonic after harmonic (rec64 with h = 0, 1, ... by all
// lanes together).
struct CSWarp {
    const double2* table;         // the component's records, n_lm consecutive ones per cell
    double2* rows;                // this warp's rows in shared memory
    int lane, n_lm;
    mutable double2 next[AGB_CYL_WORDS];       // this lane's words of the next harmonic's records
    int word[AGB_CYL_WORDS];                   // and where they are for h = 0

    __device__ __forceinline__ CSWarp(const DevComp& c, int cell, double2* smem)
        : table(reinterpret_cast<const double2*>(c.table)), rows(smem), lane(threadIdx.x & 31),
          n_lm(c.n_lm)
    {
        #pragma unroll
        for (int j = 0; j < AGB_CYL_WORDS; ++j) {
            const int i = j * 32 + lane;
            word[j] = __shfl_sync(0xffffffffu, cell, i / AGB_CYL_WORDS) * n_lm * AGB_CYL_WORDS + i % AGB_CYL_WORDS;
        }
        fetch(0);
    }
    __device__ __forceinline__ void fetch(int h) const
    {
        #pragma unroll
        for (int j = 0; j < AGB_CYL_WORDS; ++j) next[j] = __ldg(table + word[j] + h * AGB_CYL_WORDS);
    }
    // harmonic h's records into the rows, the loads of h + 1 on their way, then this lane's row
    __device__ __forceinline__ void rec64(int h, double v[16]) const
    {
        __syncwarp();
        #pragma unroll
        for (int j = 0; j < AGB_CYL_WORDS; ++j) {
            const int i = j * 32 + lane;
            rows[(i / AGB_CYL_WORDS) * AGB_CYL_ROW + i % AGB_CYL_WORDS] = next[j];
        }
        __syncwarp();
        if (h + 1 < n_lm) fetch(h + 1);
        #pragma unroll
        for (int q = 0; q < AGB_CYL_WORDS; ++q) {
            const double2 w = rows[lane * AGB_CYL_ROW + q];
            v[2 * q] = w.x; v[2 * q + 1] = w.y;
        }
    }
};

template <int MODE, bool DYN>
__global__ void __launch_bounds__(AGB_CYL_BLOCK, cyl_min_blocks(MODE))
agb_cyl_kernel(const __grid_constant__ EvalArgs a)
{
    __shared__ DevLeaf dyn_leaves[DYN ? AGB_MAX_LEAVES : 1];
    __shared__ double2 rows[AGB_CYL_BLOCK * AGB_CYL_ROW];
    if (DYN) {
        for (int q = threadIdx.x; q < a.n_leaves; q += blockDim.x) dyn_leaves[q] = a.dleaves[q];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const long long lo = (long long)blockIdx.x * a.chunk;
    const long long hi = lo + a.chunk < a.n ? lo + a.chunk : a.n;
    // every lane of a warp makes the same number of passes
    for (long long first = lo + threadIdx.x - lane; first < hi; first += blockDim.x) {
        const long long pos = first + lane;
        const bool live = pos < hi;
        const long long at = live ? pos : hi - 1;
        const double x = a.xyz[3 * at], y = a.xyz[3 * at + 1], z = a.xyz[3 * at + 2];
        double phi = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0;
        double h[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int L = 0; L < a.n_leaves; ++L) {
            const DevLeaf& lf = DYN ? dyn_leaves[L] : a.leaves[L];
            if (lf.ampl == 0.0) continue;
            const DevComp& c = a.comps[lf.comp];
            const double lx = lf.sigma * x - lf.g0;
            const double ly = lf.sigma * y - lf.g1;
            const double lz = lf.sigma * z - lf.g2;
            PointOut o;
            o.phi = 0.0; o.rho = 0.0;
            o.g[0] = o.g[1] = o.g[2] = 0.0;
            #pragma unroll
            for (int q = 0; q < 6; ++q) o.h[q] = 0.0;
            if (c.kind == AGB_KIND_CYLSPLINE) {
                CSPlace q;
                const bool in = cs_place(c, lx, ly, lz, q);
                if (!in) {                  // a lane beyond the grid takes part with cell 0
                    q.iR = q.iz = 0;
                    q.tR = q.tz = 0.0;
                    q.hR = q.hz = 1.0;
                    q.R_at_hi = q.z_at_hi = false;
                }
                if (__any_sync(0xffffffffu, in)) {
                    const double cph = (q.R > 0.0) ? lx / q.R : 1.0;
                    const double sph = (q.R > 0.0) ? ly / q.R : 0.0;
                    CSSums s;
                    double2* mine = rows + (threadIdx.x >> 5) * 32 * AGB_CYL_ROW;
                    cs_harmonics<MODE>(c, q, cph, sph, CSWarp(c, q.iR * (c.nz - 1) + q.iz, mine), s);
                    if (in) cs_close<MODE, false>(c, lx, ly, lz, q, s, o);
                }
                if (!in) cs_outer<MODE>(c, lx, ly, lz, o);
            } else {
                eval_component<MODE, double, false, true>(c, lx, ly, lz, o);
            }
            const double A = lf.ampl;
            phi += A * o.phi;
            if (MODE != AGB_MODE_POT) {
                const double As = A * lf.sigma;
                g0 += As * o.g[0]; g1 += As * o.g[1]; g2 += As * o.g[2];
                if (MODE == AGB_MODE_HESS) {
                    const double As2 = As * lf.sigma;
                    #pragma unroll
                    for (int q = 0; q < 6; ++q) h[q] += As2 * o.h[q];
                }
            }
        }
        if (live) eval_write<MODE>(a, pos, pos, phi, g0, g1, g2, h, 0.0);
    }
}

// false where the general kernel is the better one: force calls that it holds in one wave of 16
// warps an SM while most warps here make a second pass (71041 to 75776 points; 33 against 39 us
// at 75776, 35 against 31 at 76000, 33 against 31 at 64000, where a quarter of the warps do)
template <int MODE, bool DYN>
static bool launch_cyl(EvalArgs& a, cudaStream_t st)
{
    static std::atomic<int> per_sm[AGB_MAX_DEVICES];
    const int occ = blocks_per_sm(per_sm, agb_cyl_kernel<MODE, DYN>, AGB_CYL_BLOCK);
    const long long want = (a.n + AGB_CYL_BLOCK - 1) / AGB_CYL_BLOCK, slots = (long long)num_sms() * occ;
    if (MODE == AGB_MODE_GRAD && a.n > slots * (AGB_CYL_BLOCK + 32) && a.n <= num_sms() * 512LL) return false;
    const long long grid = want < slots ? want : slots;
    a.chunk = ((a.n + grid - 1) / grid + 31) / 32 * 32;
    agb_cyl_kernel<MODE, DYN><<<(int)((a.n + a.chunk - 1) / a.chunk), AGB_CYL_BLOCK, 0, st>>>(a);
    return true;
}

// FP64 calls of trees of cell-major CylSplines and analytic leaves, points unsorted, the default
// launch shape.  (A density is a trace that cancels: batches and single calls agree in it only
// with the same kernel code, so densities stay with the general kernel.)
bool agb_launch_cyl(int mode, bool mixed, EvalArgs& a, cudaStream_t st)
{
    if (mixed || a.soa || a.perm || a.stage || (a.out_flags & AGB_OUT_SHAPE_BITS)) return false;
    bool any = false;
    for (const DevComp& c : a.comps) {
        if (c.kind == AGB_KIND_MULTIPOLE) return false;
        if (c.kind != AGB_KIND_CYLSPLINE) continue;
        if (c.layout != 1) return false;
        // 32-bit word offsets into the table
        if ((long long)(c.n_int - 1) * (c.nz - 1) * c.n_lm * 8 > 0x7fffffffLL) return false;
        any = true;
    }
    if (!any) return false;
    switch (mode) {
    case AGB_MODE_POT:  return a.dleaves ? launch_cyl<AGB_MODE_POT, true>(a, st) : launch_cyl<AGB_MODE_POT, false>(a, st);
    case AGB_MODE_GRAD: return a.dleaves ? launch_cyl<AGB_MODE_GRAD, true>(a, st) : launch_cyl<AGB_MODE_GRAD, false>(a, st);
    case AGB_MODE_HESS: return a.dleaves ? launch_cyl<AGB_MODE_HESS, true>(a, st) : launch_cyl<AGB_MODE_HESS, false>(a, st);
    default: return false;
    }
}
