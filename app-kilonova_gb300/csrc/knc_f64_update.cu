// knc_f64_update.cu — flux, source and update of the plain FP64 stage
// (compiled with --fmad=false, src/scheme.rs:90-157).
//
// Every FP64 warp instruction occupies its SM partition's FP64 unit for 64 to
// 76 cycles, idle lanes or not, so the kernel's time is the number of FP64
// warp instructions of the busiest partition. Hence
//   - one warp owns an update item {slot, i0, j0, rows} of 32 columns and
//     marches down its rows: no barrier, no idle halo lane, every radial
//     face, slope difference and row load made once;
//   - polar neighbours come through shuffles. What a warp cannot form from its
//     own columns (the flux through its right edge, the state left of its
//     first column, the slope difference across its left edge) is formed for
//     all its rows at once before the march, one lane per row, and kept in
//     shared memory: one more face pass per item instead of one per row;
//   - divisions, square roots, comparisons and supersonic faces take the
//     forms of knc_physics64.cuh;
//   - the items' rows follow the work left (f64_items in knc_api.cu): large
//     grids start with 16 rows, which amortise an item's first faces, and end
//     with 2, so that the last items leave no partition idle.
#include <algorithm>

#include "knc_internal.h"
#include "knc_physics.cuh"
#include "knc_physics64.cuh"
#include "knc_stage.cuh"

namespace knc {

constexpr int ROWS64_WARPS = 4;    // warps per CTA, one per SM partition
constexpr int ROWS64_MAX = 32;     // rows of an item: one lane per row before the march

// What an item keeps per row (lane order before the march, row order in it).
struct Edge64 {
    double flux[NFIELD][ROWS64_MAX];    // through the face right of the last column
    double left[NFIELD][ROWS64_MAX];    // reconstructed state left of the first column
    double diff[NFIELD][ROWS64_MAX];    // theta (P(j0) - P(j0 - 1))
};

__device__ __forceinline__ void load_row64(const double* P, int64_t pn, int64_t off, bool ok, double v[NFIELD]) {
#pragma unroll
    for (int q = 0; q < NFIELD; ++q) v[q] = ok ? P[q * pn + off] : 0.0;
}

// A product with a power of two joins the sum that follows it (or follows the
// sum) exactly unless it falls below the normal range or overflows.
__device__ __forceinline__ bool odd_average(double x) {
    return (hi_word(x) & 0x7fffffffu) - (64u << 20) > (1900u << 20) && magnitude(x) != 0ull;
}

// face64 out of line for the relativistic faces, whose four uses in an item
// then share one copy of their code (2048 x 512 jet fold 5.46 -> 5.22 ms, 450 x
// 230 RK3 HLLC 1.13 -> 1.10 ms); the shorter Newtonian ones are faster inline
// (4.12 against 4.29 ms).
struct State64 {
    double v[NFIELD];
};
template <bool SRHD, bool HLLC>
static __device__ __noinline__ State64 face_call(const PhysT<double> ph, float gmf, float ghf, const State64 l,
                                                 const State64 r, int axis) {
    State64 f;
    face64<SRHD, HLLC>(ph, gmf, ghf, l.v, r.v, axis, f.v);
    return f;
}
template <bool SRHD, bool HLLC>
__device__ __forceinline__ void item_face(const StageArgs& a, const PhysT<double>& ph, const double* pl,
                                          const double* pr, int axis, double out[NFIELD]) {
    if constexpr (!SRHD) {
        face64<SRHD, HLLC>(ph, a.gm_f, a.gh_f, pl, pr, axis, out);
    } else {
        State64 l, r;
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            l.v[q] = pl[q];
            r.v[q] = pr[q];
        }
        const State64 f = face_call<SRHD, HLLC>(ph, a.gm_f, a.gh_f, l, r, axis);
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) out[q] = f.v[q];
    }
}

// out x c x A in that order (c is 1 for Newtonian hydro)
template <bool SRHD>
__device__ __forceinline__ void through_area(double out[NFIELD], double c, double A) {
#pragma unroll
    for (int q = 0; q < NFIELD; ++q) out[q] = (SRHD ? out[q] * c : out[q]) * A;
}

template <bool SRHD, bool HLLC>
__device__ __forceinline__ void edges64(const StageArgs& a, const PhysT<double>& ph, const DevBlock& B, int i0, int j0,
                                        int rows, Edge64& E) {
    const int lane = threadIdx.x & 31;
    const int nr = B.nr, nq = B.nq, i = i0 + lane;
    const double* P = reinterpret_cast<const double*>(B.P);
    const int64_t pn = (int64_t)(nr + 4) * nq;
    const double th = ph.theta;
    if (lane >= rows) return;
    const double* row = P + (int64_t)(i + 2) * nq;
    if (j0 > 0) {
        // zone j0 - 1: its column is at least 31, never the block's first or last
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            const double* p = row + q * pn + j0;
            const double pa = p[-2], pb = p[-1], pc = p[0];
            const double z = th * (pc - pb);
            E.diff[q][lane] = z;
            E.left[q][lane] = pb + half_slope64(th * (pb - pa), pc - pa, z);
        }
    }
    const int jr = j0 + 32;   // the face between columns jr - 1 and jr
    double f[NFIELD] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (jr < nq) {
        double pl[NFIELD], pr[NFIELD];
        const bool last = jr == nq - 1;   // zero slope on the block's last column
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            const double* p = row + q * pn + jr;
            const double pa = p[-2], pb = p[-1], pc = p[0], pd = last ? pc : p[1];
            const double z = th * (pc - pb);
            pl[q] = pb + half_slope64(th * (pb - pa), pc - pa, z);
            pr[q] = pc - (last ? 0.0 : half_slope64(z, pd - pb, th * (pd - pc)));
        }
        item_face<SRHD, HLLC>(a, ph, pl, pr, 1, f);
        through_area<SRHD>(f, a.cflux, B.aq[(int64_t)i * (nq + 1) + jr]);
    }
#pragma unroll
    for (int q = 0; q < NFIELD; ++q) E.flux[q][lane] = f[q];
}

// Sources, conserved update and RK average of zone (i, j) with primitive P0:
// radial fluxes Flo, Fhi, polar flux difference D.
template <bool SRHD>
__device__ __forceinline__ void update_zone64(const StageArgs& a, const PhysT<double>& ph, const DevBlock& B, int i,
                                              int j, const double* P0, const double* Flo, const double* Fhi,
                                              const double* D, bool one_d, double dt) {
    const int64_t n = (int64_t)B.nr * B.nq, z = (int64_t)i * B.nq + j;
    const double* Uin = B.buf[a.sel_in];
    double* Uout = B.buf[a.sel_out];
    double s1, s2, res[NFIELD];
    const double dV = B.dv[z];
    sources64<SRHD>(ph, P0, B.rc[i], B.cot[j], s1, s2);
    s1 = (SRHD ? s1 * a.cflux : s1) * dV;
    s2 = (SRHD ? s2 * a.cflux : s2) * dV;
#pragma unroll
    for (int q = 0; q < NFIELD; ++q) {
        const double R = Fhi[q] - Flo[q];
        double du;
        // (S - dF_r - dF_q) dt; without a source the exact negative of (dF_r + dF_q) dt
        if (q == 1 || q == 2) {
            const double sc = q == 1 ? s1 : s2;
            du = (one_d ? sc - R : sc - R - D[q]) * dt;
        } else {
            du = -((one_d ? R : R + D[q]) * dt);
        }
        res[q] = Uin[q * n + z] + du;
    }
    if (a.sel_base >= 0) {
        // res w1 + U0 b
        const double* U0 = B.buf[a.sel_base];
        bool odd = false;
        double u0[NFIELD];
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            u0[q] = U0[q * n + z];
            odd = odd || odd_average(res[q]) || odd_average(u0[q]);
        }
        if (odd || !(a.avg_half || a.w1 == 0.25)) {
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) res[q] = res[q] * a.w1 + u0[q] * a.bf;
        } else if (a.avg_half) {
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) res[q] = half64(res[q] + u0[q]);
        } else {
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) res[q] = __fma_rn(res[q], 0.25, u0[q] * a.bf);
        }
    }
#pragma unroll
    for (int q = 0; q < NFIELD; ++q) Uout[q * n + z] = res[q];
}

template <bool SRHD, bool HLLC>
__device__ __forceinline__ void update_rows64(const StageArgs& a, const PhysT<double>& ph, const int4 it, Edge64& E) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const DevBlock& B = a.blocks[it.x];
    const int nr = B.nr, nq = B.nq, i0 = it.y, j0 = it.z, rows = it.w;
    const int j = j0 + lane;
    const bool jin = j < nq;
    const bool one_d = a.one_dimensional != 0;
    const double* P = reinterpret_cast<const double*>(B.P);
    const int64_t pn = (int64_t)(nr + 4) * nq;
    const double th = ph.theta, c = a.cflux;
    const double dt = stage_dt<double>(a);
    const bool pedge = j <= 0 || j >= nq - 1;   // zero polar slope on the block's first and last column
    // the column a first or last lane reads beyond the warp's
    const int je = lane == 0 ? j0 - 1 : j0 + 32;
    const bool eok = (lane == 0 && j0 > 0) || (lane == 31 && je < nq);

    if (!one_d) edges64<SRHD, HLLC>(a, ph, B, i0, j0, rows, E);
    __syncwarp();

    // rows i0 and i0 + 1, the half slope of row i0, theta (P(i0 + 1) - P(i0)), the flux through face i0
    double P0[NFIELD], P1[NFIELD], x1[NFIELD], g0[NFIELD], Flo[NFIELD] = {0.0, 0.0, 0.0, 0.0, 0.0};
    {
        double Pa[NFIELD], Pb[NFIELD], pl[NFIELD], pr[NFIELD];
        const int64_t o = (int64_t)i0 * nq + j;   // padded row i0 is zone row i0 - 2
        load_row64(P, pn, o, jin, Pa);
        load_row64(P, pn, o + nq, jin, Pb);
        load_row64(P, pn, o + 2 * (int64_t)nq, jin, P0);
        load_row64(P, pn, o + 3 * (int64_t)nq, jin, P1);
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            const double x = th * (P0[q] - Pb[q]);
            x1[q] = th * (P1[q] - P0[q]);
            g0[q] = half_slope64(x, P1[q] - Pb[q], x1[q]);
            pl[q] = Pb[q] + half_slope64(th * (Pb[q] - Pa[q]), P0[q] - Pa[q], x);
            pr[q] = P0[q] - g0[q];
        }
        if (jin) {
            item_face<SRHD, HLLC>(a, ph, pl, pr, 0, Flo);
            through_area<SRHD>(Flo, c, B.ar[(int64_t)i0 * nq + j]);
        }
    }
    for (int s = 0; s < rows; ++s) {
        const int i = i0 + s;
        const int64_t o = (int64_t)(i + 2) * nq + j;
        double P2[NFIELD];
        load_row64(P, pn, o + 2 * (int64_t)nq, jin, P2);
        // ---- polar faces j (own) and j + 1 (the next lane's)
        double D[NFIELD];   // F(j + 1) - F(j)
        if (!one_d) {
            double Pe[NFIELD], pl[NFIELD], pr[NFIELD], f[NFIELD] = {0.0, 0.0, 0.0, 0.0, 0.0};
            load_row64(P, pn, o + (je - j), eok, Pe);
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) {
                double left = __shfl_up_sync(full, P0[q], 1), right = __shfl_down_sync(full, P0[q], 1);
                if (lane == 0) left = Pe[q];
                if (lane == 31) right = Pe[q];
                const double dz = th * (right - P0[q]);
                double dx = __shfl_up_sync(full, dz, 1);
                if (lane == 0) dx = E.diff[q][s];
                const double g = pedge ? 0.0 : half_slope64(dx, right - left, dz);
                pl[q] = __shfl_up_sync(full, P0[q] + g, 1);
                if (lane == 0) pl[q] = E.left[q][s];
                pr[q] = P0[q] - g;
            }
            if (j > 0 && jin) {
                item_face<SRHD, HLLC>(a, ph, pl, pr, 1, f);
                through_area<SRHD>(f, c, B.aq[(int64_t)i * (nq + 1) + j]);
            }
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) {
                double up = __shfl_down_sync(full, f[q], 1);
                if (lane == 31) up = E.flux[q][s];
                D[q] = up - f[q];
            }
        }
        // ---- radial face i + 1
        double Fhi[NFIELD] = {0.0, 0.0, 0.0, 0.0, 0.0};
        {
            double pl[NFIELD], pr[NFIELD];
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) {
                const double dz = th * (P2[q] - P1[q]);
                const double g1 = half_slope64(x1[q], P2[q] - P0[q], dz);
                pl[q] = P0[q] + g0[q];
                pr[q] = P1[q] - g1;
                x1[q] = dz;
                g0[q] = g1;
            }
            if (jin) {
                item_face<SRHD, HLLC>(a, ph, pl, pr, 0, Fhi);
                through_area<SRHD>(Fhi, c, B.ar[(int64_t)(i + 1) * nq + j]);
            }
        }
        if (jin) update_zone64<SRHD>(a, ph, B, i, j, P0, Flo, Fhi, D, one_d, dt);
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            Flo[q] = Fhi[q];
            P0[q] = P1[q];
            P1[q] = P2[q];
        }
    }
    __syncwarp();   // E is free for the warp's next item
}

template <bool SRHD, bool HLLC>
__global__ void __launch_bounds__(ROWS64_WARPS * 32, 3)
    update_rows64_kernel(const __grid_constant__ StageArgs a, const int4* __restrict__ items, int nitems) {
    __shared__ Edge64 sE[ROWS64_WARPS];
    // A failed c2p in this or an earlier stage stops the step: keep the
    // input state untouched so the failure can be reported from it.
    if (stopped(a)) return;   // (the same for a warp's lanes, and its warps are on their own)
    const PhysT<double> ph = make_phys<double>(a);
    const int w = threadIdx.x >> 5;
    for (int k = blockIdx.x * ROWS64_WARPS + w; k < nitems; k += gridDim.x * ROWS64_WARPS)
        update_rows64<SRHD, HLLC>(a, ph, items[k], sE[w]);
}

// ---- small grids ------------------------------------------------------------------
// A march does an item's faces one after the other: with a few rows per SM
// partition its length, not the FP64 pipe, sets the kernel's time. Here a CTA of
// 4 warps takes a tile of at most TILE64_ROWS rows x 31 columns and its warps
// claim face passes, the rows' 32 polar faces first, then the rows + 1 rows of
// radial faces; fluxes meet in shared memory, then a warp per row updates it.
// Slopes are formed by the faces on both of their sides (25 FP64 instructions
// more per face than in the march), with the same roundings.
constexpr int TILE64_ROWS = 2;

struct Tile64 {
    double P[NFIELD][TILE64_ROWS + 4][TILE64_COLS + 4];
    double Fr[NFIELD][TILE64_ROWS + 1][32];
    double Fq[NFIELD][TILE64_ROWS][32];
    unsigned claim;
};

template <bool SRHD, bool HLLC>
__global__ void __launch_bounds__(ROWS64_WARPS * 32, 3)
    update_tile64_kernel(const __grid_constant__ StageArgs a, const int4* __restrict__ items) {
    __shared__ Tile64 T;
    const PhysT<double> ph = make_phys<double>(a);
    const int4 it = items[blockIdx.x];
    const DevBlock& B = a.blocks[it.x];
    const int nr = B.nr, nq = B.nq, i0 = it.y, j0 = it.z, rows = it.w;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool one_d = a.one_dimensional != 0;
    const double th = ph.theta;
    {
        const double* P = reinterpret_cast<const double*>(B.P);
        const int64_t pn = (int64_t)(nr + 4) * nq;
        constexpr int PC = TILE64_COLS + 4;
        for (int k = threadIdx.x; k < (rows + 4) * PC; k += ROWS64_WARPS * 32) {
            const int r = k / PC, c = k - r * PC, j = j0 - 2 + c;
            const bool ok = j >= 0 && j < nq;
            const int64_t o = (int64_t)(i0 + r) * nq + j;   // padded row i0 is zone row i0 - 2
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) T.P[q][r][c] = ok ? P[q * pn + o] : 0.0;
        }
        if (threadIdx.x == 0) T.claim = ROWS64_WARPS;
    }
    // after a failure the CTA leaves as one (the barrier is needed anyway)
    if (__syncthreads_or(stopped(a))) return;
    const unsigned polar = one_d ? 0u : (unsigned)rows, passes = polar + (unsigned)rows + 1u;
    const int j = j0 + lane;
    // A warp's first pass is rotated with the CTA: a warp stays on its SM
    // partition, and the polar faces cost more than supersonic radial ones.
    unsigned p = (warp + blockIdx.x) % ROWS64_WARPS;
    while (p < passes) {
        const bool radial = p >= polar;
        const int r = (int)(radial ? p - polar : p);   // radial face i0 + r, or row i0 + r
        const bool exists = radial ? lane < TILE64_COLS && j < nq : j > 0 && j < nq;
        double f[NFIELD] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (exists) {
            // the face lies between the second and third of its four zones
            const bool zl = !radial && j - 1 == 0, zr = !radial && j == nq - 1;   // zero polar slope on the edge columns
            double pl[NFIELD], pr[NFIELD];
#pragma unroll
            for (int q = 0; q < NFIELD; ++q) {
                const double* s = radial ? &T.P[q][r][lane + 2] : &T.P[q][r + 2][lane];
                const int st = radial ? TILE64_COLS + 4 : 1;
                const double s0 = s[0], s1 = s[st], s2 = s[2 * st], s3 = s[3 * st];
                const double mid = th * (s2 - s1);
                pl[q] = s1 + (zl ? 0.0 : half_slope64(th * (s1 - s0), s2 - s0, mid));
                pr[q] = s2 - (zr ? 0.0 : half_slope64(mid, s3 - s1, th * (s3 - s2)));
            }
            item_face<SRHD, HLLC>(a, ph, pl, pr, radial ? 0 : 1, f);
            through_area<SRHD>(f, a.cflux, radial ? B.ar[(int64_t)(i0 + r) * nq + j] : B.aq[(int64_t)(i0 + r) * (nq + 1) + j]);
        }
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) (radial ? T.Fr[q][r] : T.Fq[q][r])[lane] = f[q];
        if (lane == 0) p = atomicAdd(&T.claim, 1u);
        p = __shfl_sync(0xffffffffu, p, 0);
    }
    __syncthreads();
    if (warp < rows && lane < TILE64_COLS && j < nq) {
        const int r = warp;
        double P0[NFIELD], lo[NFIELD], hi[NFIELD], D[NFIELD];
#pragma unroll
        for (int q = 0; q < NFIELD; ++q) {
            P0[q] = T.P[q][r + 2][lane + 2];
            lo[q] = T.Fr[q][r][lane];
            hi[q] = T.Fr[q][r + 1][lane];
            D[q] = one_d ? 0.0 : T.Fq[q][r][lane + 1] - T.Fq[q][r][lane];
        }
        update_zone64<SRHD>(a, ph, B, i0 + r, j, P0, lo, hi, D, one_d, stage_dt<double>(a));
    }
}

cudaError_t launch_update_f64(const StageArgs& a, cudaStream_t s) {
    const int4* items = a.strips ? a.strips : a.utiles;
    const int n = a.strips ? a.nstrips : a.nutiles;
    if (n <= 0) return cudaSuccess;
    if (a.f64_tiles) {
        auto k = a.srhd ? (a.hllc ? update_tile64_kernel<true, true> : update_tile64_kernel<true, false>)
                        : (a.hllc ? update_tile64_kernel<false, true> : update_tile64_kernel<false, false>);
        k<<<n, ROWS64_WARPS * 32, 0, s>>>(a, items);
        return cudaGetLastError();
    }
    const int grid = (n + ROWS64_WARPS - 1) / ROWS64_WARPS;
    auto k = a.srhd ? (a.hllc ? update_rows64_kernel<true, true> : update_rows64_kernel<true, false>)
                    : (a.hllc ? update_rows64_kernel<false, true> : update_rows64_kernel<false, false>);
    k<<<grid, ROWS64_WARPS * 32, 0, s>>>(a, items, n);
    return cudaGetLastError();
}

}  // namespace knc
