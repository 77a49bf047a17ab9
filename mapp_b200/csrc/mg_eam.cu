// Tabulated EAM (ff_eam.cpp:44-356) and analytic Finnis-Sinclair
// (ff_fs.cpp:379-684) force / energy kernels.
//
// Layout of work: one lane per listed pair of the compact list (pairs sorted by
// i), so every lane carries work however many neighbours an atom has.  The
// forces and densities of a warp's pairs are added up through shared memory
// (rows_scatter for the atoms j, rows_runs for the atoms i; owned j only, as in
// the reference: ghost j receive nothing and their pair energy and virial count
// one half).
// Energy and virial go to per-block partial rows reduced deterministically at
// the end; the grids are persistent, so there are a few thousand rows at most.
//
// Pass 1 stores -drho/dr / r for both sides of every pair (one 16-byte item per
// pair) like drhoi_dr / drhoj_dr (ff_eam.cpp:172-173); pass 2 reads F'(rho) of a
// ghost j from its owner (the ghost refresh atoms->update(rho_n),
// ff_eam.cpp:194, fused into the load).
//
// What bounds the pair passes: the L1 data stage takes one cycle per lane of a
// gather (positions, 32-byte spline knots), per line of a reduction and per
// shuffle.  With one warp per atom, two 64-byte knot rows, the species gather and
// four single reductions a pair cost 10 of them and 256000 atoms took 380 us
// (pass 1) and 286 us (pass 2); here the derivative comes from the value's
// coefficients, one species needs no gather, and the reductions share lines:
// 177 us and 115 us (L1 data stage 84 % and 76 % busy; 798 -> 352 us a call).
#include "mg_reduce.cuh"
#include "mg_launch.cuh"
#include "mg_dmd_common.cuh"

namespace mg {

namespace {

// Resident blocks per SM of the pair passes (64 registers a thread at 4).
#ifndef MG_EAM_MINB
#define MG_EAM_MINB 4
#endif

// f(p, valid, i) for the compact pairs, a warp's lanes together
template <typename F>
__device__ __forceinline__ void for_pairs(const Dev& d, F f)
{
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; b < d.npairs; b += stride) {
        const long long p = b + lane;
        const bool valid = p < d.npairs;
        f(p, valid, valid ? d.pair_i[p] : -1);
    }
}

// the sums of a warp's pairs: value q < 3 of a row is a force component, q = 3 a density
__device__ __forceinline__ void add_value(const Dev& d, int row, int q, double x)
{
    atomicAdd(q < 3 ? d.f + (size_t)row * 3 + q : d.rho + row, x);
}

__device__ __forceinline__ void add_virial(double (&acc)[7], double w, double dx0, double dx1, double dx2)
{
    acc[1] -= w * dx0 * dx0;
    acc[2] -= w * dx1 * dx1;
    acc[3] -= w * dx2 * dx2;
    acc[4] -= w * dx1 * dx2;
    acc[5] -= w * dx2 * dx0;
    acc[6] -= w * dx0 * dx1;
}

// EAM pass 1 (ff_eam.cpp:95-177).  kEnergyOnly skips forces and stored
// derivatives (ForceField_eam::energy_calc, ff_eam.cpp:297-338); kOne: one
// species, whose index is not read and whose two densities are the same.
template <bool kEnergyOnly, bool kOne>
__global__ void __launch_bounds__(kFFBlock, MG_EAM_MINB) k_eam_pass1(Dev d, int st_clc, int row0)
{
    dep_sync();
    constexpr int NV = kEnergyOnly ? 1 : 4;
    __shared__ RowBuf<NV> sh[kFFWarps];
    RowBuf<NV>& buf = sh[threadIdx.x >> 5];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for_pairs(d, [&](long long p, bool valid, int i) {
        // the pair's shares: of atom j its force and density (the other way round, of atom i)
        double v[NV], rho_i = 0.0, pi_ = 0.0, pj_ = 0.0;
#pragma unroll
        for (int q = 0; q < NV; q++) v[q] = 0.0;
        int row = -1;
        if (valid) {
            const int j = d.pair_j[p];
            const double4 xi = d.pos[i], xj = d.pos[j];
            const double dx0 = xi.x - xj.x, dx1 = xi.y - xj.y, dx2 = xi.z - xj.z;
            const double rsq = __dadd_rn(__dadd_rn(__dmul_rn(dx0, dx0), __dmul_rn(dx1, dx1)), __dmul_rn(dx2, dx2));
            if (rsq < d.cut_sq) {
                const int ti = kOne ? 0 : d.type[i], tj = kOne ? 0 : d.type[j];
                const double r = sqrt(rsq);
                const double r_inv = 1.0 / r;
                double q = r * d.dr_inv;
                const int m = min((int)q, d.nr - 2);
                q -= m;
                q = fmin(q, 1.0);
                // knots of rho(ti, tj) and phi side by side (Dev::pk64)
                const double* kt = d.pk64 + ((size_t)(ti * d.nt + tj) * d.nr + m) * 8;
                const double4 cf = knot4(kt), ch = knot4(kt + 4);
                const double4 cg = kOne || tj == ti ? cf : knot4(d.pk64 + ((size_t)(tj * d.nt + ti) * d.nr + m) * 8);
                const double rho_jv = ((cg.w * q + cg.z) * q + cg.y) * q + cg.x;
                const double z2 = ((ch.w * q + ch.z) * q + ch.y) * q + ch.x;
                const double phi = z2 * r_inv;
                const bool own_j = j < d.natms;
                const double w = own_j ? 1.0 : 0.5;
                rho_i = kOne ? rho_jv : ((cf.w * q + cf.z) * q + cf.y) * q + cf.x;
                v[NV - 1] = rho_jv;
                if (own_j) row = j;
                acc[0] += w * phi;
                if (!kEnergyOnly) {
                    const double z2p = ((3.0 * ch.w * q + 2.0 * ch.z) * q + ch.y) * d.dr_inv;
                    const double dphi = z2p * r_inv - phi * r_inv;
                    const double fpair = -dphi * r_inv;
                    v[0] = -fpair * dx0;
                    v[1 % NV] = -fpair * dx1;
                    v[2 % NV] = -fpair * dx2;
                    if (st_clc) add_virial(acc, w * fpair, dx0, dx1, dx2);
                    pj_ = -((3.0 * cg.w * q + 2.0 * cg.z) * q + cg.y) * d.dr_inv * r_inv;
                    pi_ = kOne ? pj_ : -((3.0 * cf.w * q + 2.0 * cf.z) * q + cf.y) * d.dr_inv * r_inv;
                }
            }
            if (!kEnergyOnly) __stcs(reinterpret_cast<double2*>(d.pr) + p, make_double2(pi_, pj_));
        }
        rows_put<NV>(buf, v, i);
        rows_scatter<NV>(buf, row, [&](int r, int q, double x) { add_value(d, r, q + 4 - NV, x); });
        if (!kOne) {  // atom i's density is not atom j's
            __syncwarp();
            buf.v[(threadIdx.x & 31) * RowBuf<NV>::PITCH + NV - 1] = rho_i;
            __syncwarp();
        }
        rows_runs<NV>(buf, [&](int r, int q, double x) { add_value(d, r, q + 4 - NV, q + 4 - NV < 3 ? -x : x); });
    });
    block_partials<7>(acc, d.partial, row0 + blockIdx.x);
}

// Embedding energy F(rho) and F'(rho) per owned atom (ff_eam.cpp:178-190);
// the index clamp uses nr-2 like the reference (ff_eam.cpp:180).
template <bool kEnergyOnly>
__global__ void __launch_bounds__(kFFBlock) k_eam_embed(Dev d, int row0)
{
    dep_sync();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    if (i < d.natms) {
        double rv = d.rho[i];
        double p = rv * d.drho_inv;
        int m = max(0, min((int)p, d.nr - 2));  // lower clamp: never index before the table
        p -= m;
        p = fmin(p, 1.0);
        const double* cf = d.FT + ((size_t)d.type[i] * (d.nrho + 1) + m) * d.Fw;
        double tmp1 = (cf[6] * p + cf[5]) * p + cf[4];
        double tmp0 = ((cf[3] * p + cf[2]) * p + cf[1]) * p + cf[0];
        if (rv > d.rho_max) tmp0 += tmp1 * (rv - d.rho_max);
        acc[0] = tmp0;
        if (!kEnergyOnly) d.rho[i] = tmp1;
    }
    block_partials<7>(acc, d.partial, row0 + blockIdx.x);
}

// EAM / FS pass 2: embedding forces from the stored pair derivatives
// (ff_eam.cpp:196-250, ff_fs.cpp:531-588).
__global__ void __launch_bounds__(kFFBlock, MG_EAM_MINB) k_embed_pass2(Dev d, int st_clc, int row0)
{
    dep_sync();
    constexpr int NV = 3;
    __shared__ RowBuf<NV> sh[kFFWarps];
    RowBuf<NV>& buf = sh[threadIdx.x >> 5];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for_pairs(d, [&](long long p, bool valid, int i) {
        double f[3] = {0, 0, 0};
        int row = -1;
        if (valid) {
            const int j = d.pair_j[p];
            const double2 dr = __ldcs(reinterpret_cast<const double2*>(d.pr) + p);
            if (dr.x != 0.0 || dr.y != 0.0) {
                const double4 xi = d.pos[i], xj = d.pos[j];
                const double fpair = d.rho[i] * dr.x + d.rho[owner(d, j)] * dr.y;
                const double dx0 = xi.x - xj.x, dx1 = xi.y - xj.y, dx2 = xi.z - xj.z;
                f[0] = -dx0 * fpair;
                f[1] = -dx1 * fpair;
                f[2] = -dx2 * fpair;
                const bool own_j = j < d.natms;
                if (own_j) row = j;
                if (st_clc) add_virial(acc, (own_j ? 1.0 : 0.5) * fpair, dx0, dx1, dx2);
            }
        }
        rows_put<3>(buf, f, i);
        rows_scatter<3>(buf, row, [&](int r, int q, double x) { add_value(d, r, q, x); });
        rows_runs<3>(buf, [&](int r, int q, double x) { add_value(d, r, q, -x); });
    });
    block_partials<7>(acc, d.partial, row0 + blockIdx.x);
}

// Analytic FS pass 1 (ff_fs.cpp:424-527).
template <bool kEnergyOnly>
__global__ void __launch_bounds__(kFFBlock, MG_EAM_MINB) k_fs_pass1(Dev d, int st_clc, int row0)
{
    dep_sync();
    constexpr int NV = kEnergyOnly ? 1 : 4;
    __shared__ RowBuf<NV> sh[kFFWarps];
    RowBuf<NV>& buf = sh[threadIdx.x >> 5];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for_pairs(d, [&](long long p, bool valid, int i) {
        double v[NV], rho_i = 0.0, pi_ = 0.0, pj_ = 0.0;
#pragma unroll
        for (int q = 0; q < NV; q++) v[q] = 0.0;
        int row = -1;
        if (valid) {
            const int j = d.pair_j[p];
            const int ti = d.type[i], tj = d.type[j];
            const int cs = comp_idx(ti, tj);
            if (d.fs_chk[cs]) {
                const double4 xi = d.pos[i], xj = d.pos[j];
                const double dx0 = xi.x - xj.x, dx1 = xi.y - xj.y, dx2 = xi.z - xj.z;
                const double rsq = __dadd_rn(__dadd_rn(__dmul_rn(dx0, dx0), __dmul_rn(dx1, dx1)), __dmul_rn(dx2, dx2));
                if (rsq < d.fs_cut_sq[cs]) {
                    const double r = sqrt(rsq);
                    const double r_inv = 1.0 / r;
                    const bool own_j = j < d.natms;
                    const double w = own_j ? 1.0 : 0.5;
                    if (own_j) row = j;
                    if (r < d.fs_cut_rho[cs]) {
                        const double dr_ = r - d.fs_cut_rho[cs];
                        rho_i = dr_ * dr_ * (d.fst1[tj][ti] + d.fst2[tj][ti] * dr_);
                        v[NV - 1] = dr_ * dr_ * (d.fst1[ti][tj] + d.fst2[ti][tj] * dr_);
                        pi_ = -r_inv * dr_ * (d.fst1[tj][ti] + 1.5 * d.fst2[tj][ti] * dr_);
                        pj_ = -r_inv * dr_ * (d.fst1[ti][tj] + 1.5 * d.fst2[ti][tj] * dr_);
                    }
                    if (r < d.fs_cut_phi[cs]) {
                        const double dp = r - d.fs_cut_phi[cs];
                        const double poly = d.fsk1[cs] + d.fsk2[cs] * r + d.fsk3[cs] * rsq;
                        acc[0] += w * (dp * dp * poly);
                        if (!kEnergyOnly) {
                            double pc = 2.0 * dp * poly + dp * dp * (d.fsk2[cs] + 2.0 * d.fsk3[cs] * r);
                            pc *= -r_inv;
                            v[0] = -dx0 * pc;
                            v[1 % NV] = -dx1 * pc;
                            v[2 % NV] = -dx2 * pc;
                            if (st_clc) add_virial(acc, w * pc, dx0, dx1, dx2);
                        }
                    }
                }
            }
            if (!kEnergyOnly) __stcs(reinterpret_cast<double2*>(d.pr) + p, make_double2(pi_, pj_));
        }
        rows_put<NV>(buf, v, i);
        rows_scatter<NV>(buf, row, [&](int r, int q, double x) { add_value(d, r, q + 4 - NV, x); });
        {  // atom i's density is not atom j's
            __syncwarp();
            buf.v[(threadIdx.x & 31) * RowBuf<NV>::PITCH + NV - 1] = rho_i;
            __syncwarp();
        }
        rows_runs<NV>(buf, [&](int r, int q, double x) { add_value(d, r, q + 4 - NV, q + 4 - NV < 3 ? -x : x); });
    });
    block_partials<7>(acc, d.partial, row0 + blockIdx.x);
}

// FS embedding: F = -A sqrt(rho), stores 2 F'(rho) = -A / sqrt(rho) (ff_fs.cpp:524-526).
template <bool kEnergyOnly>
__global__ void __launch_bounds__(kFFBlock) k_fs_embed(Dev d, int row0)
{
    dep_sync();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    if (i < d.natms) {
        double rs = sqrt(d.rho[i]);
        double A = d.fsA[d.type[i]];
        acc[0] = -(A * rs);
        if (!kEnergyOnly) d.rho[i] = -A / rs;
    }
    block_partials<7>(acc, d.partial, row0 + blockIdx.x);
}

}  // namespace

cudaError_t launch_eam_force(const Dev& d, int st_clc, int* nblocks_out, cudaStream_t st)
{
    const int g1 = persistent_grid(d.npairs, MG_EAM_MINB), g2 = div_up(d.natms, kFFBlock);
    if (d.nt == 1) launch_dep(k_eam_pass1<false, true>, g1, kFFBlock, 0, st, d, st_clc, 0);
    else launch_dep(k_eam_pass1<false, false>, g1, kFFBlock, 0, st, d, st_clc, 0);
    launch_dep(k_eam_embed<false>, g2, kFFBlock, 0, st, d, g1);
    launch_dep(k_embed_pass2, g1, kFFBlock, 0, st, d, st_clc, g1 + g2);
    *nblocks_out = 2 * g1 + g2;
    return cudaGetLastError();
}

cudaError_t launch_eam_energy(const Dev& d, int* nblocks_out, cudaStream_t st)
{
    const int g1 = persistent_grid(d.npairs, MG_EAM_MINB), g2 = div_up(d.natms, kFFBlock);
    if (d.nt == 1) launch_dep(k_eam_pass1<true, true>, g1, kFFBlock, 0, st, d, 0, 0);
    else launch_dep(k_eam_pass1<true, false>, g1, kFFBlock, 0, st, d, 0, 0);
    launch_dep(k_eam_embed<true>, g2, kFFBlock, 0, st, d, g1);
    *nblocks_out = g1 + g2;
    return cudaGetLastError();
}

cudaError_t launch_fs_force(const Dev& d, int st_clc, int* nblocks_out, cudaStream_t st)
{
    const int g1 = persistent_grid(d.npairs, MG_EAM_MINB), g2 = div_up(d.natms, kFFBlock);
    launch_dep(k_fs_pass1<false>, g1, kFFBlock, 0, st, d, st_clc, 0);
    launch_dep(k_fs_embed<false>, g2, kFFBlock, 0, st, d, g1);
    launch_dep(k_embed_pass2, g1, kFFBlock, 0, st, d, st_clc, g1 + g2);
    *nblocks_out = 2 * g1 + g2;
    return cudaGetLastError();
}

cudaError_t launch_fs_energy(const Dev& d, int* nblocks_out, cudaStream_t st)
{
    const int g1 = persistent_grid(d.npairs, MG_EAM_MINB), g2 = div_up(d.natms, kFFBlock);
    launch_dep(k_fs_pass1<true>, g1, kFFBlock, 0, st, d, 0, 0);
    launch_dep(k_fs_embed<true>, g2, kFFBlock, 0, st, d, g1);
    *nblocks_out = g1 + g2;
    return cudaGetLastError();
}

}  // namespace mg
