// Device build of the STO overlap S and the extended-Hueckel h for one
// nuclear configuration.
//
// One thread per atom pair (ia >= ib).  Each thread writes its whole AO
// block of S and h and the transposed block, so every element of the two
// N x N matrices is written exactly once (no memset, no atomics).
//
//   lined-up overlaps ... sto_pair.cuh (SOLAP, overlap_D.f:701-962, for l <= 1)
//   rotation ............ ROTAR for l <= 1 (overlap_D.f:983-1027): its matrix
//                         elements are the direction cosines of the pair
//   normalisation ....... GET_ANOR / GET_ANOR_DIVISOR (overlap_D.f:464-517), one
//                         factor per AO and exponent, formed when the basis is
//                         laid out (sto_norm)
//   assembly ............ BUILD_OVERLAP_MATRIX (overlap_D.f:228-291), diag 1
//   Hueckel ............. h_ij = X_ij S_ij, weighted Wolfsberg-Helmholz
//                         (hamiltonians.f:33-63, ElHl_Chebyshev.f:313-321)
//
// Supported basis: n <= 3, l <= 1, one or two zetas (the H/C/O EHT basis of
// the workloads).
//
// Bound: the FP64 unit (64-76 cycles per warp instruction), and for a few dozen
// atoms one thread's chain of them.  So the kernel counts FP64 instructions, and
// divides, takes roots and multiplies constants outside the pair loop.
#include "elhl_internal.cuh"
#include "sto_pair.cuh"

namespace elhl {
namespace {

constexpr int kMaxShell = 4;                // radial shells per atom handled per shell pair

// constants of the basic integrals and of the 1F1 series (sto_pair.cuh), filled
// once per device by init_build_tables
__device__ double g_cell[sto::kCellTable];
__device__ double g_series[sto::kSeriesTable];

__global__ void init_tables_kernel() {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < sto::kCellTable) g_cell[i] = sto::cell_constant(i);
    if (i < sto::kSeriesTable) g_series[i] = sto::series_constant(i);
}

__device__ __forceinline__ sto::Tables tables() { return sto::Tables{g_cell, g_series}; }

__device__ __forceinline__ double x_ij(double ipi, double ipj, double vi, double vj, double ki, double kj) {
    const double c1 = ipi - ipj, c2 = ipi + ipj;
    const double c3 = (c1 / c2) * (c1 / c2);
    const double c4 = (vi + vj) * 0.5;
    const double k = (ki + kj) * 0.5;
    const double keff = k + c3 + c3 * c3 * (1.0 - k);
    return keff * c2 * 0.5 + c4;
}

// Shells of one atom: runs of consecutive AOs with the same n, l, zetas and
// coefficients (the m components of one radial function).  The lined-up
// overlaps depend on the shells only, so they are computed once per shell pair
// and the rotation is applied per AO pair.

__device__ bool same_radial(const DevBasis &b, int x, int y) {
    return b.ao_n[x] == b.ao_n[y] && b.ao_l[x] == b.ao_l[y] && b.ao_nzeta[x] == b.ao_nzeta[y] &&
           b.ao_zeta[2 * x] == b.ao_zeta[2 * y] && b.ao_zeta[2 * x + 1] == b.ao_zeta[2 * y + 1] &&
           b.ao_coef[2 * x] == b.ao_coef[2 * y] && b.ao_coef[2 * x + 1] == b.ao_coef[2 * y + 1];
}

// shell index of every AO of an atom (ao0, nao); returns the shell count, or
// -1 when the atom has more than kMaxShell shells.  first[s] = first AO of shell s.
__device__ int atom_shells(const DevBasis &b, int ao0, int nao, int *first, int *shell_of) {
    int ns = 0;
    for (int j = 0; j < nao; ++j) {
        if (j == 0 || !same_radial(b, ao0 + j, ao0 + j - 1)) {
            if (ns == kMaxShell) return -1;
            first[ns++] = ao0 + j;
        }
        shell_of[j] = ns - 1;
    }
    return ns;
}

// normalised, contracted lined-up overlaps <aa|bb>_m, m = 0..min(la, lb)
// (the SOLAP + GET_ANOR part of BUILD_OVERLAP_MATRIX, overlap_D.f:228-280)
__device__ void contracted_overlap(const DevBasis &b, int aa, int bb, double R, double *solnorm) {
    solnorm[0] = solnorm[1] = 0.0;
    for (int j = 0; j < b.ao_nzeta[bb]; ++j) {
        for (int i = 0; i < b.ao_nzeta[aa]; ++i) {
            const int na = b.ao_n[aa], la = b.ao_l[aa], nb = b.ao_n[bb], lb = b.ao_l[bb];
            double sol[2];
            if (sto::supported(na, la) && sto::supported(nb, lb)) {
                sto::PairTable t;
                sto::pair_table(tables(), b.ao_zeta[2 * aa + i], b.ao_zeta[2 * bb + j], R, sto::reach(na, la, nb, lb), t);
                sto::lined_up(t, na, la, nb, lb, sol);
            } else {
                sol[0] = sol[1] = __longlong_as_double(0x7ff8000000000000ULL);  // NaN marks unsupported
            }
            const double nn = b.ao_norm[2 * aa + i] * b.ao_norm[2 * bb + j];
            solnorm[0] += nn * sol[0];
            if (la == 1 && lb == 1) solnorm[1] += nn * sol[1];
        }
    }
}

// the single exponent carried by every shell (first AOs first[0..ns)) of an atom, if there is one
__device__ bool uniform_zeta(const DevBasis &b, const int *first, int ns, double *z) {
    const double z0 = b.ao_zeta[2 * first[0]];
    for (int s = 0; s < ns; ++s)
        if (b.ao_nzeta[first[s]] != 1 || b.ao_zeta[2 * first[s]] != z0) return false;
    *z = z0;
    return true;
}

// S block of atoms ia != ib for B - A = (xab, yab, zab) (Angstrom): calls
// out(ja, jb, s) for every AO pair (a0 + ja of ia, b0 + jb of ib), jb outermost; s = 0
// beyond the cutoff.  Lined-up overlaps once per shell pair (from one table where
// every shell of an atom carries one exponent, the H/C/O EHT basis), then
//   <s|s> = s0, <s|p_i> = u_i s0, <p_i|s> = u_i s0, <p_i|p_j> = u_i u_j s0 + (d_ij - u_i u_j) s1
// with the direction cosines u: ROTATIONOVERLAP's matrices (overlap_D.f:520-583,
// :983-1027) for l <= 1, whose p row is (y, z, x) for m = -1, 0, 1.
template <typename Out>
__device__ void pair_overlap_block(const DevBasis &b, int ia, int ib, double xab, double yab, double zab,
                                   double cutoff, Out &&out) {
    const int a0 = b.atom_ao0[ia], na_ao = b.atom_nao[ia];
    const int b0 = b.atom_ao0[ib], nb_ao = b.atom_nao[ib];
    const double R = sqrt(xab * xab + yab * yab + zab * zab);
    if (R > cutoff) {
        for (int jb = 0; jb < nb_ao; ++jb)
            for (int ja = 0; ja < na_ao; ++ja) out(ja, jb, 0.0);
        return;
    }
    const double Rinv = 1.0 / R;
    const double u[3] = {yab * Rinv, zab * Rinv, xab * Rinv};  // by m + 1

    int fa[kMaxShell], fb[kMaxShell], sha[16], shb[16];
    const int nsa = na_ao <= 16 ? atom_shells(b, a0, na_ao, fa, sha) : -1;
    const int nsb = nb_ao <= 16 ? atom_shells(b, b0, nb_ao, fb, shb) : -1;
    const bool shells = nsa > 0 && nsb > 0;
    double sn[kMaxShell][kMaxShell][2];
    if (shells) {
        double za = 0.0, zb = 0.0;
        bool shared = uniform_zeta(b, fa, nsa, &za) && uniform_zeta(b, fb, nsb, &zb);
        sto::Reach need{0, 0, 0};
        for (int p = 0; p < nsa && shared; ++p)
            for (int q = 0; q < nsb; ++q) {
                const int na = b.ao_n[fa[p]], la = b.ao_l[fa[p]], nb = b.ao_n[fb[q]], lb = b.ao_l[fb[q]];
                shared = shared && sto::supported(na, la) && sto::supported(nb, lb);
                need = sto::widest(need, sto::reach(na, la, nb, lb));
            }
        if (shared) {
            sto::PairTable t;
            sto::pair_table(tables(), za, zb, R, need, t);
            for (int q = 0; q < nsb; ++q)
                for (int p = 0; p < nsa; ++p) {
                    sto::lined_up(t, b.ao_n[fa[p]], b.ao_l[fa[p]], b.ao_n[fb[q]], b.ao_l[fb[q]], sn[p][q]);
                    const double nn = b.ao_norm[2 * fa[p]] * b.ao_norm[2 * fb[q]];
                    sn[p][q][0] *= nn;
                    sn[p][q][1] *= nn;
                }
        } else {
            for (int q = 0; q < nsb; ++q)
                for (int p = 0; p < nsa; ++p) contracted_overlap(b, fa[p], fb[q], R, sn[p][q]);
        }
    }
    for (int jb = 0; jb < nb_ao; ++jb) {
        const int bb = b0 + jb, lb = b.ao_l[bb], mb = b.ao_m[bb];
        for (int ja = 0; ja < na_ao; ++ja) {
            const int aa = a0 + ja, la = b.ao_l[aa], ma = b.ao_m[aa];
            double two[2];
            const double *so = two;
            if (shells) so = sn[sha[ja]][shb[jb]];
            else contracted_overlap(b, aa, bb, R, two);
            double s = so[0];
            if (la) s *= u[ma + 1];
            if (lb) s *= u[mb + 1];
            if (la && lb) s += so[1] * ((ma == mb ? 1.0 : 0.0) - u[ma + 1] * u[mb + 1]);
            out(ja, jb, s);
        }
    }
}

// One thread per atom pair.  Threads walk the pairs in b.atom_order (atoms
// grouped by kind), so that the lanes of a warp mostly take the same shell and
// zeta loops; each pair is computed as (ia, ib) with ia >= ib in the input order,
// the same arithmetic whatever the walk.
__global__ void build_sh_kernel(DevBasis b, const double *__restrict__ coords, double cutoff,
                                double *__restrict__ S, double *__restrict__ h, int ld) {
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    if (py >= b.natoms || px >= b.natoms || px > py) return;
    int ia = b.atom_order ? b.atom_order[py] : py, ib = b.atom_order ? b.atom_order[px] : px;
    if (ib > ia) {
        const int t = ia;
        ia = ib;
        ib = t;
    }
    const int a0 = b.atom_ao0[ia], na_ao = b.atom_nao[ia];
    const int b0 = b.atom_ao0[ib], nb_ao = b.atom_nao[ib];

    if (ia == ib) {  // diagonal block: S = 1, h = IP + V_shift; same-atom off-diagonals 0
        for (int jb = 0; jb < nb_ao; ++jb)
            for (int ja = 0; ja < na_ao; ++ja) {
                const int r = a0 + ja, c = b0 + jb;
                const size_t o = (size_t)c * ld + r;
                S[o] = (r == c) ? 1.0 : 0.0;
                h[o] = (r == c) ? b.ao_ip[r] + b.ao_vshift[r] : 0.0;
            }
        return;
    }
    // B - A vector, lined-up frame (ROTATIONOVERLAP, overlap_D.f:558-574)
    const double xab = coords[3 * ib] - coords[3 * ia];
    const double yab = coords[3 * ib + 1] - coords[3 * ia + 1];
    const double zab = coords[3 * ib + 2] - coords[3 * ia + 2];
    // X_ij (a division) once per run of AOs with the same parameters on either atom
    auto same = [&](int x, int y) {
        return b.ao_ip[x] == b.ao_ip[y] && b.ao_vshift[x] == b.ao_vshift[y] && b.ao_kwh[x] == b.ao_kwh[y];
    };
    constexpr int kRow = 16;
    double xrow[kRow];  // X of (ja, the current run of ib's AOs)
    double x = 0.0;
    pair_overlap_block(b, ia, ib, xab, yab, zab, cutoff, [&](int ja, int jb, double s) {
        const int aa = a0 + ja, bb = b0 + jb;
        if (jb > 0 && ja < kRow && same(bb, bb - 1))
            x = xrow[ja];
        else if (!(ja > 0 && same(aa, aa - 1)))
            x = x_ij(b.ao_ip[aa], b.ao_ip[bb], b.ao_vshift[aa], b.ao_vshift[bb], b.ao_kwh[aa], b.ao_kwh[bb]);
        if (ja < kRow) xrow[ja] = x;
        const double hv = x * s;
        S[(size_t)bb * ld + aa] = s;
        S[(size_t)aa * ld + bb] = s;
        h[(size_t)bb * ld + aa] = hv;
        h[(size_t)aa * ld + bb] = hv;
    });
}

// Pulay (overlap-derivative) force terms of the Ehrenfest force
// (Ehrenfest, diabatic-Ehren.f:163-230): for every atom pair K < L with
// R_KL < cutoff and every direction, dS(j in L, i in K)/dR_K by central
// differences of the S block rebuilt with atom K displaced by +-delta
// (PULAY_OVERLAP, overlap_D.f:314-463), and
//   F[K][L][xyz] = -sum_{j in L} sum_{i in K} dS_ji/dR_K Kernel(i, j)
// (Kernel column-major, ld = ldk); F is natoms x natoms x 3, written for K < L only.
// One lane per (pair, direction, sign), five pairs a warp: one lane did the six
// builds of a pair before, so that 200 atoms were one warp per SM sub-partition and
// the run one warp's chain of FP64 instructions.  Pairs in atom_order (grouped by
// kind), like build_sh_kernel's.
constexpr int kMaxAoAtom = 16;
constexpr int kPulayPairs = 5;  // pairs per warp

__global__ void __launch_bounds__(128) pulay_pairs_kernel(DevBasis b, const double *__restrict__ coords, double cutoff,
                                                          double delta, const double *__restrict__ kernel, int ldk,
                                                          double *__restrict__ F) {
    const int lane = threadIdx.x & 31, slot = lane / 6, sub = lane % 6, xyz = sub >> 1;
    const bool minus = sub & 1;
    const int nat = b.natoms;
    const long long npairs = (long long)nat * (nat - 1) / 2;
    const long long pair = ((long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * kPulayPairs + slot;
    const bool valid = slot < kPulayPairs && pair < npairs;
    int L = 1, K = 0;
    if (valid) {  // pair = y (y - 1) / 2 + x, x < y
        long long y = (long long)((1.0f + sqrtf(1.0f + 8.0f * (float)pair)) * 0.5f);
        while (y * (y - 1) / 2 > pair) --y;
        while (y * (y + 1) / 2 <= pair) ++y;
        const int py = (int)y, px = (int)(pair - y * (y - 1) / 2);
        const int a = b.atom_order ? b.atom_order[py] : py, c = b.atom_order ? b.atom_order[px] : px;
        L = max(a, c);
        K = min(a, c);
    }
    double blk[kMaxAoAtom * kMaxAoAtom];  // S block, entry jb * na + ja (ja in L, jb in K)
    int na = 0, ne = 0, a0 = 0, b0 = 0;
    if (valid) {
        const double l[3] = {coords[3 * L], coords[3 * L + 1], coords[3 * L + 2]};
        double k[3] = {coords[3 * K], coords[3 * K + 1], coords[3 * K + 2]};
        const double dx = k[0] - l[0], dy = k[1] - l[1], dz = k[2] - l[2];
        a0 = b.atom_ao0[L];
        b0 = b.atom_ao0[K];
        na = b.atom_nao[L];
        const int nb = b.atom_nao[K];
        if (sqrt(dx * dx + dy * dy + dz * dz) < cutoff && na <= kMaxAoAtom && nb <= kMaxAoAtom) {
            ne = na * nb;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (c == xyz) k[c] = minus ? k[c] - delta : k[c] + delta;
            pair_overlap_block(b, L, K, k[0] - l[0], k[1] - l[1], k[2] - l[2], cutoff,
                               [&](int ja, int jb, double s) { blk[jb * na + ja] = s; });
        }
    }
    __syncwarp();
    const int nmax = __reduce_max_sync(0xffffffffu, ne);
    const double inv = 1.0 / (2.0 * delta);
    double f = 0.0;
    for (int e = 0, ja = 0, jb = 0; e < nmax; ++e) {  // the + and - lanes of a direction are neighbours
        const double v = e < ne ? blk[e] : 0.0;
        const double o = __shfl_xor_sync(0xffffffffu, v, 1);
        if (e < ne) f = f - (v - o) * inv * kernel[(size_t)(a0 + ja) * ldk + (b0 + jb)];
        if (++ja == na) {
            ja = 0;
            ++jb;
        }
    }
    if (valid && !minus) F[((size_t)K * nat + L) * 3 + xyz] = f;
}

// Extended-Hueckel Hamiltonian with environment fields (even_more_extended_Huckel
// and Huckel_with_FIELDS, hamiltonians.f:69-264), one thread per atom pair
// ia > ib closer than the cutoff: for i in ia, j in ib
//   h_ij = X_ij S_ij - [S_ij DP_1 + (mu_ij - (r0 - R_i) S_ij) . DP_2..4]   (|S_ij| > 1e-7)
// with r0 the midpoint of the two atoms, mu = dp_ao (the AO dipole matrix,
// N x N x 3, ld N) and DP the 4-vector (potential, field) of the pair, dp4
// (natoms x natoms x 4, entry (ia, ib)); h_ji = h_ij, h_ii = IP_i + V_shift_i.
// h must be zero on entry (blocks beyond the cutoff and same-atom off-diagonals stay 0).
__global__ void huckel_fields_kernel(DevBasis b, const double *__restrict__ coords, double cutoff,
                                     const double *__restrict__ S, int lds, const double *__restrict__ dp_ao,
                                     const double *__restrict__ dp4, double *__restrict__ h, int ldh) {
    const int ia = blockIdx.y * blockDim.y + threadIdx.y;
    const int ib = blockIdx.x * blockDim.x + threadIdx.x;
    const int nat = b.natoms, n = b.nao;
    if (ia >= nat || ib >= nat || ib > ia) return;
    const int a0 = b.atom_ao0[ia], na_ao = b.atom_nao[ia];
    const int b0 = b.atom_ao0[ib], nb_ao = b.atom_nao[ib];
    if (ia == ib) {
        for (int ja = 0; ja < na_ao; ++ja) h[(size_t)(a0 + ja) * ldh + a0 + ja] = b.ao_ip[a0 + ja] + b.ao_vshift[a0 + ja];
        return;
    }
    const double dx = coords[3 * ib] - coords[3 * ia], dy = coords[3 * ib + 1] - coords[3 * ia + 1],
                 dz = coords[3 * ib + 2] - coords[3 * ia + 2];
    if (sqrt(dx * dx + dy * dy + dz * dz) > cutoff) return;
    const double Ri[3] = {coords[3 * ia], coords[3 * ia + 1], coords[3 * ia + 2]};
    const double r0[3] = {(coords[3 * ia] + coords[3 * ib]) / 2.0, (coords[3 * ia + 1] + coords[3 * ib + 1]) / 2.0,
                          (coords[3 * ia + 2] + coords[3 * ib + 2]) / 2.0};
    const size_t nn = (size_t)nat * nat;
    const double DP[4] = {dp4[(size_t)ib * nat + ia], dp4[nn + (size_t)ib * nat + ia],
                          dp4[2 * nn + (size_t)ib * nat + ia], dp4[3 * nn + (size_t)ib * nat + ia]};
    const size_t n2 = (size_t)n * n;
    for (int jb = 0; jb < nb_ao; ++jb) {
        const int j = b0 + jb;
        for (int ja = 0; ja < na_ao; ++ja) {
            const int i = a0 + ja;
            const double sij = S[(size_t)j * lds + i];
            double v = x_ij(b.ao_ip[i], b.ao_ip[j], b.ao_vshift[i], b.ao_vshift[j], b.ao_kwh[i], b.ao_kwh[j]) * sij;
            if (fabs(sij) > 1.0e-7) {
                double vec[3];
                for (int c = 0; c < 3; ++c) vec[c] = dp_ao[c * n2 + (size_t)j * n + i] - (r0[c] - Ri[c]) * sij;
                v = v - (sij * DP[0] + (vec[0] * DP[1] + vec[1] * DP[2] + vec[2] * DP[3]));
            }
            h[(size_t)j * ldh + i] = v;
            h[(size_t)i * ldh + j] = v;
        }
    }
}

// force(a)[xyz] = scale * (sum_{L > a} F[a][L] - sum_{K < a} F[K][a]), one warp each,
// fixed order (the atom(i)%Ehrenfest sum over F_snd, diabatic-Ehren.f:140-148 with 216-223)
__global__ void pulay_reduce_kernel(const double *__restrict__ F, int nat, double scale, double *__restrict__ force) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
    if (t >= 3 * nat) return;
    const int a = t / 3, xyz = t % 3;
    double s = 0.0;
    for (int q = lane; q < nat; q += 32) {
        if (q > a) s = s + F[((size_t)a * nat + q) * 3 + xyz];
        else if (q < a) s = s - F[((size_t)q * nat + a) * 3 + xyz];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) force[t] = scale * s;
}

}  // namespace

double sto_norm(double zeta, int n, int l) { return sto::norm(zeta, n, l); }

cudaError_t init_build_tables() {
    init_tables_kernel<<<(sto::kTableMax + 255) / 256, 256>>>();
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return e;
}

cudaError_t launch_pulay_forces(const DevBasis &b, const double *d_coords, double cutoff, double delta,
                                const double *d_kernel, int ldk, double *d_F, double scale, double *d_force,
                                cudaStream_t st) {
    if (b.natoms <= 0) return cudaSuccess;
    const long long warps = ((long long)b.natoms * (b.natoms - 1) / 2 + kPulayPairs - 1) / kPulayPairs;
    if (warps > 0) {
        pulay_pairs_kernel<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(b, d_coords, cutoff, delta, d_kernel, ldk, d_F);
        count_launch();
    }
    pulay_reduce_kernel<<<(3 * b.natoms + 3) / 4, 128, 0, st>>>(d_F, b.natoms, scale, d_force);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_huckel_fields(const DevBasis &b, const double *d_coords, double cutoff, const double *d_S, int lds,
                                 const double *d_dp_ao, const double *d_dp4, double *d_h, int ldh, cudaStream_t st) {
    if (b.natoms <= 0) return cudaSuccess;
    dim3 block(16, 8);
    dim3 grid((b.natoms + block.x - 1) / block.x, (b.natoms + block.y - 1) / block.y);
    huckel_fields_kernel<<<grid, block, 0, st>>>(b, d_coords, cutoff, d_S, lds, d_dp_ao, d_dp4, d_h, ldh);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_build_sh(const DevBasis &b, const double *d_coords, double cutoff, double *d_S,
                            double *d_h, int ld, cudaStream_t st) {
    if (b.natoms <= 0) return cudaSuccess;
    dim3 block(16, 8);
    dim3 grid((b.natoms + block.x - 1) / block.x, (b.natoms + block.y - 1) / block.y);
    build_sh_kernel<<<grid, block, 0, st>>>(b, d_coords, cutoff, d_S, d_h, ld);
    count_launch();
    return cudaGetLastError();
}

}  // namespace elhl
