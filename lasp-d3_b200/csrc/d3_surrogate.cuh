// Descriptors of the learned ATM surrogate and their backward pass.
// Included by d3_engine.cu after the kernel parameter block and the traversal helper.
//
// For atom i, neighbour-element channel c and radial function k (32 per channel):
//     G_i[c][k] = sum_{j,T: 0 < r_ij <= rc_ATM, chan(j) = c} C6_ij psi_k(r_ij)
//     psi_k(r) = exp(-(r - mu_k)^2 / (2 sigma^2)) fc(r),  fc(r) = (1 + cos(pi r / rc)) / 2
// with mu_k uniform in [0.8, 21] A and sigma = 0.7 A (in bohr here), C6_ij the exact
// CN-dependent coefficient of the pair. The smooth cutoff keeps energies continuous.
//
// Backward, given dE/dG for every atom (E = sum_i E_i(G_i), E in the engine's stored sign):
//     a_ij = C6_ij sum_k dE_i/dG_i[c_j][k] psi_k'(r),   b_ij = sum_k dE_i/dG_i[c_j][k] psi_k(r)
//     force (gradient) on i:  sum_j (a_ij + a_ji) (x_i - x_j) / r_ij
//     dE/dCN_i:               sum_j (b_ij + b_ji) dC6_ij/dCN_i
//     virial:                 -(x_i - x_j) (x) (x_i - x_j) (a_ij + a_ji) / (2 V r) per ordered pair
// Forward: one warp per atom, one lane per radial function; backward: one lane per
// neighbour. Neighbours come from the rc_ATM stencil. The cutoff function is evaluated in
// FP32 (sincospif) in both passes.

constexpr int SURR_NRBF = 32;
constexpr int SURR_MAXCH = 8;
constexpr int SURR_WARPS = 4; // warps (atoms) per CTA of the descriptor kernels

struct SurrDesc {
    const int *chan;   // channel of each handle type (-1: not covered)
    int nch;
    float mu0, dmu;    // bohr
    float inv2s2;      // 1 / (2 sigma^2), bohr^-2
    float *G;          // [n][nch][32], binned order
    const float *dEdG; // [n][nch][32], binned order (backward input)
    int *center;       // [n] channel of each atom (binned order), -1: not a channel
};

// smooth cutoff fc(r) = (1 + cos(pi r / rc)) / 2 and its derivative, FP32 (the same
// values in the forward and the backward pass)
__device__ __forceinline__ void surr_cutoff(float r, float inv_rc, float &fc, float &dfc) {
    float sn, cs;
    sincospif(r * inv_rc, &sn, &cs);
    fc = 0.5f * (1.0f + cs);
    dfc = -0.5f * 3.14159265358979f * inv_rc * sn;
}

// In-range neighbours of an atom, compacted: every stencil candidate is only tested for
// distance; those within the cutoff go to a per-warp queue (separation and atom), and
// batch(valid) is called (converged) with 32 of them, one per lane at q[lane], the last time
// with the remainder. C6, root and cutoff function are then evaluated by full warps only:
// about 12 of 32 candidates of a chunk are in range. Both passes share this walk.
struct SurrNb {
    double dx, dy, dz, d2;
    int j, pad;
};

template <class F>
__device__ __forceinline__ void surr_neighbours(const KP &p, const SG &g, int i, const double4 &xi, SurrNb *q, F &&batch) {
    const int lane = threadIdx.x & 31;
    const int4 si = p.shift[i];
    // without atoms given outside the cell the image box is a test of the image alone
    const bool box_pair = g.box_mode && p.anyshift[p.sid[i]];
    int count = 0; // queued neighbours (warp-uniform)
    traverse(p, g, p.bin_s[i], p.stencils + g.sta_off, g.sta_n, [&](int j, int Tx, int Ty, int Tz, const double3 &sh, bool act) {
        if (g.box_mode && !box_pair && (abs(Tx) > g.half[0] || abs(Ty) > g.half[1] || abs(Tz) > g.half[2])) return;
        bool keep = false;
        SurrNb nb;
        if (act) {
            const double4 xj = p.xs[j];
            nb.dx = xi.x - (xj.x + sh.x);
            nb.dy = xi.y - (xj.y + sh.y);
            nb.dz = xi.z - (xj.z + sh.z);
            nb.d2 = nb.dx * nb.dx + nb.dy * nb.dy + nb.dz * nb.dz;
            nb.j = j;
            keep = nb.d2 <= p.ratm2 && nb.d2 > 0.0 && (!box_pair || in_box(g, si, p.shift[j], Tx, Ty, Tz));
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) q[count + __popc(m & ((1u << lane) - 1u))] = nb;
        count += __popc(m);
        if (count >= 32) {
            __syncwarp();
            batch(true);
            __syncwarp();
            if (lane < count - 32) q[lane] = q[32 + lane];
            count -= 32;
            __syncwarp();
        }
    });
    __syncwarp();
    if (count > 0) batch(lane < count);
}

// Forward: lane k of the atom's warp owns radial function k. The batch's neighbours, one per
// lane, go on to a queue per channel; a channel with 32 of them is summed in one unrolled loop
// of broadcast loads (independent exponentials; walking them through ballots and shuffles left
// each waiting for the one before) and added to its sum in shared memory. 30,000-atom box,
// forward pass with the network: 9.9 -> 5.9 ms.
template <int NR>
__global__ void __launch_bounds__(SURR_WARPS * 32) k_desc_fwd(KP p, SurrDesc sd) {
    __shared__ SurrNb Q[SURR_WARPS][64];
    __shared__ float2 C[SURR_WARPS][SURR_MAXCH][64]; // r, C6 fc of the neighbours of a channel
    __shared__ int N[SURR_WARPS][SURR_MAXCH];
    __shared__ float A[SURR_WARPS][SURR_MAXCH][32];
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (i >= p.n) return;
    const SG &g = p.sg[p.sid[i]];
    SurrNb *q = Q[warp];
    const double4 xi = p.xs[i];
    const int ti = (int)xi.w;
    if (lane == 0) sd.center[i] = sd.chan[ti];
    double wi[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a) wi[a] = p.w[(size_t)i * NR + a];
    const float mu_k = sd.mu0 + sd.dmu * lane;
    const float inv_rc = (float)(1.0 / sqrt(p.ratm2));
    const int nch = sd.nch;
    for (int c = 0; c < nch; ++c) A[warp][c][lane] = 0.f;
    if (lane < nch) N[warp][lane] = 0;
    __syncwarp();
    // add the first m queued neighbours of channel c
    auto add = [&](int c, int m) {
        const float2 *e = C[warp][c];
        float s0 = 0.f, s1 = 0.f;
        int k = 0;
#pragma unroll 1
        for (; k + 8 <= m; k += 8) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float2 v = e[k + u];
                const float d = v.x - mu_k;
                float &s = (u & 1) ? s1 : s0;
                s = fmaf(v.y, __expf(-d * d * sd.inv2s2), s);
            }
        }
        for (; k < m; ++k) {
            const float2 v = e[k];
            const float d = v.x - mu_k;
            s0 = fmaf(v.y, __expf(-d * d * sd.inv2s2), s0);
        }
        A[warp][c][lane] += s0 + s1;
    };
    surr_neighbours(p, g, i, xi, q, [&](bool valid) {
        float r = 0.f, wgt = 0.f;
        int ch = -1;
        if (valid) {
            const SurrNb nb = q[lane];
            const int cj = sd.chan[(int)p.xs[nb.j].w];
            if (cj >= 0) {
                const double *yj = p.Y + ((size_t)nb.j * p.ne + ti) * NR;
                double c6 = 0.0;
#pragma unroll
                for (int b = 0; b < NR; ++b) c6 += yj[b] * wi[b];
                r = (float)sqrt(nb.d2);
                float fc, dfc;
                surr_cutoff(r, inv_rc, fc, dfc);
                wgt = (float)c6 * fc;
                ch = cj;
            }
        }
        const unsigned same = __match_any_sync(0xffffffffu, ch);
        const int rank = __popc(same & ((1u << lane) - 1u)), base = ch >= 0 ? N[warp][ch] : 0;
        __syncwarp();
        if (ch >= 0) {
            C[warp][ch][base + rank] = make_float2(r, wgt);
            if (rank == 0) N[warp][ch] = base + __popc(same);
        }
        __syncwarp();
        unsigned ready = __ballot_sync(0xffffffffu, lane < nch && N[warp][lane < nch ? lane : 0] >= 32);
        while (ready) {
            const int c = __ffs(ready) - 1;
            ready &= ready - 1u;
            add(c, 32);
            const int left = N[warp][c] - 32;
            __syncwarp();
            if (lane < left) C[warp][c][lane] = C[warp][c][32 + lane];
            if (lane == 0) N[warp][c] = left;
            __syncwarp();
        }
    });
    __syncwarp();
    float *out = sd.G + (size_t)i * nch * SURR_NRBF;
    for (int c = 0; c < nch; ++c) {
        add(c, N[warp][c]);
        out[c * SURR_NRBF + lane] = A[warp][c][lane];
    }
}

// Backward, one warp per atom and one neighbour per lane. With phi_k = exp(-(r - mu_k)^2
// / (2 sigma^2)), psi_k = phi_k fc and g_k = dE/dG_i[c_j][k] + dE/dG_j[c_i][k]:
//     sum_k g_k psi_k  = fc S0,   sum_k g_k psi_k' = dfc S0 - 2 fc S1 / (2 sigma^2)
//     S0 = sum_k g_k phi_k,       S1 = sum_k g_k phi_k (r - mu_k)
// so each neighbour costs 32 exponentials and two FMAs per radial function; the atom's own
// dE/dG rows sit in shared memory (rows padded to 33 floats: lanes reading different
// channels at the same k hit different banks), the neighbour's row is read as 8 float4
// (copying whole rows to shared memory first, coalesced: 12.4 ms instead of 8.7).
template <int NR>
__global__ void __launch_bounds__(SURR_WARPS * 32, 4) k_desc_bwd(KP p, SurrDesc sd) {
    constexpr int PITCH = SURR_NRBF + 1;
    __shared__ float Ds[SURR_WARPS][SURR_MAXCH * PITCH];
    __shared__ SurrNb Q[SURR_WARPS][64];
    const int warp_in_block = threadIdx.x >> 5;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const SG &g = p.sg[p.sid[i]];
    float *Dw = Ds[warp_in_block];
    SurrNb *q = Q[warp_in_block];
    const float *din = sd.dEdG + (size_t)i * sd.nch * SURR_NRBF;
    for (int c = 0; c < sd.nch; ++c) Dw[c * PITCH + lane] = din[c * SURR_NRBF + lane];
    __syncwarp();
    const double4 xi = p.xs[i];
    const int ti = (int)xi.w;
    const int chi = sd.chan[ti];
    double wi[NR], dwi[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a) {
        wi[a] = p.w[(size_t)i * NR + a];
        dwi[a] = p.dw[(size_t)i * NR + a];
    }
    const float inv_rc = (float)(1.0 / sqrt(p.ratm2));
    const float a2 = sd.inv2s2;
    double fx = 0, fy = 0, fz = 0, gcn = 0, vxx = 0, vyy = 0, vzz = 0, vxy = 0, vxz = 0, vyz = 0;
    // one queued neighbour per lane: the radial sums and their contributions
    auto process = [&](bool valid) {
        if (!valid || chi < 0) return;
        const SurrNb nb = q[lane];
        const int ch = sd.chan[(int)p.xs[nb.j].w];
        if (ch < 0) return;
        const double *yj = p.Y + ((size_t)nb.j * p.ne + ti) * NR;
        double c6d = 0.0, dc6d = 0.0;
#pragma unroll
        for (int b = 0; b < NR; ++b) {
            c6d += yj[b] * wi[b];
            dc6d += yj[b] * dwi[b]; // dC6_ij/dCN_i
        }
        const float r = (float)sqrt(nb.d2), c6 = (float)c6d, dc6 = (float)dc6d;
        float fc, dfc;
        surr_cutoff(r, inv_rc, fc, dfc);
        const float4 *gj = reinterpret_cast<const float4 *>(sd.dEdG + ((size_t)nb.j * sd.nch + chi) * SURR_NRBF);
        const float *gi = Dw + ch * PITCH;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int qd = 0; qd < SURR_NRBF / 4; ++qd) {
            const float4 v = __ldg(gj + qd);
            const float gv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int k = 4 * qd + t;
                const float u = r - (sd.mu0 + sd.dmu * k);
                const float w = (gv[t] + gi[k]) * __expf(-u * u * a2);
                s0 += w;
                s1 = fmaf(w, u, s1);
            }
        }
        // dE/dr / r and dE/dC6_ij
        const double fs = (double)c6 * ((double)dfc * s0 - 2.0 * (double)a2 * (double)fc * s1) / (double)r;
        const double dx = (float)nb.dx, dy = (float)nb.dy, dz = (float)nb.dz;
        fx += fs * dx;
        fy += fs * dy;
        fz += fs * dz;
        vxx += fs * dx * dx;
        vyy += fs * dy * dy;
        vzz += fs * dz * dz;
        vxy += fs * dx * dy;
        vxz += fs * dx * dz;
        vyz += fs * dy * dz;
        gcn += (double)(fc * s0) * (double)dc6; // dE/dC6_ij dC6_ij/dCN_i
    };
    surr_neighbours(p, g, i, xi, q, process);
    fx = warp_sum(fx);
    fy = warp_sum(fy);
    fz = warp_sum(fz);
    gcn = warp_sum(gcn);
    vxx = warp_sum(vxx);
    vyy = warp_sum(vyy);
    vzz = warp_sum(vzz);
    vxy = warp_sum(vxy);
    vxz = warp_sum(vxz);
    vyz = warp_sum(vyz);
    if (lane == 0) {
        // the surrogate's share enters through the ATM apex arrays (entry arrays stay zero
        // for atoms the surrogate covers)
        p.fa[3 * i] += fx;
        p.fa[3 * i + 1] += fy;
        p.fa[3 * i + 2] += fz;
        p.ga[i] += gcn;
        const double sc = -1.0 / (2.0 * g.vol);
        double *v = p.va + 6 * (size_t)i;
        v[0] += vxx * sc;
        v[1] += vyy * sc;
        v[2] += vzz * sc;
        v[3] += vxy * sc;
        v[4] += vxz * sc;
        v[5] += vyz * sc;
    }
}
