// ATM three-body kernel, FP64, block-pair schedule: every triplet visited once. Included by
// d3_engine.cu after d3_atm.cuh (same entries, term and weights as k_atm64).
//
// Per (apex, split) item: the entries of the half list are sorted along a Hilbert curve (in a
// fixed order, so that the splits of an apex agree on its blocks) and cut into blocks of 32.
// A warp takes (block A, part of the blocks B >= A) units; lane L owns entry x = A[L] and at
// step s visits y = B[(L + s) mod 32] (diagonal blocks: steps 1..16, step 16 on lanes 0..15
// only), so no two lanes of a step touch one y. The distance tests of all steps run first (FP32;
// pairs near a limit again in FP64) and steps without a pair in range are skipped. x sums stay in registers over
// the unit; y sums travel with their y by shuffles (as many lanes as steps have passed) and
// are added once per block pair to the entry's accumulators in this CTA's scratch (L2
// atomics). The y block (records, and for every type the entry's C6 row Y, derivative row D
// and r0^2 from the YD64 table) is staged in shared memory by cp.async.
//   C6_xy = Y_y[t_x] . w_x, dC6_xy/dCN_x = Y_y[t_x] . dw_x, dC6_xy/dCN_y = D_y[t_x] . w_x
//
// Against k_atm64 (two visits a triplet, 83 FP64 operations each, nearly all lanes busy):
// one visit of 100 operations with 70 % of the lanes in range. Bound: latency of the visit's
// chain with three warps per scheduler (8, 9, 10, 12 warps a CTA: 162, 153, 147, 138 ms on 8,000
// atoms; the shared memory and 168 registers hold no more), beside it instruction issue (47 %
// busy, an FP64 instruction counting twice) and the shared-memory pipe (59 %). Testing every
// step just before its visit took 186 ms instead of 157.
// ATM pass on a B200, k_atm64 -> this kernel: 96-atom water box 2.65 -> 2.11 ms, 777 atoms 20.7
// -> 17.9 ms, 2,000 atoms 50.0 -> 44.3 ms, 20,000-atom box 443 -> 394 ms (383 with two
// CTAs per SM), batch of 48 structures 106 -> 98 ms.

constexpr int ATM64B_WARPS = 12;   // warps per SM at most (168 registers a thread)
constexpr int ATM64B_MCAP = 4096;  // longest list at most (KP::atmb_mcap; longer ones: k_atm64)
constexpr int ATM64B_NACC = 8;     // accumulators per entry: E, dE/dCN, force, virial coefficient
constexpr int ATM64B_STATIC = 2560;

__host__ __device__ inline size_t atm64b_fixed(int ne, int NR) {
    size_t b = 2 * (size_t)(ATM64B_MCAP / 32) * sizeof(float4); // block boxes
    b += (size_t)((ne * NR + 1) & ~1) * sizeof(double) + (size_t)((ne * ne + 1) & ~1) * sizeof(double);
    return (b + 15) & ~(size_t)15;
}
// per warp: rows of the y block, its records and FP32 positions, virial carries (weighted kind)
__host__ __device__ inline size_t atm64b_warp(int ne, int NR, bool simple) {
    return 32 * ((size_t)ne * atm64b_row(NR) * sizeof(double) + 3 * sizeof(double2) + sizeof(float4) + (simple ? 0 : 6 * sizeof(double)));
}
// scratch of one CTA: atmb_mcap entries, then their accumulators
constexpr size_t ATM64B_ENTRY_BYTES = sizeof(Atm64Row) + ATM64B_NACC * sizeof(double);

template <int NR, bool SIMPLE>
__global__ void __launch_bounds__(ATM64B_WARPS * 32, 1) k_atm64b(KP p, unsigned char *scratch) {
    extern __shared__ __align__(16) unsigned char sm64b[];
    constexpr int RW = atm64b_row(NR) / 2; // double2 words per row
    const int ne = p.ne, nw = blockDim.x >> 5;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4 *box = reinterpret_cast<float4 *>(sm64b);                   // [MCAP / 32][2]
    double *yapex = reinterpret_cast<double *>(box + 2 * (ATM64B_MCAP / 32)); // [ne][NR]
    double *r0sq = yapex + ((ne * NR + 1) & ~1);                       // [ne][ne]
    unsigned char *stage = sm64b + atm64b_fixed(ne, NR);
    double2 *yR = reinterpret_cast<double2 *>(stage + (size_t)warp * atm64b_warp(ne, NR, SIMPLE)); // [ne][RW][32]
    double2 *yA = yR + (size_t)ne * RW * 32;                           // [3][32]: vx vy | vz id | p g
    float4 *yF = reinterpret_cast<float4 *>(yA + 96);                  // [32] FP32 position, atom
    double *carry = reinterpret_cast<double *>(yF + 32) + lane;        // [6][32]: virial cross terms
    // while the entries are sorted the staging area holds the cells and the entry numbers
    int *cells = reinterpret_cast<int *>(stage), *order = cells + ATM64_CELLS;
    __shared__ int s_item, s_unit, s_tot[ATM64B_WARPS];
    __shared__ double red[ATM64B_WARPS][12];
    if (warp_uniform(p.atm_off[p.n] > p.atm_cap ? 1 : 0)) return; // list overflowed: the host grows it and re-runs
    for (int k = tid; k < ne * ne; k += blockDim.x) r0sq[k] = p.r0ab[k] * p.r0ab[k];
    Atm64Row *entries = reinterpret_cast<Atm64Row *>(scratch + blockIdx.x * (ATM64B_ENTRY_BYTES * p.atmb_mcap));
    double (*acc)[ATM64B_NACC] = reinterpret_cast<double (*)[ATM64B_NACC]>(entries + p.atmb_mcap);
    const double rc = sqrt(p.ratm2), cinv = 16.0 / (2.0 * rc);
    const float half = (float)(0.5 * p.ratm2 * (1.0 + 1e-5)), sure = half * (1.0f - 4e-5f);
    const float rc_hi = (float)(p.ratm2 * (1.0 + 1e-4));
    unsigned long long visits = 0;
    while (true) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(p.work, 1);
        __syncthreads();
        const int S = p.atmb_split;
        const int got = warp_uniform(s_item), split = got % S, item = (got / S) * p.shard_world + p.shard_rank;
        if (item >= p.n) break;
        const int a = p.sorted_of[p.n - 1 - item];
        const SG &g = p.sg[p.sid[a]];
        const long long e0 = p.atm_off[a];
        const int m = warp_uniform((int)(p.atm_off[a + 1] - e0));
        if (m > p.atmb_mcap || warp_uniform(g.atm_simple) != (SIMPLE ? 1 : 0)) continue; // k_atm64's, the other instance's
        const bool ref = !SIMPLE && atm_reference_order(p, g, p.sid[a]);
        const double4 xa = p.xs[a];
        for (int k = tid; k < ne * NR; k += blockDim.x) yapex[k] = p.Y[(size_t)a * ne * NR + k];
        // ---- entries in Hilbert order (counting sort, each cell by entry number)
        const int hs = m >= 1024 ? 0 : (m >= 128 ? 3 : 6), ncell = ATM64_CELLS >> hs;
        auto cell_of = [&](const int2 ent) {
            const double3 v = atm64_pos(p, g, xa, ent, p.xs[ent.x]);
            const int cx = min(15, max(0, (int)((v.x + rc) * cinv)));
            const int cy = min(15, max(0, (int)((v.y + rc) * cinv)));
            const int cz = min(15, max(0, (int)((v.z + rc) * cinv)));
            return atmb_hilbert(cx, cy, cz) >> hs;
        };
        for (int k = tid; k < ncell; k += blockDim.x) cells[k] = 0;
        if (tid == 0) s_unit = 0;
        __syncthreads();
        for (int k = tid; k < m; k += blockDim.x) atomicAdd(&cells[cell_of(p.atm_ent[e0 + k])], 1);
        __syncthreads();
        atm64_scan(cells, ncell, s_tot);
        __syncthreads();
        for (int k = tid; k < m; k += blockDim.x) order[atomicAdd(&cells[cell_of(p.atm_ent[e0 + k])], 1)] = k;
        __syncthreads();
        for (int c = tid; c < ncell; c += blockDim.x) {
            const int lo = c ? cells[c - 1] : 0, hi = cells[c];
            for (int q = lo + 1; q < hi; ++q) {
                const int v = order[q];
                int r = q - 1;
                while (r >= lo && order[r] > v) {
                    order[r + 1] = order[r];
                    --r;
                }
                order[r + 1] = v;
            }
        }
        __syncthreads();
        for (int k = tid; k < m; k += blockDim.x) {
            entries[k] = atm64_entry<NR>(p, g, xa, a, p.atm_ent[e0 + order[k]], yapex, r0sq + (int)xa.w * ne, true);
#pragma unroll
            for (int q = 0; q < 6; ++q) __stcg(&acc[k][q], 0.0);
        }
        __syncthreads();
        const int nb = (m + 31) >> 5;
        for (int b = warp_uniform(warp); b < nb; b += nw) {
            const Atm64Row *r = entries + min(32 * b + lane, m - 1);
            float lo[3] = {r->f[0], r->f[1], r->f[2]}, hi[3] = {lo[0], lo[1], lo[2]};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    lo[q] = fminf(lo[q], __shfl_xor_sync(0xffffffffu, lo[q], o));
                    hi[q] = fmaxf(hi[q], __shfl_xor_sync(0xffffffffu, hi[q], o));
                }
            if (lane == 0) {
                box[2 * b] = make_float4(lo[0], lo[1], lo[2], 0.f);
                box[2 * b + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
            }
        }
        if (!SIMPLE)
#pragma unroll
            for (int q = 0; q < 6; ++q) carry[32 * q] = 0.0;
        __syncthreads();
        // ---- units (A, q): block A with blocks B = A + q, A + q + Q, ... in order of A, Q parts
        // so that the splits' warps all find some
        const int Q = max(1, min(16, (4 * nw * S + nb - 1) / max(1, nb)));
        for (;;) {
            int u = 0;
            if (lane == 0) u = split + S * atomicAdd(&s_unit, 1);
            u = warp_uniform(u);
            if (u >= nb * Q) break;
            const int A = u / Q;
            const int xe = 32 * A + lane;
            const bool xv = xe < m;
            const Atm64Row *X = entries + min(xe, m - 1);
            const double vx = X->v[0], vy = X->v[1], vz = X->v[2], id1 = X->id, h1 = 0.75 * id1;
            const double d1 = vx * vx + vy * vy + vz * vz;
            const double p1 = X->p, g1 = X->g * (6.0 * 4294967296.0 / 43046721.0); // 6 (4/3)^16
            const int jx = X->j;
            const float fx = xv ? X->f[0] : 3e18f, fy = X->f[1], fz = X->f[2];
            const double2 *yRx = yR + (size_t)X->t * RW * 32;
            double wx[NR], dwx[NR];
#pragma unroll
            for (int b = 0; b < NR; ++b) {
                wx[b] = p.w[(size_t)jx * NR + b];
                dwx[b] = p.dw[(size_t)jx * NR + b];
            }
            // x sums: E, dE/dCN part, wf (f1 + f3), wf f3 v_y (3); weighted kind: (w - wf) times
            // (f1 + f3) and f3 v_y
            double SE = 0, SD = 0, SF = 0, Wx = 0, Wy = 0, Wz = 0, SC = 0, Ux = 0, Uy = 0, Uz = 0;
            const float4 la = box[2 * A], ha = box[2 * A + 1];
            for (int B = A + (u - A * Q); B < nb; B += Q) {
                const float4 lb = box[2 * B], hb = box[2 * B + 1];
                const float nx = fmaxf(0.f, fmaxf(la.x - hb.x, lb.x - ha.x)), ny = fmaxf(0.f, fmaxf(la.y - hb.y, lb.y - ha.y)),
                            nz = fmaxf(0.f, fmaxf(la.z - hb.z, lb.z - ha.z));
                if (warp_uniform(nx * nx + ny * ny + nz * nz > rc_hi ? 1 : 0)) continue;
                // ---- stage block B (entries past the last one: copies of it, far FP32 position)
                const int ye = 32 * B + lane;
                const Atm64Row *Y = entries + min(ye, m - 1);
                __syncwarp(); // every lane is done with the previous block
                {
                    const char *src = reinterpret_cast<const char *>(p.YD64 + (size_t)Y->j * ne * atm64b_row(NR));
                    for (int t = 0; t < ne * RW; ++t) atmb_cp16(yR + 32 * t + lane, src + 16 * t);
                    const char *rec = reinterpret_cast<const char *>(Y);
#pragma unroll
                    for (int q = 0; q < 3; ++q) atmb_cp16(yA + 32 * q + lane, rec + 16 * q);
                    atmb_cp_commit();
                    yF[lane] = make_float4(ye < m ? Y->f[0] : -3e18f, Y->f[1], Y->f[2], __int_as_float(Y->j));
                    atmb_cp_wait<0>();
                }
                __syncwarp();
                const bool diag = A == B;
                // y sums (travelling): E, dE/dCN part, minus the force; weighted: (w - wf)(f2 + f3)
                double yE = 0, yD = 0, yX = 0, yY = 0, yZ = 0, yC = 0;
                // steps of this lane in range (bit s), all 32 tested ahead of the visits
                unsigned my = 0;
                bool edge = false;
#pragma unroll
                for (int s = 0; s < 32; ++s) {
                    const float4 f = yF[(lane + s) & 31];
                    const float dx = fx - f.x, dy = fy - f.y, dz = fz - f.z;
                    const float off = fabsf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - half);
                    my |= off <= half ? 1u << s : 0u;
                    edge |= off <= half && off >= sure;
                }
                if (diag) my &= lane < 16 ? 0x1fffeu : 0xfffeu;
                if (warp_uniform(edge ? 1 : 0)) {
                    for (unsigned left = my; left; left &= left - 1) {
                        const int s = __ffs(left) - 1, k = (lane + s) & 31;
                        const double2 A0 = yA[k];
                        const double rx = vx - A0.x, ry = vy - A0.y, rz = vz - yA[32 + k].x;
                        const double d3 = fma(rx, rx, fma(ry, ry, rz * rz));
                        if (!(d3 <= p.ratm2 && d3 >= 1e-12)) my &= ~(1u << s);
                    }
                    __syncwarp();
                }
                visits += 2u * __popc(my);
                int at = 0; // step the travelling sums are aligned to
                unsigned todo = __reduce_or_sync(0xffffffffu, my);
#pragma unroll 1
                while (todo) {
                    const int s = __ffs(todo) - 1, k = (lane + s) & 31;
                    todo &= todo - 1;
                    const bool act = (my >> s) & 1;
                    const double2 A0 = yA[k], A1 = yA[32 + k], A2 = yA[64 + k];
                    const double rx = vx - A0.x, ry = vy - A0.y, rz = vz - A1.x;
                    double d3 = fma(rx, rx, fma(ry, ry, rz * rz));
                    d3 = act ? d3 : 1.0;
                    // align the travelling sums with this step's y
                    {
                        const int src = (lane + s - at) & 31;
                        at = s;
                        yE = __shfl_sync(0xffffffffu, yE, src);
                        yD = __shfl_sync(0xffffffffu, yD, src);
                        yX = __shfl_sync(0xffffffffu, yX, src);
                        yY = __shfl_sync(0xffffffffu, yY, src);
                        yZ = __shfl_sync(0xffffffffu, yZ, src);
                        if (!SIMPLE) yC = __shfl_sync(0xffffffffu, yC, src);
                    }
                    double r[2 * RW];
#pragma unroll
                    for (int b = 0; b < RW; ++b) {
                        const double2 v = yRx[32 * b + k];
                        r[2 * b] = v.x;
                        r[2 * b + 1] = v.y;
                    }
                    double c6 = r[0] * wx[0], dcx = r[0] * dwx[0], dcy = r[NR] * wx[0];
#pragma unroll
                    for (int b = 1; b < NR; ++b) {
                        c6 = fma(r[b], wx[b], c6);
                        dcx = fma(r[b], dwx[b], dcx);
                        dcy = fma(r[NR + b], wx[b], dcy);
                    }
                    const double id2 = A1.y, d2 = fma(A0.x, A0.x, fma(A0.y, A0.y, A1.x * A1.x));
                    const double cd = c6 * d3, q = rsqrt_nr(cd), q2 = q * q, id3 = c6 * q2;
                    const double C = (act ? p1 : 0.0) * A2.x * (cd * q * (id3 * id3));
                    const double u3 = r[2 * NR] * id3;
                    const double g3 = u3 * u3 * u3 * rcbrt_nr(u3);
                    const double fd = rcp_nr(fma(g1 * A2.y, g3, 1.0));
                    const double H = h1 * id2 * id3;
                    const double t1 = d1 + d2 - d3, m12 = d1 - d2, t2 = m12 + d3, t3 = d3 - m12;
                    const double t12 = t1 * t2, t13 = t1 * t3, t23 = t2 * t3;
                    const double uu = t12 * t3 * H;
                    const double Bu = fma(0.5, uu, 1.0);
                    const double Ef = C * fd;
                    const double Sf = Ef * fma(fma(16.0 / 3.0, fd, -16.0 / 3.0), Bu, fma(2.5, uu, 3.0));
                    const double V = Ef * H, dt = t23 - t12;
                    double f1 = fma(-V, t13 + dt, id1 * Sf);
                    double f2 = fma(-V, t12 + t23 - t13, id2 * Sf);
                    double f3 = fma(-V, t13 - dt, id3 * Sf);
                    double E = Ef * Bu; // minus the energy
                    if (!SIMPLE) {
                        double w, wf;
                        const int jy = __float_as_int(yF[k].w);
                        atm_weights(jx == jy, jx == a, jy == a, ref, p.atm_force_scaled != 0, w, wf);
                        const double dw = w - wf, d3w = dw * f3;
                        SC = fma(dw, f1 + f3, SC);
                        yC = fma(dw, f2 + f3, yC);
                        Ux = fma(d3w, A0.x, Ux);
                        Uy = fma(d3w, A0.y, Uy);
                        Uz = fma(d3w, A1.x, Uz);
                        E *= w;
                        f1 *= wf;
                        f2 *= wf;
                        f3 *= wf;
                    }
                    const double El = E * (d3 * q2); // E / C6_xy
                    SE += E;
                    SD = fma(El, dcx, SD);
                    SF += f1 + f3;
                    Wx = fma(f3, A0.x, Wx);
                    Wy = fma(f3, A0.y, Wy);
                    Wz = fma(f3, A1.x, Wz);
                    const double f23 = f2 + f3;
                    yE += E;
                    yD = fma(El, dcy, yD);
                    yX = fma(f3, vx, fma(-f23, A0.x, yX));
                    yY = fma(f3, vy, fma(-f23, A0.y, yY));
                    yZ = fma(f3, vz, fma(-f23, A1.x, yZ));
                }
                // lane L holds the sums of B[(L + at) mod 32] (no bit set: not visited; a triplet
                // may have forces and no energy)
                const int e = 32 * B + ((lane + at) & 31);
                const long long any = __double_as_longlong(yE) | __double_as_longlong(yX) | __double_as_longlong(yY) | __double_as_longlong(yZ);
                if (e < m && any != 0) {
                    double *o = acc[e];
                    atomicAdd(o, yE);
                    atomicAdd(o + 1, yD);
                    atomicAdd(o + 2, -yX);
                    atomicAdd(o + 3, -yY);
                    atomicAdd(o + 4, -yZ);
                    if (!SIMPLE && yC != 0.0) atomicAdd(o + 5, yC);
                }
            }
            if (xv) {
                double *o = acc[xe];
                atomicAdd(o, SE);
                atomicAdd(o + 1, SD);
                atomicAdd(o + 2, SF * vx - Wx);
                atomicAdd(o + 3, SF * vy - Wy);
                atomicAdd(o + 4, SF * vz - Wz);
                if (!SIMPLE) {
                    if (SC != 0.0) atomicAdd(o + 5, SC);
                    // cross terms of the apex virial that the force weights miss
                    carry[0] -= 2.0 * vx * Ux;
                    carry[32] -= 2.0 * vy * Uy;
                    carry[64] -= 2.0 * vz * Uz;
                    carry[96] -= vx * Uy + vy * Ux;
                    carry[128] -= vx * Uz + vz * Ux;
                    carry[160] -= vy * Uz + vz * Uy;
                }
            }
        }
        __syncthreads();
        // ---- per entry: atom shares (FP64 atomics) and the apex's sums (force -sum F_e, virial
        // sum v_e (x) F_e: each triplet's terms depend on relative positions only)
        double out[11] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (!SIMPLE)
#pragma unroll
            for (int k = 0; k < 6; ++k) out[5 + k] = carry[32 * k];
        for (int e = tid; e < m; e += blockDim.x) {
            const double E = -__ldcg(&acc[e][0]), D = -__ldcg(&acc[e][1]);
            const double Fx = __ldcg(&acc[e][2]), Fy = __ldcg(&acc[e][3]), Fz = __ldcg(&acc[e][4]);
            const Atm64Row *r = entries + e;
            const double vx = r->v[0], vy = r->v[1], vz = r->v[2], c = SIMPLE ? 0.0 : __ldcg(&acc[e][5]);
            const int j = r->j;
            atomicAdd(&p.eb[j], E * (1.0 / 3.0));
            atomicAdd(&p.gb[j], 0.5 * (r->lam_ea * E + D));
            atomicAdd(&p.fb[3 * j], Fx);
            atomicAdd(&p.fb[3 * j + 1], Fy);
            atomicAdd(&p.fb[3 * j + 2], Fz);
            out[0] += E * (1.0 / 6.0);
            out[1] += 0.5 * r->lam_ae * E;
            out[2] -= Fx;
            out[3] -= Fy;
            out[4] -= Fz;
            out[5] += vx * fma(c, vx, Fx);
            out[6] += vy * fma(c, vy, Fy);
            out[7] += vz * fma(c, vz, Fz);
            out[8] += 0.5 * (vx * Fy + vy * Fx) + c * vx * vy;
            out[9] += 0.5 * (vx * Fz + vz * Fx) + c * vx * vz;
            out[10] += 0.5 * (vy * Fz + vz * Fy) + c * vy * vz;
        }
#pragma unroll
        for (int k = 0; k < 11; ++k) {
            const double v = warp_sum(out[k]);
            if (lane == 0) red[warp][k] = v;
        }
        __syncthreads();
        if (tid < 11) {
            double t = 0;
            for (int w = 0; w < nw; ++w) t += red[w][tid];
            double *dst = tid == 0 ? p.ea + a : (tid == 1 ? p.ga + a : (tid < 5 ? p.fa + 3 * (size_t)a + tid - 2 : p.va + 6 * (size_t)a + tid - 5));
            if (tid >= 5) t *= -1.0 / g.vol;
            if (S == 1)
                *dst = t;
            else // the apex's other splits add theirs (the arrays start at zero)
                atomicAdd(dst, t);
        }
    }
    for (int o = 16; o > 0; o >>= 1) visits += __shfl_xor_sync(0xffffffffu, visits, o);
    if (lane == 0 && p.counters) atomicAdd(p.counters, visits);
}
