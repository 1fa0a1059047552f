// ATM three-body kernel, FP64 (replaces the reference's atm_kernel, src/d3_kernel.cu:1199-1509).
// Included by d3_engine.cu after the kernel parameter block and the shared helpers.
//
// Enumeration: for each apex a, the half list L_a = {(j, T) before (a, 0) (atm_before):
// 1e-12 <= r^2 <= rc_ATM^2} built by k_atm_list; a triplet is an unordered pair of
// distinct entries {x, y} of L_a with 1e-12 <= r_xy^2 <= rc_ATM^2. With the reference's
// order (entries j <= a in caller order) this is its (b, T_b, c, T_c) loop with c <= b
// (src/d3_kernel.cu:1235-1327). Repeated atoms change the weights (atm_weights).
//
// Schedule: persistent CTAs pull (apex, split) items from a work counter; the splits of an apex share its entries x (rows) between CTAs, so that systems of
// few apexes fill the GPU. A warp owns one row x at a time. It tests x against the staged
// partners 32 at a time (FP32 positions; pairs near a limit again in FP64) and queues the
// ones in range; when 32 are queued, all 32 lanes visit one partner y each. Every visit
// slot then does work whatever the shape of the lists, and everything that belongs to x is
// the same in all lanes, so its sums cost one warp reduction per row and partner tile.
// Every unordered pair is visited from both of its entries, so nothing is added to y.
//
// The queue has eight classes, k mod 8 for partner k, and a class feeds the four lanes l
// with l mod 8 equal to it: the eight lanes that share a 128-byte wavefront of a 16-byte
// shared-memory load then read eight different bank groups, whatever the gaps between the
// queued partners are. The partners' C6 rows are staged for as many element types as fit
// with all partners of the apex (at least one), and the rows x of those types are walked
// before the next types are staged.
//
// With C = s1 s2 s3 / (r1 r2 r3)^3 (s = sqrt(C6), sides a-x, a-y, x-y), d_k = r_k^2,
// H = 3/4 / (d1 d2 d3), t1 = d1 + d2 - d3 ..., u = t1 t2 t3 H and fd the damping,
//     E   = -C fd (1 + u/2)
//     f_k = S / d_k - C fd H n_k,   S = C fd (3 + 5/2 u - 16/3 (1 - fd) (1 + u/2)),
// n_k = t_k-derivative of t1 t2 t3 by d_k (16/3 (1 - fd) fd is the derivative of the
// damping, since 6 x fd = 1 - fd). That is the reference's angular and damping derivative
// (:1367-1392) regrouped: 83 FP64 operations a visit, two visits a triplet.
//
// Bound: the FP64 pipe (a warp instruction takes two cycles of a scheduler's pipe), 40 %
// busy on the 20,000-atom box; the rest is latency of the test and queue steps.
// ATM pass on a B200, one thread per entry with a private partner mask before -> now:
// 16-atom metal cell 26.8 -> 0.51 ms, 96-atom water box 36.2 -> 3.4 ms (their few apexes
// are split over all CTAs), 777 atoms 49.4 -> 25.5 ms, 20,000-atom box 745 -> 630 ms.

// ---- refined reciprocal roots ------------------------------------------------------
__device__ __forceinline__ double rsqrt_nr(double x) {
    // x^(-1/2): the hardware's double-precision approximation (relative error ~2^-20,
    // no conversions) and one third-order step, y (1 + e/2 + 3/8 e^2) with e = 1 - x y^2
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

__device__ __forceinline__ double rcp_nr(double x) {
    // 1/x: hardware approximation and one third-order step, y (1 + e + e^2), e = 1 - x y
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double rcbrt_nr(double x) {
    // x^(-1/3): float seed 2^(-log2(x)/3), one Newton step z + z e / 3, e = 1 - x z^3
    const double z = (double)sfu_exp2(sfu_log2((float)x) * (-1.0f / 3.0f));
    const double e = fma(-x * z, z * z, 1.0);
    return fma(z * e, 1.0 / 3.0, z);
}

// two steps: the per-entry set-up
__device__ __forceinline__ double rsqrt_nr2(double x) {
    const double y = rsqrt_nr(x);
    return y * fma(-0.5 * x * y, y, 1.5);
}

__device__ __forceinline__ double rcp_nr2(double x) {
    const double y = rcp_nr(x);
    return fma(fma(-x, y, 1.0), y, y);
}

__device__ __forceinline__ double rcbrt_nr2(double x) {
    const double z = rcbrt_nr(x);
    return fma(z * fma(-x * z, z * z, 1.0), 1.0 / 3.0, z);
}

constexpr int ATM64_THREADS = 384;  // threads of all CTAs of an SM together
constexpr int ATM64_ROWS = 4096;    // entries whose rows are listed at once, over the CTAs of an SM
constexpr int ATM64_SEG = 128;      // partners tested before the queue is looked at
constexpr int ATM64_QCAP = 64;      // queue slots per class and warp (at least 8 + ATM64_SEG / 8)
constexpr int ATM64_STATIC = 2048;  // bytes left for the static arrays

// apex kinds, one instance each: weight-free structures (no atom twice in a list), the
// others, and the surrogate fallback's centre mode (apexes from p.atm_apex, full lists,
// every triplet weighted 1/3 for energy and forces alike)
enum { ATM64_SIMPLE = 0, ATM64_WEIGHTED = 1, ATM64_CENTER = 2 };

// double2 words of a partner's C6 row at one type: NR values and r0^2 of the type pair. The
// word counts of the staged records (3; 3 or 5) are odd, so that partners with different
// k mod 8 lie in different bank groups.
__host__ __device__ constexpr int atm64_rowq(int NR) { return NR == 5 ? 3 : 5; }
__host__ __device__ constexpr size_t atm64_partner_bytes(int NR, int types) {
    return 3 * sizeof(double2) + sizeof(float4) + (size_t)types * atm64_rowq(NR) * sizeof(double2);
}
__host__ __device__ inline size_t atm64_fixed_bytes(int ne, int NR, int warps, int nrows) {
    size_t b = (size_t)((ne * NR + 1) & ~1) * sizeof(double) + (size_t)((ne * ne + 1) & ~1) * sizeof(double);
    b += (size_t)warps * 8 * ATM64_QCAP * sizeof(unsigned short);
    b += (size_t)nrows * sizeof(unsigned short) + (size_t)((2 * ne + 2 + 3) & ~3) * sizeof(int);
    return (b + 15) & ~(size_t)15;
}

// one entry of the apex as a row
struct Atm64Row {
    double v[3], id, p, g; // position from the apex, 1/d, sqrt(C6)/r^3, (r0^2/d)^(8/3)
    double lam_ea, lam_ae; // dC6/dCN over C6: of the entry, of the apex
    int j, t;
};

// per-entry set-up (FP64 C6 of the apex pair, its CN derivatives, damping ratio)
template <int NR>
__device__ __forceinline__ Atm64Row atm64_entry(const KP &p, const SG &g, const double4 &xa, int a, const int2 ent,
                                                const double *yapex, const double *r0a, bool derivatives) {
    Atm64Row r;
    const double4 xj = p.xs[ent.x];
    r.j = ent.x;
    r.t = (int)xj.w;
    double sx, sy, sz;
    image_vec(g, sext8(ent.y & 0xff), sext8((ent.y >> 8) & 0xff), sext8((ent.y >> 16) & 0xff), sx, sy, sz);
    r.v[0] = xj.x + sx - xa.x;
    r.v[1] = xj.y + sy - xa.y;
    r.v[2] = xj.z + sz - xa.z;
    const double d = r.v[0] * r.v[0] + r.v[1] * r.v[1] + r.v[2] * r.v[2];
    const double ir = rsqrt_nr2(d);
    r.id = ir * ir;
    const double *ya = yapex + r.t * NR; // C6_ae = y_{a,te} . w_e
    const double *wj = p.w + (size_t)r.j * NR;
    double c6 = 0;
#pragma unroll
    for (int b = 0; b < NR; ++b) c6 += ya[b] * wj[b];
    const double is = rsqrt_nr2(c6);
    r.p = c6 * is * ir * r.id;
    const double u = r0a[r.t] * r.id;
    r.g = u * u * u * rcbrt_nr2(u);
    r.lam_ea = r.lam_ae = 0;
    if (derivatives) {
        const double *yq = p.Y + ((size_t)r.j * p.ne + (int)xa.w) * NR; // dC6_ae/dCN_a = y_{e,ta} . dw_a
        const double *dwj = p.dw + (size_t)r.j * NR, *dwa = p.dw + (size_t)a * NR;
        double dca = 0, dcq = 0;
#pragma unroll
        for (int b = 0; b < NR; ++b) {
            dcq += ya[b] * dwj[b];
            dca += yq[b] * dwa[b];
        }
        r.lam_ea = dcq * is * is;
        r.lam_ae = dca * is * is;
    }
    return r;
}

// one exchange of the row reduction: keep v on the lower lanes and w on the upper ones of
// each pair `o` apart, adding what the other lane holds of it
__device__ __forceinline__ double atm64_fold(double v, double w, int o) {
    const bool up = (threadIdx.x & o) != 0;
    return (up ? w : v) + __shfl_xor_sync(0xffffffffu, up ? v : w, o);
}
// sums of eight values over the warp; lane l returns the sum of value ((l >> 2) & 7) with
// its three bits reversed, i.e. value i is on lane atm64_lane(i)
__device__ __forceinline__ double atm64_reduce8(const double v[8]) {
    double a[4], b[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = atm64_fold(v[k], v[k + 4], 16);
#pragma unroll
    for (int k = 0; k < 2; ++k) b[k] = atm64_fold(a[k], a[k + 2], 8);
    double c = atm64_fold(b[0], b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    return c + __shfl_xor_sync(0xffffffffu, c, 1);
}
__device__ __forceinline__ constexpr int atm64_lane(int i) {
    return ((i & 4) << 2) | ((i & 2) << 2) | ((i & 1) << 2);
}

// One visit: triplet (apex, x, y) with x in the arguments and y in the staged records A and
// R. Branch-free, so that two of them overlap.
struct Atm64Visit {
    double E, lam, f1, f3, vx, vy, vz; // -E, dC6_xy/dCN_x over C6_xy, force scalars, y
};
template <int NR>
__device__ __forceinline__ void atm64_visit(double vx, double vy, double vz, double d1, double id1, double h1, double p1,
                                            double g1, const double *wx, const double *dwx, const double2 *A,
                                            const double2 *R, Atm64Visit &V) {
    const double2 A0 = A[0], A1 = A[1], A2 = A[2];
    double2 Rq[(NR + 1) / 2];
#pragma unroll
    for (int b = 0; b < (NR + 1) / 2; ++b) Rq[b] = R[b];
    const double rx = vx - A0.x, ry = vy - A0.y, rz = vz - A1.x, id2 = A1.y;
    const double d3 = fma(rx, rx, fma(ry, ry, rz * rz));
    const double d2 = fma(A0.x, A0.x, fma(A0.y, A0.y, A1.x * A1.x));
    // C6_xy = y_{y,tx} . w_x and its derivative by CN_x
    double c6 = Rq[0].x * wx[0], dc6 = Rq[0].x * dwx[0];
#pragma unroll
    for (int b = 1; b < NR; ++b) {
        const double y = (b & 1) ? Rq[b >> 1].y : Rq[b >> 1].x;
        c6 = fma(y, wx[b], c6);
        dc6 = fma(y, dwx[b], dc6);
    }
    // one root for 1/d3, 1/C6 and sqrt(C6) / r3^3
    const double cd = c6 * d3, q = rsqrt_nr(cd), q2 = q * q;
    const double id3 = c6 * q2;
    V.lam = d3 * q2 * dc6;
    const double C = p1 * A2.x * (cd * q * (id3 * id3));
    const double u3 = Rq[NR / 2].y * id3;
    const double g3 = u3 * u3 * u3 * rcbrt_nr(u3);
    const double fd = rcp_nr(fma(g1 * A2.y, g3, 1.0));
    const double H = h1 * id2 * id3;
    const double s = d1 + d2, m12 = d1 - d2;
    const double t1 = s - d3, t2 = m12 + d3, t3 = d3 - m12;
    const double t12 = t1 * t2, t13 = t1 * t3, t23 = t2 * t3;
    const double uu = t12 * t3 * H;
    const double B = fma(0.5, uu, 1.0);
    const double Ef = C * fd;
    const double Sf = Ef * fma(fma(16.0 / 3.0, fd, -16.0 / 3.0), B, fma(2.5, uu, 3.0));
    const double W = Ef * H, dt = t23 - t12;
    V.f1 = fma(-W, t13 + dt, id1 * Sf);
    V.f3 = fma(-W, t13 - dt, id3 * Sf);
    V.E = Ef * B;
    V.vx = A0.x;
    V.vy = A0.y;
    V.vz = A1.x;
}

template <int NR, int KIND>
__global__ void __launch_bounds__(ATM64_THREADS, 1) k_atm64(KP p, Atm64Row *scratch, int nrows, int tile_bytes, int tile_max) {
    extern __shared__ __align__(16) unsigned char sm64[];
    constexpr int RQ = atm64_rowq(NR);
    const int ne = p.ne, nw = blockDim.x >> 5;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *yapex = reinterpret_cast<double *>(sm64);              // [ne][NR]
    double *r0sq = yapex + ((ne * NR + 1) & ~1);                   // [ne][ne] r0ab^2
    int *toff = reinterpret_cast<int *>(r0sq + ((ne * ne + 1) & ~1)); // [ne + 1] rows of each type, [ne] fill positions
    int *tpos = toff + ne + 1;
    unsigned short *rowperm = reinterpret_cast<unsigned short *>(toff + ((2 * ne + 2 + 3) & ~3)); // [nrows]
    unsigned short *queue = rowperm + nrows + warp * 8 * ATM64_QCAP; // [slot][class]
    unsigned char *area = sm64 + atm64_fixed_bytes(ne, NR, nw, nrows);
    __shared__ int s_item, s_row;
    __shared__ double red[ATM64_THREADS / 32][11];
    if (p.atm_off[p.n] > p.atm_cap) return; // list overflowed: the host grows it and re-runs
    for (int k = tid; k < ne * ne; k += blockDim.x) r0sq[k] = p.r0ab[k] * p.r0ab[k];
    Atm64Row *rows = scratch + (size_t)blockIdx.x * nrows;
    const double third = 1.0 / 3.0;
    // FP32 range test: |d3 - half| <= half in range, but within `slack` of either end of
    // [0, 2 half] the pair is tested again in FP64. The rounded positions put d3 off by at
    // most about 5e-7 rc^2.
    const float half = (float)(0.5 * p.ratm2 * (1.0 + 1e-5)), sure = half * (1.0f - 4e-5f);
    const int cls = lane & 7, member = lane >> 3;
    const unsigned cls_bits = 0x01010101u << cls, below = cls_bits & ((1u << lane) - 1u);
    unsigned long long visits = 0;
    while (true) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(p.work, 1);
        __syncthreads();
        const int S = KIND == ATM64_CENTER ? 1 : p.atmb_split;
        const int split = s_item % S, unit = s_item / S;
        const int item = KIND == ATM64_CENTER ? unit : unit * p.shard_world + p.shard_rank;
        if (item >= (KIND == ATM64_CENTER ? *p.atm_napex : p.n)) break;
        const int a = KIND == ATM64_CENTER ? p.atm_apex[item] : p.sorted_of[p.n - 1 - item];
        const SG &g = p.sg[p.sid[a]];
        if (KIND != ATM64_CENTER && (g.atm_simple != 0) != (KIND == ATM64_SIMPLE)) continue; // the other instance's
        const bool ref = KIND == ATM64_WEIGHTED && atm_reference_order(p, g, p.sid[a]);
        const long long e0 = p.atm_off[a];
        const int m = (int)(p.atm_off[a + 1] - e0);
        const double4 xa = p.xs[a];
        const double *r0a = r0sq + (int)xa.w * ne;
        for (int k = tid; k < ne * NR; k += blockDim.x) yapex[k] = p.Y[(size_t)a * ne * NR + k];
        // types staged together and partner tile: all partners of the apex with as many
        // types as fit, else one type and the largest tile (one record more is the dummy
        // partner of idle lanes)
        int types = ne, tile = 0;
        for (;; --types) {
            tile = min(tile_max, (int)(tile_bytes / atm64_partner_bytes(NR, types) - 1) & ~(ATM64_SEG - 1));
            if (types == 1 || tile >= m) break;
        }
        tile = min(tile, (m + ATM64_SEG - 1) & ~(ATM64_SEG - 1));
        double2 *sA = reinterpret_cast<double2 *>(area);              // [tile + 1][3]: vx vy | vz id | p g
        float4 *sF = reinterpret_cast<float4 *>(sA + 3 * (tile + 1)); // [tile + 1]: FP32 position, atom
        double2 *sR = reinterpret_cast<double2 *>(sF + tile + 1);     // [types][tile + 1][RQ]
        double acc = 0; // this lane's apex sum (lanes 0..10: energy, dE/dCN, force, virial)
        for (int b0 = 0; b0 < m; b0 += nrows) {
            // rows of this split, listed by type
            const int bn = min(nrows, m - b0);
            __syncthreads();
            for (int k = tid; k <= ne; k += blockDim.x) toff[k] = 0;
            __syncthreads();
            const int first = (split - b0 % S + S) % S; // entries b0 + k with (b0 + k) % S == split
            for (int k = first + tid * S; k < bn; k += blockDim.x * S) {
                const Atm64Row r = atm64_entry<NR>(p, g, xa, a, p.atm_ent[e0 + b0 + k], yapex, r0a, true);
                rows[k] = r;
                atomicAdd(&toff[r.t + 1], 1);
            }
            __syncthreads();
            if (tid == 0)
                for (int t = 0; t < ne; ++t) {
                    tpos[t] = toff[t];
                    toff[t + 1] += toff[t];
                }
            __syncthreads();
            for (int k = first + tid * S; k < bn; k += blockDim.x * S)
                rowperm[atomicAdd(&tpos[rows[k].t], 1)] = (unsigned short)k;
            __syncthreads();
            if (toff[ne] == 0) continue; // no row of this split
            for (int p0 = 0; p0 < m; p0 += tile) {
                const int cnt = min(tile, m - p0);
                for (int t0 = 0; t0 < ne; t0 += types) {
                    const int tn = min(types, ne - t0);
                    __syncthreads(); // the previous phase is done with the staged data and s_row
                    const int r1 = toff[t0 + tn];
                    if (toff[t0] == r1 && !(t0 == 0)) continue;
                    if (tid == 0) s_row = toff[t0];
                    for (int k = tid; k < cnt; k += blockDim.x) {
                        const int2 ent = p.atm_ent[e0 + p0 + k];
                        int j = ent.x, tj;
                        if (t0 == 0) {
                            const Atm64Row r = atm64_entry<NR>(p, g, xa, a, ent, yapex, r0a, false);
                            sA[3 * k] = make_double2(r.v[0], r.v[1]);
                            sA[3 * k + 1] = make_double2(r.v[2], r.id);
                            sA[3 * k + 2] = make_double2(r.p, r.g);
                            sF[k] = make_float4((float)r.v[0], (float)r.v[1], (float)r.v[2], __int_as_float(j));
                            tj = r.t;
                        } else {
                            tj = (int)p.xs[j].w;
                        }
                        const double *Y = p.Y + ((size_t)j * ne + t0) * NR;
                        for (int t = 0; t < tn; ++t) {
                            double q[NR + 1];
#pragma unroll
                            for (int b = 0; b < NR; ++b) q[b] = Y[t * NR + b];
                            q[NR] = r0sq[(t0 + t) * ne + tj];
                            double2 *dst = sR + ((size_t)t * (tile + 1) + k) * RQ;
#pragma unroll
                            for (int b = 0; b < (NR + 1) / 2; ++b) dst[b] = make_double2(q[2 * b], q[2 * b + 1]);
                        }
                    }
                    // the tail of the last segment lies out of range of every row; the dummy
                    // partner of idle lanes has p = 0, which makes its terms vanish
                    for (int k = cnt + tid; k < ((cnt + ATM64_SEG - 1) & ~(ATM64_SEG - 1)); k += blockDim.x) sF[k] = make_float4(3e18f, 3e18f, 3e18f, 0.f);
                    if (tid < tn) {
                        if (tid == 0) {
                            sA[3 * tile] = make_double2(3e4, 3e4);
                            sA[3 * tile + 1] = make_double2(3e4, 1.0);
                            sA[3 * tile + 2] = make_double2(0.0, 1.0);
                            sF[tile] = make_float4(3e18f, 3e18f, 3e18f, __int_as_float(-1));
                        }
                        double2 *dst = sR + ((size_t)tid * (tile + 1) + tile) * RQ;
#pragma unroll
                        for (int b = 0; b < (NR + 1) / 2; ++b) dst[b] = make_double2(1.0, 1.0);
                    }
                    __syncthreads();
                    for (;;) {
                        int r = 0;
                        if (lane == 0) r = atomicAdd(&s_row, 1);
                        r = __shfl_sync(0xffffffffu, r, 0);
                        if (r >= r1) break;
                        const Atm64Row *X = rows + rowperm[r];
                        const double vx = X->v[0], vy = X->v[1], vz = X->v[2];
                        const double id1 = X->id, p1 = X->p, h1 = 0.75 * id1;
                        const double g1 = X->g * (6.0 * 4294967296.0 / 43046721.0); // 6 (4/3)^16
                        const double d1 = vx * vx + vy * vy + vz * vz;
                        const int jx = X->j;
                        double wx[NR], dwx[NR];
#pragma unroll
                        for (int b = 0; b < NR; ++b) {
                            wx[b] = p.w[(size_t)jx * NR + b];
                            dwx[b] = p.dw[(size_t)jx * NR + b];
                        }
                        const float fx = (float)vx, fy = (float)vy, fz = (float)vz;
                        const double2 *sRx = sR + (size_t)(X->t - t0) * RQ * (tile + 1);
                        // sums over this row's visits: w E', w E' lam_xy, wf (f1 + f3),
                        // wf f3 v_y (3), wf f1; v[7] unused
                        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        // weighted kind: (w - wf) (f1 + f3), (w - wf) f3 v_y
                        double dv[4] = {0, 0, 0, 0};
                        int head = 0, tail = 0; // of this lane's class
                        for (int c0 = 0; c0 < cnt; c0 += ATM64_SEG) {
                            // test ATM64_SEG partners, queue those in range
                            bool in[ATM64_SEG / 32];
                            bool edge = false;
                            const float4 *sFc = sF + c0 + lane;
#pragma unroll
                            for (int c = 0; c < ATM64_SEG / 32; ++c) {
                                const float4 f = sFc[32 * c];
                                const float dx = fx - f.x, dy = fy - f.y, dz = fz - f.z;
                                const float off = fabsf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - half);
                                in[c] = off <= half;
                                edge |= in[c] & (off >= sure);
                            }
                            if (__any_sync(0xffffffffu, edge)) {
#pragma unroll
                                for (int c = 0; c < ATM64_SEG / 32; ++c)
                                    if (in[c]) {
                                        const double2 *A = sA + 3 * (c0 + 32 * c + lane);
                                        const double rx = vx - A[0].x, ry = vy - A[0].y, rz = vz - A[1].x;
                                        const double d3 = fma(rx, rx, fma(ry, ry, rz * rz));
                                        in[c] = d3 <= p.ratm2 && d3 >= 1e-12; // also drops x == y
                                    }
                            }
#pragma unroll
                            for (int c = 0; c < ATM64_SEG / 32; ++c) {
                                const unsigned bits = __ballot_sync(0xffffffffu, in[c]);
                                const int slot = ((tail + __popc(bits & below)) & (ATM64_QCAP - 1)) * 8 + cls;
                                if (in[c]) queue[slot] = (unsigned short)(c0 + 32 * c + lane);
                                tail += __popc(bits & cls_bits);
                            }
                            __syncwarp();
                            // two visits per lane while all lanes are busy (after the last
                            // partners: while any is), and while a class could overflow next
                            const int least = c0 + ATM64_SEG >= cnt ? 0 : 8;
                            for (;;) {
                                const int pend = tail - head;
                                if (least ? !(__all_sync(0xffffffffu, pend >= 8) ||
                                              __any_sync(0xffffffffu, pend > ATM64_QCAP - ATM64_SEG / 8))
                                          : !__any_sync(0xffffffffu, pend > 0))
                                    break;
                                int k[2];
                                Atm64Visit V[2];
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const int i = head + member + 4 * h;
                                    k[h] = queue[(i & (ATM64_QCAP - 1)) * 8 + cls];
                                    k[h] = i < tail ? k[h] : tile;
                                }
                                head = min(head + 8, tail);
#pragma unroll
                                for (int h = 0; h < 2; ++h)
                                    atm64_visit<NR>(vx, vy, vz, d1, id1, h1, p1, g1, wx, dwx, sA + 3 * k[h], sRx + RQ * k[h], V[h]);
                                if (KIND == ATM64_WEIGHTED) {
                                    const int jy[2] = {__float_as_int(sF[k[0]].w), __float_as_int(sF[k[1]].w)};
                                    if (jx == jy[0] || jx == jy[1] || jx == a || jy[0] == a || jy[1] == a) {
#pragma unroll
                                        for (int h = 0; h < 2; ++h) {
                                            double w, wf;
                                            atm_weights(jx == jy[h], jx == a, jy[h] == a, ref, p.atm_force_scaled != 0, w, wf);
                                            const double d3w = (w - wf) * V[h].f3;
                                            const double2 *A = sA + 3 * k[h];
                                            dv[0] = fma(w - wf, V[h].f1 + V[h].f3, dv[0]);
                                            dv[1] = fma(d3w, A[0].x, dv[1]);
                                            dv[2] = fma(d3w, A[0].y, dv[2]);
                                            dv[3] = fma(d3w, A[1].x, dv[3]);
                                            V[h].E *= w;
                                            V[h].f1 *= wf;
                                            V[h].f3 *= wf;
                                        }
                                    }
                                }
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    v[0] += V[h].E;
                                    v[1] = fma(V[h].E, V[h].lam, v[1]);
                                    v[2] += V[h].f1 + V[h].f3;
                                    v[3] = fma(V[h].f3, V[h].vx, v[3]);
                                    v[4] = fma(V[h].f3, V[h].vy, v[4]);
                                    v[5] = fma(V[h].f3, V[h].vz, v[5]);
                                    v[6] += V[h].f1;
                                }
                            }
                            __syncwarp();
                        }
                        if (member == 0) visits += (unsigned)tail;
                        if (KIND == ATM64_CENTER) {
#pragma unroll
                            for (int k = 0; k < 7; ++k) v[k] *= third;
                        }
                        // the row's sums: entry shares (atomics by lanes 11..15) and apex sums
                        const double tot = atm64_reduce8(v);
                        const double SE = -__shfl_sync(0xffffffffu, tot, atm64_lane(0));
                        const double SD = -__shfl_sync(0xffffffffu, tot, atm64_lane(1));
                        const double SF = __shfl_sync(0xffffffffu, tot, atm64_lane(2));
                        const double Wx = __shfl_sync(0xffffffffu, tot, atm64_lane(3));
                        const double Wy = __shfl_sync(0xffffffffu, tot, atm64_lane(4));
                        const double Wz = __shfl_sync(0xffffffffu, tot, atm64_lane(5));
                        const double SA = __shfl_sync(0xffffffffu, tot, atm64_lane(6));
                        double Sv = SF, Ux = Wx, Uy = Wy, Uz = Wz; // virial sums (weights w)
                        if (KIND == ATM64_WEIGHTED && __any_sync(0xffffffffu, dv[0] != 0.0 || dv[1] != 0.0 || dv[2] != 0.0 || dv[3] != 0.0)) {
                            Sv += warp_sum(dv[0]);
                            Ux += warp_sum(dv[1]);
                            Uy += warp_sum(dv[2]);
                            Uz += warp_sum(dv[3]);
                        }
                        // component of each lane: force lanes 2..4 and 13..15, virial lanes
                        // 5..10 (xx yy zz xy xz yz)
                        const int ca = lane < 5 ? lane - 2 : (lane < 8 ? lane - 5 : (lane < 10 ? 0 : (lane == 10 ? 1 : lane - 13)));
                        const int cb = lane < 8 ? ca : (lane == 8 ? 1 : 2);
                        const double va = ca == 0 ? vx : (ca == 1 ? vy : vz), vb = cb == 0 ? vx : (cb == 1 ? vy : vz);
                        const double Ua = ca == 0 ? Ux : (ca == 1 ? Uy : Uz), Ub = cb == 0 ? Ux : (cb == 1 ? Uy : Uz);
                        const double Wa = ca == 0 ? Wx : (ca == 1 ? Wy : Wz);
                        // apex: energy E/3 per pair and dE/dCN E/2 lam over both visits of a
                        // pair, force -f1 v_x per visit, virial f r (x) r with the x-y side's
                        // cross part split evenly between the two visits
                        if (lane == 0)
                            acc += SE * (0.5 * third);
                        else if (lane == 1)
                            acc += 0.5 * X->lam_ae * SE;
                        else if (lane < 5)
                            acc -= SA * va;
                        else if (lane < 11)
                            acc += Sv * va * vb - 0.5 * (Ua * vb + Ub * va);
                        else if (lane == 11)
                            atomicAdd(&p.eb[jx], SE * third);
                        else if (lane == 12)
                            atomicAdd(&p.gb[jx], 0.5 * (X->lam_ea * SE + SD));
                        else if (lane < 16)
                            atomicAdd(&p.fb[3 * jx + ca], SF * va - Wa);
                    }
                }
            }
        }
        // apex sums over the CTA's warps (fixed order)
        if (lane < 11) red[warp][lane] = acc;
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
    // in-range visits (each unordered triplet counted twice)
    for (int o = 16; o > 0; o >>= 1) visits += __shfl_xor_sync(0xffffffffu, visits, o);
    if (lane == 0 && p.counters) atomicAdd(p.counters, visits);
}
