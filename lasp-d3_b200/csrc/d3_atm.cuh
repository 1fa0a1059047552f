// ATM three-body kernel, FP64 (replaces the reference's atm_kernel, src/d3_kernel.cu:1199-1509).
// Included by d3_engine.cu after the kernel parameter block and the shared helpers.
//
// Enumeration: for each apex a, the half list L_a = {(j, T) before (a, 0) (atm_before):
// 1e-12 <= r^2 <= rc_ATM^2} built by k_atm_list; a triplet is an unordered pair of
// distinct entries {x, y} of L_a with 1e-12 <= r_xy^2 <= rc_ATM^2. With the reference's
// order (entries j <= a in caller order) this is its (b, T_b, c, T_c) loop with c <= b
// (src/d3_kernel.cu:1235-1327). Repeated atoms change the weights (atm_weights).
//
// Schedule: persistent CTAs pull (apex, split) items from a work counter; the splits of an
// apex share its entries x (rows) between CTAs, so that systems of few apexes fill the GPU.
// The entries are sorted along a Hilbert curve and staged in shared memory as partners, 32
// consecutive ones a chunk with a bounding sphere. A warp owns one row x at a time:
//  1. each lane compares x with the sphere of one chunk: out of range, all in range, or mixed;
//  2. chunks all in range are visited as they are, one partner y per lane;
//  3. partners of mixed chunks are tested (FP32 positions; pairs near a limit again in FP64),
//     the ones in range are queued, and whole warps of them are visited.
// Nearly every visit slot then does work whatever the shape of the lists, and everything
// that belongs to x is the same in all lanes, so its sums cost one warp reduction per row
// and partner tile. Every unordered pair is visited from both of its entries, so nothing is
// added to y.
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
// Bound: instruction issue, where an FP64 instruction counts twice (its pipe takes a warp in
// two cycles). A visit alone costs 200 cycles of a scheduler (83 FP64 and 24 other
// instructions), on the 20,000-atom box 310 with everything else: of the ATM pass 31 % are
// visits of whole chunks, 37 % of queued partners (15 % of their lanes idle), 13 % range
// tests, 10 % row set-up and sums, 4 % set-up of the apex.
// ATM pass on a B200, one thread per entry with a private partner mask -> this kernel:
// 16-atom metal cell 26.8 -> 0.38 ms, 96-atom water box 36.2 -> 2.65 ms (their few apexes
// are split over all CTAs), 777 atoms 49.4 -> 20.7 ms, 2,000 atoms 73.3 -> 50.0 ms,
// 20,000-atom box 745 -> 441 ms. Large systems take k_atm64b (d3_atm64b.cuh), which visits a
// triplet once; this kernel keeps few apexes, short lists, lists beyond k_atm64b's capacity,
// many types and the surrogate fallback.

constexpr int ATM64_THREADS = 512;  // threads of all CTAs of an SM together
constexpr int ATM64_ENTRIES = 4096; // entries set up at once at most (longer lists: in parts)
constexpr int ATM64_CHUNKS = 64;    // chunks of 32 partners in a tile at most
constexpr int ATM64_SEG = 4;        // chunks tested together
constexpr int ATM64_GROUP = 32;     // mixed chunks of a row queued at once (a multiple of ATM64_SEG)
constexpr int ATM64_QCAP = 4 * ATM64_GROUP; // queue slots per class and warp
constexpr int ATM64_LIST = ATM64_CHUNKS + ATM64_SEG; // a row's chunks: all in range from the front, mixed from the back
constexpr int ATM64_CELLS = 4096;   // sort cells: 16^3, fewer for short lists
constexpr int ATM64_STATIC = 5120;  // bytes left for the static arrays

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
// tile bytes: the partners, 32 far positions (the first of them the dummy partner of idle
// lanes, with a record and rows of its own), the chunk bounds
__host__ __device__ constexpr size_t atm64_tile_fixed(int NR, int types) {
    return atm64_partner_bytes(NR, types) + 31 * sizeof(float4) + 2 * ATM64_CHUNKS * sizeof(float4);
}
__host__ __device__ inline size_t atm64_fixed_bytes(int ne, int NR, int warps) {
    size_t b = (size_t)((ne * NR + 1) & ~1) * sizeof(double) + (size_t)((ne * ne + 1) & ~1) * sizeof(double);
    b += (size_t)warps * (8 * ATM64_QCAP + ATM64_LIST * sizeof(unsigned short));
    b += (size_t)((2 * ne + 2 + 3) & ~3) * sizeof(int);
    return (b + 15) & ~(size_t)15;
}

// one entry of the apex: the first three words are its record as a partner
struct __align__(16) Atm64Row {
    double v[3], id, p, g; // position from the apex, 1/d, sqrt(C6)/r^3, (r0^2/d)^(8/3)
    double lam_ea, lam_ae; // dC6/dCN over C6: of the entry, of the apex
    int j, t, k, pad;      // atom, type, entry number
    float f[4];            // rounded position
};
// a row x: its entry and C6 weights
struct Atm64X {
    Atm64Row e;
    double w[MAX_NREF + 1], dw[MAX_NREF + 1];
};
// scratch of one CTA: the rows of its split by type, then the entries set up at once
struct Atm64Scratch {
    unsigned char *p;
    unsigned int stride, first; // bytes per CTA, of its rows
    int entries;
};

// position of an entry relative to the apex
__device__ __forceinline__ double3 atm64_pos(const KP &p, const SG &g, const double4 &xa, const int2 ent, const double4 &xj) {
    double sx, sy, sz;
    image_vec(g, sext8(ent.y & 0xff), sext8((ent.y >> 8) & 0xff), sext8((ent.y >> 16) & 0xff), sx, sy, sz);
    return make_double3(xj.x + sx - xa.x, xj.y + sy - xa.y, xj.z + sz - xa.z);
}

// per-entry set-up (FP64 C6 of the apex pair, its CN derivatives, damping ratio)
template <int NR>
__device__ __forceinline__ Atm64Row atm64_entry(const KP &p, const SG &g, const double4 &xa, int a, const int2 ent,
                                                const double *yapex, const double *r0a, bool derivatives) {
    Atm64Row r;
    const double4 xj = p.xs[ent.x];
    r.j = ent.x;
    r.t = (int)xj.w;
    const double3 v = atm64_pos(p, g, xa, ent, xj);
    r.v[0] = v.x;
    r.v[1] = v.y;
    r.v[2] = v.z;
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
    r.f[0] = (float)v.x;
    r.f[1] = (float)v.y;
    r.f[2] = (float)v.z;
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

// a value that all lanes agree on, through the warp reduction whose result the hardware
// keeps once per warp: loops bounded by it need no divergence checks at every vote and
// shuffle inside
__device__ __forceinline__ int warp_uniform(int v) { return (int)__reduce_max_sync(0xffffffffu, v); }

// exclusive scan of the cell counts by the whole CTA: a run of 32 cells per warp and step
__device__ __forceinline__ void atm64_scan(int *cells, int ncell, int *s_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int run = (ncell / 32 + nw - 1) / nw; // steps per warp
    int carry = 0;
    for (int r = 0; r < run; ++r) {
        const int c = (warp * run + r) * 32 + lane;
        const int n = c < ncell ? cells[c] : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (c < ncell) cells[c] = carry + incl - n;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_tot[warp] = carry;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += s_tot[w];
    for (int r = 0; r < run; ++r) {
        const int c = (warp * run + r) * 32 + lane;
        if (c < ncell) cells[c] += before;
    }
}

// one exchange of the row reduction: keep v on the lower lanes and w on the upper ones of
// each pair `o` apart, adding what the other lane holds of it
__device__ __forceinline__ double atm64_fold(double v, double w, int o) {
    const bool up = (threadIdx.x & o) != 0;
    return (up ? w : v) + __shfl_xor_sync(0xffffffffu, up ? v : w, o);
}
// sums of eight values over the warp; lane l returns the sum of value ((l >> 2) & 7) with
// its three bits reversed
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

// Row sums in shared memory: [0..6] the reduced sums, then v_x, 1, 0, lam_ae, lam_ea and the
// weighted kind's virial sums. Output of lane l from entries S, A, B, U, V, M (s_rule) and
// coefficients c (s_coef): c0 M sum0 + c1 sum1 + c2 S A B - c3 (U B + V A).
//   0 energy share of the apex (E/3 per pair, half of it per visit), 1 its dE/dCN, 2..4 its
//   force -f1 v_x, 5..10 virial f r (x) r with the x-y side's cross part split evenly between
//   the two visits of a pair (xx yy zz xy xz yz), 11..15 energy, dE/dCN and force of the entry
enum { ATM64_SV = 8, ATM64_S1 = 11, ATM64_S0 = 12, ATM64_SAE = 13, ATM64_SEA = 14, ATM64_SVIR = 15, ATM64_SR = 20 };
__device__ inline void atm64_rules(bool weighted, int l, unsigned long long &rule, double c[4]) {
    const int Z = ATM64_S0;
    int q[6] = {Z, Z, Z, Z, Z, Z}; // S A B U V M
    c[0] = c[1] = c[2] = c[3] = 0;
    if (l == 0 || l == 11) {
        c[0] = l == 0 ? -1.0 / 6.0 : -1.0 / 3.0;
        q[5] = ATM64_S1;
    } else if (l == 1 || l == 12) {
        c[0] = -0.5;
        q[5] = l == 1 ? ATM64_SAE : ATM64_SEA;
        if (l == 12) c[1] = -0.5;
    } else if (l < 5) {
        c[2] = -1.0;
        q[0] = 6;
        q[1] = ATM64_SV + l - 2;
        q[2] = ATM64_S1;
    } else if (l < 11) {
        const int a = l < 8 ? l - 5 : (l < 10 ? 0 : 1), b = l < 8 ? a : (l == 8 ? 1 : 2);
        const int vir = weighted ? (int)ATM64_SVIR : 2;
        c[2] = 1.0;
        c[3] = 0.5;
        q[0] = vir;
        q[1] = ATM64_SV + a;
        q[2] = ATM64_SV + b;
        q[3] = vir + 1 + a;
        q[4] = vir + 1 + b;
    } else {
        c[2] = c[3] = 1.0;
        q[0] = 2;
        q[1] = ATM64_SV + l - 13;
        q[2] = ATM64_S1;
        q[3] = 3 + l - 13;
    }
    rule = 0;
    for (int k = 0; k < 6; ++k) rule |= (unsigned long long)q[k] << (8 * k);
}

// One visit: triplet (apex, x, y) with x in the arguments and y in the staged records A and
// R. Branch-free.
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
__global__ void __launch_bounds__(ATM64_THREADS, 1) k_atm64(KP p, Atm64Scratch scratch, int tile_bytes, int tile_max) {
    extern __shared__ __align__(16) unsigned char sm64[];
    constexpr int RQ = atm64_rowq(NR);
    const int ne = p.ne, nw = blockDim.x >> 5;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *yapex = reinterpret_cast<double *>(sm64);                 // [ne][NR]
    double *r0sq = yapex + ((ne * NR + 1) & ~1);                      // [ne][ne] r0ab^2
    int *toff = reinterpret_cast<int *>(r0sq + ((ne * ne + 1) & ~1)); // [ne + 1] rows of each type, [ne] fill positions
    int *tpos = toff + ne + 1;
    unsigned char *queue = reinterpret_cast<unsigned char *>(toff + ((2 * ne + 2 + 3) & ~3)) +
                           (size_t)warp * (8 * ATM64_QCAP + ATM64_LIST * sizeof(unsigned short)); // [slot][class]
    unsigned short *list = reinterpret_cast<unsigned short *>(queue + 8 * ATM64_QCAP);             // [ATM64_LIST]
    unsigned char *area = sm64 + atm64_fixed_bytes(ne, NR, nw);
    int *cells = reinterpret_cast<int *>(area); // [ATM64_CELLS] while the entries are sorted
    // (the entries' address and number, needed between the visits only, are read from shared
    // memory there: in registers they made 2,000 atoms of 12 types and 7 references 1 % slower)
    __shared__ Atm64Row *volatile s_entries;
    __shared__ volatile int s_ecap;
    __shared__ int s_item, s_row, s_tot[ATM64_THREADS / 32];
    __shared__ double red[ATM64_THREADS / 32][11], s_sums[ATM64_THREADS / 32][ATM64_SR], s_coef[16][4];
    __shared__ unsigned long long s_rule[16];
    double *sr = s_sums[warp];
    if (tid == 0) {
        s_entries = reinterpret_cast<Atm64Row *>(scratch.p + (size_t)blockIdx.x * scratch.stride + scratch.first);
        s_ecap = scratch.entries;
    }
    if (tid < 16) atm64_rules(KIND == ATM64_WEIGHTED, tid, s_rule[tid], s_coef[tid]);
    if (lane == 0) {
        sr[ATM64_S1] = 1.0;
        sr[ATM64_S0] = 0.0;
    }
    if (warp_uniform(p.atm_off[p.n] > p.atm_cap ? 1 : 0)) return; // list overflowed: the host grows it and re-runs
    for (int k = tid; k < ne * ne; k += blockDim.x) r0sq[k] = p.r0ab[k] * p.r0ab[k];
    Atm64X *rows = reinterpret_cast<Atm64X *>(scratch.p + (size_t)blockIdx.x * scratch.stride);
    const double third = 1.0 / 3.0;
    const double rc = sqrt(p.ratm2), cinv = 16.0 / (2.0 * rc);
    // FP32 range test: |d3 - half| <= half in range, but near either end of [0, 2 half] the
    // pair is tested again in FP64 (the rounded positions put d3 off by at most about
    // 5e-7 rc^2). Chunk spheres: distances off by less than 1e-5 rc.
    const float half = (float)(0.5 * p.ratm2 * (1.0 + 1e-5)), sure = half * (1.0f - 4e-5f);
    const float rcf = (float)rc, slack = 1e-4f * rcf, rc_hi = rcf * rcf * (1.0f + 1e-4f), rc_lo = rcf * rcf * (1.0f - 1e-4f);
    const int cls = lane & 7, member = lane >> 3;
    const unsigned cls_bits = 0x01010101u << cls, below = cls_bits & ((1u << lane) - 1u);
    unsigned long long visits = 0;
    while (true) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(p.work, 1);
        __syncthreads();
        const int S = KIND == ATM64_CENTER ? 1 : p.atmb_split;
        const int got = warp_uniform(s_item), split = got % S, unit = got / S;
        const int item = KIND == ATM64_CENTER ? unit : unit * p.shard_world + p.shard_rank;
        if (item >= (KIND == ATM64_CENTER ? warp_uniform(*p.atm_napex) : p.n)) break;
        const int a = KIND == ATM64_CENTER ? p.atm_apex[item] : p.sorted_of[p.n - 1 - item];
        const SG &g = p.sg[p.sid[a]];
        if (KIND != ATM64_CENTER && warp_uniform(g.atm_simple) != (KIND == ATM64_SIMPLE ? 1 : 0)) continue; // the other instance's
        const long long e0 = p.atm_off[a];
        const int m = warp_uniform((int)(p.atm_off[a + 1] - e0));
        if (KIND != ATM64_CENTER && m <= p.atm_min_m) continue; // k_atm64b's
        const double4 xa = p.xs[a];
        const bool ref = KIND == ATM64_WEIGHTED && atm_reference_order(p, g, p.sid[a]);
        const double *r0a = r0sq + (int)xa.w * ne;
        for (int k = tid; k < ne * NR; k += blockDim.x) yapex[k] = p.Y[(size_t)a * ne * NR + k];
        // types staged together and partner tile: all partners of the apex with as many
        // types as fit, else one type and the fewest tiles of equal length
        int types = ne, tile = 0;
        for (;; --types) {
            tile = min(min(tile_max, 32 * ATM64_CHUNKS),
                       (int)(((unsigned)tile_bytes - (unsigned)atm64_tile_fixed(NR, types)) / (unsigned)atm64_partner_bytes(NR, types)) & ~31);
            if (types == 1 || tile >= m) break;
        }
        if (m > 0) {
            const int tiles = (m + tile - 1) / tile;
            tile = ((m + tiles - 1) / tiles + 31) & ~31;
        }
        double2 *sA = reinterpret_cast<double2 *>(area);              // [tile + 1][3]: vx vy | vz id | p g
        float4 *sF = reinterpret_cast<float4 *>(sA + 3 * (tile + 1)); // [tile + 32]: FP32 position, atom
        float4 *sC = sF + tile + 32;                                  // [ATM64_CHUNKS][2]: box of each chunk, sphere radius
        double2 *sR = reinterpret_cast<double2 *>(sC + 2 * ATM64_CHUNKS); // [types][tile + 1][RQ]
        double acc = 0; // this lane's apex sum (lanes 0..10: energy, dE/dCN, force, virial)
        for (int b0 = 0; b0 < m; b0 += s_ecap) {
            // set up the entries in Hilbert order (counting sort on a 16^3, 8^3 or 4^3 grid,
            // whose curves are prefixes of one another) and list this split's rows by type
            const int bn = min(s_ecap, m - b0);
            Atm64Row *entries = s_entries;
            const int hs = bn >= 1024 ? 0 : (bn >= 128 ? 3 : 6), ncell = ATM64_CELLS >> hs;
            auto cell_of = [&](const int2 ent) {
                const double3 v = atm64_pos(p, g, xa, ent, p.xs[ent.x]);
                const int cx = min(15, max(0, (int)((v.x + rc) * cinv)));
                const int cy = min(15, max(0, (int)((v.y + rc) * cinv)));
                const int cz = min(15, max(0, (int)((v.z + rc) * cinv)));
                return atmb_hilbert(cx, cy, cz) >> hs;
            };
            __syncthreads();
            for (int k = tid; k <= ne; k += blockDim.x) toff[k] = 0;
            for (int k = tid; k < ncell; k += blockDim.x) cells[k] = 0;
            __syncthreads();
            for (int k = tid; k < bn; k += blockDim.x) atomicAdd(&cells[cell_of(p.atm_ent[e0 + b0 + k])], 1);
            __syncthreads();
            atm64_scan(cells, ncell, s_tot);
            __syncthreads();
            for (int k = tid; k < bn; k += blockDim.x) {
                const int2 ent = p.atm_ent[e0 + b0 + k];
                Atm64Row r = atm64_entry<NR>(p, g, xa, a, ent, yapex, r0a, true);
                r.k = b0 + k;
                entries[atomicAdd(&cells[cell_of(ent)], 1)] = r;
                if (r.k % S == split) atomicAdd(&toff[r.t + 1], 1);
            }
            __syncthreads();
            if (tid == 0)
                for (int t = 0; t < ne; ++t) {
                    tpos[t] = toff[t];
                    toff[t + 1] += toff[t];
                }
            __syncthreads();
            for (int k = tid; k < bn; k += blockDim.x)
                if (entries[k].k % S == split) {
                    Atm64X *r = rows + atomicAdd(&tpos[entries[k].t], 1);
                    r->e = entries[k];
#pragma unroll
                    for (int b = 0; b < NR; ++b) {
                        r->w[b] = p.w[(size_t)entries[k].j * NR + b];
                        r->dw[b] = p.dw[(size_t)entries[k].j * NR + b];
                    }
                }
            if (warp_uniform(toff[ne]) == 0) continue; // no row of this split
            for (int p0 = 0; p0 < m; p0 += tile) {
                const int cnt = min(tile, m - p0), nchunk = (cnt + 31) >> 5;
                for (int t0 = 0; t0 < ne; t0 += types) {
                    const int tn = min(types, ne - t0);
                    __syncthreads(); // the previous phase is done with the staged data and s_row
                    const int r0 = warp_uniform(toff[t0]), r1 = warp_uniform(toff[t0 + tn]);
                    if (r0 == r1 && t0 != 0) continue;
                    if (tid == 0) s_row = r0;
                    const Atm64Row *staged = s_entries;
                    for (int k = tid; k < cnt; k += blockDim.x) {
                        int j, tj;
                        if (m <= s_ecap) {
                            const Atm64Row *src = staged + p0 + k;
                            j = src->j;
                            tj = src->t;
                            if (t0 == 0) {
                                const double2 *q = reinterpret_cast<const double2 *>(src);
                                const double2 q0 = q[0], q1 = q[1];
                                sA[3 * k] = q0;
                                sA[3 * k + 1] = q1;
                                sA[3 * k + 2] = q[2];
                                sF[k] = make_float4((float)q0.x, (float)q0.y, (float)q1.x, __int_as_float(j));
                            }
                        } else {
                            const int2 ent = p.atm_ent[e0 + p0 + k];
                            j = ent.x;
                            tj = (int)p.xs[j].w;
                            if (t0 == 0) {
                                const Atm64Row r = atm64_entry<NR>(p, g, xa, a, ent, yapex, r0a, false);
                                sA[3 * k] = make_double2(r.v[0], r.v[1]);
                                sA[3 * k + 1] = make_double2(r.v[2], r.id);
                                sA[3 * k + 2] = make_double2(r.p, r.g);
                                sF[k] = make_float4((float)r.v[0], (float)r.v[1], (float)r.v[2], __int_as_float(j));
                            }
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
                    // far positions after the last partner and at tile .. tile + 31 (out of
                    // range of every row); the dummy partner's p = 0 makes its terms vanish
                    if (tid < 32) {
                        if (cnt + tid < 32 * nchunk) sF[cnt + tid] = make_float4(3e18f, 3e18f, 3e18f, 0.f);
                        sF[tile + tid] = make_float4(3e18f, 3e18f, 3e18f, __int_as_float(-1));
                    }
                    if (tid < tn) {
                        if (tid == 0) {
                            sA[3 * tile] = make_double2(3e4, 3e4);
                            sA[3 * tile + 1] = make_double2(3e4, 1.0);
                            sA[3 * tile + 2] = make_double2(0.0, 1.0);
                        }
                        double2 *dst = sR + ((size_t)tid * (tile + 1) + tile) * RQ;
#pragma unroll
                        for (int b = 0; b < (NR + 1) / 2; ++b) dst[b] = make_double2(1.0, 1.0);
                    }
                    __syncthreads();
                    if (t0 == 0) {
                        // bounding box of each chunk and the radius of its sphere about the box centre
                        for (int c = warp_uniform(warp); c < nchunk; c += nw) {
                            const float4 f = sF[min(32 * c + lane, cnt - 1)];
                            float lo[3] = {f.x, f.y, f.z}, hi[3] = {f.x, f.y, f.z};
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                                for (int q = 0; q < 3; ++q) {
                                    lo[q] = fminf(lo[q], __shfl_xor_sync(0xffffffffu, lo[q], o));
                                    hi[q] = fmaxf(hi[q], __shfl_xor_sync(0xffffffffu, hi[q], o));
                                }
                            const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
                            float r2 = (f.x - cx) * (f.x - cx) + (f.y - cy) * (f.y - cy) + (f.z - cz) * (f.z - cz);
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
                            if (lane == 0) {
                                sC[2 * c] = make_float4(lo[0], lo[1], lo[2], sqrtf(r2));
                                sC[2 * c + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
                            }
                        }
                        __syncthreads();
                    }
                    for (;;) {
                        int r = 0;
                        if (lane == 0) r = atomicAdd(&s_row, 1);
                        r = warp_uniform(r); // (the other lanes hold 0)
                        if (r >= r1) break;
                        const Atm64Row *X = &rows[r].e;
                        const double vx = X->v[0], vy = X->v[1], vz = X->v[2];
                        const double id1 = X->id, p1 = X->p, h1 = 0.75 * id1;
                        const double g1 = X->g * (6.0 * 4294967296.0 / 43046721.0); // 6 (4/3)^16
                        const double d1 = vx * vx + vy * vy + vz * vz;
                        const int jx = X->j;
                        double wx[NR], dwx[NR];
#pragma unroll
                        for (int b = 0; b < NR; ++b) {
                            wx[b] = rows[r].w[b];
                            dwx[b] = rows[r].dw[b];
                        }
                        const float fx = X->f[0], fy = X->f[1], fz = X->f[2];
                        const double2 *sRx = sR + (size_t)(X->t - t0) * RQ * (tile + 1);
                        // sums over this row's visits: w E', w E' lam_xy, wf (f1 + f3),
                        // wf f3 v_y (3), wf f1; v[7] unused
                        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                        // weighted kind: (w - wf) (f1 + f3), (w - wf) f3 v_y
                        double dv[4] = {0, 0, 0, 0};
                        // one visit per lane, of partner k
                        auto visit = [&](int k) {
                            Atm64Visit V;
                            atm64_visit<NR>(vx, vy, vz, d1, id1, h1, p1, g1, wx, dwx, sA + 3 * k, sRx + RQ * k, V);
                            if (KIND == ATM64_WEIGHTED) {
                                const int jy = __float_as_int(sF[k].w);
                                if (jx == jy || jx == a || jy == a) {
                                    double w, wf;
                                    atm_weights(jx == jy, jx == a, jy == a, ref, p.atm_force_scaled != 0, w, wf);
                                    const double d3w = (w - wf) * V.f3;
                                    dv[0] = fma(w - wf, V.f1 + V.f3, dv[0]);
                                    dv[1] = fma(d3w, V.vx, dv[1]);
                                    dv[2] = fma(d3w, V.vy, dv[2]);
                                    dv[3] = fma(d3w, V.vz, dv[3]);
                                    V.E *= w;
                                    V.f1 *= wf;
                                    V.f3 *= wf;
                                }
                            }
                            v[0] += V.E;
                            v[1] = fma(V.E, V.lam, v[1]);
                            v[2] += V.f1 + V.f3;
                            v[3] = fma(V.f3, V.vx, v[3]);
                            v[4] = fma(V.f3, V.vy, v[4]);
                            v[5] = fma(V.f3, V.vz, v[5]);
                            v[6] += V.f1;
                        };
                        // classify the chunks (lane l: chunks l and l + 32) and list them. A
                        // chunk is all in range only when it is whole and x lies outside its
                        // box (no pair closer than 0.1 bohr)
                        int nfull = 0, nmixed = 0;
                        __syncwarp();
#pragma unroll
                        for (int h = 0; h < ATM64_CHUNKS / 32; ++h) {
                            const int c = 32 * h + lane;
                            bool none = true, all = false;
                            if (c < nchunk) {
                                // nearest and farthest points of its box, its sphere
                                const float4 L = sC[2 * c], H = sC[2 * c + 1];
                                const float ax = fx - L.x, bx = H.x - fx, ay = fy - L.y, by = H.y - fy, az = fz - L.z, bz = H.z - fz;
                                const float nx = fmaxf(0.f, -fminf(ax, bx)), ny = fmaxf(0.f, -fminf(ay, by)), nz = fmaxf(0.f, -fminf(az, bz));
                                const float gx = fmaxf(ax, bx), gy = fmaxf(ay, by), gz = fmaxf(az, bz);
                                const float near2 = nx * nx + ny * ny + nz * nz, far2 = gx * gx + gy * gy + gz * gz;
                                const float d2 = 0.25f * ((ax - bx) * (ax - bx) + (ay - by) * (ay - by) + (az - bz) * (az - bz));
                                const float past = rcf + L.w + slack, inside = fmaxf(0.f, rcf - L.w - slack);
                                none = near2 > rc_hi || d2 > past * past;
                                all = (far2 < rc_lo || d2 < inside * inside) && near2 > 0.01f && 32 * c + 32 <= cnt;
                            }
                            const unsigned fb = __ballot_sync(0xffffffffu, all), mb = __ballot_sync(0xffffffffu, !all && !none);
                            const unsigned lt = (1u << lane) - 1u;
                            if (all) list[nfull + __popc(fb & lt)] = (unsigned short)(32 * c);
                            if (!all && !none) list[ATM64_LIST - 1 - (nmixed + __popc(mb & lt))] = (unsigned short)(32 * c);
                            nfull = warp_uniform(nfull + __popc(fb));
                            nmixed = warp_uniform(nmixed + __popc(mb));
                        }
                        // (the mixed list is filled up with the far positions)
                        if (lane < ATM64_SEG - 1 && nmixed + lane < ((nmixed + ATM64_SEG - 1) & ~(ATM64_SEG - 1)))
                            list[ATM64_LIST - 1 - (nmixed + lane)] = (unsigned short)tile;
                        __syncwarp();
                        if (lane == 0) visits += 32 * nfull;
#pragma unroll 1
                        for (int i = 0; i < nfull; ++i) visit(list[i] + lane);
#pragma unroll 1
                        for (int i0 = 0; i0 < nmixed; i0 += ATM64_GROUP) {
                            // test the partners of up to ATM64_GROUP mixed chunks, queue those
                            // in range (k / 8: the class is k mod 8)
                            const int i1 = min(nmixed, i0 + ATM64_GROUP);
                            int tail = 0; // queued partners of this lane's class
                            __syncwarp();
#pragma unroll 1
                            for (int i = i0; i < i1; i += ATM64_SEG) {
                                unsigned bits[ATM64_SEG];
                                int k[ATM64_SEG];
                                bool edge = false;
#pragma unroll
                                for (int c = 0; c < ATM64_SEG; ++c) {
                                    k[c] = list[ATM64_LIST - 1 - (i + c)] + lane;
                                    const float4 f = sF[k[c]];
                                    const float dx = fx - f.x, dy = fy - f.y, dz = fz - f.z;
                                    const float off = fabsf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - half);
                                    bits[c] = __ballot_sync(0xffffffffu, off <= half);
                                    edge |= off <= half && off >= sure;
                                }
                                if (warp_uniform(edge ? 1 : 0)) {
#pragma unroll
                                    for (int c = 0; c < ATM64_SEG; ++c) {
                                        const double2 *A = sA + 3 * min(k[c], tile);
                                        const double rx = vx - A[0].x, ry = vy - A[0].y, rz = vz - A[1].x;
                                        const double d3 = fma(rx, rx, fma(ry, ry, rz * rz));
                                        bits[c] &= __ballot_sync(0xffffffffu, d3 <= p.ratm2 && d3 >= 1e-12); // also drops x == y
                                    }
                                }
#pragma unroll
                                for (int c = 0; c < ATM64_SEG; ++c) {
                                    if (bits[c] & (1u << lane))
                                        queue[(tail + __popc(bits[c] & below)) * 8 + cls] = (unsigned char)(k[c] >> 3);
                                    tail += __popc(bits[c] & cls_bits);
                                }
                            }
                            __syncwarp();
                            const int rounds = warp_uniform((tail + 3) >> 2);
#pragma unroll 1
                            for (int i = 0; i < rounds; ++i) {
                                const int q = 4 * i + member;
                                int k = queue[q * 8 + cls] * 8 + cls;
                                k = q < tail ? k : tile;
                                visit(k);
                            }
                            if (member == 0) visits += (unsigned)tail;
                        }
                        if (KIND == ATM64_CENTER) {
#pragma unroll
                            for (int k = 0; k < 7; ++k) v[k] *= third;
                        }
                        // the row's sums; then each of 16 lanes forms one output from them (rule
                        // and coefficients in s_rule, s_coef): lanes 0..10 apex sums, 11..15
                        // the entry's energy, dE/dCN and force
                        const double tot = atm64_reduce8(v);
                        if ((lane & 3) == 0) sr[((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = tot;
                        if (lane == 1) {
                            sr[ATM64_SV] = vx;
                            sr[ATM64_SV + 1] = vy;
                            sr[ATM64_SV + 2] = vz;
                            sr[ATM64_SAE] = X->lam_ae;
                            sr[ATM64_SEA] = X->lam_ea;
                        }
                        __syncwarp();
                        if (KIND == ATM64_WEIGHTED) {
                            // virial sums (weights w)
                            double d[4] = {0, 0, 0, 0};
                            if (warp_uniform(dv[0] != 0.0 || dv[1] != 0.0 || dv[2] != 0.0 || dv[3] != 0.0))
#pragma unroll
                                for (int k = 0; k < 4; ++k) d[k] = warp_sum(dv[k]);
                            if (lane == 0)
#pragma unroll
                                for (int k = 0; k < 4; ++k) sr[ATM64_SVIR + k] = sr[2 + k] + d[k];
                            __syncwarp();
                        }
                        if (lane < 16) {
                            const unsigned long long rule = s_rule[lane];
                            auto at = [&](int q) { return sr[(rule >> (8 * q)) & 0xff]; };
                            const double va = at(1), vb = at(2);
                            const double val = s_coef[lane][0] * at(5) * sr[0] + s_coef[lane][1] * sr[1] +
                                               s_coef[lane][2] * at(0) * va * vb - s_coef[lane][3] * (at(3) * vb + at(4) * va);
                            if (lane < 11)
                                acc += val;
                            else
                                atomicAdd(lane == 11 ? p.eb + jx : (lane == 12 ? p.gb + jx : p.fb + 3 * (size_t)jx + (lane - 13)), val);
                        }
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
