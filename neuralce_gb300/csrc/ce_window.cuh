// Windowed sign-parity kernel of the cluster-expansion chunk (one basis site per cell, binary point functions +-1).
// Included by ce_engine.cu, whose job descriptor, proposals and chunk end it shares.
//
// What bounds a chunk is the Markov chain: each step's dE depends on every earlier accepted swap.  But a swap moves
// only the dE of swaps whose neighbourhoods hold one of its two sites, so the CTA of a replica evaluates a window of up
// to 32 steps (at most 16 of them between different species) at once.  Each swap is evaluated on the state that the
// earlier swaps of the window would leave if they went as predicted (as they went when a former window evaluated them;
// a new one as most of this replica's swaps went).  Then the window is decided in step order up to the first step that
// a wrongly predicted swap touches (or that shares a site with an accepted one): all steps before it have been
// evaluated on exactly the state that the step-by-step chain reaches, so every decision is the chain's.  The next
// window starts there.
//
// Evaluation is bit-sliced over the window's sites: word n of the window holds, for every one of the up to 32 sites
// (2 per swap), the species bit of its neighbourhood entry n (one ballot per entry, a site a lane).  The parity of one
// row product for all sites is then the XOR of at most three words.  A lane XORs kWinRows rows of one cluster-vector
// column and compresses them with full adders into three words (weights 1, 2, 4); a 32 x 32 bit transpose across the
// warp turns 32 lanes' words into one word a site, whose popcount over a column's lanes is that column's count of odd
// products.  Flipping a site negates every product that holds it, so a swap of a and b (b flipped first, then a with b
// already flipped) moves column c by 2 sgn (odd_a - odd_b): the integers n_c of the step-by-step kernel, and dE their
// exact fixed-point sum (float64) or the same float32 sum in the same order.

constexpr int kWinRows = 7;              // rows a lane: 7 = the most that three adder words hold
constexpr int kWinSwaps = 16;            // swaps evaluated at once: two sites each fill the 32 bits of a word
constexpr int kWinBatch = 9;             // neighbourhood entries a warp loads at once (141 entries on 16 warps: all)
constexpr int kWinSegs = 4;               // column segments of a row block
constexpr int kWinNone = 0x7fffffff;     // "no neighbour": no window index has this value

// per-model tables (device)
struct WinTab {
    int32_t n_ent;                       // neighbourhood entries, entry 0 the site itself; entry n_ent reads as 0
    int32_t aliases;                     // some displacement has two entries (tiny cells)
    int32_t n_blk;                       // row blocks of 32 lanes x kWinRows rows
    int32_t lo[3], ext[3];               // offsets per axis lie in [-lo, ext - 1 - lo], ext <= d
    const int4 *ent;                     // (n_ent) offset (u0, u1, u2 in [0, d)) and its window index
    const uint32_t *desc;                // (n_blk, kWinRows, 32) three word indices x 4: bits 2.., 12.., 22..
    const uint2 *seg;                    // (n_blk, kWinSegs) (lanes of the block, 33 x column), lanes 0 when unused
    const int16_t *nbr;                  // entry at each displacement of the window, -1 none
    const int16_t *alias;                // (n_ent) next entry at the same displacement (tiny cells), -1 none
    const int32_t *csign;                // (n_cols) +-2: twice the sign of a column's products for species bits as stored
};

struct WinLayout {                       // dynamic shared memory
    size_t words, cnt, desc, seg, ent, dcv, nsw, ring, total;
    __host__ __device__ static WinLayout make(int n_ent, int n_blk, int n_cols) {
        WinLayout L; size_t o = 0;
        auto al = [](size_t x) { return (x + 15) / 16 * 16; };
        L.words = o; o = al(o + 4 * (size_t)(n_ent + 1));
        L.cnt = o; o = al(o + 4 * 33 * (size_t)n_cols);
        L.desc = o; o = al(o + 4 * 32 * (size_t)kWinRows * n_blk);
        L.seg = o; o = al(o + 8 * (size_t)kWinSegs * n_blk);
        L.ent = o; o = al(o + 16 * (size_t)n_ent);
        L.dcv = o; o = al(o + 4 * (size_t)n_cols);
        L.nsw = o; o = al(o + 2 * (size_t)kWinSwaps * n_cols);
        L.ring = o; o = al(o + (size_t)kWinRing * (16 + 16 + 8 + 4 + 4));
        L.total = o;
        return L;
    }
};

struct WinCtl {
    int32_t s, n_w, nv;                  // first step of the window, its steps, its evaluated swaps
    uint32_t pred;                       // swaps predicted to be accepted
    int4 site[32];                       // per site: k0, k1, k2, site index
    int32_t del[32];                     // window index of the partner b from site a; kWinNone for b and far pairs
    int32_t step[2][kWinSwaps];          // step within the window, per swap (windows in turn)
    int32_t spa[kWinSwaps];              // species of site a
    long long part[kWinSwaps];           // dE: fixed point or the bits of a float64
    int32_t flags[kWinSwaps];            // 1 accepted, 2 near its threshold
    int32_t nbr[kWinSwaps], same[kWinSwaps];   // first later step whose dE the swap moves; first that shares a site with it
    uint8_t known[kWinRing];             // how a former window decided a step it could not settle: 0 unknown, 1 yes, 2 no
};

// ring of proposals: coordinates and site index of a and b, uniform, its logarithm, window index of b seen from a
struct WinRing { int4 *a, *b; unsigned long long *u; float *lnu; int32_t *del; };

// displacement x -> y as an index of the displacement window, kWinNone when outside it
__device__ __forceinline__ int32_t win_disp(const CEJob &jb, const WinTab &wt, const int4 &x, const int4 &y) {
    const int32_t z0 = y.x - x.x + wt.lo[0], z1 = y.y - x.y + wt.lo[1], z2 = y.z - x.z + wt.lo[2];
    // z in (-d, 2 d): the representative in [0, d) is the least of z, z + d, z - d as unsigned numbers
    const uint32_t a0 = min(min((uint32_t)z0, (uint32_t)(z0 + jb.d0)), (uint32_t)(z0 - jb.d0));
    const uint32_t a1 = min(min((uint32_t)z1, (uint32_t)(z1 + jb.d1)), (uint32_t)(z1 - jb.d1));
    const uint32_t a2 = min(min((uint32_t)z2, (uint32_t)(z2 + jb.d2)), (uint32_t)(z2 - jb.d2));
    const bool in = a0 < (uint32_t)wt.ext[0] && a1 < (uint32_t)wt.ext[1] && a2 < (uint32_t)wt.ext[2];
    return in ? (int32_t)((a0 * (uint32_t)wt.ext[1] + a1) * (uint32_t)wt.ext[2] + a2) : kWinNone;
}

// neighbourhood entry of site x that is site y, -1 none (aliases: wt.alias)
__device__ __forceinline__ int win_entry(const CEJob &jb, const WinTab &wt, const int4 &x, const int4 &y) {
    const int32_t i = win_disp(jb, wt, x, y);
    const int n = __ldg(wt.nbr + (i == kWinNone ? 0 : i));
    return i == kWinNone ? -1 : n;
}

__device__ __forceinline__ void win_propose(const CEJob &jb, const WinTab &wt, const WinRing &ring, int64_t g0, int32_t s, int32_t t) {
    LfProp P;
    lf_propose(jb, g0, s, t, P);
    const int i = win_slot(s, 0);
    const int4 a = make_int4(P.ka[0], P.ka[1], P.ka[2], (int32_t)P.ia), b = make_int4(P.kb[0], P.kb[1], P.kb[2], (int32_t)P.ib);
    ring.a[i] = a; ring.b[i] = b;
    ring.u[i] = jb.prop_a ? (unsigned long long)__double_as_longlong(P.uh) : (unsigned long long)P.um;
    // (a host uniform below 0 or NaN has no logarithm: the float64 rule takes it, and rejects)
    ring.lnu[i] = jb.prop_a && !(P.uh >= 0.0) ? nanf("") : P.lnu;
    ring.del[i] = win_disp(jb, wt, a, b);
}

// float64 logarithm of the stored uniform, as the step-by-step kernels form it
__device__ __noinline__ double win_log(bool host, unsigned long long u) {
    return log(host ? __longlong_as_double((long long)u) : (double)(u + 1ull) * 1.1102230246251565404236316680908203125e-16);
}

// Metropolis decision and near-threshold flag of dE.  float32 settles a swap whose |beta dE + ln u| exceeds its own error
// (below 1e-6 + 1e-6 (|beta dE| + |ln u|)) and the near band (tol_near); the others (about one in 10^5) take the exact
// rule: the fixed-point threshold ceil(-ln u / beta 2^S) (float64) or ln u < -beta dE in float64 (float32).  So does every
// swap at a beta below 0 or NaN, where the fixed-point rule has no such threshold and the band no width.
__device__ __forceinline__ int win_decide_fix(const CEJob &jb, long long part, unsigned long long u, float lnu, float beta_f,
                                              float scale_f, float tol_near) {
    const float bd = beta_f * ((float)part * scale_f), y = bd + lnu;
    const float tol = tol_near + 1e-6f * (fabsf(bd) + fabsf(lnu));
    if (y < -tol) return 1;
    if (y > tol) return 0;
    const double logu = win_log(jb.prop_a != nullptr, u), beta = (double)beta_f;
    long long thr;
    if (beta > 0.0) {
        const double xs = -logu / beta * ldexp(1.0, jb.fix_shift);
        thr = xs >= 4.611686018427388e18 ? 4611686018427387904ll : (long long)ceil(xs);
    } else {
        thr = logu < 0.0 ? 4611686018427387904ll : -4611686018427387904ll;
    }
    const long long dd = part - thr;
    return (part < thr ? 1 : 0) | ((dd < 0 ? -dd : dd) < (long long)jb.near_fix ? 2 : 0);
}

__device__ __forceinline__ int win_decide_f32(const CEJob &jb, double dE, unsigned long long u, float lnu, float beta_f,
                                              float tol_near) {
    const float bd = beta_f * (float)dE, y = bd + lnu;
    const float tol = tol_near + 1e-6f * (fabsf(bd) + fabsf(lnu));
    if (y < -tol) return 1;
    if (y > tol) return 0;
    const double logu = win_log(jb.prop_a != nullptr, u), beta = (double)beta_f;
    return (logu < -beta * dE ? 1 : 0) | (beta > 0.0 && fabs(dE + logu / beta) < jb.near_eV ? 2 : 0);
}

// One CTA per replica.  Warp 0 decides and lists windows while warp 1 keeps the books, the last warp draws proposals while the
// others count rows; all warps gather the window's words and sum the swaps' dE.  Four barriers a window.  A window takes
// about 6.9 k cycles on an SM of its own (2,048 sites: words 2.6 k, rows 1.9 k, dE 1.1 k, decision and list 1.4 k), at the hottest
// replica 20 steps; with one warp keeping everything, 64 registers a thread and uneven column segments it took 10.5 k
// (1,000 steps of 32 replicas: 281 -> 211 us; 1,048,576 sites x 64, 500 steps: 152 -> 103 us).
template <typename Acc, int MINB>
__global__ void __launch_bounds__(512, MINB) ce_win_chunk_kernel(const __grid_constant__ CEBatch bt) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool FIX = std::is_same<Acc, double>::value;
    __shared__ CEJob sjob;
    __shared__ WinTab wt;
    __shared__ WinCtl X;
    const int j = find_job(bt, blockIdx.x);
    copy_job(bt, j, sjob);
    const CEJob &jb = sjob;
    const int r = blockIdx.x - jb.cta_base;
    if (r >= jb.R) return;
    const int tid = threadIdx.x, nt = blockDim.x, nw = nt >> 5, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < (int)(sizeof(WinTab) / 4); i += nt)
        reinterpret_cast<int *>(&wt)[i] = reinterpret_cast<const int *>(jb.win)[i];
    __syncthreads();
    const int n_ent = wt.n_ent, n_cols = jb.n_cols, n_blk = wt.n_blk;
    const WinLayout L = WinLayout::make(n_ent, n_blk, n_cols);
    uint32_t *words = reinterpret_cast<uint32_t *>(smem + L.words);
    int32_t *cnt = reinterpret_cast<int32_t *>(smem + L.cnt);               // [column][site], rows of 33
    uint32_t *desc = reinterpret_cast<uint32_t *>(smem + L.desc);
    uint2 *seg = reinterpret_cast<uint2 *>(smem + L.seg);
    int4 *ent = reinterpret_cast<int4 *>(smem + L.ent);
    int32_t *dcv = reinterpret_cast<int32_t *>(smem + L.dcv);
    int16_t *nsw = reinterpret_cast<int16_t *>(smem + L.nsw);                // [swap][column] of the evaluated swaps
    WinRing ring;
    ring.a = reinterpret_cast<int4 *>(smem + L.ring); ring.b = ring.a + kWinRing;
    ring.u = reinterpret_cast<unsigned long long *>(ring.b + kWinRing);
    ring.lnu = reinterpret_cast<float *>(ring.u + kWinRing); ring.del = reinterpret_cast<int32_t *>(ring.lnu + kWinRing);
    int8_t *gsig = jb.sigma + (int64_t)r * jb.N;
    for (int i = tid; i < n_blk * kWinRows * 32; i += nt) desc[i] = __ldg(wt.desc + i);
    for (int i = tid; i < n_blk * kWinSegs; i += nt) seg[i] = __ldg(wt.seg + i);
    for (int i = tid; i < n_ent; i += nt) ent[i] = __ldg(wt.ent + i);
    for (int i = tid; i < 33 * n_cols; i += nt) cnt[i] = 0;
    for (int i = tid; i <= n_ent; i += nt) words[i] = 0;
    for (int c = tid; c < n_cols; c += nt) dcv[c] = 0;
    for (int i = tid; i < kWinRing; i += nt) X.known[i] = 0;
    const bool track = jb.cv != nullptr;
    const int32_t t = jb.slot_of_rep[r];
    const float beta_f = jb.beta_slot[t];
    const int32_t T = (int32_t)jb.n_steps;
    const int64_t g0 = jb.step_dev ? *jb.step_dev : jb.step0;
    const double fscale = ldexp(1.0, -jb.fix_shift);
    const float scale_f = ldexpf(1.0f, -jb.fix_shift);
    // (beta below 0 or NaN: nothing is settled in float32)
    const float tol_near = beta_f >= 0.0f ? 1e-6f + 1.001f * beta_f * ((float)jb.near_eV + (FIX ? 4.0f * scale_f : 0.0f)) : HUGE_VALF;
    const int32_t si = jb.E_samples && jb.sample_interval <= T ? (int32_t)jb.sample_interval : 0;
    int32_t left = si;                                       // steps from the window's start to the next sample
    const double E0 = jb.E[r];
    double E = E0, Emin = jb.E_min_rep[r];                  // float32: carried energy and running minimum (warp 1)
    long long dsum = 0, dmin = 0;                            // float64: the chunk's energy change; this lane's minimum of it
    int32_t nacc = 0, nnear = 0, s_cur = 0, score = 0;
    uint32_t drawn = 96;
    for (int q = tid; q < min(96, T); q += nt) win_propose(jb, wt, ring, g0, q, t);
    // this lane's columns (lane, lane + 32) of the dE sum; further columns, if any, are read where they are used
    const int c0 = lane, c1 = lane + 32;
    auto col_e = [&](int c) -> Acc {
        return FIX ? Acc(0) : (c < n_cols ? __ldg(reinterpret_cast<const Acc *>(jb.ecol2) + c) : Acc(0));
    };
    auto col_fix = [&](int c) -> long long { return FIX && c < n_cols ? (long long)__ldg(jb.ecol_fix + c) : 0ll; };
    const float e0 = (float)col_e(c0), e1 = (float)col_e(c1);
    const long long f0 = col_fix(c0), f1 = col_fix(c1);
    const int cs0 = c0 < n_cols ? __ldg(wt.csign + c0) : 0, cs1 = c1 < n_cols ? __ldg(wt.csign + c1) : 0;
    __syncthreads();
    // transpose constants of this lane: byte selectors of the 16- and 8-steps, rotations and keep masks of 4, 2, 1
    const uint32_t sel16 = (lane & 16) ? 0x3276u : 0x5410u, sel8 = (lane & 8) ? 0x3715u : 0x6240u;
    const int rot4 = (lane & 4) ? 28 : 4, rot2 = (lane & 2) ? 30 : 2, rot1 = (lane & 1) ? 31 : 1;
    const uint32_t keep4 = (lane & 4) ? 0xf0f0f0f0u : 0x0f0f0f0fu, keep2 = (lane & 2) ? 0xccccccccu : 0x33333333u,
                   keep1 = (lane & 1) ? 0xaaaaaaaau : 0x55555555u;
    auto transpose = [&](uint32_t x) -> uint32_t {           // bit r of lane p <- bit p of lane r
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16);
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8);
        uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4); y = __funnelshift_l(y, y, rot4); x = (x & keep4) | (y & ~keep4);
        y = __shfl_xor_sync(0xffffffffu, x, 2); y = __funnelshift_l(y, y, rot2); x = (x & keep2) | (y & ~keep2);
        y = __shfl_xor_sync(0xffffffffu, x, 1); y = __funnelshift_l(y, y, rot1); x = (x & keep1) | (y & ~keep1);
        return x;
    };
    int par = 1;                                              // parity of the window in X.step
    // warp 0: the window that starts at step s_cur, on the present occupancy, into X (X.step of the other parity)
    auto list_window = [&]() {
        const int avail = min(32, T - s_cur);
        const int i = win_slot(s_cur, lane);
        int sa = 0, sb = 0, known = 0, del = 0;
        int4 a = make_int4(0, 0, 0, 0), b = a;
        if (lane < avail) {
            a = ring.a[i]; b = ring.b[i]; known = X.known[i]; del = ring.del[i];
            sa = gsig[a.w]; sb = gsig[b.w];
        }
        const unsigned V = __ballot_sync(0xffffffffu, sa != sb);
        const int rank = __popc(V & ((1u << lane) - 1u));
        const unsigned over = __ballot_sync(0xffffffffu, sa != sb && rank == kWinSwaps);   // the 17th swap ends the window
        const int n_w = over ? __ffs(over) - 1 : avail;
        const int nv = min(__popc(V), kWinSwaps);
        const bool in = sa != sb && lane < n_w, yes = in && (known == 1 || (known == 0 && score > 0));
        const unsigned pred = __reduce_or_sync(0xffffffffu, yes ? 1u << rank : 0u);
        if (lane >= 2 * nv) {                                 // unused sites read the first cell's neighbourhood
            X.site[lane] = make_int4(0, 0, 0, 0); X.del[lane] = kWinNone;
        }
        if (in) {
            X.site[2 * rank] = a; X.site[2 * rank + 1] = b;
            X.del[2 * rank] = del; X.del[2 * rank + 1] = kWinNone;
            X.step[par ^ 1][rank] = lane; X.spa[rank] = sa;
        }
        if (lane == 0) { X.s = s_cur; X.n_w = n_w; X.nv = nv; X.pred = pred; }
    };
    if (warp == 0) list_window();
    for (;;) {
        __syncthreads();                                      // the window is listed
        const int n_w = X.n_w, nv = X.nv, s_w = X.s;
        const uint32_t pred = X.pred;
        if (n_w == 0) break;
        par ^= 1;
        const int32_t *step = X.step[par];
        // what swap v changes, once accepted: the first later swap whose neighbourhood holds one of its sites and the
        // first later step that shares a site with it; apply: flip its two sites in the later swaps' words
        auto touch = [&](int v, const int4 &own, bool apply) {
            const int4 a = X.site[2 * v], b = X.site[2 * v + 1];
            const int q = step[v];
            const int na = win_entry(jb, wt, own, a), nb = win_entry(jb, wt, own, b);
            const bool later = lane >= 2 * v + 2 && lane < 2 * nv;
            const unsigned hit = __ballot_sync(0xffffffffu, later && (na >= 0 || nb >= 0));
            if (apply && later) {
                if (na >= 0) atomicXor(&words[na], 1u << lane);
                if (nb >= 0) atomicXor(&words[nb], 1u << lane);
                if (wt.aliases) {
                    for (int n = na; n >= 0 && (n = __ldg(wt.alias + n)) >= 0;) atomicXor(&words[n], 1u << lane);
                    for (int n = nb; n >= 0 && (n = __ldg(wt.alias + n)) >= 0;) atomicXor(&words[n], 1u << lane);
                }
            }
            const int i = win_slot(s_w, lane);
            bool eq = false;
            if (lane > q && lane < n_w) {
                const int pa = ring.a[i].w, pb = ring.b[i].w;
                eq = pa == a.w || pa == b.w || pb == a.w || pb == b.w;
            }
            const unsigned same = __ballot_sync(0xffffffffu, eq);
            if (lane == 0) {
                X.nbr[v] = hit ? step[(__ffs(hit) - 1) >> 1] : 32;
                X.same[v] = same ? __ffs(same) - 1 : 32;
            }
        };
        if (nv > 0) {
            // 1. words: entry n of every site's neighbourhood, b seen from a already flipped, swaps predicted to be
            //    accepted flipped in the later swaps' words (XORs into zeroed words: in any order)
            const int4 own = X.site[lane];
            const int del = X.del[lane];
            bool touched = false;
            for (int n0 = 1 + warp; n0 < n_ent; n0 += kWinBatch * nw) {      // (no row lists its own site)
                uint32_t mine = 0;
                int at[kWinBatch]; int8_t v[kWinBatch];
#pragma unroll
                for (int i = 0; i < kWinBatch; ++i) {
                    const int4 e = ent[min(n0 + i * nw, n_ent - 1)];
                    uint32_t q0 = (uint32_t)(own.x + e.x), q1 = (uint32_t)(own.y + e.y), q2 = (uint32_t)(own.z + e.z);
                    q0 = min(q0, q0 - (uint32_t)jb.d0); q1 = min(q1, q1 - (uint32_t)jb.d1); q2 = min(q2, q2 - (uint32_t)jb.d2);
                    at[i] = e.w;
                    v[i] = gsig[(q0 * (uint32_t)jb.d1 + q1) * (uint32_t)jb.d2 + q2];
                }
                if (!touched) {                                  // (while the loads are on their way)
                    touched = true;
                    for (int t = warp; t < nv; t += nw)
                        if ((pred >> t) & 1u) touch(t, own, true);
                }
#pragma unroll
                for (int i = 0; i < kWinBatch; ++i) {
                    const uint32_t w = __ballot_sync(0xffffffffu, (v[i] != 0) != (at[i] == del));
                    if (lane == i) mine = w;
                }
                if (lane < kWinBatch && n0 + lane * nw < n_ent) atomicXor(&words[n0 + lane * nw], mine);
            }
            if (!touched)                                        // (a warp without entries)
                for (int t = warp; t < nv; t += nw)
                    if ((pred >> t) & 1u) touch(t, own, true);
            __syncthreads();
            // 2. rows: odd products per column and site (the last warp draws proposals: 64 steps ahead of the window's
            //    start stay drawn, whatever the window's progress; at most 128 are in the ring)
            for (int blk = warp; blk < n_blk; blk += nw) {
                const uint32_t *dp = desc + blk * (kWinRows * 32) + lane;
                uint32_t v[kWinRows];
                const char *wb = reinterpret_cast<const char *>(words);
#pragma unroll
                for (int h = 0; h < kWinRows; ++h) {
                    const uint32_t dd = dp[h * 32];
                    v[h] = *reinterpret_cast<const uint32_t *>(wb + (dd & 0xffcu)) ^
                           *reinterpret_cast<const uint32_t *>(wb + ((dd >> 10) & 0xffcu)) ^
                           *reinterpret_cast<const uint32_t *>(wb + ((dd >> 20) & 0xffcu));
                }
                // seven rows into three words by four full adders
                const uint32_t s0 = v[0] ^ v[1] ^ v[2], k0 = (v[0] & v[1]) | (v[2] & (v[0] | v[1]));
                const uint32_t s1 = v[3] ^ v[4] ^ v[5], k1 = (v[3] & v[4]) | (v[5] & (v[3] | v[4]));
                const uint32_t w1 = s0 ^ s1 ^ v[6], k2 = (s0 & s1) | (v[6] & (s0 | s1));
                const uint32_t w2 = k0 ^ k1 ^ k2, w4 = (k0 & k1) | (k2 & (k0 | k1));
                uint2 sg[kWinSegs];                              // (a block has at most kWinSegs segments, padded with empty ones)
#pragma unroll
                for (int g = 0; g < kWinSegs; ++g) sg[g] = seg[blk * kWinSegs + g];
                const uint32_t t1 = transpose(w1), t2 = transpose(w2), t4 = transpose(w4);
#pragma unroll
                for (int g = 0; g < kWinSegs; ++g)
                    if (sg[g].x) atomicAdd(&cnt[sg[g].y + lane], __popc(t1 & sg[g].x) + 2 * __popc(t2 & sg[g].x) + 4 * __popc(t4 & sg[g].x));
            }
        }
        if (warp == nw - 1 && win_draws(drawn, s_w) && win_in_chunk(drawn, lane, T)) {
            win_propose(jb, wt, ring, g0, (int32_t)drawn + lane, t);
            X.known[win_slot((int32_t)drawn, lane)] = 0;
        }
        if (win_draws(drawn, s_w)) drawn += 32;
        __syncthreads();
        if (nv > 0) {
            // 3. dE of each swap and its decision; what a swap accepted against its prediction changes
            for (int i = tid; i < n_ent; i += nt) words[i] = 0;
            for (int v = warp; v < kWinSwaps; v += nw) {
                int32_t *ca = cnt + 2 * v, *cb = ca + 1;
                if (v < nv) {
                    const int i = win_slot(s_w, step[v]);
                    const int sgn = X.spa[v] ? -1 : 1;
                    const unsigned long long u = ring.u[i];
                    const float lnu = ring.lnu[i];
                    long long part = 0; float pf = 0.0f;
                    int n0 = 0, n1 = 0, flags;
                    if (c0 < n_cols) n0 = sgn * cs0 * (ca[c0 * 33] - cb[c0 * 33]);
                    if (c1 < n_cols) n1 = sgn * cs1 * (ca[c1 * 33] - cb[c1 * 33]);
                    if (track) {
                        if (c0 < n_cols) nsw[v * n_cols + c0] = (int16_t)n0;
                        if (c1 < n_cols) nsw[v * n_cols + c1] = (int16_t)n1;
                    }
                    if (FIX) part = (long long)n0 * f0 + (long long)n1 * f1;
                    else { pf += e0 * (float)n0; pf += e1 * (float)n1; }
                    for (int c = lane + 64; c < n_cols; c += 32) {
                        const int n = sgn * __ldg(wt.csign + c) * (ca[c * 33] - cb[c * 33]);
                        if (FIX) part += (long long)n * col_fix(c); else pf += (float)col_e(c) * (float)n;
                        if (track) nsw[v * n_cols + c] = (int16_t)n;
                    }
                    if (FIX) {
                        part = warp_sum_i64(part);
                        flags = win_decide_fix(jb, part, u, lnu, beta_f, scale_f, tol_near);
                    } else {
                        const double dE = (double)warp_sum(pf);
                        part = __double_as_longlong(dE);
                        flags = win_decide_f32(jb, dE, u, lnu, beta_f, tol_near);
                    }
                    if ((flags & 1) && !((pred >> v) & 1u)) touch(v, X.site[lane], false);
                    if (lane == 0) { X.part[v] = part; X.flags[v] = flags; }
                }
                for (int c = lane; c < n_cols; c += 32) { ca[c * 33] = 0; cb[c * 33] = 0; }
            }
        }
        __syncthreads();
        // 4. the window in step order (warp 0), and the next one listed.  A swap that went as predicted ends the window
        //    only at a later step that shares a site with it (once accepted); one that did not, at the first later step
        //    whose dE it moves.  (That step lies after the swap, so the least of these over all swaps of the window is
        //    the least over the decided ones.)
        //    Warp 0 only writes the accepted swaps and lists the next window; warp 1 keeps energies, samples and counts.
        if (warp < 2) {
            long long part = 0;
            int flags = 0, q = 32, first = 32;
            if (lane < nv) {
                flags = X.flags[lane]; q = step[lane];
                const int a = flags & 1, p = (pred >> lane) & 1;
                if (a) first = X.same[lane];
                if (a != p) first = min(first, X.nbr[lane]);
            }
            const int limit = min(n_w, (int)__reduce_min_sync(0xffffffffu, (unsigned)first));
            const bool mine = (flags & 1) && q < limit;
            const unsigned acc = __ballot_sync(0xffffffffu, mine);
            if (warp == 0) {
                // the two sites of each accepted swap, a lane a site
                if ((acc >> (lane >> 1)) & 1u) {
                    const int sa = X.spa[lane >> 1];
                    gsig[X.site[lane].w] = (int8_t)((lane & 1) ? sa : 1 - sa);
                }
                if (lane < nv && q >= limit) X.known[win_slot(s_w, q)] = (flags & 1) ? 1 : 2;
                const unsigned decided = __ballot_sync(0xffffffffu, lane < nv && q < limit);
                score = max(-64, min(64, score + 2 * __popc(acc) - __popc(decided)));
                s_cur = s_w + limit;
                __syncwarp();
                list_window();
            } else {
                if (lane < nv) part = X.part[lane];
                nnear += __popc(__ballot_sync(0xffffffffu, (flags & 2) && q < limit));
                nacc += __popc(acc);
                if (track)                                      // tracked sums: each changed row moves its column by +-2
                    for (unsigned m = acc; m; m &= m - 1)
                        for (int c = lane; c < n_cols; c += 32) dcv[c] += 2 * (int)nsw[(__ffs(m) - 1) * n_cols + c];
                const bool sample = si > 0 && left <= limit;
                long long pre = dsum; double Epre = E;          // energy after this lane's step (when sampled)
                if (FIX) {
                    long long run = mine ? part : 0;            // inclusive sum over the accepted swaps
#pragma unroll
                    for (int o = 1; o < kWinSwaps; o <<= 1) {
                        const long long y = __shfl_up_sync(0xffffffffu, run, o);
                        if (lane >= o) run += y;
                    }
                    if (mine) dmin = min(dmin, dsum + run);
                    if (sample)
                        for (unsigned m = acc; m; m &= m - 1) {
                            const int v = __ffs(m) - 1;
                            const long long y = __shfl_sync(0xffffffffu, run, v);
                            if (__shfl_sync(0xffffffffu, q, v) <= lane) pre = dsum + y;
                        }
                    dsum += __shfl_sync(0xffffffffu, run, kWinSwaps - 1);
                } else {
                    if (s_w == 0 && !(acc && __shfl_sync(0xffffffffu, q, __ffs(acc) - 1) == 0)) Emin = fmin(Emin, E);
                    for (unsigned m = acc; m; m &= m - 1) {
                        const int v = __ffs(m) - 1;
                        E += __longlong_as_double(__shfl_sync(0xffffffffu, part, v));
                        Emin = fmin(Emin, E);
                        if (__shfl_sync(0xffffffffu, q, v) <= lane) Epre = E;
                    }
                }
                if (sample && win_samples(left, si, lane, limit))
                    jb.E_samples[(int64_t)((s_w + lane + 1) / si - 1) * jb.R + t] = FIX ? E0 + (double)pre * fscale : Epre;
                if (si > 0) left = win_left(left, si, limit);
            }
        }
    }
    if (FIX)                                                    // warp 1: the minimum over its lanes
        for (int o = 16; o > 0; o >>= 1) dmin = min(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    if (track)
        for (int c = tid; c < n_cols; c += nt) jb.cv[(int64_t)r * n_cols + c] += dcv[c];
    __syncthreads();                                           // the replica's outputs are written before it is counted
    if (tid == 32) {
        if (FIX) { E = E0 + (double)dsum * fscale; if (T > 0) Emin = fmin(Emin, E0 + (double)dmin * fscale); }
        jb.E[r] = E; jb.E_min_rep[r] = Emin; jb.n_acc[r] += nacc;
        if (jb.n_near) jb.n_near[r] += nnear;
    }
    if (warp == 1 && jb.ex_sync) fused_chunk_end(jb, g0, lane);
}
