// The small levels of an instance on one CTA.  Included by learn.cu inside its namespaces.
//
// A level of a few hundred candidates costs the whole-GPU queue 20 to 50 us, nearly all of it
// round trips between SMs (claims, plans, hash slots, completion counters in L2).  Here one CTA
// holds the instance's level starts, its plan, its fingerprints and a hash set in shared memory and
// goes through the levels with block barriers: every unit's fingerprints, then every candidate's
// place in the set (one thread each), then the rows of the new ones written and the matches
// verified word by word.  Rows and parents go to global memory as everywhere, so the level
// kernel can take over at any level (local_handoff).  A level is taken only if its candidates
// could all be new and still fit: this CTA's tables, and the rows, cache and hash slots that the
// instance has in the level kernel, so that a search that passes one of those ends as it does there.
//
// A learn of 40 short traces to cost 3 took 168 us of which 43 on the device and the rest in launches,
// copies and waits; with its set-up and levels in this one kernel, one copy down and one back, 80.
//
// Exact keys and 64-bit fingerprints, fused block order, levels below 63.
constexpr int LT_ONE = 1024;    // threads when one instance has the GPU to itself
constexpr int LT_BATCH = 512;   // threads per instance of a batch, two CTAs an SM
constexpr int LROWS = LOCAL_ROWS;  // rows the CTA can hold fingerprints of
constexpr int LTAB = 16384;     // hash slots (row + 1, or LCAND | candidate of the current round)
constexpr u32 LCAND = 0x8000u;
constexpr int LC = 1024;        // candidates per round (256 units of 4)
constexpr int LPITCH = 1024;    // words per row at most
constexpr int LCOST = 62;       // last level
static_assert(LCOST + 3 <= LOCAL_COSTS, "level arrays");
constexpr int LSEGS = 4 + 3 * 32;

// Consecutive units of a level: rows [r0, r0 + nr) under unary operators, or pairs of left rows
// [l0, l0 + nl) and right rows [r0, r0 + nr), right rows fastest.
struct LocalSeg {
    int mode, op;        // M_UNARY or M_ALL; the candidates that exist (bit t): operator slots, or & | lUr rUl
    int l0, nl, r0, nr;
    int upos[4];         // block position of each
    int unit0;           // its first unit in the level
};

struct Local {
    InstArgs A;
    u64 fp[LROWS];
    u64 sum[LC];               // fingerprints of the round's candidates
    u64 meta[LPITCH];
    unsigned short tab[LTAB];
    u32 at[LC];                // a claim's row; a match's row, or LMATCH | candidate
    unsigned short idx[LC];    // slot a candidate stands at
    unsigned char fail[LC];    // F_* bits, then 1: differs from its match
    unsigned short claim[LC], verify[LC], retry[2][LC];
    unsigned short ul[LC / 4], ur[LC / 4];  // the round's units: operand rows,
    unsigned char useg[LC / 4];             // segment,
    unsigned char uops[LC / 4];             // candidates (operators) to evaluate
    u32 nclaim, nverify, nretry[2];
    LocalSeg seg[LSEGS];
    int ls[LCOST + 3];
    u64 lc[LCOST + 3];         // candidates of the levels done
    int nseg, units;
    u32 nrows;
    u64 cand;
    u64 found_key;             // smallest block position << 32 | candidate of the level
    u64 found_parent;
    u64 evaluated;
    u32 skipped;               // candidates of the level behind its find
    int ok;
    u32 every, some;           // batches: letters that hold first in every positive / some negative
};
constexpr u32 LMATCH = 0x80000000u;
enum : u32 { F_FAIL = 1u, F_DEAD = 2u };

// ---- plan: the level's segments, in the order of the whole-GPU plan (unary first).  Warp 0.
__device__ void local_plan(Local &S, int c, int lane) {
    const InstArgs &A = S.A;
    const int c1 = A.cf[0];
    auto lo = [&](int k) { return k >= c1 && k < c ? S.ls[k] : 0; };
    auto hi = [&](int k) { return k >= c1 && k < c ? S.ls[k + 1] : 0; };
    const int uop = unary_slot_op(lane & 3), uk = c - A.cf[uop + 1];
    bool uex = lane < 4 && hi(uk) > lo(uk);
    if (uop == OP_NEG && !(A.neg_type == 1 || (A.neg_type == 2 && uk == c1))) uex = false;
    const u32 um = __ballot_sync(FULL, uex) & 15u;
    const bool fuse2 = A.cf[OP_AND + 1] == A.cf[OP_OR + 1], fuse3 = fuse2 && A.cf[OP_AND + 1] == A.cf[OP_U + 1];
    // splits of operator op: lane i - c1 is split (i, c - i - cop)
    auto splits = [&](int op) {
        const int i = c1 + lane, j = c - i - A.cf[op + 1];
        return __ballot_sync(FULL, 2 * i <= c - A.cf[op + 1] && hi(i) > lo(i) && hi(j) > lo(j));
    };
    const u32 ma = splits(OP_AND), mo = splits(OP_OR), mu = splits(OP_U);
    int upos[4] = {POS_NONE, POS_NONE, POS_NONE, POS_NONE}, pos = 0;
    if (um & 1u) upos[0] = pos++;
    const int pos_and = pos, pos_or = pos_and + __popc(ma);
    pos = pos_or + __popc(mo);
    for (int j = 1; j < 4; ++j)
        if ((um >> j) & 1u) upos[j] = pos++;
    const int pos_u = pos;
    // unary segments: one per source range
    int nu = 0;
    {
        const int k0 = __shfl_sync(FULL, uk, 0), k1 = __shfl_sync(FULL, uk, 1), k2 = __shfl_sync(FULL, uk, 2),
                  k3 = __shfl_sync(FULL, uk, 3);
        const int k[4] = {k0, k1, k2, k3};
        for (int j = 0; j < 4; ++j) {
            if (!((um >> j) & 1u)) continue;
            bool seen = false;
            for (int q = 0; q < j; ++q) seen |= ((um >> q) & 1u) && k[q] == k[j];
            if (seen) continue;
            if (lane == 0) {
                LocalSeg &g = S.seg[nu];
                g.mode = M_UNARY;
                g.op = 0;
                for (int q = 0; q < 4; ++q) {
                    const bool in = ((um >> q) & 1u) && k[q] == k[j];
                    g.op |= in ? 1 << q : 0;
                    g.upos[q] = in ? upos[q] : POS_NONE;
                }
                g.l0 = 0;
                g.nl = 1;
                g.r0 = lo(k[j]);
                g.nr = hi(k[j]) - lo(k[j]);
            }
            ++nu;
        }
    }
    int nseg = nu;
    auto binary = [&](int op, int mask, u32 m, int first) {
        const int i = c1 + lane, j = c - i - A.cf[op + 1];
        if ((m >> lane) & 1u) {
            const int rank = __popc(m & ((1u << lane) - 1u));
            LocalSeg &g = S.seg[nseg + rank];
            g.mode = M_ALL;
            g.op = mask;
            g.l0 = lo(i);
            g.nl = hi(i) - lo(i);
            g.r0 = lo(j);
            g.nr = hi(j) - lo(j);
            const bool fused = (mask & 3) == 3;
            g.upos[0] = first + rank;
            g.upos[1] = fused ? pos_or + rank : first + rank;
            g.upos[2] = g.upos[3] = fused ? pos_u + rank : first + rank;
        }
        nseg += __popc(m);
    };
    if (fuse3) {
        binary(OP_AND, 15, ma, pos_and);
    } else {
        if (fuse2) {
            binary(OP_AND, 3, ma, pos_and);
        } else {
            binary(OP_AND, 1, ma, pos_and);
            binary(OP_OR, 2, mo, pos_or);
        }
        binary(OP_U, 12, mu, pos_u);
    }
    __syncwarp();
    int units = 0;
    u64 cand = 0;
    for (int base = 0; base < nseg; base += 32) {
        const int q = base + lane;
        u64 n = 0, m = 0;  // units can pass 32 bits before the level is refused
        if (q < nseg) {
            const LocalSeg &g = S.seg[q];
            n = (u64)g.nl * (u64)g.nr;
            m = n * (u64)__popc((unsigned)g.op);
        }
        u64 incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        if (q < nseg) S.seg[q].unit0 = (int)min((u64)INT_MAX, (u64)units + incl - n);
        units = (int)min((u64)INT_MAX, (u64)units + __shfl_sync(FULL, incl, 31));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(FULL, m, o);
        cand += m;
    }
    if (lane == 0) {
        S.nseg = nseg;
        S.units = units;
        S.cand = cand;
    }
    __syncwarp();
}

// A unit's operands: unit `u` of the round, decoded into shared memory by one thread each.
struct LocalUnit {
    const LocalSeg *g;
    int l, r;
};
__device__ __forceinline__ void local_decode(Local &S, int u, int unit) {
    int lo = 0, hi = S.nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (S.seg[mid].unit0 <= unit)
            lo = mid;
        else
            hi = mid - 1;
    }
    const LocalSeg &g = S.seg[lo];
    const u32 q = (u32)(unit - g.unit0), l = g.mode == M_UNARY ? 0u : q / (u32)g.nr;
    S.ul[u] = (unsigned short)(g.l0 + (int)l);
    S.ur[u] = (unsigned short)(g.r0 + (int)(q - l * (u32)g.nr));
    S.useg[u] = (unsigned char)lo;
    // once a round has found and the search ends here, only the operators whose blocks come before the find
    u32 ops = (u32)g.op;
    if (S.A.stop_at_found && S.found_key != ~0ull) {
        for (int t = 0; t < 4; ++t)
            if (g.upos[t] >= (int)(S.found_key >> 32)) ops &= ~(1u << t);
        if (ops != (u32)g.op) atomicAdd(&S.skipped, (u32)__popc((u32)g.op & ~ops));
    }
    S.uops[u] = (unsigned char)ops;
}
__device__ __forceinline__ LocalUnit local_unit(const Local &S, int u) {
    return LocalUnit{&S.seg[S.useg[u]], (int)S.ul[u], (int)S.ur[u]};
}
__device__ __forceinline__ int local_wop(const LocalSeg &g, int t) {
    return g.mode == M_UNARY ? unary_slot_op(t) : mode_swapped(M_ALL, t) ? (int)W_URL : mode_op(M_ALL, t, 0);
}
__device__ __forceinline__ u64 local_parent(const LocalUnit &x, int t) {
    if (x.g->mode == M_UNARY) return pack_parent(unary_slot_op(t), (u64)x.r, 0);
    return mode_swapped(M_ALL, t) ? pack_parent(OP_U, (u64)x.r, (u64)x.l)
                                  : pack_parent(mode_op(M_ALL, t, 0), (u64)x.l, (u64)x.r);
}
// What a candidate is made of: its operand rows (unary: right only) and its operator (W_URL, or a code).
// & | U are one formula on a = l | r under word masks: a & ((y & (l | n)) | (~(a + y) & u) | o), y the
// operand U reaches (r, or l for r U l), so that one loop without branches serves them.
struct LocalCand {
    const ulonglong2 *l, *r;
    u64 n, u, o;
    int wop;
    bool un, rl;
    __device__ __forceinline__ u64 pair(u64 x, u64 z) const {
        const u64 a = x | z, y = rl ? x : z;
        return a & ((y & (x | n)) | (~(a + y) & u) | o);
    }
    __device__ __forceinline__ u64 word(u64 x, u64 z, u64 m) const { return un ? row_unary(wop, z, m & LENMASK) : pair(x, z); }
};
__device__ __forceinline__ LocalCand local_form(bool un, int wop) {  // without its rows
    LocalCand k;
    k.l = k.r = nullptr;
    k.wop = wop;
    k.un = un;
    k.rl = wop == W_URL;
    k.n = wop == OP_AND ? 0ull : ~0ull;
    k.u = wop == OP_U || wop == W_URL ? ~0ull : 0ull;
    k.o = wop == OP_OR ? ~0ull : 0ull;
    return k;
}
__device__ __forceinline__ LocalCand local_cand(const Local &S, const LocalUnit &x, int t) {
    const u64 pitch = (u64)S.A.pitch;
    LocalCand k = local_form(x.g->mode == M_UNARY, local_wop(*x.g, t));
    k.l = reinterpret_cast<const ulonglong2 *>(S.A.cache + (u64)x.l * pitch);
    k.r = reinterpret_cast<const ulonglong2 *>(S.A.cache + (u64)x.r * pitch);
    return k;
}
// f(c, words of chunk c) over chunks c = gl, gl + P, ...  One chunk at a time: two or four in flight spill
// (64 registers) and made a level of 732 candidates take 34 instead of 24 us.
template <class F>
__device__ __forceinline__ void local_words(const Local &S, const LocalCand &k, int gl, int P, int nch, F f) {
#pragma unroll 1
    for (int c = gl; c < nch; c += P) {
        const ulonglong2 r = k.r[c], l = k.un ? r : k.l[c];
        f(c, k.word(l.x, r.x, S.meta[2 * c]), k.word(l.y, r.y, S.meta[2 * c + 1]));
    }
}

// Sums and acceptance of one unit over this lane's chunks (first lane gl of P lanes).
template <int MODE, int HK>
__device__ __forceinline__ void local_eval(const Local &S, const LocalUnit &x, int gl, int P, u64 (&h)[4], u32 (&fails)[4]) {
    const int nch = S.A.pitch >> 1, npos = S.A.npos, n = S.A.n, opmask = x.g->op;
    const u64 pitch = (u64)S.A.pitch;
    const ulonglong2 *R = reinterpret_cast<const ulonglong2 *>(S.A.cache + (u64)x.r * pitch);
    const ulonglong2 *L = reinterpret_cast<const ulonglong2 *>(S.A.cache + (u64)x.l * pitch);
#pragma unroll 1
    for (int c = gl; c < nch; c += P) {
        const ulonglong2 rv = R[c];
        const u64 k = (2ull * (u64)c + 1ull) * WEYL;
        const u32 p0 = 2 * c < npos ? ROW_BIT0_HI : 0u, p1 = 2 * c + 1 < npos ? ROW_BIT0_HI : 0u;
        const bool v0 = 2 * c < n, v1 = 2 * c + 1 < n;
        auto take = [&](int t, u64 w0, u64 w1) {
            h[t] += hw<HK>(w0, k, v0) + hw<HK>(w1, k + WEYL, v1);
            fails[t] |= fails2(w0, w1, p0, p1);
        };
        if constexpr (MODE == M_UNARY) {
            const u64 m0 = S.meta[2 * c] & LENMASK, m1 = S.meta[2 * c + 1] & LENMASK;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if ((opmask >> t) & 1) take(t, row_unary(unary_slot_op(t), rv.x, m0), row_unary(unary_slot_op(t), rv.y, m1));
        } else {
            pair_words<MODE>(L[c], rv, 0, 15u, take);
        }
    }
}

// Candidate j of the round into the set, from slot `idx` on.
__device__ __forceinline__ void local_probe(Local &S, int j, u32 idx) {
    const u64 fp = S.sum[j];
    const bool exact = S.A.key_mode == KEY_EXACT;
    for (;; idx = (idx + 1) & (LTAB - 1)) {
        u32 v = *(volatile unsigned short *)&S.tab[idx];
        if (v == 0u) {
            v = atomicCAS(&S.tab[idx], (unsigned short)0, (unsigned short)(LCAND | (u32)j));
            if (v == 0u) {
                const u32 row = atomicAdd(&S.nrows, 1u);
                S.fp[row] = fp;
                S.at[j] = row;
                S.idx[j] = (unsigned short)idx;
                S.claim[atomicAdd(&S.nclaim, 1u)] = (unsigned short)j;
                return;
            }
        }
        const bool cand = (v & LCAND) != 0u;
        const u32 o = cand ? v & (LCAND - 1u) : v - 1u;
        if ((cand ? S.sum[o] : S.fp[o]) != fp) continue;
        if (exact) {
            S.at[j] = cand ? LMATCH | o : o;
            S.idx[j] = (unsigned short)idx;
            S.fail[j] = 0;
            S.verify[atomicAdd(&S.nverify, 1u)] = (unsigned short)j;
        }
        return;
    }
}

// Its place in the reference's order, as the level kernel's A.prio has it: block position << 40 | the reference's
// thread index (U: l U r before r U l).
__device__ __forceinline__ u64 local_prio(const LocalUnit &x, int t) {
    const LocalSeg &g = *x.g;
    const u64 pair = g.mode == M_UNARY ? (u64)(x.r - g.r0) : (u64)(x.l - g.l0) * (u64)g.nr + (u64)(x.r - g.r0);
    const bool until = g.mode != M_UNARY && mode_op(M_ALL, t, 0) == OP_U;
    return ((u64)(u32)g.upos[t] << 40) | (until ? 2 * pair + (mode_swapped(M_ALL, t) ? 1u : 0u) : pair);
}
// The row that candidate j of the round stands for: its own, or the one it matches.
__device__ __forceinline__ int local_row(const Local &S, int j) {
    const u32 at = S.at[j];
    return (int)(at & LMATCH ? S.at[at & ~LMATCH] : at);
}

// One level, already planned, by the whole CTA.  Returns with the level's rows stored, nrows and
// the find updated.  TIES: the reference's keys, kept out of the other learns' code (40 traces: 1.8% longer with it).
template <int HK, int LT, bool TIES>
__device__ void local_level(Local &S, int c, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    const InstArgs &A = S.A;
    const int nch = A.pitch >> 1;
    // lanes per unit: few, so that many units' round trips overlap
    const int P = nch <= 32 ? 8 : nch <= 64 ? 16 : 32;
    const int gl = lane & (P - 1), per_warp = 32 / P, group = tid / P, ngroups = LT / P;
    for (int u0 = 0; u0 < S.units; u0 += LC / 4) {
        const int nu = min(LC / 4, S.units - u0);
        if (tid < nu) local_decode(S, tid, u0 + tid);
        __syncthreads();
        // fingerprints and acceptance
        for (int b = warp * per_warp; b < nu; b += (LT / 32) * per_warp) {
            const int u = b + lane / P;
            u64 h[4] = {0, 0, 0, 0};
            u32 fails[4] = {0, 0, 0, 0}, valid = 0;
            if (u < nu && S.uops[u]) {
                const LocalUnit x = local_unit(S, u);
                valid = S.uops[u];
                if (x.g->mode == M_UNARY)
                    local_eval<M_UNARY, HK>(S, x, gl, P, h, fails);
                else
                    local_eval<M_ALL, HK>(S, x, gl, P, h, fails);
            }
            __syncwarp();
            u32 fb = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) fb |= (fails[t] & ROW_BIT0_HI) ? 1u << t : 0u;
            for (int o = P >> 1; o > 0; o >>= 1) fb |= __shfl_xor_sync(FULL, fb, o);
            // reduce-scatter of the four sums over the P lanes: lane gl ends with candidate 4 gl / P
            const int o1 = P >> 1, o2 = P >> 2;
            const bool up1 = (gl & o1) != 0, up2 = (gl & o2) != 0;
            const u64 a = (up1 ? h[2] : h[0]) + __shfl_xor_sync(FULL, up1 ? h[0] : h[2], o1);
            const u64 d = (up1 ? h[3] : h[1]) + __shfl_xor_sync(FULL, up1 ? h[1] : h[3], o1);
            u64 sum = (up2 ? d : a) + __shfl_xor_sync(FULL, up2 ? a : d, o2);
            for (int o = P >> 3; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
            if (u < nu && (gl & (o2 - 1)) == 0) {
                const int t = gl / o2, j = 4 * u + t;
                S.sum[j] = fmix64(sum);
                S.fail[j] = (unsigned char)(((valid >> t) & 1u) ? (fb >> t) & 1u : F_DEAD);
            }
        }
        __syncthreads();
        // acceptance, the find, the hash set
        u64 mine[LC / LT];
#pragma unroll
        for (int q = 0; q < LC / LT; ++q) {
            const int j = tid + q * LT;
            mine[q] = ~0ull;
            if (j >= 4 * nu) continue;
            const u32 f = S.fail[j];
            if (f & F_DEAD) continue;
            if (!f) {
                const LocalUnit x = local_unit(S, j >> 2);
                mine[q] = ((u64)(u32)x.g->upos[j & 3] << 32) | (u32)(4 * u0 + j);
                atomicMin(&S.found_key, mine[q]);
                if (A.stop_at_found) continue;  // the last level: no dedupe
            }
            local_probe(S, j, (u32)S.sum[j] & (LTAB - 1));
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < LC / LT; ++q)
            if (mine[q] != ~0ull && mine[q] == S.found_key)
                S.found_parent = local_parent(local_unit(S, (tid + q * LT) >> 2), tid & 3);
        // new rows written, matches compared; a match that differs goes on along the set
        for (int p = 0;; p ^= 1) {
            const int nc = (int)S.nclaim, n = nc + (int)S.nverify;
            for (int i = group; i < n; i += ngroups) {
                const bool write = i < nc;
                const int j = write ? S.claim[i] : S.verify[i - nc];
                const LocalUnit x = local_unit(S, j >> 2);
                const LocalCand k = local_cand(S, x, j & 3);
                const u32 at = S.at[j];
                if (write) {
                    ulonglong2 *row = reinterpret_cast<ulonglong2 *>(A.cache + (u64)at * (u64)A.pitch);
                    u32 pm = 0, nh = 0;
                    local_words(S, k, gl, P, nch, [&](int q, u64 x0, u64 x1) {
                        row[q] = make_ulonglong2(x0, x1);
                        if (A.lstats) {
                            const u32 p0 = 2 * q < A.npos ? ROW_BIT0_HI : 0u, p1 = 2 * q + 1 < A.npos ? ROW_BIT0_HI : 0u;
                            pm |= pmiss2(x0, x1, p0, p1);
                            nh |= nhit2(x0, x1, p0, p1);
                        }
                    });
                    if (A.lstats) {  // a learn that counts row statistics: one vote per group
                        const u32 gm = P == 32 ? FULL : ((1u << P) - 1u) << (lane & ~(P - 1));
                        const bool anyp = __any_sync(gm, pm), anyn = __any_sync(gm, nh);
                        if (gl == 0) {
                            if (!anyp) atomicAdd(A.lstats + (u64)c * LSTATS, 1ull);
                            if (!anyn) atomicAdd(A.lstats + (u64)c * LSTATS + 1, 1ull);
                        }
                    }
                    if (gl == 0) {
                        S.tab[S.idx[j]] = (unsigned short)(at + 1u);
                        A.parents[at] = local_parent(x, j & 3);
                        if (TIES) A.prio[at] = local_prio(x, j & 3) << 1;
                        if (A.keys) {
                            A.keys[2 * (u64)at] = S.sum[j];
                            A.keys[2 * (u64)at + 1] = 0;
                        }
                    }
                } else {
                    u64 diff = 0;
                    if (at & LMATCH) {  // a claim of this round: compared as it is made
                        const int o = (int)(at & ~LMATCH);
                        const LocalCand m = local_cand(S, local_unit(S, o >> 2), o & 3);
#pragma unroll 1
                        for (int q = gl; q < nch; q += P) {
                            const ulonglong2 r = k.r[q], l = k.un ? r : k.l[q], z = m.r[q], y = m.un ? z : m.l[q];
                            diff |= k.word(l.x, r.x, S.meta[2 * q]) ^ m.word(y.x, z.x, S.meta[2 * q]);
                            diff |= k.word(l.y, r.y, S.meta[2 * q + 1]) ^ m.word(y.y, z.y, S.meta[2 * q + 1]);
                        }
                    } else {
                        const ulonglong2 *row = reinterpret_cast<const ulonglong2 *>(A.cache + (u64)at * (u64)A.pitch);
                        local_words(S, k, gl, P, nch, [&](int q, u64 x0, u64 x1) {
                            const ulonglong2 b = row[q];
                            diff |= (x0 ^ b.x) | (x1 ^ b.y);
                        });
                    }
                    if (diff) S.fail[j] = 1;
                }
            }
            __syncthreads();
            for (int i = tid; i < n - nc; i += LT) {
                const int j = S.verify[i];
                if (S.fail[j])
                    S.retry[p][atomicAdd(&S.nretry[p], 1u)] = (unsigned short)j;
                else if (TIES && local_row(S, j) >= S.ls[c])
                    atomicMin(A.prio + local_row(S, j), local_prio(local_unit(S, j >> 2), j & 3) << 1);
            }
            __syncthreads();
            if (TIES)  // of the candidates in one row of the level, the first in the reference's order gives its parents
                for (int i = tid; i < n - nc; i += LT) {
                    const int j = S.verify[i], row = local_row(S, j);
                    const LocalUnit x = local_unit(S, j >> 2);
                    if (!S.fail[j] && row >= S.ls[c] && ld_volatile(A.prio + row) == local_prio(x, j & 3) << 1)
                        A.parents[row] = local_parent(x, j & 3);
                }
            const int nr = (int)S.nretry[p];
            if (tid == 0) {
                S.nclaim = 0;
                S.nverify = 0;
                S.nretry[p ^ 1] = 0;
            }
            __syncthreads();
            if (nr == 0) break;
            for (int i = tid; i < nr; i += LT) {
                const int j = S.retry[p][i];
                local_probe(S, j, (S.idx[j] + 1u) & (LTAB - 1));
            }
            __syncthreads();
        }
    }
}

// ---- set-up of an instance: letters and word metadata from its step masks, the level arrays and
// the control block.  Any number of threads (tid of nt) over any number of CTAs.
__device__ void init_traces(const InstArgs &A, const StartIn &in, u64 *meta, int tid, int nt) {
    if (in.width == 1)
        init_traces_of<unsigned char>(A, in, meta, tid, nt);
    else if (in.width == 2)
        init_traces_of<unsigned short>(A, in, meta, tid, nt);
    else
        init_traces_of<u32>(A, in, meta, tid, nt);
}
__device__ void init_state(const InstArgs &A, int tid, int nt) {
    for (int k = tid; k < A.max_cost + 3; k += nt) {
        A.ls[k] = 0;
        A.level_cands[k] = 0;
        if (A.lstats)
            for (int q = 0; q < LSTATS; ++q) A.lstats[(u64)k * LSTATS + q] = 0;
        if (A.level_ns)
            for (int q = 0; q < LEVEL_TRACE; ++q) A.level_ns[(u64)k * LEVEL_TRACE + q] = 0;
    }
    if (tid == 0) {
        InstCtl c{};
        c.row_count = (u64)A.nalpha;
        c.found_key = NO_FIND;
        c.plan.cost = A.cf[0];
        c.t_start = globaltimer();
        *A.ctl = c;
    }
}
__global__ void init_kernel(const InstArgs *__restrict__ args, const StartIn *__restrict__ in) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    init_traces(*args, *in, nullptr, tid, nt);
    init_state(*args, tid, nt);
}

// The letters into the CTA's hash set, in letter order (a duplicate letter stays a row, the set keeps
// the first).  The rows are in place.
template <int HK, int LT>
__device__ void local_letters(Local &S, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    const InstArgs &A = S.A;
    const int nch = A.pitch >> 1, nalpha = A.nalpha;
    for (int j = warp; j < nalpha; j += LT / 32) {
        const ulonglong2 *row = reinterpret_cast<const ulonglong2 *>(A.cache + (u64)j * (u64)A.pitch);
        u64 h[1] = {0};
        u32 pm = 0, nh = 0;
        for (int c = lane; c < nch; c += 32) {
            const u64 k = (2ull * (u64)c + 1ull) * WEYL;
            const ulonglong2 w = row[c];
            h[0] += hw<HK>(w.x, k, 2 * c < A.n) + hw<HK>(w.y, k + WEYL, 2 * c + 1 < A.n);
            const u32 p0 = 2 * c < A.npos ? ROW_BIT0_HI : 0u, p1 = 2 * c + 1 < A.npos ? ROW_BIT0_HI : 0u;
            pm |= pmiss2(w.x, w.y, p0, p1);
            nh |= nhit2(w.x, w.y, p0, p1);
        }
        const u64 fp = fmix64(reduce_to_lane<1>(h, lane));
        if (A.lstats) count_stats(A.lstats + (u64)A.cf[0] * LSTATS, !__any_sync(FULL, pm), !__any_sync(FULL, nh), lane);
        if (lane == 0) {
            S.fp[j] = fp;
            A.parents[j] = pack_parent(OP_ATOM, 0, 0);
            if (A.keys) {
                A.keys[2 * j] = fp;
                A.keys[2 * j + 1] = 0;
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
        for (int j = 0; j < nalpha; ++j) {
            const u64 fp = S.fp[j];
            for (u32 idx = (u32)fp & (LTAB - 1);; idx = (idx + 1) & (LTAB - 1)) {
                const u32 v = S.tab[idx];
                if (v == 0u) {
                    __syncwarp();
                    if (lane == 0) S.tab[idx] = (unsigned short)(j + 1);
                    break;
                }
                const u32 o = v - 1u;
                if (S.fp[o] != fp) continue;
                bool diff = false;
                if (A.key_mode == KEY_EXACT) {
                    const u64 *a = A.cache + (u64)j * (u64)A.pitch, *b = A.cache + (u64)o * (u64)A.pitch;
                    for (int i = lane; i < A.pitch; i += 32) diff |= a[i] != b[i];
                }
                if (!__any_sync(FULL, diff)) break;
            }
            __syncwarp();
        }
    }
    __syncthreads();
}

// Starts S for an instance whose arguments are in S.A (all threads): an empty set, the letters.
template <int HK, int LT>
__device__ void local_begin(Local &S, int tid) {
    for (int i = tid; i < LTAB / 2; i += LT) reinterpret_cast<u32 *>(S.tab)[i] = 0u;
    for (int k = tid; k < LCOST + 3; k += LT) S.ls[k] = k > S.A.cf[0] ? S.A.nalpha : 0;
    if (tid == 0) {
        S.nclaim = S.nverify = S.nretry[0] = S.nretry[1] = 0;
        S.nrows = (u32)S.A.nalpha;
        S.evaluated = 0;
        S.found_key = ~0ull;
        S.found_parent = 0;
    }
    __syncthreads();
    local_letters<HK, LT>(S, tid);
}

// The levels the CTA takes, from the first one on; `limit` bounds the work of a level (units x
// 32-chunk steps + 1).  On return the control block and the level arrays stand as before the closing
// of the last complete level (plan.cost), which close_level does; returns true when that will end
// the search, false when the next level is for the level kernel.
template <int HK, int LT, bool TIES>
__device__ bool local_run(Local &S, long long limit, int tid) {
    const InstArgs &A = S.A;
    InstCtl *C = A.ctl;
    const int lane = tid & 31, c1 = A.cf[0];
    const int its = (A.pitch + 63) >> 6;
    int c = c1 + 1, ne = 0;
    u64 found = 0;
    int found_cost = 0;
    bool over = false;
    // rows that fit this CTA and that the instance may have: its row limit, its hash set's slots
    const u64 room = min((u64)min((long long)LROWS, A.cap_rows), A.slot_mask + 1u);
    if (tid == 0 && A.level_ns) A.level_ns[(u64)c1 * LEVEL_TRACE + LT_END] = globaltimer();
    for (;; ++c) {
        // level c - 1 is complete
        if (c > A.max_cost || (found && A.stop_at_found)) {
            over = true;
            break;
        }
        if (c > LCOST) break;
        if (tid < 32) {
            local_plan(S, c, lane);
            if (lane == 0) {
                S.found_key = ~0ull;
                S.skipped = 0;
                S.ok = (long long)S.units * (its + 1) <= limit &&
                       (u64)S.nrows + S.cand <= room && !(A.cancel && *A.cancel);
                if (S.ok && A.level_ns && S.units) {
                    const u64 t = globaltimer();
                    u64 *ns = A.level_ns + (u64)c * LEVEL_TRACE;
                    ns[LT_PUBLISHED] = ns[LT_CLAIMED] = ns[LT_STARTED] = t;
                }
            }
        }
        __syncthreads();
        if (!S.ok) break;
        if (tid == 0) {  // close level c - 1
            A.ls[c] = S.ls[c];
            if (S.ls[c] > S.ls[c - 1]) A.ne[ne] = c - 1;
        }
        if (S.ls[c] > S.ls[c - 1]) ++ne;
        if (S.units) local_level<HK, LT, TIES>(S, c, tid);
        __syncthreads();
        if (S.found_key != ~0ull && !found) {
            found = (1ull << 63) | S.found_parent;
            found_cost = c;
            if (tid == 0) C->found_key = ((u64)(u32)c << 32) | (u32)(S.found_key >> 32);
        }
        for (int k = c + 1 + tid; k < LCOST + 3; k += LT) S.ls[k] = (int)S.nrows;
        if (tid == 0) {
            A.level_cands[c] = S.lc[c] = S.cand;
            S.evaluated += S.cand - S.skipped;
            if (A.level_ns) A.level_ns[(u64)c * LEVEL_TRACE + LT_END] = globaltimer();
        }
        __syncthreads();
    }
    if (tid == 0) {
        C->plan.cost = c - 1;
        C->row_count = (u64)S.nrows;
        C->evaluated = S.evaluated;
        C->ne_count = (u32)ne;
        C->found = found;
        C->found_cost = (u32)found_cost;
        C->last_cost = (u32)max(c1, c - 2);
    }
    __syncthreads();
    return over;
}

// The CTA's set into the instance's hash set in HBM.
template <int LT>
__device__ void local_handoff(Local &S, int tid) {
    const InstArgs &A = S.A;
    for (int i = tid; i < LTAB; i += LT) {
        const u32 v = S.tab[i];
        if (!v) continue;
        const u64 fp = S.fp[v - 1u], want = ((fp >> 40) << 40) | ((u64)A.gen << 32) | (u64)v;
        u64 idx = fp & A.slot_mask;
        for (u64 probes = 0;; idx = (idx + 1) & A.slot_mask) {
            u64 o = atomicCAS(A.slots + idx, 0ull, want);
            while (o != 0ull && slot_free(o, A.gen)) {
                const u64 w = atomicCAS(A.slots + idx, o, want);
                if (w == o) {
                    o = 0ull;
                    break;
                }
                o = w;
            }
            if (o == 0ull) break;
            if (++probes > A.slot_mask) {
                atomicOr(&A.ctl->status, ST_TABLE);
                break;
            }
        }
    }
}

// One instance from its traces: set-up, the small levels, and the plan of the first level that is
// left to the level kernel (or the end of the search).
template <int HK, bool TIES>
__global__ void __launch_bounds__(LT_ONE, 1)
    start_kernel(const InstArgs *__restrict__ args, const StartIn *__restrict__ in, long long limit) {
    constexpr int LT = LT_ONE;
    extern __shared__ __align__(128) unsigned char smem[];
    Local &S = *reinterpret_cast<Local *>(smem);
    const int tid = threadIdx.x;
    for (int w = tid; w < (int)(sizeof(InstArgs) / 8); w += LT)
        reinterpret_cast<u64 *>(&S.A)[w] = reinterpret_cast<const u64 *>(args)[w];
    __syncthreads();
    init_traces(S.A, *in, S.meta, tid, LT);
    init_state(S.A, tid, LT);
    __syncthreads();
    local_begin<HK, LT>(S, tid);
    if (!local_run<HK, LT, TIES>(S, limit, tid)) local_handoff<LT>(S, tid);
    __threadfence();
    __syncthreads();
    if (tid < 32) close_level(S.A, S.A.ctl, true, tid);
}

// The result of an instance whose search ended in local_run, as finish_instance gives it.  Warp 0;
// S still has the plan of the last level.
__device__ void local_result(const Local &S, BatchOut &o, u64 t0, int letter, int lane) {
    const InstArgs &A = S.A;
    const InstCtl *C = A.ctl;
    const int c1 = A.cf[0], last = C->plan.cost;
    const u64 found = C->found, key = C->found_key;
    const int found_cost = (int)C->found_cost;
    const bool stop_found = found && A.stop_at_found;
    u64 all = lane == 0 ? (u64)A.nalpha : 0ull;
    const int top = stop_found ? found_cost - 1 : last;
    for (int c = c1 + 1 + lane; c <= top; c += 32) all += S.lc[c];
    if (stop_found) {  // the blocks of the level of the find up to the one that holds it
        const int fpos = (int)(u32)key;
        for (int q = lane; q < S.nseg; q += 32) {
            const LocalSeg &g = S.seg[q];
            const u64 n = (u64)g.nl * (u64)g.nr;
            for (int t = 0; t < 4; ++t)
                if (((g.op >> t) & 1) && g.upos[t] <= fpos) all += n;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) all += __shfl_xor_sync(FULL, all, d);
    if (lane != 0) return;
    o.status = found || letter >= 0 ? LTLG_FOUND : LTLG_NOT_FOUND;
    o.cost = letter >= 0 ? c1 : found ? found_cost : max(c1, last);
    o.all_ltls = all;
    o.evaluated = (u64)A.nalpha + S.evaluated;
    o.rows = (long long)S.nrows;
    o.found = letter >= 0 ? 0ull : found;
    o.letter = letter;
    o.device_flags = 0;
    int count = 0, over = 0;
    if (found && letter < 0) {
        u64 *e = o.walk;
        e[0] = ~0ull;
        e[1] = found & ~(1ull << 63);
        count = 1;
        for (int head = 0; head < count && !over; ++head) {
            const u64 p = e[2 * head + 1];
            const int op = parent_op(p);
            const u64 kids[2] = {parent_left(p), parent_right(p)};
            const int nk = (op == OP_AND || op == OP_OR || op == OP_U) ? 2 : (op == OP_ATOM ? 0 : 1);
            for (int q = 0; q < nk; ++q) {
                if (kids[q] < (u64)A.nalpha) continue;
                if (count >= WALK_MAX) {
                    over = 1;
                    break;
                }
                e[2 * count] = kids[q];
                e[2 * count + 1] = A.parents[kids[q]];
                ++count;
            }
        }
    }
    o.walk_count = count;
    o.walk_overflow = over;
    o.ns = globaltimer() - t0;
}

// A batch's instances one per CTA, taken from a counter: those whose search ends on the small levels get
// their results here, the others go on the pending list, which the level kernel's slots take from (they
// start again from the letters: what is done twice is small next to what is left).  args: per CTA
// (its own rows, parents and level arrays).
template <int HK>
__global__ void __launch_bounds__(LT_BATCH, 2)
    batch_local_kernel(BatchDev *__restrict__ B, const InstArgs *__restrict__ args, long long words, long long limit) {
    constexpr int LT = LT_BATCH;
    extern __shared__ __align__(128) unsigned char smem[];
    Local &S = *reinterpret_cast<Local *>(smem);
    const int tid = threadIdx.x, lane = tid & 31;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            S.ok = (int)atomicAdd(&B->next_local, 1ull);
            S.every = ~0u;
            S.some = 0u;
        }
        for (int w = tid; w < (int)(sizeof(InstArgs) / 8); w += LT)
            reinterpret_cast<u64 *>(&S.A)[w] = reinterpret_cast<const u64 *>(args + blockIdx.x)[w];
        __syncthreads();
        const int idx = S.ok;
        if (idx >= B->count) return;
        const u64 t0 = globaltimer();
        const BatchIn &bi = B->in[idx];
        const int npos = bi.npos, n = npos + bi.nneg, nalpha = bi.nalpha;
        const int pitch = n <= 4 ? 4 : ((n + 3) & ~3);
        const u32 *steps = B->steps + bi.steps0;
        const int *offs = B->offs + bi.offs0;
        // the first letter that holds first in every positive and in no negative ends the search
        u32 every = ~0u, some = 0u;
        for (int i = tid; i < n; i += LT) {
            const u32 m = offs[i + 1] > offs[i] ? steps[offs[i]] : 0u;
            if (i < npos)
                every &= m;
            else
                some |= m;
        }
        every = __reduce_and_sync(FULL, every);
        some = __reduce_or_sync(FULL, some);
        if (lane == 0) {
            atomicAnd(&S.every, every);
            atomicOr(&S.some, some);
        }
        __syncthreads();
        int hit = -1;
        for (int j = 0; j < nalpha && hit < 0; ++j)
            if (((S.every & ~S.some) >> (bi.alpha[j] - 'a')) & 1u) hit = j;
        const int c1 = S.A.cf[0];
        BatchOut &o = B->out[idx];
        if ((hit >= 0 && S.A.stop_at_found) || n == 0 || nalpha == 0) {
            if (tid == 0) {
                const u64 all = hit >= 0 && S.A.stop_at_found ? (u64)hit + 1 : (u64)nalpha;
                o.status = hit >= 0 ? LTLG_FOUND : LTLG_NOT_FOUND;
                o.cost = hit >= 0 ? c1 : max(c1, S.A.max_cost);
                o.all_ltls = o.evaluated = all;
                o.rows = hit >= 0 && S.A.stop_at_found ? hit + 1 : 0;  // no rows of an instance without traces
                o.found = 0;
                o.letter = hit;
                o.walk_count = o.walk_overflow = 0;
                o.device_flags = 0;
                o.ns = globaltimer() - t0;
            }
            continue;
        }
        // as many rows as the CTA's share of the caches holds, and no more than a slot would have
        const long long cap = min((long long)LROWS, min(min(words, B->cache_words) / pitch, B->max_rows));
        bool over = false;
        if (pitch <= LPITCH && cap > nalpha) {
            if (tid == 0) {
                S.A.n = n;
                S.A.pitch = pitch;
                S.A.npos = npos;
                S.A.nalpha = nalpha;
                S.A.cap_rows = cap;
                InstCtl c{};
                c.found_key = NO_FIND;
                c.plan.cost = c1;
                *S.A.ctl = c;
            }
            __syncthreads();
            StartIn in;
            in.steps = steps;
            in.offs = offs;
            in.width = 4;
            for (int q = 0; q < nalpha; ++q) in.bit[q] = (char)(bi.alpha[q] - 'a');
            init_traces(S.A, in, S.meta, tid, LT);
            __syncthreads();
            local_begin<HK, LT>(S, tid);
            over = local_run<HK, LT, false>(S, limit, tid);
        }
        if (tid < 32) {
            if (over) {
                local_result(S, o, t0, hit, lane);
            } else if (lane == 0) {
                o.ns = globaltimer() - t0;
                B->order[atomicAdd(&B->pending, 1)] = idx;
            }
        }
    }
}
