// bf_local.cuh -- Bellman-Ford sweeps on per-CTA local tables (included by
// kernels_bf.cu).
//
// A step of the sweep -- one (layer, depth) -- depends on the step before it
// through the mesh's neighbourhoods only.  Each CTA owns a contiguous range of
// list slots, a patch of the mesh (LayerTemplate::slotNode), and keeps in
// shared memory the DP records of every node its in-edges can read: its own
// nodes and the halo, the neighbouring CTAs' nodes among its sources.  An
// in-edge names its source by a 16-bit index into that table, so a relaxation
// reads shared memory only, and a step's cost outside the SM is one exchange
// of the boundary records.
//
// Exchange.  A boundary record is 16 bytes -- value, step number, path origin
// and length -- written and read with single 128-bit accesses, so the step
// number tells whether the value beside it is the one waited for: no fence,
// no flag and no barrier lie between a node's store and its readers' polls.
// Two parities of records exist per depth; a CTA overwrites one only after
// every neighbour has reported that it read the record before it, two layers
// back.  That report does need an order: stepDone is published with release
// and polled with acquire semantics, a CTA barrier on either side, so that a
// neighbour's read comes before the store that replaces what it read.  Both are
// the staging warp's, once per layer.
//
// What it replaces: sources gathered from L2 per in-edge, and a release /
// acquire hand-off of per-CTA step counters with two CTA barriers around it
// (still there for more than four depths and for tables that do not fit).
// Cycles per step, before -> now (relaxation + hand-off or exchange):
//   conjugate 5,000 x 200, K = 3, 148 CTAs     6.0k + 3.8k -> 2.1k + 2.2k
//   pruned 20,000 x 500, 148 CTAs             25.7k + 5.4k -> 9.3k + 2.9k
//   plain 1,777 x 97, K = 3, 3 -> 10 CTAs      5.9k + 2.7k -> 1.8k + 1.3k
//   plain 642 x 60, K = 2, 1 -> 4 CTAs         5.5k + 0.5k -> 1.5k + 1.3k
//   64 uneven plain pairs in one launch       11.7k + 4.6k -> 2.7k + 1.5k
// What bounds it now: latency.  With a slice per warp (conjugate 5,000 x 30,
// K = 3, 148 CTAs, counters of one launch) the schedulers issue in 30 % of the
// cycles and shared memory moves 17 % of its wavefronts; of the 16.8 cycles
// between a warp's instructions it waits 5.9 at the step's barrier, for the
// CTA's slowest slice and its halo, 3.1 for L2 (the exchange's polls), 2.7 for
// fixed latencies and 1.6 for shared memory.  With few slices a CTA it is the
// dependent chain of one slice and the L2 round trip of the exchange.
//
// The sweep's other parts (set-up, wrap-around, candidates, extraction) work
// on the records in global memory: a sweep loads its tables from them and
// leaves the last two layers there.

// Requirements checked by the host (Graph::plan_local): at most four depths,
// three layers or more, local indices of 16 bits, path origins and lengths
// that fit 32 bits together, and tables that fit shared memory.

__device__ __forceinline__ void st_record(uint4* at, double v, unsigned tag, unsigned oh) {
    const unsigned long long lo = (unsigned long long)__double_as_longlong(v);
    const unsigned long long hi = ((unsigned long long)oh << 32) | tag;
    asm volatile(
        "{\n\t.reg .b128 r;\n\tmov.b128 r, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], r;\n\t}" ::"l"(at), "l"(lo),
        "l"(hi)
        : "memory");
}
__device__ __forceinline__ void ld_record(const uint4* at, double& v, unsigned& tag, unsigned& oh) {
    unsigned long long lo, hi;
    asm volatile(
        "{\n\t.reg .b128 r;\n\tld.relaxed.gpu.global.b128 r, [%2];\n\tmov.b128 {%0, %1}, r;\n\t}"
        : "=l"(lo), "=l"(hi)
        : "l"(at)
        : "memory");
    v = __longlong_as_double((long long)lo);
    tag = (unsigned)hi;
    oh = (unsigned)(hi >> 32);
}
// gid word of an own table entry: its node, bit 30 when another CTA reads it;
// negative where the slot holds no node.  Of a halo entry: its node.
constexpr int kGidExposed = 1 << 30;
constexpr int kGidNode = kGidExposed - 1;
// hslot word: the halo node's slot, and whether its slice has rows in the
// interlayer / intralayer part (then its owner publishes it in those steps).
constexpr unsigned kHaloInter = 1u << 30, kHaloIntra = 1u << 31, kHaloSlot = kHaloInter - 1u;

// Table entry (parity, local index i, depth k) is (parity * L + i) * KD + k;
// entries [0, nOwn) are the CTA's own slots, then the halo, then one entry
// that stays at +inf: the source of empty list slots.

// What the steps of a CTA read, at the start of its dynamic shared memory:
// the step loop runs in a function of its own, so that the registers of the
// set-up and the verdict around it do not spill into it, and takes everything
// from here.
struct LocalHot {
    unsigned long long bar[2];  // completion of the step buffers' copies
    const char* cost;
    const char* time;
    int* pred;
    uint4* xbuf;
    int* layerFlag;
    unsigned* stepDone;
    const int* waitIdx;         // the CTA's neighbours
    int* err;
    const unsigned* neverSet;
    double lam, lt, ub;         // lambda, lambda times the constant time, upper bound
    long long layerStride, interEntries;
    unsigned long long cyc[3];  // lead: relaxation, exchange, waits for staged streams
    // A wait of this CTA ran out in a step of that number modulo 4 (before the
    // first step: in the one before it).  Set during the step, read by every
    // warp between its barrier and the next one, and acted on before that one;
    // later steps have words of their own, so every warp leaves at the same
    // barrier.
    volatile int stop[4];
    int n, K, nY, nslots, L, nOwn, nHalo, s0, nsl, rowCap, hopBits;
    int r0[2], nrows[2], nAct[2];
    int nWait, stall, cta, ncta;
    unsigned spin;
    unsigned copySpin;          // polls of the step loop's waits for copies (0: the test hook's CTA)
    unsigned copiesOut;         // bit b: a copy into buffer b may be in flight after the sweep gave up
    unsigned oTslot, oGid, oHslot, oOh, oVal, oLsrc[2], oRec[2], oBuf[2];  // byte offsets in shared memory
};
static_assert(sizeof(LocalHot) <= kLocalHotBytes, "");
extern __shared__ double4 smemRaw[];
__device__ __forceinline__ LocalHot& local_hot() { return *reinterpret_cast<LocalHot*>(smemRaw); }
template <class T>
__device__ __forceinline__ T* local_at(unsigned offset) {
    return reinterpret_cast<T*>(reinterpret_cast<char*>(smemRaw) + offset);
}
// One slice with rows in a part: its first entry (lane 0, from the CTA's
// first), rows, table entry of lane 0, and slot of lane 0.
struct __align__(16) LocalSlice {
    int entry, nr, tab, slot;
};
// tslot word of a slice: its table slice, and whether it has interlayer rows.
constexpr unsigned kTabNone = 0x7fffu, kTabInter = 0x8000u;

// A record's path origin (a layer-0 node or a kLap* code) and length in one
// word: (origin + 2) << hopBits | length.
__device__ __forceinline__ unsigned pack_oh(int hopBits, int o, int h) {
    return ((unsigned)(o + 2) << hopBits) | (unsigned)h;
}

// Rows of a slice folded into NC = CH * NK running first minima: one per
// source depth and per row modulo CH.  Each is the reference's sequential scan
// (cand < best && cand < upper bound, as thr starts at their minimum) over its
// own candidates; an empty slot's source is the +inf entry, and its NaN cost
// gives a candidate that no comparison takes.  Several short chains instead of
// one long one: a chain's comparisons depend on each other (23 cycles each).
// Addresses are 32-bit byte offsets in shared memory; in place (STAGED false)
// the streams are read from global memory.
template <class CT, int TK, bool STAGED>
struct LocalStreams {
    unsigned ls, c, t;            // byte offsets of the lane's entries: source index, cost, time
    const CT* gc;
    const char* gt;
    using Time = std::conditional_t<TK == 2, double, float>;
    __device__ __forceinline__ CT cost(int r) const { return STAGED ? local_at<CT>(c)[r * 32] : gc[r * 32]; }
    __device__ __forceinline__ Time time(int r) const {
        if constexpr (TK == 0) return Time(0);
        else return STAGED ? local_at<Time>(t)[r * 32] : reinterpret_cast<const Time*>(gt)[r * 32];
    }
    static __device__ __forceinline__ double weight(CT c, Time t, double lam, double lt) {
        return __dsub_rn((double)c, TK == 0 ? lt : __dmul_rn(lam, (double)t));
    }
    __device__ __forceinline__ void advance(int rows) {
        constexpr int timeBytes = TK == 1 ? 4 : TK == 2 ? 8 : 0;
        ls += rows * 64;
        if constexpr (STAGED) {
            c += rows * 32 * (int)sizeof(CT);
            t += rows * 32 * timeBytes;
        } else {
            gc += rows * 32;
            if constexpr (TK != 0) gt += rows * 32 * timeBytes;
        }
    }
};

template <class CT, int TK, bool STAGED, int KD, int NK, int CH, int NR>
__device__ __forceinline__ void local_batch(const LocalStreams<CT, TK, STAGED>& q, unsigned sval, double lam, double lt,
                                            int row8, double (&thr)[CH * NK], int (&win)[CH * NK]) {
    using Streams = LocalStreams<CT, TK, STAGED>;
    unsigned si[NR];
    double d[NR][NK];
    CT cost[NR];
    typename Streams::Time time[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        cost[r] = q.cost(r);
        time[r] = q.time(r);
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) si[r] = sval + (unsigned)local_at<unsigned short>(q.ls)[r * 32] * (KD * 8);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if constexpr (NK == 2 && KD == 2) {
            // one 16-byte load: two 8-byte loads at this stride would use
            // every other bank pair
            const double2 x = *local_at<double2>(si[r]);
            d[r][0] = x.x;
            d[r][1] = x.y;
        } else {
#pragma unroll
            for (int kk = 0; kk < NK; ++kk) d[r][kk] = local_at<double>(si[r])[kk];
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const double w = Streams::weight(cost[r], time[r], lam, lt);
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
            const double cand = __dadd_rn(d[r][kk], w);
            const int c = (r % CH) * NK + kk;
            if (cand < thr[c]) {
                thr[c] = cand;
                win[c] = row8 + (r * 8 + kk);
            }
        }
    }
}

template <class CT, int TK, bool STAGED, int KD, int NK, int CH, int NR>
__device__ __forceinline__ void local_tail(const LocalStreams<CT, TK, STAGED>& q, unsigned sval, double lam, double lt,
                                           int row8, int nr, double (&thr)[CH * NK], int (&win)[CH * NK]) {
    if constexpr (NR > 1) {
        if (nr < NR) {
            local_tail<CT, TK, STAGED, KD, NK, CH, NR - 1>(q, sval, lam, lt, row8, nr, thr, win);
            return;
        }
    }
    local_batch<CT, TK, STAGED, KD, NK, CH, NR>(q, sval, lam, lt, row8, thr, win);
}

// Rows per batch and chains per depth (CH divides the batch): the batch's
// loads are in flight together; registers bound both, and every further chain
// costs seven instructions where the chains meet.
__host__ __device__ constexpr int local_batch_rows(int nk) { return nk <= 2 ? 8 : nk == 3 ? 6 : 4; }
__host__ __device__ constexpr int local_chains(int nk) { return nk == 1 ? 2 : 1; }

// What a step keeps in registers from step to step.  The tables are written
// between the reads, so values left in shared memory would be loaded again
// for every slice; a step's issue slots, not its arithmetic, are what it runs
// out of.
struct LocalRegs {
    double lam, lt, ub;
    unsigned val, oh, gid;  // byte offsets
    int L, n, K, nslots, hopBits;
    int* pred;
    uint4* xbuf;
};

// A warp's first slice of a part, in registers for the whole sweep (most warps
// have one).
struct LocalFirst {
    LocalSlice rec;
    int g;
};

// One step (l, k) over the warp's slices with rows in its part.  `buf` (or
// gcost, gtime) holds the step's streams from the CTA's first row on,
// `timeOfs` the times' offset there; predOff is the index of the step's first
// predecessor, `step` its number, the tag of the records it publishes.
// Returns whether the thread improved a node.
template <class CT, int TK, int KD, int NK, bool STAGED>
__device__ __forceinline__ bool local_relax(const LocalRegs& R, const LocalFirst& first, int warp, int nwarps,
                                            unsigned rec0, int count, unsigned lsrc, unsigned buf, unsigned timeOfs, const char* gcost,
                                            const char* gtime, int l, int k, int predOff, unsigned step) {
    constexpr int CH = local_chains(NK), NC = CH * NK, NR = local_batch_rows(NK);
    constexpr int timeBytes = TK == 1 ? 4 : TK == 2 ? 8 : 0;
    constexpr int part = NK == KD ? 0 : 1;
    const int lane = threadIdx.x & 31;
    const int curBase = (l & 1) * R.L, srcBase = part ? curBase : R.L - curBase;
    const int kofs = part ? k - 1 : 0;
    const unsigned sval = R.val + (unsigned)(srcBase * KD + kofs) * 8u;
    bool any = false;
    LocalSlice rec = first.rec;
    int g = first.g;
    for (int i = warp; i < count; i += nwarps) {
        if (i != warp) {
            rec = local_at<LocalSlice>(rec0)[i];
            g = local_at<int>(R.gid)[rec.tab + lane];
        }
        int nr = rec.nr;
        const unsigned at = (unsigned)((curBase + rec.tab + lane) * KD + k);
        double thr[NC];
        int win[NC];
        thr[0] = R.ub;
        if (l == 0) {
            const double kept = local_at<double>(R.val)[at];
            if (kept < thr[0]) thr[0] = kept;
        }
        win[0] = -1;
#pragma unroll
        for (int c = 1; c < NC; ++c) {
            thr[c] = thr[0];
            win[c] = -1;
        }
        const unsigned e0 = (unsigned)(rec.entry + lane), ls0 = lsrc + e0 * 2u;
        LocalStreams<CT, TK, STAGED> q;
        q.ls = ls0;
        if constexpr (STAGED) {
            q.c = buf + e0 * (unsigned)sizeof(CT);
            q.t = timeOfs + e0 * (unsigned)timeBytes;
        } else {
            q.gc = reinterpret_cast<const CT*>(gcost) + e0;
            q.gt = gtime + (size_t)(e0 * (unsigned)timeBytes);
        }
        int row8 = 0;
        for (; nr >= NR; nr -= NR, row8 += NR * 8) {
            local_batch<CT, TK, STAGED, KD, NK, CH, NR>(q, sval, R.lam, R.lt, row8, thr, win);
            q.advance(NR);
        }
        if (nr) local_tail<CT, TK, STAGED, KD, NK, CH, NR - 1>(q, sval, R.lam, R.lt, row8, nr, thr, win);
        // the first minimum over the chains: ties go to the earlier position
#pragma unroll
        for (int c = 1; c < NC; ++c)
            if (thr[c] < thr[0] || (thr[c] == thr[0] && (unsigned)win[c] < (unsigned)win[0])) {
                thr[0] = thr[c];
                win[0] = win[c];
            }
        if (g < 0) continue;
        const int v = g & kGidNode;
        double best = thr[0];
        unsigned oh = 0;  // (kLapUnknown, 0)
        if (win[0] >= 0) {
            const int bk = kofs + (win[0] & 7);
            const unsigned bs = *local_at<unsigned short>(ls0 + (unsigned)(win[0] >> 3) * 64u);
            const int node = local_at<int>(R.gid)[bs] & kGidNode;
            const int srcLayer = part ? l : l - 1;
            R.pred[predOff + v] = node + (srcLayer * R.K + bk) * R.n;
            oh = srcLayer == 0 && bk == 0 ? pack_oh(R.hopBits, node, 1)
                                          : local_at<unsigned>(R.oh)[(srcBase + (int)bs) * KD + bk] + 1u;
            any = true;
        } else {
            best = kInfD;
            if (l == 0) {
                // layer 0 keeps an older value and its older predecessor, one
                // of the node's own intralayer sources
                best = local_at<double>(R.val)[at];
                const int pe = __ldcg(R.pred + predOff + v);
                const int ps = pe - (k - 1) * R.n;
                if (pe < 0) {
                    oh = pack_oh(R.hopBits, kLapEnd, 0);
                } else if (ps >= 0 && ps < R.n) {
                    if (k == 1) {
                        oh = pack_oh(R.hopBits, ps, 1);
                    } else {
                        for (int r = 0; r < rec.nr; ++r) {
                            const int bs = *local_at<unsigned short>(ls0 + (unsigned)r * 64u);
                            if (bs != R.L - 1 && (local_at<int>(R.gid)[bs] & kGidNode) == ps) {
                                oh = local_at<unsigned>(R.oh)[(curBase + bs) * KD + k - 1] + 1u;
                                break;
                            }
                        }
                    }
                }
            }
        }
        local_at<double>(R.val)[at] = best;
        local_at<unsigned>(R.oh)[at] = oh;
        if (g & kGidExposed) st_record(R.xbuf + ((l & 1) * KD + k) * R.nslots + rec.slot + lane, best, step, oh);
    }
    return any;
}

// One more unsuccessful poll of a bounded wait; true when it gives up: its
// polls ran out, or another CTA raised the error word.
__device__ __forceinline__ bool local_give_up(LocalHot& H, unsigned step, unsigned& spins) {
    ++spins;
    if (spins > H.spin || ((spins & 63u) == 0 && *(volatile int*)H.err)) {
        atomicExch(H.err, 1);
        H.stop[step & 3] = 1;
        return true;
    }
    if (spins > 512) __nanosleep(32);
    return false;
}

// Takes the halo records that step (l, k), number `step`, produced.
template <int KD>
__device__ __forceinline__ void local_take_halo(int l, int k, unsigned step, int nthreads) {
    LocalHot& H = local_hot();
    const unsigned need = k == 0 ? kHaloInter : kHaloIntra;
    for (int i = (int)threadIdx.x; i < H.nHalo; i += nthreads) {
        const unsigned hs = local_at<unsigned>(H.oHslot)[i];
        const unsigned at = (unsigned)(((l & 1) * H.L + H.nOwn + i) * KD + k);
        if (hs & need) {
            const uint4* in = H.xbuf + ((l & 1) * KD + k) * H.nslots + (int)(hs & kHaloSlot);
            double v;
            unsigned tag, oh, spins = 0;
            for (;;) {
                ld_record(in, v, tag, oh);
                if (tag == step || local_give_up(H, step, spins)) break;
            }
            local_at<double>(H.oVal)[at] = v;
            local_at<unsigned>(H.oOh)[at] = oh;
        } else if (l == 2 && k == 0) {
            // the parity still holds layer 0's start value
            local_at<double>(H.oVal)[at] = kInfD;
            local_at<unsigned>(H.oOh)[at] = 0;
        }
    }
}

// Stages step (l, k)'s costs and times into buffer b, or, when no buffer
// fits, brings them into L2 for the step's reads in place.  One thread.
template <class CT, int TK>
__device__ __forceinline__ void local_stage_issue(int b, int l, int k) {
    constexpr int costBytes = sizeof(CT), timeBytes = TK == 1 ? 4 : TK == 2 ? 8 : 0;
    LocalHot& H = local_hot();
    const int part = k == 0 ? 0 : 1;
    const int rows = H.nrows[part];
    if (rows == 0) return;
    const size_t base =
        (size_t)l * (size_t)H.layerStride + (part ? (size_t)H.interEntries : 0) + (size_t)H.r0[part] * 32;
    const unsigned bc = (unsigned)rows * 32 * costBytes, bt = (unsigned)rows * 32 * timeBytes;
    if (H.rowCap == 0) {
        bulk_prefetch_l2(H.cost + base * costBytes, bc);
        if (TK) bulk_prefetch_l2(H.time + base * timeBytes, bt);
        return;
    }
    char* dst = local_at<char>(H.oBuf[b]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect(H.bar + b, bc + bt);
    bulk_load(dst, H.cost + base * costBytes, bc, H.bar + b);
    if (TK) bulk_load(dst + (size_t)H.rowCap * 32 * costBytes, H.time + base * timeBytes, bt, H.bar + b);
}

// At the start of a call: the CTA's tables and its in-edges' local source indices.
__device__ __forceinline__ void local_begin(const BfParams& p, const Team& t, int s0, int s1, int costBytes,
                                            int timeBytes) {
    LocalHot& H = local_hot();
    const LocalLayout o = local_layout(p.maxCtaSlices, p.localL, p.localHalo, p.localRows[0], p.localRows[1], p.localKD);
    unsigned short* tslot = local_at<unsigned short>((unsigned)o.tslot);
    const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, nsl = s1 - s0;
    if (threadIdx.x < 32) {
        // table slices, and per part the slices with rows, in order
        int base = 0, act[2] = {0, 0};
        for (int i0 = 0; i0 < nsl; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < nsl;
            const bool used = in && __ldg(p.sliceUsed + s0 + i) != 0;
            const unsigned m = __ballot_sync(0xffffffffu, used), below = (1u << lane) - 1u;
            const unsigned tab = used ? (unsigned)(base + __popc(m & below)) : kTabNone;
            base += __popc(m);
            unsigned inter = 0;
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const int* sp = part ? p.spIntra : p.spInter;
                const int first = __ldg(sp + s0), a = in ? __ldg(sp + s0 + i) : 0, b = in ? __ldg(sp + s0 + i + 1) : 0;
                const bool rows = b > a;
                const unsigned mr = __ballot_sync(0xffffffffu, rows);
                if (rows)
                    local_at<LocalSlice>((unsigned)o.rec[part])[act[part] + __popc(mr & below)] =
                        LocalSlice{(a - first) * 32, b - a, (int)tab * 32, (s0 + i) * 32};
                act[part] += __popc(mr);
                if (part == 0 && rows) inter = kTabInter;
            }
            if (in) tslot[i] = (unsigned short)(tab | inter);
        }
        if (lane == 0) {
            mbar_init(H.bar);
            mbar_init(H.bar + 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            H.cost = (const char*)p.cost;
            H.time = (const char*)p.time;
            H.pred = p.pred;
            H.xbuf = p.xbuf;
            H.layerFlag = p.layerFlag;
            H.stepDone = p.stepDone;
            const int w0 = __ldg(p.waitPtr + t.cta);
            H.waitIdx = p.waitIdx + w0;
            H.nWait = __ldg(p.waitPtr + t.cta + 1) - w0;
            H.err = t.err;
            H.neverSet = &p.ctl->neverSet;
            H.stall = t.cta == p.stallCta ? 1 : 0;
            H.lam = p.lambda;
            H.lt = __dmul_rn(p.lambda, p.tconst);
            H.ub = p.ub;
            H.layerStride = p.layerStride;
            H.interEntries = p.interEntries;
            H.n = p.n;
            H.K = p.K;
            H.nY = p.nY;
            H.nslots = p.nslots;
            H.nOwn = 32 * base;
            H.nHalo = t.ncta > 1 ? __ldg(p.haloCnt + t.cta) : 0;
            H.L = H.nOwn + H.nHalo + 1;
            H.s0 = s0;
            H.nsl = nsl;
            H.rowCap = p.rowCap;
            H.hopBits = p.hopBits;
            for (int part = 0; part < 2; ++part) {
                const int* sp = part ? p.spIntra : p.spInter;
                H.r0[part] = __ldg(sp + s0);
                H.nrows[part] = __ldg(sp + s1) - H.r0[part];
                H.nAct[part] = act[part];
                H.oLsrc[part] = (unsigned)o.lsrc[part];
                H.oRec[part] = (unsigned)o.rec[part];
                H.oBuf[part] = (unsigned)(o.total + (size_t)part * p.rowCap * 32 * (costBytes + timeBytes));
            }
            H.stop[0] = H.stop[1] = H.stop[2] = H.stop[3] = 0;
            H.cta = t.cta;
            H.ncta = t.ncta;
            H.spin = p.spinLimit;
            H.copySpin = t.cta == p.stallCopyCta ? 0u : p.spinLimit;
            H.copiesOut = 0;
            H.oTslot = (unsigned)o.tslot;
            H.oGid = (unsigned)o.gid;
            H.oHslot = (unsigned)o.hslot;
            H.oOh = (unsigned)o.oh;
            H.oVal = (unsigned)o.val;
        }
    }
    __syncthreads();
    int* gid = local_at<int>(H.oGid);
    for (int i = (int)(threadIdx.x >> 5); i < nsl; i += nwarps) {
        const unsigned ts = tslot[i] & kTabNone;
        if (ts == kTabNone) continue;
        const int v = __ldg(p.slotNode + (size_t)(s0 + i) * 32 + lane);
        const unsigned ex = t.ncta > 1 ? __ldcg(p.exposed + s0 + i) : 0u;
        gid[ts * 32 + lane] = v < 0 ? -1 : (v | (((ex >> lane) & 1u) ? kGidExposed : 0));
    }
    unsigned* hslot = local_at<unsigned>(H.oHslot);
    for (int i = (int)threadIdx.x; i < H.nHalo; i += blockDim.x) {
        const unsigned hs = __ldg(p.haloSlot + (size_t)t.cta * p.haloCap + i);
        hslot[i] = hs;
        gid[H.nOwn + i] = __ldg(p.slotNode + (hs & kHaloSlot));
    }
    for (int part = 0; part < 2; ++part) {
        if (part == 1 && p.localRows[1] == 0) break;
        const int words = H.nrows[part] * 16;
        const unsigned* in = reinterpret_cast<const unsigned*>(p.lsrc[part]) + (size_t)H.r0[part] * 16;
        unsigned* to = local_at<unsigned>(H.oLsrc[part]);
        for (int i = (int)threadIdx.x; i < words; i += blockDim.x) to[i] = __ldg(in + i);
    }
    if (threadIdx.x == 0) gid[H.L - 1] = 0;
    __syncthreads();
}

// The tables at the start of a sweep: layer 0's parity from the records in
// global memory, the other parity unreached.
__device__ __forceinline__ void local_load(const BfParams& p) {
    const LocalHot& H = local_hot();
    const int L = H.L, n = p.n, Kp = p.Kp, KD = p.localKD;
    const int* gid = local_at<int>(H.oGid);
    double* val = local_at<double>(H.oVal);
    unsigned* ohs = local_at<unsigned>(H.oOh);
    for (int i = (int)threadIdx.x; i < L; i += blockDim.x) {
        const int g = gid[i];
        const bool real = i < L - 1 && g >= 0;
        const int v = g & kGidNode;
        for (int k = 0; k < KD; ++k) {
            double x = kInfD;
            unsigned oh = 0;
            if (real) {
                x = __ldcg(p.dv + (size_t)v * Kp + k);
                const int2 e = __ldcg(p.doh + (size_t)k * n + v);
                oh = pack_oh(p.hopBits, e.x, e.y);
            }
            val[i * KD + k] = x;
            ohs[i * KD + k] = oh;
            val[(L + i) * KD + k] = kInfD;
            ohs[(L + i) * KD + k] = 0;
        }
    }
}

// Layers nY - 1 and nY of the CTA's own nodes into global memory: what the
// sweep's verdict and the next sweep read.  A node without a table entry is
// never reached.
__device__ __forceinline__ void local_store(const BfParams& p) {
    const LocalHot& H = local_hot();
    const int n = p.n, Kp = p.Kp, L = H.L, KD = p.localKD, s0 = H.s0, nsl = H.nsl;
    const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const unsigned short* tslot = local_at<unsigned short>(H.oTslot);
    const double* val = local_at<double>(H.oVal);
    const unsigned* ohs = local_at<unsigned>(H.oOh);
    for (int i = (int)(threadIdx.x >> 5); i < nsl; i += nwarps) {
        const unsigned ts = tslot[i] & kTabNone;
        const int v = __ldg(p.slotNode + (size_t)(s0 + i) * 32 + lane);
        if (v < 0) continue;
        for (int par = 0; par < 2; ++par) {
            const bool last = par == (p.nY & 1);
            const size_t base = (size_t)par * n * Kp;
            for (int k = 0; k < KD; ++k) {
                double x = kInfD;
                int2 e = make_int2(kLapUnknown, 0);
                if (ts != kTabNone && !(last && k > 0)) {
                    const int at = (par * L + (int)ts * 32 + lane) * KD + k;
                    x = val[at];
                    const unsigned w = ohs[at];
                    e = make_int2((int)(w >> p.hopBits) - 2, (int)(w & ((1u << p.hopBits) - 1u)));
                }
                p.dv[base + (size_t)v * Kp + k] = x;
                p.doh[base + (size_t)k * n + v] = e;
            }
        }
    }
}

// All steps of one sweep from step number `step` on.  The CTA's last warp
// stages the streams and waits for the neighbours' progress; the others relax
// and take the halo; one CTA barrier ends each step.  `phase`: bit b is the
// parity of step buffer b's next completion (kept by the last warp).  Returns
// the new phases, bit 2 set when a wait ran out; the copies are waited for once
// more then, and H.copiesOut says whether that ran out too.  SITE keeps the
// instances of kernels with different register budgets apart.
template <class CT, int TK, int KD, int SITE>
__device__ __noinline__ unsigned local_sweep(int stamp, unsigned step, unsigned phase) {
    LocalHot& H = local_hot();
    const int warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5) - 1;
    const int nY = H.nY;
    const bool staged = H.rowCap > 0;
    const unsigned staging = staged ? (H.nrows[0] ? 1u : 0u) | (H.nrows[1] ? 2u : 0u) : 0u;  // parts with copies
    int sb = 0;
    bool ok = true;
    if (warp == nwarps) {
        // Copies are issued a step ahead and waited for here, before the
        // barrier that opens their step: the relaxing warps read the buffer
        // without a wait of their own.
        const int lane = threadIdx.x & 31;
        unsigned out = 0;  // bit b: a copy into buffer b is in flight
        auto stage = [&](int b, int l, int k) {
            if (lane == 0) local_stage_issue<CT, TK>(b, l, k);
            const unsigned copy = (staging >> (k == 0 ? 0 : 1)) & 1u;
            out |= copy << b;
            return copy != 0;
        };
        auto wait = [&](int b, unsigned spin) {
            if (!__all_sync(0xffffffffu, mbar_wait(H.bar + b, (phase >> b) & 1u, spin))) return false;
            phase ^= 1u << b;
            out &= ~(1u << b);
            return true;
        };
        auto landed = [&](int b) {
            if (wait(b, H.copySpin)) return;
            atomicExch(H.err, 1);
            H.stop[step & 3] = 1;
        };
        if (stage(0, KD > 1 ? 0 : 1, KD > 1 ? 1 : 0)) landed(0);
        __syncthreads();
        int stopped = H.stop[step & 3];
        for (int l = KD > 1 ? 0 : 1; l <= nY && ok; ++l) {
            for (int k = l == 0 ? 1 : 0; k < (l == nY ? 1 : KD); ++k) {  // the closing layer has no intralayer edges
                if (stopped) {
                    ok = false;
                    break;
                }
                const unsigned t0 = (unsigned)clock();
                ++step;
                if (l < nY) {
                    const bool copy = k + 1 < KD ? stage(sb ^ 1, l, k + 1) : stage(sb ^ 1, l + 1, 0);
                    if (H.ncta > 1 && k + 1 == KD) {
                        // the next layer overwrites the records of the layer
                        // before this one, which the neighbours have read when
                        // they have finished that layer; the stall hook's word
                        // is one that nothing writes
                        const int nWait = H.nWait;
                        for (int i = lane; i < nWait + H.stall; i += 32) {
                            const unsigned* f =
                                i < nWait ? H.stepDone + (size_t)__ldg(H.waitIdx + i) * kStepDoneStride : H.neverSet;
                            const int want = i < nWait ? (int)step - KD : (int)step;
                            unsigned spins = 0;
                            while ((int)ld_acquire_u32(f) < want)
                                if (local_give_up(H, step, spins)) break;
                        }
                    }
                    if (copy) landed(sb ^ 1);
                    if (lane == 0 && H.cta == 0) H.cyc[2] += (unsigned)clock() - t0;
                }
                __syncthreads();
                // release: the halo reads of the CTA's threads, before the
                // barrier, come before what the neighbours store after they
                // have seen this.  Of the closing layer too: with one depth the
                // next sweep's first wait is for it.
                if (lane == 0 && H.ncta > 1 && (k + 1 == KD || l == nY))
                    st_release_u32(H.stepDone + (size_t)H.cta * kStepDoneStride, step);
                sb ^= 1;
                stopped = H.stop[step & 3];
            }
        }
        if (ok && !stopped) return phase;
        for (int b = 0; b < 2; ++b)
            if ((out >> b) & 1u) wait(b, H.spin);
        if (lane == 0) H.copiesOut = out;
        return phase | 4u;
    }
    __syncthreads();  // the first step's streams have landed
    const bool lead = H.cta == 0 && threadIdx.x == 0;
    const bool team = H.ncta > 1;
    const LocalRegs R{H.lam, H.lt, H.ub, H.oVal, H.oOh, H.oGid, H.L, H.n, H.K, H.nslots, H.hopBits, H.pred, H.xbuf};
    const unsigned rec[2] = {H.oRec[0], H.oRec[1]}, lsrc[2] = {H.oLsrc[0], H.oLsrc[1]};
    const int nAct[2] = {H.nAct[0], H.nAct[1]};
    const unsigned buf0 = H.oBuf[0], bufBytes = H.oBuf[1] - buf0, timeOfs = (unsigned)H.rowCap * 32u * (unsigned)sizeof(CT);
    LocalFirst first[2];
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        first[part] = LocalFirst{};
        if (warp < nAct[part]) {
            first[part].rec = local_at<LocalSlice>(rec[part])[warp];
            first[part].g = local_at<int>(R.gid)[first[part].rec.tab + (threadIdx.x & 31)];
        }
    }
    const int predStep = (KD > 1 ? 1 : R.K) * R.n;
    int stopped = H.stop[step & 3];
    int predOff = predStep;
    for (int l = KD > 1 ? 0 : 1; l <= nY && ok; ++l) {
        for (int k = l == 0 ? 1 : 0; k < (l == nY ? 1 : KD); ++k) {
            unsigned t0 = 0, t2 = 0;
            if (lead) t0 = (unsigned)clock();
            const bool inter = KD == 1 || k == 0;
            ++step;
            bool any;
            if (staged) {
                const unsigned buf = buf0 + (sb ? bufBytes : 0u);
                if (inter)
                    any = local_relax<CT, TK, KD, KD, true>(R, first[0], warp, nwarps, rec[0], nAct[0], lsrc[0], buf, buf + timeOfs,
                                                            nullptr, nullptr, l, k, predOff, step);
                else
                    any = local_relax<CT, TK, KD, 1, true>(R, first[1], warp, nwarps, rec[1], nAct[1], lsrc[1], buf, buf + timeOfs,
                                                           nullptr, nullptr, l, k, predOff, step);
            } else {
                const size_t off = (size_t)l * (size_t)H.layerStride + (inter ? 0 : (size_t)H.interEntries) +
                                   (size_t)H.r0[inter ? 0 : 1] * 32;
                const char* cost = H.cost + off * sizeof(CT);
                const char* time = TK == 0 ? nullptr : H.time + off * (TK == 1 ? 4 : 8);
                if (inter)
                    any = local_relax<CT, TK, KD, KD, false>(R, first[0], warp, nwarps, rec[0], nAct[0], lsrc[0], 0, 0, cost, time,
                                                             l, k, predOff, step);
                else
                    any = local_relax<CT, TK, KD, 1, false>(R, first[1], warp, nwarps, rec[1], nAct[1], lsrc[1], 0, 0, cost, time,
                                                            l, k, predOff, step);
            }
            // a layer without an improved node leaves every later one
            // unreached, so the last layer before the closing one tells
            if (l == nY - 1 && any) H.layerFlag[l] = stamp;
            if (l == 2 && inter) {
                // own entries without interlayer rows: the parity still holds
                // layer 0's start values
                const unsigned short* tslot = local_at<unsigned short>(H.oTslot);
                for (int i = (int)threadIdx.x; i < H.nsl * 32; i += nwarps * 32) {
                    const unsigned ts = tslot[i >> 5];
                    if ((ts & kTabInter) || (ts & kTabNone) == kTabNone) continue;
                    const int at = ((int)ts * 32 + (i & 31)) * KD;
                    local_at<double>(R.val)[at] = kInfD;
                    local_at<unsigned>(R.oh)[at] = 0;
                }
            }
            if (lead) t2 = (unsigned)clock();
            if (team && l < nY) local_take_halo<KD>(l, k, step, nwarps * 32);
            if (stopped) {
                ok = false;
                break;
            }
            __syncthreads();
            if (lead) {
                H.cyc[0] += t2 - t0;  // 32-bit clock differences
                H.cyc[1] += (unsigned)clock() - t2;
            }
            sb ^= 1;
            predOff += predStep;
            stopped = H.stop[step & 3];
        }
    }
    return phase | (ok && !stopped ? 0u : 4u);
}
