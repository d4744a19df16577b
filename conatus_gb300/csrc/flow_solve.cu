// Scheduled solve of the factored tau systems: the column sweeps' own operations, in an order fixed per
// system at the factorization.
//
// A column sweep applies its updates y_i -= l_ij y_j column by column, one warp per system: a chain of
// 2 n columns, each two FP64 instructions, shared-memory round trips and two warp barriers deep, with
// few of the lanes at work. But an update only waits for y_j's own updates and for the earlier ones
// of y_i. Every operation of a solve is therefore given the first time slot after those it needs (list
// scheduling: Graham 1966; sparse triangular solves by levels: Anderson and Saad 1989), `flow_ops` of
// them to a slot, and a warp runs slot after slot, a lane per (operation, component). An operation is
// a fused multiply-add v_dst = -c v_src + v_dst (or + 0). The rows of the vector v stay where they are:
// the interchanges only decide which rows an operation names (a row is named by the column it ends up
// the pivot row of, so the solution comes out in order). The border's sums, the small LU solve
// and the correction x - W z are operations as well (the rows behind the system's hold the partial
// sums). L and U take about n / 2 slots each: the two parities of the Chebyshev modes are independent,
// and so are most rows of a column.
// Every entry sees the operations of the column sweeps in their order, the border's sums in the order
// of 16 or 32 lanes, so the results are theirs bit for bit.
//
// The values are those of the real form (real_form.cuh), the components of a complex right-hand side (and
// of a shared pair's two) being right-hand sides of one real system: one fused multiply-add where the
// complex update takes four.
//
// What bounds it: few systems, the chain of a slot (a shared-memory read, a fused multiply-add of 64
// cycles, a write, two warp barriers: 140 cycles, from RB 256 x 64's 25.3 us for 354 slots and Burgers' 12.2 us
// for 160 at 2.07 GHz, 2800 cycles beside the slots); many, the FP64 unit (channel 192 x 129 x 192: 657 us, a
// slot per 23 cycles and SM, of which the unit takes 16).
#include "flow_solve.cuh"

#include <algorithm>
#include <utility>

#include "real_form.cuh"

namespace cng {

constexpr int kSlots = 16;                       // slots of a chunk of the operation stream
constexpr int kRing = 3;                         // chunks staged in shared memory (4: 8 warps an SM instead of
                                                 // 9, channel 128 x 129 x 128 351 us against 298)
constexpr int kFlowWarps = 4;                    // most systems of a block
constexpr size_t kFlowSmem = 220 * 1024;
constexpr size_t kFlowLoose = 64 << 20;           // bytes of operations laid out at their most and left so
constexpr int kMaxBorder = 64;
constexpr unsigned kFresh = 0x80000000u;         // the operation's sum starts from 0

__host__ __device__ constexpr int flow_ops(int ncr) { return 32 / ncr; }        // operations of a slot
// a chunk: values -c [kSlots][ops], then rows [kSlots][ops] (read | written << 16 | kFresh)
__host__ __device__ constexpr int flow_chunk(int ncr, int elem) { return kSlots * flow_ops(ncr) * (elem + 4); }

FlowForm::~FlowForm() {
    for (void* p : {(void*)data[0], (void*)data[1], (void*)nchunk, (void*)row, (void*)flags}) dev_free(p);
}

// ---- build ---------------------------------------------------------------------------------------
template <class T>
struct FlowIn {
    FlowSource s;
    int kv, ncr, rows, cap;                      // rows of the vector, slots allowed
    const T* ab;
    const T* vt;
    const T* w;
    const T* slu;
    const unsigned char* mask;                   // [r][n]: V^T's entries, the union over the batch
};
struct FlowOut {
    unsigned char* data;
    size_t sb;
    unsigned short* row;
};

__device__ __forceinline__ int phase_of(const unsigned char* p, int i) { return p ? p[i] : 0; }
__device__ __forceinline__ bool pure_imag(double) { return false; }
__device__ __forceinline__ bool pure_imag(zd v) { return v.re == 0.0 && v.im != 0.0; }

// The schedule of one system, by one warp. `ready` of a row: the slot after its last write; `read`: the
// last slot that reads it (a slot reads before it writes).
template <bool COUNT>
struct FlowPlan {
    int *ready, *read;
    unsigned short* next;                        // where to look for room from a slot on
    unsigned char* cnt;                          // operations of a slot
    unsigned char* data;
    int ops, chunk, cap, lane, end = 0;
    bool over = false;
    // v_dst = -c v_src + (fresh ? 0 : v_dst), one per lane where `has`, the dst all different
    __device__ void operator()(bool has, int src, int dst, double c, bool fresh) {
        int t = has ? max(max(ready[src], ready[dst]), read[dst]) : 0;
        bool open = has;
        while (__any_sync(0xffffffffu, open)) {
            if (open)                            // past the full slots (the links halve as they are followed)
                while (t < cap && next[t] != t) {
                    const int u = next[t];
                    next[t] = next[min(u, cap)];
                    t = u;
                }
            __syncwarp();
            if (open && t >= cap) {
                over = true;
                open = has = false;
            }
            const unsigned same = __match_any_sync(0xffffffffu, open ? t : -1);
            const int rank = __popc(same & ((1u << lane) - 1));
            const int at = open ? cnt[t] : 0;
            __syncwarp();
            if (open && rank == 0) {
                cnt[t] = (unsigned char)min(ops, at + __popc(same));
                if (at + __popc(same) >= ops) next[t] = (unsigned short)(t + 1);
            }
            __syncwarp();
            if (open && at + rank < ops) {
                if constexpr (!COUNT) {
                    unsigned char* ch = data + (size_t)(t / kSlots) * chunk;
                    const int e = (t % kSlots) * ops + at + rank;
                    reinterpret_cast<double*>(ch)[e] = -c;
                    reinterpret_cast<unsigned*>(ch + (size_t)kSlots * ops * sizeof(double))[e] =
                        (unsigned)src | (unsigned)dst << 16 | (fresh ? kFresh : 0u);
                }
                open = false;
            } else if (open) {
                ++t;
            }
        }
        if (has) {
            ready[dst] = t + 1;
            atomicMax(&read[src], t);
            end = max(end, t + 1);
        }
        __syncwarp();
    }
};

// One warp per system: its slots into nslot and, unless COUNT, its operations.
// stat[0]: not of the form, stat[1]: more slots than allowed.
// What bounds it: the latency of one warp, 1.7 ms for n = 522, whatever the number of systems. So the
// operations are written without a counting pass, at their most, and packed where that is more than 64 MB; the
// counting pass is for host-built handles, whose bytes are limited, and where the device has no room.
template <class T, bool COUNT>
__global__ void __launch_bounds__(32) k_flow_build(FlowIn<T> in, int* nslot, int* stat, FlowOut o) {
    extern __shared__ __align__(16) unsigned char fsm[];
    const int n = in.s.n, r = in.s.r, kl = in.s.kl, kv = in.kv, ldab = in.s.ldab, rows = in.rows, LS = in.s.lanes;
    const int sys = blockIdx.x, lane = threadIdx.x;
    FlowPlan<COUNT> put;
    put.ready = reinterpret_cast<int*>(fsm);
    put.read = put.ready + rows;
    unsigned short* ord = reinterpret_cast<unsigned short*>(put.read + rows);      // row at a position
    unsigned short* piv = ord + n;
    unsigned short* name = piv + n;
    put.next = name + n;
    put.cnt = reinterpret_cast<unsigned char*>(put.next + in.cap + 1);
    unsigned char* rowph = put.cnt + in.cap;
    put.data = COUNT ? nullptr : o.data + (size_t)sys * o.sb;
    put.ops = flow_ops(in.ncr);
    put.chunk = flow_chunk(in.ncr, (int)sizeof(double));
    put.cap = in.cap;
    put.lane = lane;
    const T* ab = in.ab + (size_t)sys * n * ldab;
    const int* ipiv = in.s.ipiv + (size_t)sys * n;
    const unsigned char *p = in.s.rowp, *q = in.s.colp;
    int bad = 0;
    for (int i = lane; i < rows; i += 32) put.ready[i] = put.read[i] = 0;
    for (int i = lane; i < n; i += 32) ord[i] = (unsigned short)i;
    for (int t = lane; t <= in.cap; t += 32) put.next[t] = (unsigned short)t;
    for (int t = lane; t < in.cap; t += 32) put.cnt[t] = 0;
    __syncwarp();
    // phase of the row that becomes row j of U, from 1 / u_jj = i^{q_j - p} r
    for (int j = lane; j < n; j += 32) {
        piv[j] = (unsigned short)ipiv[j];
        rowph[j] = (unsigned char)(phase_of(q, j) ^ (pure_imag(ab[(size_t)j * ldab + kv]) ? 1 : 0));
    }
    __syncwarp();
    if (lane == 0) {                             // where every row ends up
        for (int j = 0; j + 1 < n; ++j) {
            const int l = piv[j];
            const unsigned short t = ord[j];
            ord[j] = ord[l];
            ord[l] = t;
        }
        for (int j = 0; j < n; ++j) name[ord[j]] = (unsigned short)j;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        ord[i] = name[i];                        // from here on the name of the row at a position
        if constexpr (!COUNT) o.row[(size_t)sys * n + i] = name[i];
        // the solve applies the batch's phase of row i: this system's has to be the same (the batch's are
        // found on a sample of the systems)
        if (rowph[name[i]] != phase_of(p, i)) bad = 1;
    }
    __syncwarp();
    auto dinv_of = [&](int j) { return real_part_of(ab[(size_t)j * ldab + kv], phase_of(q, j) - rowph[j], bad); };
    // the columns' first 32 entries are read a column ahead
    auto low = [&](int j, int t) { return j + 1 < n && t < min(kl, n - 1 - j) ? ab[(size_t)j * ldab + kv + 1 + t] : T(0.0); };
    auto high = [&](int j, int d) { return j >= 0 && d <= min(kv, j) ? ab[(size_t)j * ldab + kv - d] : T(0.0); };
    T ahead = low(0, lane);
    for (int j = 0; j + 1 < n; ++j) {            // L
        T a = ahead;
        ahead = low(j + 1, lane);
        const int l = piv[j];
        if (lane == 0 && l != j) {
            const unsigned short t = ord[j];
            ord[j] = ord[l];
            ord[l] = t;
        }
        __syncwarp();
        const int src = ord[j];
        for (int t0 = 0; t0 < min(kl, n - 1 - j); t0 += 32) {
            const int t = t0 + lane;
            if (t0) a = low(j, t);
            const int dst = j + 1 + t < n ? ord[j + 1 + t] : src;
            const double v = real_part_of(a, rowph[dst] - rowph[j], bad);
            put(v != 0.0, src, v != 0.0 ? dst : 0, v, false);
        }
    }
    ahead = high(n - 1, 1 + lane);
    T diag = ab[(size_t)(n - 1) * ldab + kv];
    for (int j = n - 1; j >= 0; --j) {           // U: y_i -= (u_ij / u_jj) y_j
        T a = ahead;
        const double dinv = real_part_of(diag, phase_of(q, j) - rowph[j], bad);
        ahead = high(j - 1, 1 + lane);
        if (j) diag = ab[(size_t)(j - 1) * ldab + kv];
        const int qj = phase_of(q, j), src = ord[j];
        for (int d0 = 1; d0 <= min(kv, j); d0 += 32) {
            const int d = d0 + lane;
            if (d0 > 1) a = high(j, d);
            const double v = is_zero(a) ? 0.0 : real_part_of(a, rowph[j - d] - qj, bad) * dinv;
            put(v != 0.0, src, v != 0.0 ? ord[j - d] : 0, v, false);
        }
    }
    for (int j0 = 0; j0 < n; j0 += 32) {         // x_j = y_j / u_jj, in y_j's row
        const int j = j0 + lane, at = j < n ? j : 0;
        put(j < n, at, at, j < n ? -dinv_of(j) : 0.0, true);
    }
    // the border: rows n + a LS + l hold the partial sums of border row a, row n + r LS + i a product
    const T* vt = in.vt + (size_t)sys * r * n;
    for (int a = 0; a < r; ++a) {
        const int sum = n + a * LS;
        int e0 = 0;                              // union entries so far
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + lane;
            const bool in_union = j < n && in.mask[(size_t)a * n + j];
            const unsigned m = __ballot_sync(0xffffffffu, in_union);
            const int e = e0 + __popc(m & ((1u << lane) - 1)), l = e % LS;
            const double v = in_union ? real_part_of(vt[(size_t)a * n + j], phase_of(p, a) - phase_of(q, j), bad) : 0.0;
            // the first entry of each sum is fresh; LS entries at a time keep the sums' order
            for (int h = 0; h < 32; h += LS) {
                const bool mine = v != 0.0 && e - e0 >= h && e - e0 < h + LS;
                const bool fresh = mine && put.ready[sum + l] == 0;
                put(mine, mine ? j : 0, mine ? sum + l : 0, -v, fresh);
            }
            e0 += __popc(m);
        }
        for (int m = LS / 2; m > 0; m >>= 1) {   // the lanes' sums, halved: an empty one adds nothing
            const bool from = lane < m && put.ready[sum + lane + m] != 0, to = lane < m && put.ready[sum + lane] != 0;
            __syncwarp();
            put(from, from ? sum + lane + m : 0, from ? sum + lane : 0, -1.0, from && !to);
        }
        const bool none = put.ready[sum] == 0;   // no entry at all: the sum is 0
        __syncwarp();
        put(none && lane == 0, rows - 1, sum, 0.0, true);
    }
    // z = S^-1 v: row i of the small LU works on the sum that its pivoting puts there
    if (r > 0) {
        const T* S = in.slu + (size_t)sys * r * r;
        const int* spiv = in.s.spiv + (size_t)sys * r;
        __shared__ unsigned char order[kMaxBorder];
        if (lane == 0) {
            for (int i = 0; i < r; ++i) order[i] = (unsigned char)i;
            for (int k = 0; k < r; ++k) {
                const unsigned char t = order[k];
                order[k] = order[spiv[k]];
                order[spiv[k]] = t;
            }
        }
        __syncwarp();
        auto z = [&](int i) { return n + order[i] * LS; };
        // S_ab = i^{p_a - p_b}: L rows against pivot rows, 1 / u_ii, U rows against columns
        auto entry = [&](int i, int k) {
            const int pi = phase_of(p, order[i]), pk = phase_of(p, order[k]), ck = phase_of(p, k);
            return real_part_of(S[k * r + i], i > k ? pi - pk : (i == k ? ck - pi : pi - ck), bad);
        };
        // z_i -= round(s z_k): the product in a row of its own
        auto eliminate = [&](int k, int i, bool has) {
            const double v = has ? entry(i, k) : 0.0;
            const bool on = v != 0.0;
            const int t = n + r * LS + (on ? i : 0);
            put(on, on ? z(k) : 0, t, -v, true);
            put(on, t, on ? z(i) : 0, 1.0, false);
        };
        for (int k = 0; k < r; ++k)
            for (int i0 = k + 1; i0 < r; i0 += 32) eliminate(k, i0 + lane, i0 + lane < r);
        for (int k = r - 1; k >= 0; --k) {
            put(lane == 0, z(k), z(k), lane == 0 ? -entry(k, k) : 0.0, true);
            for (int i0 = 0; i0 < k; i0 += 32) eliminate(k, i0 + lane, i0 + lane < k);
        }
        // x_j -= W_jk z_k, k ascending: z_k is the k-th unknown
        const T* w = in.w + (size_t)sys * r * n;
        for (int k = 0; k < r; ++k)
            for (int j0 = 0; j0 < n; j0 += 32) {
                const int j = j0 + lane;
                const double v = j < n ? real_part_of(w[(size_t)k * n + j], phase_of(q, j) - phase_of(p, k), bad) : 0.0;
                put(v != 0.0, z(k), v != 0.0 ? j : 0, v, false);
            }
    }
    const int end = __reduce_max_sync(0xffffffffu, put.end);
    if (lane == 0) nslot[sys] = end;
    if (bad) stat[0] = 1;
    if (put.over) stat[1] = 1;
}

// unused operations name the last row, which stays zero
__global__ void k_flow_clear(unsigned char* data, size_t sb, int batch, int chunks, int chunk, int vbytes, unsigned none) {
    const size_t per = (size_t)chunks * (chunk / 4);
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < per * batch; e += (size_t)gridDim.x * blockDim.x) {
        const size_t sys = e / per, w = e - sys * per;
        reinterpret_cast<unsigned*>(data + sys * sb)[w] = (int)(w % (chunk / 4)) * 4 < vbytes ? 0u : none;
    }
}

// a system's first bytes, laid out closer
__global__ void k_flow_pack(const int4* __restrict__ in, size_t from, int4* __restrict__ out, size_t to, size_t total) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t sys = e / to;
        out[e] = in[sys * from + (e - sys * to)];
    }
}

// the FP32 copies: the same rows, the values rounded; `per` operations to a chunk
__global__ void k_flow_demote(const unsigned char* __restrict__ in, unsigned char* __restrict__ out, long long total, int per) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const long long g = e / per;
        const int i = (int)(e - g * per);
        const unsigned char* a = in + g * per * 12;
        unsigned char* b = out + g * per * 8;
        reinterpret_cast<float*>(b)[i] = (float)reinterpret_cast<const double*>(a)[i];
        reinterpret_cast<unsigned*>(b)[per + i] = reinterpret_cast<const unsigned*>(a)[2 * per + i];
    }
}

template <class T>
__global__ void k_flow_union(const T* __restrict__ vt, int batch, int rn, unsigned char* __restrict__ mask) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= rn) return;
    for (int k = blockIdx.y; k < batch; k += gridDim.y)
        if (!is_zero(vt[(size_t)k * rn + q])) {
            mask[q] = 1;                         // whichever block is first
            return;
        }
}

__global__ void k_flow_flags(int n, const int* perm, const unsigned char* rowp, const unsigned char* colp,
                             const unsigned char* flip_r, const unsigned char* flip_c, unsigned char* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = (unsigned char)(phase_of(rowp, i) | (flip_r ? flip_r[perm[i]] << 1 : 0));
    out[n + i] = (unsigned char)(phase_of(colp, i) | (flip_c ? flip_c[i] << 1 : 0));
}

// shared memory of a system: the ring, the vector; 16-byte multiples
static size_t flow_smem(int rows, int ncr, int elem) {
    return (size_t)kRing * flow_chunk(ncr, elem) + ((size_t)rows * ncr * elem + 15) / 16 * 16;
}

// One handle's build: its kernels are launched and their outcome fetched in separate calls, so that the
// builds of several handles run side by side (each takes a warp's latency, whatever its systems).
struct FlowBuild {
    FlowSource s;
    cudaStream_t st;
    std::unique_ptr<FlowForm> f = std::make_unique<FlowForm>();
    int* d = nullptr;                            // [batch] slots, the two verdicts, the union of V^T's entries
    int cap = 0, chunk = 0, per = 0;
    size_t smem = 0;
    bool large = false, counted = false;
    unsigned char* loose = nullptr;              // the operations at their most, once they are packed
    std::vector<int> h;

    FlowBuild(const FlowSource& src, cudaStream_t stream) : s(src), st(stream), h(src.batch + 2) {}
    FlowBuild(FlowBuild&& o) : s(o.s), st(o.st), f(std::move(o.f)), d(std::exchange(o.d, nullptr)), h(std::move(o.h)) {}
    ~FlowBuild() {
        dev_free(d);
        dev_free(loose);
    }
    static int blocks(size_t items) { return (int)std::min<size_t>((items + 255) / 256, 152 * 32); }

    template <bool COUNT>
    void launch(const FlowOut& o) {
        auto go = [&](auto zero) {
            using T = decltype(zero);
            ensure_smem_attr((const void*)k_flow_build<T, COUNT>, (int)kFlowSmem);
            const FlowIn<T> in{s, s.kl + s.ku, f->ncr, f->rows, cap, static_cast<const T*>(s.ab), static_cast<const T*>(s.vt),
                               static_cast<const T*>(s.w), static_cast<const T*>(s.slu),
                               reinterpret_cast<const unsigned char*>(d + s.batch + 2)};
            k_flow_build<T, COUNT><<<s.batch, 32, smem, st>>>(in, d, d + s.batch, o);
            CNG_LAUNCH("k_flow_build");
        };
        if (s.dtype) go(zd(0.0));
        else go(0.0);
    }
    void fetch() {
        CNG_CUDA(cudaMemcpyAsync(h.data(), d, sizeof(int) * h.size(), cudaMemcpyDeviceToHost, st));
        CNG_CUDA(cudaStreamSynchronize(st));
        if (h[s.batch]) throw InvalidArgument("scheduled solve: the factors are not real up to powers of i");
        if (h[s.batch + 1]) throw InvalidArgument("scheduled solve: too many operations per column");
        for (int k = 0; k < s.batch; ++k) h[k] = ceil_div(h[k], kSlots);
    }
    void begin() {
        const int n = s.n, r = s.r, B = s.batch;
        if (r > kMaxBorder || n > 32000) throw InvalidArgument("scheduled solve: too many border rows or columns");
        if (s.dtype && !s.rowp) throw InvalidArgument("scheduled solve: the systems are not real up to powers of i");
        f->n = n; f->batch = B; f->dtype = s.dtype; f->lanes = s.lanes;
        f->ncr = (s.dtype ? 2 : 1) * (s.flip_r ? 2 : 1);
        f->rows = n + r * s.lanes + r + 1;
        f->perm = s.in_order ? nullptr : s.perm;
        if (f->rows > 32000 || flow_smem(f->rows, f->ncr, 8) > kFlowSmem)
            throw InvalidArgument("scheduled solve: system too large for shared memory");
        const int ops = flow_ops(f->ncr);
        cap = std::min(65000, kFlowColumnBytes * (n + 64) / (12 * ops) / kSlots * kSlots);
        smem = (size_t)f->rows * 8 + (size_t)n * 7 + (size_t)cap * 3 + 2;
        if (smem > kFlowSmem) throw InvalidArgument("scheduled solve: system too large");
        const int rn = std::max(1, r * n);
        d = static_cast<int*>(dev_alloc(sizeof(int) * (B + 2) + rn));
        CNG_CUDA(cudaMemsetAsync(d, 0, sizeof(int) * (B + 2) + rn, st));
        unsigned char* mask = reinterpret_cast<unsigned char*>(d + B + 2);
        const dim3 grid(ceil_div(r * n, 64), std::min(B, 64));     // a zero entry is read in every system
        if (r && s.dtype) k_flow_union<zd><<<grid, 64, 0, st>>>(static_cast<const zd*>(s.vt), B, r * n, mask);
        else if (r) k_flow_union<double><<<grid, 64, 0, st>>>(static_cast<const double*>(s.vt), B, r * n, mask);
        CNG_LAUNCH("k_flow_union");
        chunk = flow_chunk(f->ncr, 8);
        per = kSlots * ops;
        f->chunks = ceil_div(cap, kSlots);
        large = (size_t)B * f->chunks * chunk > kFlowLoose;
        if (large && !s.most) {                  // at their most, packed below, where there is room
            try {
                f->data[0] = static_cast<unsigned char*>(dev_alloc((size_t)B * f->chunks * chunk));
            } catch (const DeviceMemoryFull&) {
            }
        }
        counted = large && !f->data[0];
        if (counted) launch<true>(FlowOut{});
    }
    void write() {
        const int n = s.n, B = s.batch;
        if (counted) {
            fetch();
            f->chunks = *std::max_element(h.begin(), h.begin() + B);
        }
        const size_t each = (size_t)f->chunks * (chunk + (s.fp32 ? flow_chunk(f->ncr, 4) : 0)) + 2 * (size_t)n + sizeof(int);
        if (s.most && each * B > s.most) throw InvalidArgument("scheduled solve: too much memory");
        FlowOut o{};
        f->row = o.row = static_cast<unsigned short*>(dev_alloc(2 * (size_t)B * n));
        f->flags = static_cast<unsigned char*>(dev_alloc(2 * (size_t)n));
        f->nchunk = static_cast<int*>(dev_alloc(sizeof(int) * B));
        k_flow_flags<<<ceil_div(n, 128), 128, 0, st>>>(n, s.perm, s.rowp, s.colp, s.flip_r, s.flip_c, f->flags);
        CNG_LAUNCH("k_flow_flags");
        f->sb[0] = o.sb = (size_t)f->chunks * chunk;
        if (!f->data[0]) f->data[0] = static_cast<unsigned char*>(dev_alloc(std::max<size_t>((size_t)B * o.sb, 16)));
        o.data = f->data[0];
        const size_t words = (size_t)B * o.sb / 4;
        if (words)
            k_flow_clear<<<blocks(words), 256, 0, st>>>(o.data, o.sb, B, f->chunks, chunk, per * 8,
                                                        (unsigned)(f->rows - 1) * 0x10001u);
        CNG_LAUNCH("k_flow_clear");
        launch<false>(o);
    }
    void pack() {                                // what was written at its most, where that saves half or more
        const size_t B = (size_t)s.batch;
        fetch();
        const int used = *std::max_element(h.begin(), h.begin() + B);
        if (!large || 2 * used > f->chunks) return;
        const size_t to = (size_t)used * chunk;
        loose = std::exchange(f->data[0], nullptr);
        f->data[0] = static_cast<unsigned char*>(dev_alloc(std::max<size_t>(B * to, 16)));
        if (used)
            k_flow_pack<<<blocks(B * to / 16), 256, 0, st>>>(reinterpret_cast<const int4*>(loose), f->sb[0] / 16,
                                                            reinterpret_cast<int4*>(f->data[0]), to / 16, B * to / 16);
        CNG_LAUNCH("k_flow_pack");
        f->sb[0] = to;
        f->chunks = used;
    }
    void finish() {
        const int B = s.batch;
        if (loose) {
            CNG_CUDA(cudaStreamSynchronize(st));
            dev_free(std::exchange(loose, nullptr));
        }
        if (s.fp32) {
            f->sb[1] = (size_t)f->chunks * flow_chunk(f->ncr, 4);
            f->data[1] = static_cast<unsigned char*>(dev_alloc(std::max<size_t>((size_t)B * f->sb[1], 16)));
            const long long total = (long long)B * f->chunks * per;
            if (total) k_flow_demote<<<blocks((size_t)total), 256, 0, st>>>(f->data[0], f->data[1], total, per);
            CNG_LAUNCH("k_flow_demote");
        }
        for (int k = 0; k < B; ++k) {
            f->used[0] += (size_t)h[k] * chunk;
            if (s.fp32) f->used[1] += (size_t)h[k] * flow_chunk(f->ncr, 4);
        }
        CNG_CUDA(cudaMemcpyAsync(f->nchunk, h.data(), sizeof(int) * B, cudaMemcpyHostToDevice, st));
        CNG_CUDA(cudaStreamSynchronize(st));
    }
};

// up to kMost streams beside `main`, ordered after its work
struct SideStreams {
    static constexpr int kMost = 7;
    cudaStream_t side[kMost] = {};
    int n = 0;
    SideStreams(int want, cudaStream_t main) {
        if (want <= 0) return;
        EventPair ev;
        CNG_CUDA(cudaEventRecord(ev.e0, main));
        for (; n < std::min(want, kMost); ++n) {
            CNG_CUDA(cudaStreamCreateWithFlags(&side[n], cudaStreamNonBlocking));
            const cudaError_t e = cudaStreamWaitEvent(side[n], ev.e0, 0);
            if (e != cudaSuccess) {
                for (int k = 0; k <= n; ++k) cudaStreamDestroy(side[k]);
                CNG_CUDA(e);
            }
        }
    }
    ~SideStreams() {
        for (int k = 0; k < n; ++k) cudaStreamDestroy(side[k]);
    }
};

// One warp a system takes 1.7 ms for n = 522, whatever the other handles do, and 3.0 where a handle has more
// systems than the SMs hold warps: channel 96 x 129 x 96, four handles (2209 systems the largest), 11.7 ms one
// after another and counted first, 6.5 side by side, 4.4 with the largest written at its most and packed.
std::vector<std::unique_ptr<FlowForm>> flow_build(const std::vector<FlowSource>& sources, cudaStream_t st) {
    const SideStreams side((int)sources.size() - 1, st);
    std::vector<FlowBuild> b;
    b.reserve(sources.size());
    for (size_t k = 0; k < sources.size(); ++k) {
        const int q = (int)(k % (side.n + 1));
        b.emplace_back(sources[k], q ? side.side[q - 1] : st);
    }
    struct Wait {                                // also where a build is refused with others in flight
        const std::vector<FlowBuild>& b;
        ~Wait() {
            for (const auto& x : b) cudaStreamSynchronize(x.st);
        }
    } wait{b};
    for (auto& x : b) x.begin();
    for (auto& x : b) x.write();
    for (auto& x : b) x.pack();
    for (auto& x : b) x.finish();
    std::vector<std::unique_ptr<FlowForm>> out;
    for (auto& x : b) out.push_back(std::move(x.f));
    return out;
}

// ---- solve ---------------------------------------------------------------------------------------
struct FlowArgs {
    int n, rows, ncr, batch, s0, s1;
    size_t sb;
    const unsigned char* data;
    const int *nchunk, *perm;
    const unsigned short* row;
    const unsigned char *in, *out;               // per row and column: phase | partner's sign << 1
    SolveIo io, io2;
};
struct FlowMulti {
    int nb;
    int start[kMaxGrp + 1];
    FlowArgs a[kMaxGrp];
};
__device__ __forceinline__ double flow_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float flow_fma(float a, float b, float c) { return fmaf(a, b, c); }

// A warp per system or shared pair. NCR: right-hand sides of a factor (1: real, 2: complex, 4: a pair)
template <class R, int NCR, int IO>
__device__ __forceinline__ void flow_body(const FlowArgs& a, int block, int smem_sys) {
    extern __shared__ __align__(16) unsigned char fsm[];
    constexpr int NC = NCR == 1 ? 1 : 2;         // components of an entry
    constexpr int OPS = flow_ops(NCR), CHB = flow_chunk(NCR, (int)sizeof(R));
    static_assert(CHB % 512 == 0, "a warp copies whole rows of a chunk");
    using V = std::conditional_t<NC == 1, double, std::conditional_t<sizeof(R) == 8, zd, zf>>;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int sys = a.s0 + block * ((int)blockDim.x / 32) + wib;
    if (sys >= a.s1) return;                     // the whole warp
    const int n = a.n;
    unsigned char* ring = fsm + (size_t)wib * smem_sys;
    R* y = reinterpret_cast<R*>(ring + kRing * CHB);
    const unsigned char* data = a.data + (size_t)sys * a.sb;
    const int nch = a.nchunk[sys];
    auto stage = [&](int c) {                    // one commit group per chunk
        if (c < nch) {
            const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(ring + (c % kRing) * CHB + lane * 16));
            const unsigned char* g = data + (size_t)c * CHB + lane * 16;
#pragma unroll
            for (int e = 0; e < CHB; e += 512)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + e), "l"(g + e) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int c = 0; c < kRing - 1; ++c) stage(c);
    // the right-hand sides, rows in solver order, times i^-p and the partner's signs
    constexpr int kU = 8;                        // rows in flight a lane
    const unsigned short* row = a.row + (size_t)sys * n;
    for (int i0 = lane; i0 < n; i0 += kU * 32) {
        int p[kU], at[kU];
        unsigned char fl[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = min(i0 + u * 32, n - 1);                // the last row again: the same value
            p[u] = a.perm ? a.perm[i] : i;
            at[u] = row[i];
            fl[u] = a.in[i];
        }
        V v[kU], v2[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            v2[u] = V(0.0);
            if constexpr (IO == IO_MIXED) {
                v[u] = to_zf(static_cast<const zd*>(a.io.rhs)[(size_t)sys * n + p[u]]);
                if (NCR == 4 && a.io2.rhs) v2[u] = to_zf(static_cast<const zd*>(a.io2.rhs)[(size_t)sys * n + p[u]]);
            } else {
                v[u] = io_load<V, IO>(a.io, sys, n, p[u]);
                if (NCR == 4 && a.io2.rhs) v2[u] = io_load<V, IO>(a.io2, sys, n, p[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if constexpr (NC == 1) {
                y[at[u]] = v[u];
            } else {
                reinterpret_cast<V*>(y)[at[u] * (NCR / 2)] = phase_in(v[u], fl[u] & 1);
                if constexpr (NCR == 4) reinterpret_cast<V*>(y)[at[u] * 2 + 1] = phase_in(fl[u] & 2 ? V(flip(v2[u].re), flip(v2[u].im)) : v2[u], fl[u] & 1);
            }
        }
    }
    if (lane < NCR) y[(a.rows - 1) * NCR + lane] = R(0);
    __syncwarp();
    // the operations, slot after slot
    {
        const int op = lane / NCR;
        R* yc = y + lane % NCR;
        const R* zero = yc + (a.rows - 1) * NCR;
        for (int c = 0; c < nch; ++c) {
            stage(c + kRing - 1);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(kRing - 1) : "memory");
            __syncwarp();
            const R* val = reinterpret_cast<const R*>(ring + (c % kRing) * CHB) + op;
            const unsigned* rows = reinterpret_cast<const unsigned*>(ring + (c % kRing) * CHB + kSlots * OPS * (int)sizeof(R)) + op;
            // addresses and value of the slot at hand; the next one's are made before this one's result is
            // there (the row words are read two slots ahead)
            const R *src, *add;
            R *dst, v;
            auto decode = [&](unsigned w, R x) {
                src = yc + (w & 0xffffu) * NCR;
                dst = yc + ((w >> 16) & 0x7fffu) * NCR;
                add = w & kFresh ? zero : dst;
                v = x;
            };
            unsigned w = rows[OPS];
            R x = val[OPS];
            decode(rows[0], val[0]);
#pragma unroll
            for (int s = 0; s < kSlots; ++s) {
                const R b = *src, d = *add, f = v;
                R* to = dst;
                __syncwarp();                    // a slot may write a row that its other operations read:
                                                 // every read first (no cost seen: 128 systems of n = 262
                                                 // 26.6 us without it, 26.7 with it)
                if (s + 1 < kSlots) decode(w, x);
                if (s + 2 < kSlots) {
                    w = rows[(s + 2) * OPS];
                    x = val[(s + 2) * OPS];
                }
                *to = flow_fma(f, b, d);
                __syncwarp();
            }
        }
    }
    // the solution, times i^q and the partner's signs, a lane per component
    const int comp = lane % NCR, im = comp & 1;
    const bool partner = comp >= 2;
    const SolveIo io = partner ? a.io2 : a.io;
    const size_t k0 = (size_t)sys * n;
    double* xs = static_cast<double*>(io.x) + (IO == IO_SPLIT ? 0 : im);
    for (int e0 = lane; e0 - lane < n * NCR; e0 += kU * 32) {
        unsigned char fl[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) fl[u] = a.out[min((e0 + u * 32) / NCR, n - 1)];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = min((e0 + u * 32) / NCR, n - 1);
            R v = y[i * NCR + comp];
            if constexpr (NC == 1) {
                if (e0 + u * 32 < n) io_store<double, IO>(a.io, sys, n, i, v);
            } else {
                const R other = __shfl_xor_sync(0xffffffffu, v, 1);
                if (fl[u] & 1) v = im ? other : flip(other);      // i x
                if (partner && fl[u] & 2) v = flip(v);
                if (e0 + u * 32 >= n * NCR || (partner && !io.x)) continue;
                if constexpr (IO == IO_SPLIT) {
                    xs[im ? io.cols_s[k0 + i] : io.cols[k0 + i]] = v;
                } else if constexpr (IO == IO_MIXED) {
                    double* w = xs + 2 * (k0 + i);
                    const double o = io.accumulate ? *w + (double)v : (double)v;
                    *w = o;
                    if (io.xT) static_cast<double*>(io.xT)[2 * ((size_t)i * a.batch + sys) + im] = o;
                } else {
                    const long long w = IO == IO_MAPPED && io.cols ? io.cols[k0 + i] : (long long)(k0 + i);
                    xs[2 * w] = v;
                }
            }
        }
    }
}

template <class R, int IO>
__global__ void __launch_bounds__(32 * kFlowWarps) k_solve_flow(const __grid_constant__ FlowMulti ms, int smem_sys) {
    int bk = 0;
    while (bk + 1 < ms.nb && (int)blockIdx.x >= ms.start[bk + 1]) ++bk;
    const FlowArgs& a = ms.a[bk];
    const int block = (int)blockIdx.x - ms.start[bk];
    if (a.ncr == 4) flow_body<R, 4, IO>(a, block, smem_sys);
    else flow_body<R, 2, IO>(a, block, smem_sys);
}
template <int IO>
__global__ void __launch_bounds__(32 * kFlowWarps) k_solve_flow_real(const __grid_constant__ FlowMulti ms, int smem_sys) {
    flow_body<double, 1, IO>(ms.a[0], (int)blockIdx.x, smem_sys);
}

template <class R, class Kernel>
static void launch_flow(const std::vector<FlowJob>& jobs, Kernel kernel, cudaStream_t st) {
    if (jobs.size() > (size_t)kMaxGrp) throw InvalidArgument("scheduled solve: at most 8 handles per launch");
    constexpr int V = sizeof(R) == 8 ? 0 : 1;
    FlowMulti ms{};
    ms.nb = (int)jobs.size();
    size_t smem = 0;
    int systems = 0;
    for (const auto& j : jobs) {
        if (!j.form->data[V]) throw InvalidArgument("scheduled solve: call cng_banded_make_fp32 first");
        smem = std::max(smem, flow_smem(j.form->rows, j.form->ncr, (int)sizeof(R)));
        systems += j.s1 - j.s0;
    }
    // systems of a block: the count that keeps the most warps resident on an SM, where there are that many
    int per = 1;
    auto resident = [&](int w) { return (int)(227 * 1024 / (w * smem + 1024)) * w; };
    for (int w = 2; w <= kFlowWarps; ++w)
        if (w * smem <= kFlowSmem && resident(w) > resident(per) && systems >= w * sm_count()) per = w;
    int total = 0;
    for (int k = 0; k < ms.nb; ++k) {
        const FlowForm& f = *jobs[k].form;
        ms.start[k] = total;
        ms.a[k] = FlowArgs{f.n, f.rows, f.ncr, f.batch, jobs[k].s0, jobs[k].s1, f.sb[V], f.data[V], f.nchunk, f.perm, f.row,
                           f.flags, f.flags + f.n, jobs[k].io, jobs[k].io2};
        total += ceil_div(jobs[k].s1 - jobs[k].s0, per);
    }
    ms.start[ms.nb] = total;
    if (total <= 0) return;
    ensure_smem_attr((const void*)kernel, (int)kFlowSmem);
    kernel<<<total, 32 * per, smem * per, st>>>(ms, (int)smem);
    CNG_LAUNCH("k_solve_flow");
}

template <int IO>
static void flow_io(const std::vector<FlowJob>& jobs, cudaStream_t st) {
    if (jobs[0].form->dtype == 0) {
        if constexpr (IO == IO_PLAIN || IO == IO_MAPPED) launch_flow<double>(jobs, k_solve_flow_real<IO>, st);
        else throw InvalidArgument("solve_split needs complex (complex128) factors");
    } else {
        using R = std::conditional_t<IO == IO_MIXED, float, double>;
        launch_flow<R>(jobs, k_solve_flow<R, IO>, st);
    }
}

void flow_solve(const std::vector<FlowJob>& jobs, int io_kind, cudaStream_t st) {
    switch (io_kind) {
        case IO_PLAIN: flow_io<IO_PLAIN>(jobs, st); break;
        case IO_MAPPED: flow_io<IO_MAPPED>(jobs, st); break;
        case IO_SPLIT: flow_io<IO_SPLIT>(jobs, st); break;
        default: flow_io<IO_MIXED>(jobs, st); break;
    }
}

}  // namespace cng
