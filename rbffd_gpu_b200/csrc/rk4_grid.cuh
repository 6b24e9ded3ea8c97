// Device-resident RK4 (included by rk4.cu): every step of an advance in one
// cooperative launch, one CTA per SM.
//
// CTA b owns a block of consecutive rows (grid_halo_whole: equal blocks, at most
// as many as SMs) and keeps, for the whole launch, its rows' weights and halo
// positions in shared memory -- as many of the stencils' 4-slot chunks as fit;
// the others are read from L2 in every stage, the first of them asked for before
// the wait below -- and its rows' u, accumulator and coefficients in registers.
// A stage is: gather from the halo buffer in shared memory, stage_update,
// publish the rows' next stage input, take the neighbours' values.  So a stage
// moves no weights that fit the SMs, and stages are separated by one exchange
// instead of a launch.
//
// The exchange needs no barrier across CTAs, flag or fence: a value travels with
// the number of its stage in one 8-byte (FP32) or 16-byte (FP64) word, written
// and read whole, and a reader polls the words of its own halo until each
// carries the stage it waits for.  Two buffers by the stage's parity: a CTA
// writes stage s + 2 over stage s only after it has the values of stage s + 1
// from every CTA that reads it, which those wrote after reading stage s (the
// host adds a word to the reader's list where only one of two CTAs reads the
// other).  Waits are bounded (GRID_POLL_LIMIT, a constant: as a parameter it cost
// stages 3 to 14%); a CTA whose wait runs out marks the launch as given up, on
// the device and for the host, and ends, as do the others when theirs run out,
// and every later launch on that state after its first stage.
//
// One lane per (row, tracer), slots in stencil order: the arithmetic of
// k_stage_scalar and k_stage_vec with one lane per row, bit for bit.
//
// What bounds it, in cycles of a stage read with clock64 (a busy warp's): a row's
// chain of gathers and multiply-adds with the update, then the exchange (a store to
// L2, polls until it is seen, a barrier).  642 nodes (n = 17, FP64): 820 and 1410;
// 4096 (31, three operators): 1340 and 1080 to 1280; 40003 (37, FP32): 2010 and 1290
// to 1400; 163842 (50, FP64), with the L2 reads of what does not fit: 17000 and 1700
// to 2000.  Where the per-stage kernels are faster is at grid_geom (rk4.cu).
#pragma once

constexpr int GRID_POLL_LIMIT = 1 << 21;  // polls of one word (about a second)

template <typename T>
struct GridParams {
    const int* rows;               // [blocks + 1] first row of each block
    const int* ptr;                // [blocks + 1] halo offsets
    const int* nodes;              // node at each halo position
    const unsigned short* lidx;    // sliced ELL: halo position of each slot
    const int* rptr;               // [blocks + 1] offsets into rnode / rpos
    const int* rnode;              // nodes read from other blocks
    const unsigned short* rpos;    // their halo positions
    const T* w[3];                 // the operators streamed (sliced ELL)
    const T* cu;
    const T* cv;
    T* u;                          // state [N][T_tr]
    float* comp;                   // compensated FP32 state, or nullptr
    void* word[2];                 // stage inputs with their stage numbers, by parity; before them grid_gave_up
    int* status;                   // host-mapped; DEV_STATUS_WAIT_TIMEOUT on a wait that ran out
    T c[4];                        // dt/2, dt/2, dt, dt/6
    T kappa;
    int nc, T_tr, R, cs, H, nr, nsteps;  // cs: chunks in shared memory; H: halo positions; nr: most words read
    unsigned tag;                  // stage number of the launch's first published stage
};

// Nonzero once a launch on these words gave up, for the launches that follow.  It
// lies GRID_HEAD bytes before the words, which stay on the allocation's 256-byte
// alignment: 16 bytes off it, stages took 3 to 30% longer.
constexpr int GRID_HEAD = 256;
__device__ __forceinline__ volatile int* grid_gave_up(void* word0) { return (volatile int*)((char*)word0 - GRID_HEAD); }

// One published value: value and stage number in a single access.
__device__ __forceinline__ void word_store(void* p, size_t i, double v, unsigned tag)
{
    asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"((char*)p + 16 * i),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)tag)
                 : "memory");
}
__device__ __forceinline__ bool word_load(const void* p, size_t i, unsigned tag, double& v)
{
    long long x;
    unsigned long long t;
    asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}"
                 : "=l"(x), "=l"(t)
                 : "l"((const char*)p + 16 * i)
                 : "memory");
    v = __longlong_as_double(x);
    return (unsigned)t == tag;
}
__device__ __forceinline__ void word_store(void* p, size_t i, float v, unsigned tag)
{
    const unsigned long long x = (unsigned long long)tag << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"((char*)p + 8 * i), "l"(x) : "memory");
}
__device__ __forceinline__ bool word_load(const void* p, size_t i, unsigned tag, float& v)
{
    unsigned long long x;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(x) : "l"((const char*)p + 8 * i) : "memory");
    v = __uint_as_float((unsigned)x);
    return (unsigned)(x >> 32) == tag;
}

// Four weights of a row's chunk in shared memory.  FP32: one 16-byte vector per
// row; FP64: two planes of 16-byte vectors, so that a warp's reads are
// consecutive.  off: the row's vector in the chunk; R: rows per plane.
__device__ __forceinline__ void grid_w4(const float* p, int off, int R, float (&w)[4]) { ld_w4_shared(p + 4 * off, w); }
__device__ __forceinline__ void grid_w4(const double* p, int off, int R, double (&w)[4])
{
    const double2 a = reinterpret_cast<const double2*>(p)[off], b = reinterpret_cast<const double2*>(p)[R + off];
    w[0] = a.x;
    w[1] = a.y;
    w[2] = b.x;
    w[3] = b.y;
}
__device__ __forceinline__ void grid_w4_put(float* p, int off, int R, const float (&w)[4])
{
    reinterpret_cast<float4*>(p)[off] = make_float4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void grid_w4_put(double* p, int off, int R, const double (&w)[4])
{
    reinterpret_cast<double2*>(p)[off] = make_double2(w[0], w[1]);
    reinterpret_cast<double2*>(p)[R + off] = make_double2(w[2], w[3]);
}

// Shared memory of a launch: weights and positions of cs chunks, two halo
// buffers (one position more, for words read only to order the exchange), the
// lists of words read.
template <typename T>
static size_t grid_smem(int K, int cs, int R, int H, int T_tr, int nr)
{
    return (size_t)cs * R * (4 * K * sizeof(T) + 8) + round_up((int)(2 * (size_t)(H + 1) * T_tr * sizeof(T)), 16) +
           (size_t)nr * 6 + 16;
}

// 32-bit registers of one chunk of one item: weights and four 16-bit positions.
__host__ __device__ constexpr int grid_chunk_regs(int K, int es) { return K * es + 2; }

// Chunks an item keeps in registers: only where two items per thread leave room
// (640 threads of at most 102 registers) and the weights do not fit shared
// memory anyway.  Small blocks gain nothing: with 255 registers the cosine
// bell's stage took 1.68 us against 1.42 us from shared memory, its one warp per
// SM waiting for the unrolled code instead.
__host__ __device__ constexpr int grid_reg_chunks(int K, int es, int ipt)
{
    return (ipt == 2 ? 24 : 0) / (ipt * grid_chunk_regs(K, es));
}

// One chunk of one item: halo positions and the operators' weights.
template <typename T, int K>
struct GridChunk {
    ushort4 l;
    T w[K][4];
};

// VEC consecutive values of a node record in shared memory.
template <typename T, int VEC>
__device__ __forceinline__ void grid_gather(const T* p, T (&x)[VEC])
{
    if constexpr (VEC == 1) {
        x[0] = *p;
    } else {
        typedef typename std::conditional<std::is_same<T, float>::value, float4, double2>::type V;
        static_assert(sizeof(V) == VEC * sizeof(T), "16-byte vectors");
        const V v = *reinterpret_cast<const V*>(p);
        memcpy(x, &v, sizeof(V));
    }
}

// VEC: tracers of one item (a row and VEC consecutive tracers: one, or a
// 16-byte vector, which shares the row's weights and positions); IPT: items per
// thread; MAXT: most threads.
template <typename T, int KIND, bool HV, int VEC, int IPT, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_rk4_grid(GridParams<T> gp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int K = KIND == KIND_HEAT ? 1 : (HV ? 3 : 2);
    constexpr int NREG = grid_reg_chunks(K, sizeof(T), IPT);
    // a streamed chunk in flight during the wait
    constexpr bool AHEAD = IPT * grid_chunk_regs(K, sizeof(T)) <= (MAXT > 640 ? 10 : 26);
    __shared__ int s_fail;
    const int R = gp.R, nc = gp.nc, TT = gp.T_tr, TV = TT / VEC;
    // a row's chunks in order: ns read from L2 in every stage, cs in shared memory, nr in registers
    const int nr = min(NREG, nc), cs = gp.cs, ns = nc - nr - cs;
    T* const hb = reinterpret_cast<T*>(smem_raw);                      // [2][(H + 1) T_tr]
    const int hstride = (gp.H + 1) * TT;
    T* const ws = reinterpret_cast<T*>(smem_raw + ((2 * (size_t)hstride * sizeof(T) + 15) & ~(size_t)15));  // [cs][K][R][4]
    ushort4* const lx = reinterpret_cast<ushort4*>(ws + (size_t)cs * K * R * 4);  // [cs][R]
    int* const rn = reinterpret_cast<int*>(lx + (size_t)cs * R);                  // [nr]
    unsigned short* const rp = reinterpret_cast<unsigned short*>(rn + gp.nr);     // [nr]
    const int b = blockIdx.x, tid = threadIdx.x, TH = blockDim.x;
    const int row0 = gp.rows[b], nrows = gp.rows[b + 1] - row0;  // row0 is a multiple of 32
    const int r0 = gp.rptr[b], nread = gp.rptr[b + 1] - r0;
    if (tid == 0) s_fail = *grid_gave_up(gp.word[0]);
    auto load = [&](int r, int c, GridChunk<T, K>& g) {
        const size_t o = sell_off(row0 + r, c, nc);
        g.l = __ldg(reinterpret_cast<const ushort4*>(gp.lidx + o));
#pragma unroll
        for (int k = 0; k < K; k++) ld_w4(gp.w[k] + o, g.w[k]);
    };
    for (int e = tid; e < cs * R; e += TH) {
        const int c = e / R, r = e - c * R;
        if (r < nrows) {
            GridChunk<T, K> g;
            load(r, ns + c, g);
            lx[e] = g.l;
#pragma unroll
            for (int k = 0; k < K; k++) grid_w4_put(ws + ((size_t)c * K + k) * R * 4, r, R, g.w[k]);
        }
    }
    for (int e = tid; e < nread; e += TH) {
        rn[e] = gp.rnode[r0 + e];
        rp[e] = gp.rpos[r0 + e];
    }
    const int h0 = gp.ptr[b], hn = gp.ptr[b + 1] - h0;
    for (int e = tid; e < hn * TT; e += TH) {
        const int h = e / TT;
        hb[e] = gp.u[(size_t)gp.nodes[h0 + h] * TT + (e - h * TT)];
    }
    // this thread's items
    T u[IPT][VEC], acc[IPT][VEC], cm[IPT][VEC], cu[IPT], cv[IPT];
    int own[IPT], rr[IPT], tt[IPT];  // halo element of the item's own values (-1: no item), its row and first tracer
    GridChunk<T, K> reg[IPT][NREG > 0 ? NREG : 1];
    GridChunk<T, K> ahead[AHEAD ? IPT : 1];
#pragma unroll
    for (int q = 0; q < IPT; q++) {
        const int it = tid + q * TH, r = it / TV, t = (it - r * TV) * VEC;
        const bool on = r < nrows;
        const int i = row0 + (on ? r : 0);
        rr[q] = on ? r : 0;  // an idle item beside a busy one works on row 0 and publishes nothing
        tt[q] = t;
        cu[q] = on && KIND == KIND_ADVECT ? gp.cu[i] : T(0);
        cv[q] = on && KIND == KIND_ADVECT ? gp.cv[i] : T(0);
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            u[q][v] = on ? gp.u[(size_t)i * TT + t + v] : T(0);
            acc[q][v] = T(0);
            cm[q][v] = T(0);
            if (std::is_same<T, float>::value && gp.comp && on) cm[q][v] = (T)gp.comp[(size_t)i * TT + t + v];
        }
        own[q] = on ? (int)gp.lidx[sell_off(i, 0, nc)] * TT + t : -1;  // the stencil's first slot is its centre
#pragma unroll
        for (int c = 0; c < NREG; c++)
            if (c < nr) load(rr[q], ns + cs + c, reg[q][c]);
        if (AHEAD && ns > 0) load(rr[q], 0, ahead[q]);
    }
    __syncthreads();
    bool live = false;  // warps without items only take neighbours' values
#pragma unroll
    for (int q = 0; q < IPT; q++) live |= own[q] >= 0;
    live = __any_sync(0xffffffffu, live);
    StageParams<T> p = {};
    p.kappa = gp.kappa;
    const int total = 4 * gp.nsteps;
    for (int st = 0; st < total; st++) {
        const int stage = st & 3;
        const T* const hin = hb + (st & 1) * hstride;
        T* const hout = hb + ((st & 1) ^ 1) * hstride;
        const unsigned tag = gp.tag + (unsigned)st;
        void* const word = gp.word[tag & 1];
        p.c = stage == 0 ? gp.c[0] : (stage == 1 ? gp.c[1] : (stage == 2 ? gp.c[2] : gp.c[3]));
        p.stage = stage;
        const bool publish = st + 1 < total;
        T d[IPT][3][VEC];
#pragma unroll
        for (int q = 0; q < IPT; q++)
#pragma unroll
            for (int v = 0; v < VEC; v++) d[q][0][v] = d[q][1][v] = d[q][2][v] = T(0);
        auto apply = [&](int q, const GridChunk<T, K>& g) {
            const T* const x = hin + tt[q];
            const int l[4] = {g.l.x, g.l.y, g.l.z, g.l.w};
            T xj[4][VEC];
#pragma unroll
            for (int s = 0; s < 4; s++) grid_gather<T, VEC>(x + l[s] * TT, xj[s]);
#pragma unroll
            for (int k = 0; k < K; k++)
#pragma unroll
                for (int s = 0; s < 4; s++)
#pragma unroll
                    for (int v = 0; v < VEC; v++) d[q][k][v] = Ar<T>::fma(g.w[k][s], xj[s][v], d[q][k][v]);
        };
        if (live) {
            if (AHEAD) {
#pragma unroll 2
                for (int c = 0; c < ns; c++) {
                    GridChunk<T, K> now[IPT];
#pragma unroll
                    for (int q = 0; q < IPT; q++) {
                        now[q] = ahead[AHEAD ? q : 0];
                        load(rr[q], c + 1 < ns ? c + 1 : 0, ahead[AHEAD ? q : 0]);  // the last: the next stage's first
                    }
#pragma unroll
                    for (int q = 0; q < IPT; q++) apply(q, now[q]);
                }
            } else {
                for (int c = 0; c < ns; c++)
#pragma unroll
                    for (int q = 0; q < IPT; q++) {
                        GridChunk<T, K> g;
                        load(rr[q], c, g);
                        apply(q, g);
                    }
            }
#pragma unroll(MAXT <= 256 ? 4 : 2)
            for (int c = 0; c < cs; c++)
#pragma unroll
                for (int q = 0; q < IPT; q++) {
                    GridChunk<T, K> g;
                    g.l = lx[c * R + rr[q]];
#pragma unroll
                    for (int k = 0; k < K; k++) grid_w4(ws + ((size_t)c * K + k) * R * 4, rr[q], R, g.w[k]);
                    apply(q, g);
                }
#pragma unroll
            for (int c = 0; c < NREG; c++)
                if (c < nr)
#pragma unroll
                    for (int q = 0; q < IPT; q++) apply(q, reg[q][c]);
        }
#pragma unroll
        for (int q = 0; q < IPT; q++)
            if (own[q] >= 0)
#pragma unroll
                for (int v = 0; v < VEC; v++) {
                    T next = T(0);
                    p.u = &u[q][v];
                    p.acc = &acc[q][v];
                    p.xnext = &next;
                    p.comp = std::is_same<T, float>::value && gp.comp && stage == 3 ? &cm[q][v] : nullptr;
                    stage_update<T, KIND, HV>(p, 0, 0, d[q][0][v], d[q][1][v], d[q][2][v], cu[q], cv[q]);
                    if (publish) {
                        const T x = stage == 3 ? u[q][v] : next;
                        word_store(word, (size_t)(row0 + rr[q]) * TT + tt[q] + v, x, tag);
                        hout[own[q] + v] = x;
                    }
                }
        if (!publish) break;
        // the neighbours' values of this stage: one word per thread, or four in flight
        bool late = false;
        const int words = nread * TT;
        if (words <= TH) {
            if (tid < words) {
                const int k = tid / TT, t = tid - k * TT;
                const size_t i = (size_t)rn[k] * TT + t;
                T v;
                int tries = 0;
                while (!word_load(word, i, tag, v))
                    if (++tries > GRID_POLL_LIMIT) {
                        late = true;
                        break;
                    }
                hout[rp[k] * TT + t] = v;
            }
        } else for (int e0 = tid; e0 < words && !late; e0 += 4 * TH) {
            size_t i[4];
            int h[4];
            T v[4];
            unsigned wait = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int e = e0 + j * TH;
                i[j] = 0;
                h[j] = 0;
                if (e < words) {
                    const int k = e / TT, t = e - k * TT;
                    i[j] = (size_t)rn[k] * TT + t;
                    h[j] = rp[k] * TT + t;
                    wait |= 1u << j;
                }
            }
            for (int tries = 0; wait; tries++) {
                if (tries > GRID_POLL_LIMIT) {
                    late = true;
                    break;
                }
                bool ok[4];
#pragma unroll
                for (int j = 0; j < 4; j++) ok[j] = (wait >> j & 1) && word_load(word, i[j], tag, v[j]);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (ok[j]) {
                        hout[h[j]] = v[j];
                        wait &= ~(1u << j);
                    }
            }
        }
        if (late) s_fail = 1;
        __syncthreads();
        if (s_fail) {
            if (tid == 0) {
                *grid_gave_up(gp.word[0]) = 1;
                *(volatile int*)gp.status = DEV_STATUS_WAIT_TIMEOUT;
            }
            return;
        }
    }
#pragma unroll
    for (int q = 0; q < IPT; q++)
        if (own[q] >= 0)
#pragma unroll
            for (int v = 0; v < VEC; v++) {
                const size_t e = (size_t)(row0 + rr[q]) * TT + tt[q] + v;
                gp.u[e] = u[q][v];
                if (std::is_same<T, float>::value && gp.comp) gp.comp[e] = (float)cm[q][v];
            }
}
