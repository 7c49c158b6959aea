// Product kernel for clustered plans (included by cbm_engine.cu inside its anonymous namespace): rows that
// name the same columns stand next to one another in the schedule, and are worked on by one SM at about the
// same time, so that most row pieces of X come from that SM's L1 instead of L2 or DRAM.
//
// One producer thread per block claims chunks of consecutive items and brings their descriptors and delta
// entries into shared memory with bulk copies, STAGES chunks ahead; the other warps take the chunk's items
// one by one (a shared-memory ticket), read descriptor and entries as broadcasts, and have only the
// operand rows themselves left to wait for: of the dependent round trips per row (claim, descriptor,
// entries, operand rows) one remains.  A warp that finds no item left in a stage gives it back and goes
// on to the next one, without a block-wide barrier.
//
// Forward progress is that of the items kernel: chunks are claimed in increasing order and a block hands out
// the items of its chunks in increasing order, so whoever the smallest unfinished item waits for has finished.
//
// Shared memory is kept small on purpose: the lines on their way in from L2 are held in what the SM's 256 KB
// leave to L1, and a third stage cost 10 - 20 %.

// acc += sum over the `len` entries at `ent` (shared memory, 16-byte aligned) of val * X[col, columns of this
// lane], UNROLL row fetches in flight per lane.  The entries are read as broadcasts, two per instruction.
template <int UNROLL>
__device__ __forceinline__ void gather_wide(const Entry* ent, i32 len, const char* xs, unsigned ldx_bytes,
                                            float4& acc) {
    using V = Vec<true>;
    const int4* e = reinterpret_cast<const int4*>(ent);
    i32 j = 0;
    for (; j + UNROLL <= len; j += UNROLL, e += UNROLL / 2) {
        float4 t[UNROLL];
        float w[UNROLL];
#pragma unroll
        for (int k = 0; k < UNROLL; k += 2) {
            const int4 q = e[k / 2];
            w[k] = __int_as_float(q.y);
            w[k + 1] = __int_as_float(q.w);
            t[k] = V::ld_ro(reinterpret_cast<const float*>(xs + (u64)(unsigned)q.x * ldx_bytes));
            t[k + 1] = V::ld_ro(reinterpret_cast<const float*>(xs + (u64)(unsigned)q.z * ldx_bytes));
        }
#pragma unroll
        for (int k = 0; k < UNROLL; ++k) acc = V::fma(w[k], t[k], acc);
    }
    const i32 live = len - j;
    if (live > 0) {  // the last, shorter batch: the surplus fetches are switched off
        float4 t[UNROLL];
        float w[UNROLL];
#pragma unroll
        for (int k = 0; k < UNROLL; k += 2) {
            int4 q = make_int4(0, 0, 0, 0);
            if (k < live) q = e[k / 2];  // an odd last entry is followed by one of weight 0
            w[k] = __int_as_float(q.y);
            w[k + 1] = __int_as_float(q.w);
            t[k] = V::ld_ro_if(reinterpret_cast<const float*>(xs + (u64)(unsigned)q.x * ldx_bytes), k < live);
            t[k + 1] = V::ld_ro_if(reinterpret_cast<const float*>(xs + (u64)(unsigned)q.z * ldx_bytes), k + 1 < live);
        }
#pragma unroll
        for (int k = 0; k < UNROLL; ++k) acc = V::fma(w[k], t[k], acc);
    }
}

// The same sum for slabs that 2^lg < 32 lanes cover with one vector each: 32 >> lg entries are fetched
// side by side, one per group of lanes, and the groups' sums are combined by shuffles at the end, so
// that every lane holds the total of its columns.  `xs` points at the columns of lane & (2^lg - 1).
template <int UNROLL>
__device__ __forceinline__ void gather_narrow(const Entry* ent, i32 len, const char* xs, unsigned ldx_bytes, int lg,
                                              float4& acc, int lane) {
    using V = Vec<true>;
    const i32 side = 32 >> lg;  // entries side by side
    for (i32 j = lane >> lg; j - (lane >> lg) < len; j += side * UNROLL) {
        float4 t[UNROLL];
        float w[UNROLL];
#pragma unroll
        for (int k = 0; k < UNROLL; ++k) {
            const bool on = j + k * side < len;
            int2 q = make_int2(0, 0);
            if (on) q = *reinterpret_cast<const int2*>(ent + j + k * side);
            w[k] = __int_as_float(q.y);
            t[k] = V::ld_ro_if(reinterpret_cast<const float*>(xs + (u64)(unsigned)q.x * ldx_bytes), on);
        }
#pragma unroll
        for (int k = 0; k < UNROLL; ++k) acc = V::fma(w[k], t[k], acc);
    }
    for (int d = 1 << lg; d < 32; d <<= 1) acc = V::add_xor(acc, d);
}

constexpr int CONSUMERS = 15;  // warps per block that compute; one more claims and copies
constexpr int STAGES = 2;
constexpr int MAX_CHUNK_ITEMS = 32;
constexpr int CHUNK_ENTRIES = 512;
constexpr int DESC_BYTES = MAX_CHUNK_ITEMS * (int)sizeof(RowDesc);
constexpr int STAGE_BYTES = DESC_BYTES + CHUNK_ENTRIES * (int)sizeof(Entry);

template <bool RAGGED, int UNROLL, int MINB>
__global__ void __launch_bounds__((CONSUMERS + 1) * 32, MINB) cbm_chunks_kernel(const __grid_constant__ KParams p) {
    cbm::wait_before();
    using V = Vec<true>;
    __shared__ __align__(128) unsigned char smem[STAGES * STAGE_BYTES];  // descriptors, entries of each stage
    __shared__ u64 s_bar[2 * STAGES];                                    // full, then empty
    __shared__ int4 s_info[STAGES];                                      // slab, first item, items, first entry
    __shared__ unsigned s_ticket[STAGES];
    const int lane = threadIdx.x & 31;
    const unsigned bars = smem_addr(s_bar);
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bars + 8 * s, 1);
            mbar_init(bars + 8 * (STAGES + s), CONSUMERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
    }
    __syncthreads();

    if (threadIdx.x >= CONSUMERS * 32) {  // producer
        if (lane != 0) return;
        for (unsigned seq = 0;; ++seq) {
            const unsigned st = seq % STAGES;
            const u64 t = atomicAdd(p.counter, 1ULL);
            const bool last = t >= (u64)p.n_claims;
            const i32 slab = last ? 0 : (i32)((unsigned)t / (unsigned)p.claims_per_slab);
            Chunk c{0, 0, 0, 0};
            if (!last) *reinterpret_cast<int4*>(&c) = __ldg(reinterpret_cast<const int4*>(p.chunks + ((i32)t - slab * p.claims_per_slab)));
            if (seq >= STAGES &&
                !mbar_wait(bars + 8 * (STAGES + st), ((seq / STAGES) + 1) & 1, p.status, 2 * p.wait_ns, true)) {
                // Nothing may still be on its way into this block's shared memory when it retires: the
                // stages that were filled last are waited for (bounded) before leaving.
                for (unsigned q = seq - STAGES; q < seq; ++q)
                    mbar_wait(bars + 8 * (q % STAGES), (q / STAGES) & 1, p.status, p.wait_ns);
                if (last) draw_last(p, t);
                else drain(p, 0);
                return;
            }
            s_info[st] = make_int4(slab, c.first, c.count, c.e0);
            s_ticket[st] = 0;
            if (last) {  // tells the consumers to leave; they have waited for every copy before this
                mbar_arrive(bars + 8 * st);
                draw_last(p, t);
                return;
            }
            unsigned char* at = smem + st * STAGE_BYTES;
            const unsigned n_desc = (unsigned)c.count * (unsigned)sizeof(RowDesc);
            const unsigned n_ent = (unsigned)c.ne * (unsigned)sizeof(Entry);
            mbar_expect_tx(bars + 8 * st, n_desc + n_ent);
            bulk_copy_g2s(smem_addr(at), p.desc + c.first, n_desc, bars + 8 * st);
            if (n_ent) bulk_copy_g2s(smem_addr(at + DESC_BYTES), p.ent + c.e0, n_ent, bars + 8 * st);
        }
    }

    unsigned st = 0, parity = 0;
    for (;;) {
        if (!mbar_wait(bars + 8 * st, parity, p.status, 2 * p.wait_ns, true)) return;
        if (s_info[st].z == 0) return;
        for (;;) {
            unsigned tk = 0;
            if (lane == 0) tk = atomicAdd(s_ticket + st, 1u);
            tk = __shfl_sync(0xffffffffu, tk, 0);
            if (tk >= (unsigned)s_info[st].z) break;
            // What is needed again after the fetches is read again after them: registers decide how many warps
            // are resident.
            const volatile RowDesc* d = reinterpret_cast<const RowDesc*>(smem + st * STAGE_BYTES) + tk;
            V::T acc[1];
            acc[0] = V::zero();
            {
                const i32 c0 = s_info[st].x * p.slab_w;
                const i32 wcols = min(p.slab_w, p.f - c0);
                const i32 len = (d->info >> ITEM_LEN_SHIFT) & 0xff;
                const Entry* ent = reinterpret_cast<const Entry*>(smem + st * STAGE_BYTES + DESC_BYTES) + (d->beg - s_info[st].w);
                const char* xs = reinterpret_cast<const char*>(p.x + c0);
                // Lanes without columns fetch those of the last lane that has some, so that no fetch needs a
                // predicate; their sums are not stored.
                if (wcols <= 16 * V::E) {
                    const int lg = lanes_log2<V::E>(wcols);
                    const i32 li = min(lane & ((1 << lg) - 1), (wcols - 1) / V::E);
                    gather_narrow<UNROLL>(ent, len, xs + li * (V::E * 4), p.ldx_bytes, lg, acc[0], lane);
                } else {
                    gather_wide<UNROLL>(ent, len, xs + 4 * V::E * min(lane, (wcols - 1) / V::E), p.ldx_bytes, acc[0]);
                }
            }
            const volatile int4* si = s_info + st;
            const i32 slab = si->x, c0 = slab * p.slab_w;
            const bool ok[1] = {lane * V::E < min(p.slab_w, p.f - c0)};
            if (!finish_item<1, true, RAGGED>(p, slab, si->y + (i32)tk, d->out_row, d->parent_row, d->parent_pos, d->info,
                                            d->first_part, d->scale, d->inv_parent, acc, ok, c0, lane))
                return;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + 8 * (STAGES + st));
        if (++st == STAGES) {
            st = 0;
            parity ^= 1;
        }
    }
}
