// kc_part.cu -- the partition of a job's k-mers into 256 buckets: the FASTQ
// tiles are read once, every window of k valid bases becomes its canonical
// k-mer, and the k-mers are scattered by their first four bases (as string
// keys, for the counting by printed-order prefix) or by root prefix (as k-mer
// words, the reference's get_root_prefix, for global-memory tables; k <= 32).
#include <algorithm>

#include "kc_device.cuh"
#include "kc_kernels.cuh"
#include "kc_wide.cuh"

namespace kc {

namespace {

constexpr uint32_t FULLW = 0xffffffffu;
constexpr uint32_t PT_THREADS = 256;                 // one 32-byte segment per thread
constexpr uint32_t PT_BUF = TILE + HALO;             // 8224, a multiple of 16
constexpr uint32_t PT_SEGS = PT_THREADS + 1;         // the halo segment first
constexpr uint32_t PT_CHUNK = 16;                    // positions a thread rolls along
constexpr uint32_t PT_STAGE = PT_THREADS * PT_CHUNK; // most k-mers of a round

struct PartSmem {
    uint8_t tile[PT_BUF];
    unsigned long long codes[PT_SEGS + 7];   // 2-bit codes of a segment's bytes
    uint32_t good[PT_SEGS + 7];              // valid bases in sequence lines
    uint32_t chunk[2 * PT_THREADS];          // chunks holding window ends
    unsigned long long stage[PT_STAGE];      // a round's k-mers in bucket order
};

// Sum of the first `warp` of eight values.
__device__ __forceinline__ uint32_t sum_before(const uint32_t *s, int warp, uint32_t &total)
{
    const uint4 a = *reinterpret_cast<const uint4 *>(s), b = *reinterpret_cast<const uint4 *>(s + 4);
    const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        before += w < warp ? v[w] : 0u;
        all += v[w];
    }
    total = all;
    return before;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULLW, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// One tile per block at a time.  Bytes are classified per 32-byte segment;
// the 16-position chunks holding window ends are listed (header and quality
// lines have none), and a thread rolls the forward and reverse-complement
// words along one chunk, keeping its k-mers in registers while their ranks in
// their buckets come from shared-memory counters.  The k-mers are then
// written once to shared memory, in bucket order, and from there in runs of
// one bucket.  The next tile's bytes arrive while this one's k-mers are formed
// and written (the tile buffer is free once classified).
//
// String keys are rolled as complements, so that the smaller of the two is the
// key itself.
//
// Bound by instruction issue (57%) and shared-memory wavefronts (57%).  A
// kernel that staged the k-mers unsorted in shared memory first (stores 64
// bytes apart, 16 to a bank), rolled chunks of 8 with 64-bit shifts by variable
// amounts, read the file's data and line numbers when a tile had arrived and
// checked every k-mer against its bucket's region took 172 warp instructions
// per 32 k-mers at three blocks per SM, this one 117 at four: 2.4G k-mers of
// 150-base reads 21.2 -> 13.3 ms, 480M 4.25 -> 2.67, 25M 0.23 -> 0.15.
//
// BY: what a bucket is (PartBy).  By sample all k-mers of a tile have one
// bucket, and their places follow from a scan of the threads' counts.
// W: k > 16 (words reach into both halves; below, the upper half holds all).
// By sample k differs from tile to tile, and W tells every case apart itself.
template <int BY, bool W>
__global__ void __launch_bounds__(PT_THREADS, 4) k_part(ExtractArgs a)
{
    constexpr bool STRING = BY != PART_BY_ROOT, SAMPLE = BY == PART_BY_SAMPLE;
    extern __shared__ __align__(128) uint8_t pt_smem[];
    PartSmem &s = *reinterpret_cast<PartSmem *>(pt_smem);
    __shared__ __align__(8) uint64_t mbar;
    __shared__ __align__(16) uint32_t s_wnl[8], s_wbk[8];
    __shared__ uint32_t s_hist[N_BUCKETS], s_start[N_BUCKETS], s_lim[N_BUCKETS];
    __shared__ unsigned long long *s_ptr[N_BUCKETS];
    __shared__ uint32_t s_nch, s_over;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint64_t u = blockIdx.x;
    if (u >= a.n_tiles) return;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (tid == 0) {
        mbar_init(&mbar, 1);
        fence_mbar_init();
        s_over = 0;
    }
    s_hist[tid] = 0;
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&mbar, PT_BUF);
        bulk_load(s.tile, a.buf + (a.tile0 + u) * TILE - HALO, PT_BUF, &mbar);
    }
    const uint32_t blo = a.bucket_lo, bhi = a.bucket_hi ? a.bucket_hi : N_BUCKETS;
    const bool all_buckets = blo == 0 && bhi == N_BUCKETS;
    // the file a tile lies in and its first line's number (mod 4 is all that
    // counts) are read a tile ahead; the file's own data when it changes
    uint32_t seg_next = a.tile_seg[a.tile0 + u], seg_cur = 0xFFFFFFFFu;
    uint32_t line_next = (uint32_t)a.tile_prefix[a.tile0 + u], line_file = 0, k = 0, sample = 0;
    uint64_t first_tile = 0;
    for (uint32_t iter = 0; u < a.n_tiles; u += gridDim.x, ++iter) {
        const uint64_t t = a.tile0 + u;
        if (tid == 0) s_nch = 0;
        if (seg_next != seg_cur) {
            seg_cur = seg_next;
            first_tile = a.segs[seg_cur].first_tile;
            k = a.segs[seg_cur].k;
            if (SAMPLE) sample = a.segs[seg_cur].sample - a.sample0;
            line_file = (uint32_t)a.tile_prefix[first_tile];
        }
        const uint32_t line0 = line_next - line_file;
        const bool ok = mbar_wait(&mbar, iter & 1);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(&a.counters[C_FLAGS], ERR_WAIT_TIMEOUT);
            return;
        }
        const bool first = t == first_tile;
        const uint32_t fs = 64 - 2 * k;

        // ---- segments: codes, valid bases, lines
        uint64_t codes;
        uint32_t valid, nl;
        classify32(s.tile + HALO + 32 * tid, codes, valid, nl);
        const uint32_t own_nl = (uint32_t)__popc(nl);
        const uint32_t inc_nl = warp_inclusive(own_nl, lane);
        if (lane == 31) s_wnl[warp] = inc_nl;
        s.codes[tid + 1] = codes;
        if (warp == 0) {
            // the halo segment (the end of the file's previous tile), a byte per lane
            const uint32_t b = s.tile[lane], up = b & 0xDFu;
            const bool v = up == 'A' || up == 'C' || up == 'G' || up == 'T' || up == 'U';
            const uint32_t c = ((up >> 1) & 3u) ^ ((up >> 2) & 1u);
            const uint32_t hn = __ballot_sync(FULLW, b == '\n'), hv = __ballot_sync(FULLW, v);
            const uint32_t lo = __reduce_or_sync(FULLW, lane < 16 ? c << (2 * lane) : 0u);
            const uint32_t hi = __reduce_or_sync(FULLW, lane >= 16 ? c << (2 * (lane - 16)) : 0u);
            if (lane == 0) {
                s.codes[0] = ((uint64_t)hi << 32) | lo;
                s.good[0] = first ? 0u : hv & line_mask(line0 - (uint32_t)__popc(hn), hn, 1);
            }
        }
        __syncthreads();
        uint32_t tot_nl;
        const uint32_t before_nl = sum_before(s_wnl, warp, tot_nl);
        s.good[tid + 1] = valid & line_mask(line0 + before_nl + inc_nl - own_nl, nl, 1);
        __syncthreads();
        // classified: the tile buffer takes the next tile
        if (u + gridDim.x < a.n_tiles) {
            if (tid == 0) {
                fence_proxy_async_smem();
                mbar_expect_tx(&mbar, PT_BUF);
                bulk_load(s.tile, a.buf + (t + gridDim.x) * TILE - HALO, PT_BUF, &mbar);
            }
            seg_next = a.tile_seg[t + gridDim.x];
            line_next = (uint32_t)a.tile_prefix[t + gridDim.x];
        }

        // ---- chunks holding ends of windows of k valid bases, in any order
        const uint32_t ends = run_ends((uint64_t)s.good[tid] | ((uint64_t)s.good[tid + 1] << 32), k);
        {
            const uint32_t e0 = ends & 0xFFFFu, e1 = ends >> 16;
            const uint32_t b0 = __ballot_sync(FULLW, e0 != 0), b1 = __ballot_sync(FULLW, e1 != 0);
            uint32_t at = 0;
            if (lane == 0 && (b0 | b1)) at = atomicAdd(&s_nch, (uint32_t)(__popc(b0) + __popc(b1)));
            at = __shfl_sync(FULLW, at, 0);
            if (e0) s.chunk[at + (uint32_t)__popc(b0 & lt)] = ((uint32_t)tid << 17) | e0;
            if (e1) s.chunk[at + (uint32_t)(__popc(b0) + __popc(b1 & lt))] = ((uint32_t)tid << 17) | 0x10000u | e1;
        }
        __syncthreads();
        const uint32_t n_ch = s_nch;
        const uint64_t topmask = k >= 32 ? ~0ULL : ~0ULL << fs;
        const uint32_t tm_hi = (uint32_t)(topmask >> 32), tm_lo = (uint32_t)topmask;

        for (uint32_t r0 = 0; r0 < n_ch; r0 += PT_THREADS) {
            uint32_t e = 0;
            uint32_t kh[PT_CHUNK], kl[PT_CHUNK], rk[PT_CHUNK / 2];
            if (r0 + tid < n_ch) {
                const uint32_t ch = s.chunk[r0 + tid];
                e = ch & 0xFFFFu;
                const uint32_t sgm = ch >> 17;
                const uint64_t prev = s.codes[sgm], cur = s.codes[sgm + 1];
                const bool half = (ch & 0x10000u) != 0;
                // the window ending just before the chunk: forward word (base
                // i at bit 64-2k+2i, stale bits below) and, from it, the
                // reverse complement's; for string keys the complements of both
                const uint32_t cw = half ? (uint32_t)(cur >> 32) : (uint32_t)cur;   // the chunk's 16 codes
                uint32_t fh = half ? (uint32_t)cur : (uint32_t)(prev >> 32);
                uint32_t fl = half ? (uint32_t)(prev >> 32) : (uint32_t)prev;
                const uint64_t rev = pair_reverse(((uint64_t)fh << 32) | fl) << fs;
                const uint64_t rc0 = STRING ? rev : ~rev & topmask;
                uint32_t rh = (uint32_t)(rc0 >> 32), rl = (uint32_t)rc0;
                const uint32_t fw = STRING ? ~cw : cw;   // the forward word's codes, the reverse one's are their complements
                if (STRING) {
                    fh = ~fh;
                    fl = ~fl;
                }
                // the reverse word's codes at the bits where the roll takes them
                // in (by sample with k <= 16 that is the upper half)
                const bool upper = SAMPLE && fs >= 32;
                const uint32_t in_sh = !W || upper ? fs - 32 : fs;
                const uint64_t nc = (uint64_t)(~fw) << in_sh;
                const uint32_t nc_hi = (uint32_t)(nc >> 32), nc_lo = (uint32_t)nc;
                const uint32_t in_mask = 3u << in_sh;
#pragma unroll
                for (uint32_t p = 0; p < PT_CHUNK; ++p) {
                    const uint32_t in = __funnelshift_r(nc_lo, nc_hi, 2 * p) & in_mask;
                    if (SAMPLE) {
                        fl = __funnelshift_r(fl, fh, 2);
                        rh = __funnelshift_l(rl, rh, 2) | (upper ? in : 0u);
                        rl = (rl << 2) | (upper ? 0u : in);
                    } else if (W) {
                        fl = __funnelshift_r(fl, fh, 2);
                        rh = __funnelshift_l(rl, rh, 2);
                        rl = (rl << 2) | in;
                    } else {
                        rh = (rh << 2) | in;
                    }
                    fh = __funnelshift_r(fh, fw >> (2 * p), 2);
                    // the canonical word is the smaller one; the string key of
                    // the canonical strand is the complement of the larger one:
                    // the smaller complement
                    const uint32_t xh = W && !SAMPLE ? fh : fh & tm_hi, xl = W ? fl & tm_lo : 0u;
                    const bool less = W ? (((uint64_t)xh << 32) | xl) < (((uint64_t)rh << 32) | rl) : xh < rh;
                    kh[p] = less ? xh : rh;
                    kl[p] = W ? (less ? xl : rl) : 0u;
                }
                if (!SAMPLE && !all_buckets) {
#pragma unroll
                    for (uint32_t p = 0; p < PT_CHUNK; ++p) {
                        const uint32_t b = kh[p] >> 24;
                        if (b < blo || b >= bhi) e &= ~(1u << p);
                    }
                }
                if (!SAMPLE) {
#pragma unroll
                    for (uint32_t p = 0; p < PT_CHUNK; ++p) {
                        uint32_t r = 0;
                        if ((e >> p) & 1u) r = atomicAdd(&s_hist[kh[p] >> 24], 1u);
                        if (p & 1) rk[p / 2] |= r << 16;
                        else rk[p / 2] = r;
                    }
                }
            }
            if (SAMPLE) {
                const uint32_t own = (uint32_t)__popc(e), inc = warp_inclusive(own, lane);
                if (lane == 31) s_wbk[warp] = inc;
                __syncthreads();
                uint32_t n;
                uint32_t at = sum_before(s_wbk, warp, n) + inc - own;
                if (tid == 0) {
                    const unsigned long long cur = a.bucket_base[sample] + atomicAdd(&a.bucket_cursor[sample], (unsigned long long)n);
                    const unsigned long long end = a.bucket_end[sample] < a.list_cap ? a.bucket_end[sample] : a.list_cap;
                    s_ptr[0] = a.list + cur;
                    s_lim[0] = cur >= end ? 0u : (uint32_t)(end - cur < n ? end - cur : n);
                }
#pragma unroll
                for (uint32_t p = 0; p < PT_CHUNK; ++p)
                    if ((e >> p) & 1u) s.stage[at++] = ((unsigned long long)kh[p] << 32) | kl[p];
                __syncthreads();
                const uint32_t lim = s_lim[0];
                unsigned long long *out = s_ptr[0];
                for (uint32_t i = tid; i < lim; i += PT_THREADS) out[i] = s.stage[i];
                if (r0 + PT_THREADS < n_ch) __syncthreads();
                continue;
            }
            __syncthreads();
            // bucket starts; the cursor update is in flight while the k-mers
            // are placed
            const uint32_t c = s_hist[tid];
            s_hist[tid] = 0;
            const unsigned long long cur = c ? atomicAdd(&a.bucket_cursor[tid], (unsigned long long)c) : 0ull;
            const uint32_t inc = warp_inclusive(c, lane);
            if (lane == 31) s_wbk[warp] = inc;
            __syncthreads();
            uint32_t n;
            const uint32_t start = sum_before(s_wbk, warp, n) + inc - c;
            s_start[tid] = start;
            __syncthreads();
#pragma unroll
            for (uint32_t p = 0; p < PT_CHUNK; ++p)
                if ((e >> p) & 1u)
                    s.stage[s_start[kh[p] >> 24] + ((rk[p / 2] >> (16 * (p & 1))) & 0xFFFFu)] =
                        ((unsigned long long)kh[p] << 32) | kl[p];
            // sorted index i of bucket b goes to s_ptr[b] + i; a bucket that
            // outgrows its estimated region is reported by its cursor and
            // redone, and only its region's part is written
            if (c) {
                const unsigned long long at = a.bucket_base[tid] + cur;
                const unsigned long long end = a.bucket_end[tid] < a.list_cap ? a.bucket_end[tid] : a.list_cap;
                s_ptr[tid] = a.list + at - start;
                s_lim[tid] = start + (uint32_t)(at >= end ? 0ull : (end - at < c ? end - at : c));
                if (at + c > end) s_over = 1;
            }
            __syncthreads();
            if (!s_over) {
#pragma unroll 4
                for (uint32_t i = tid; i < n; i += PT_THREADS) {
                    const unsigned long long key = s.stage[i];
                    s_ptr[key >> 56][i] = key;
                }
            } else {
                for (uint32_t i = tid; i < n; i += PT_THREADS) {
                    const unsigned long long key = s.stage[i];
                    const uint32_t b = (uint32_t)(key >> 56);
                    if (i < s_lim[b]) s_ptr[b][i] = key;
                }
            }
            if (r0 + PT_THREADS < n_ch) __syncthreads();   // another round: its ranks and stage follow
        }
        // s_over stays set: the launch is redone as a whole
    }
}

// k = 33..128: the same partition of kmer<N> string keys, N = 2 or 4 words.
// The tile comes with the 128 bytes before it; a chunk is 16 / N positions, so
// that a thread's k-mers fill as many registers as above.  A window's words
// are rolled one base at a time: the forward array (newest base at the top of
// word 0, older ones towards word LAST) moves down by two bits across its
// words, the reverse complement (first base's complement at the top of word 0)
// up.  The canonical array is the lexicographically smaller one
// (src/GetKmer.h:181-206), and the string key of its strand is the complement
// of the other, larger one, word by word, as for one word.
//
// CENSUS: only every (bucket_sample_mask + 1)-th tile is read and its k-mers
// are counted per bucket (and in *occ), not written.
constexpr uint32_t WP_HALO_SEGS = WIDE_HALO / 32;
constexpr uint32_t WP_SEGS = PT_THREADS + WP_HALO_SEGS;
constexpr uint32_t WP_BUF = TILE + WIDE_HALO;   // 8320, a multiple of 16

struct WidePartSmem {
    uint8_t tile[WP_BUF];
    unsigned long long codes[WP_SEGS + 4], rcodes[WP_SEGS + 4];   // rcodes: complemented codes, first at the top
    uint32_t good[WP_SEGS + 4];
    uint32_t chunk[8 * PT_THREADS];
    unsigned long long stage[PT_STAGE];   // PT_STAGE / N keys
};

template <uint32_t N, uint32_t LAST, bool CENSUS>
__global__ void __launch_bounds__(PT_THREADS, 3) k_part_wide(ExtractArgs a)
{
    constexpr uint32_t CH = 16 / N, PER_SEG = 32 / CH;   // positions of a chunk, chunks of a segment
    extern __shared__ __align__(128) uint8_t pt_smem[];
    WidePartSmem &s = *reinterpret_cast<WidePartSmem *>(pt_smem);
    __shared__ __align__(8) uint64_t mbar;
    __shared__ __align__(16) uint32_t s_wnl[8], s_wbk[8];
    __shared__ uint32_t s_hist[N_BUCKETS], s_start[N_BUCKETS], s_lim[N_BUCKETS];
    __shared__ unsigned long long *s_ptr[N_BUCKETS];
    __shared__ uint32_t s_nch, s_over;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t step = CENSUS ? a.bucket_sample_mask + 1 : 1;   // tiles between two visited ones
    const uint64_t n_visit = (a.n_tiles + step - 1) / step;
    uint64_t u = blockIdx.x;
    if (u >= n_visit) return;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (tid == 0) {
        mbar_init(&mbar, 1);
        fence_mbar_init();
        s_over = 0;
        s.codes[WP_SEGS] = 0;
        s.rcodes[WP_SEGS] = 0;
    }
    s_hist[tid] = 0;
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&mbar, WP_BUF);
        bulk_load(s.tile, a.buf + u * step * TILE - WIDE_HALO, WP_BUF, &mbar);
    }
    const uint32_t blo = a.bucket_lo, bhi = a.bucket_hi ? a.bucket_hi : N_BUCKETS;
    const bool all_buckets = blo == 0 && bhi == N_BUCKETS;
    uint32_t seg_next = a.tile_seg[u * step], seg_cur = 0xFFFFFFFFu;
    uint32_t line_next = (uint32_t)a.tile_prefix[u * step], line_file = 0, k = 0;
    uint64_t first_tile = 0;
    unsigned long long n_occ = 0;
    for (uint32_t iter = 0; u < n_visit; u += gridDim.x, ++iter) {
        const uint64_t t = u * step;
        if (tid == 0) s_nch = 0;
        if (seg_next != seg_cur) {
            seg_cur = seg_next;
            first_tile = a.segs[seg_cur].first_tile;
            k = a.segs[seg_cur].k;
            line_file = (uint32_t)a.tile_prefix[first_tile];
        }
        const uint32_t line0 = line_next - line_file;
        const bool ok = mbar_wait(&mbar, iter & 1);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(&a.counters[C_FLAGS], ERR_WAIT_TIMEOUT);
            return;
        }
        const bool first = t == first_tile;
        const uint32_t rem = k % 32, fs = rem ? 64 - 2 * rem : 0;   // unused low bits of word LAST
        const uint64_t back_mask = ~0ULL << fs;

        // ---- segments: codes, valid bases, lines
        uint64_t codes;
        uint32_t valid, nl;
        classify32(s.tile + WIDE_HALO + 32 * tid, codes, valid, nl);
        const uint32_t own_nl = (uint32_t)__popc(nl);
        const uint32_t inc_nl = warp_inclusive(own_nl, lane);
        if (lane == 31) s_wnl[warp] = inc_nl;
        s.codes[WP_HALO_SEGS + tid] = codes;
        s.rcodes[WP_HALO_SEGS + tid] = pair_reverse(~codes);
        if (warp == 7) {
            // the halo: the end of the file's previous tile (nothing for a
            // file's first one); line numbers counted back from the tile's first
            uint64_t hc = 0;
            uint32_t hv = 0, hn = 0;
            if (lane < (int)WP_HALO_SEGS && !first) classify32(s.tile + 32 * lane, hc, hv, hn);
            uint32_t x = (uint32_t)__popc(hn);
            x += __shfl_down_sync(FULLW, x, 1);
            x += __shfl_down_sync(FULLW, x, 2);   // lane j: newlines of halo segments j..3
            if (lane < (int)WP_HALO_SEGS) {
                s.codes[lane] = hc;
                s.rcodes[lane] = pair_reverse(~hc);
                s.good[lane] = first ? 0u : hv & line_mask(line0 - x, hn, 1);
            }
        }
        __syncthreads();
        uint32_t tot_nl;
        const uint32_t before_nl = sum_before(s_wnl, warp, tot_nl);
        s.good[WP_HALO_SEGS + tid] = valid & line_mask(line0 + before_nl + inc_nl - own_nl, nl, 1);
        __syncthreads();
        if (u + gridDim.x < n_visit) {
            const uint64_t tn = t + (uint64_t)gridDim.x * step;
            if (tid == 0) {
                fence_proxy_async_smem();
                mbar_expect_tx(&mbar, WP_BUF);
                bulk_load(s.tile, a.buf + tn * TILE - WIDE_HALO, WP_BUF, &mbar);
            }
            seg_next = a.tile_seg[tn];
            line_next = (uint32_t)a.tile_prefix[tn];
        }

        // ---- window ends: k > 32, so a window that ends in this segment
        // holds all its positions before that, and as many before it as are
        // missing to k
        uint32_t ends = 0;
        {
            const uint32_t g = s.good[WP_HALO_SEGS + tid];
            uint32_t run = 0;
            bool open = true;
#pragma unroll
            for (uint32_t j = 1; j <= WP_HALO_SEGS; ++j) {
                const uint32_t gj = s.good[WP_HALO_SEGS + tid - j];
                if (open) run += gj == FULLW ? 32u : (uint32_t)__clz(~gj);
                open = open && gj == FULLW;
            }
            const uint32_t lead = g == FULLW ? 32u : (uint32_t)__ffs(~g) - 1u;   // valid bases the segment starts with
            const uint32_t from = k - 1 > run ? k - 1 - run : 0u;
            if (from < lead) ends = range_mask(from, lead);
        }
        n_occ += (unsigned long long)__popc(ends);
        {
            uint32_t cnt = 0, b[PER_SEG];
#pragma unroll
            for (uint32_t q = 0; q < PER_SEG; ++q) {
                b[q] = __ballot_sync(FULLW, (ends >> (CH * q)) & ((1u << CH) - 1u));
                cnt += (uint32_t)__popc(b[q]);
            }
            uint32_t at = 0;
            if (lane == 0 && cnt) at = atomicAdd(&s_nch, cnt);
            at = __shfl_sync(FULLW, at, 0);
#pragma unroll
            for (uint32_t q = 0; q < PER_SEG; ++q) {
                const uint32_t e = (ends >> (CH * q)) & ((1u << CH) - 1u);
                if (e) s.chunk[at + (uint32_t)__popc(b[q] & lt)] = ((uint32_t)tid << 16) | (q << 8) | e;
                at += (uint32_t)__popc(b[q]);
            }
        }
        __syncthreads();
        const uint32_t n_ch = s_nch;

        for (uint32_t r0 = 0; r0 < n_ch; r0 += PT_THREADS) {
            uint32_t e = 0;
            unsigned long long key[CH][N];
            uint32_t rk[CH];
            if (r0 + tid < n_ch) {
                const uint32_t ch = s.chunk[r0 + tid];
                e = ch & 0xFFu;
                const uint32_t p0 = 32 * (WP_HALO_SEGS + (ch >> 16)) + CH * ((ch >> 8) & 0xFFu);   // the chunk's first position
                // the window ending just before the chunk
                uint64_t f[LAST + 1], r[LAST + 1];
#pragma unroll
                for (uint32_t w = 0; w <= LAST; ++w) {
                    const uint32_t en = p0 - 1 - 32 * w, es = en >> 5, eo = en & 31;
                    f[w] = eo == 31 ? s.codes[es] : (s.codes[es - 1] >> (2 * eo + 2)) | (s.codes[es] << (62 - 2 * eo));
                    const uint32_t st = p0 - k + 32 * w, ss = st >> 5, so = st & 31;
                    r[w] = so == 0 ? s.rcodes[ss] : (s.rcodes[ss] << (2 * so)) | (s.rcodes[ss + 1] >> (64 - 2 * so));
                }
                r[LAST] &= back_mask;
                const uint32_t cw = (uint32_t)(s.codes[p0 >> 5] >> (2 * (p0 & 31)));   // the chunk's codes
#pragma unroll
                for (uint32_t p = 0; p < CH; ++p) {
                    const uint64_t c = (cw >> (2 * p)) & 3u;
#pragma unroll
                    for (uint32_t w = LAST; w > 0; --w) f[w] = (f[w] >> 2) | (f[w - 1] << 62);
                    f[0] = (f[0] >> 2) | (c << 62);
#pragma unroll
                    for (uint32_t w = 0; w < LAST; ++w) r[w] = (r[w] << 2) | (r[w + 1] >> 62);
                    r[LAST] = (r[LAST] << 2) | ((c ^ 3u) << fs);
                    const uint64_t fl = f[LAST] & back_mask;
                    // the larger array, complemented
                    bool less = false, decided = false;
#pragma unroll
                    for (uint32_t w = 0; w <= LAST; ++w) {
                        const uint64_t x = w == LAST ? fl : f[w];
                        if (!decided && x != r[w]) {
                            decided = true;
                            less = x < r[w];
                        }
                    }
#pragma unroll
                    for (uint32_t w = 0; w < N; ++w) {
                        if (w > LAST) key[p][w] = 0;
                        else {
                            const uint64_t x = w == LAST ? fl : f[w];
                            key[p][w] = ~(less ? r[w] : x) & (w == LAST ? back_mask : ~0ULL);
                        }
                    }
                }
                if (!all_buckets) {
#pragma unroll
                    for (uint32_t p = 0; p < CH; ++p) {
                        const uint32_t b = (uint32_t)(key[p][0] >> 56);
                        if (b < blo || b >= bhi) e &= ~(1u << p);
                    }
                }
#pragma unroll
                for (uint32_t p = 0; p < CH; ++p) {
                    rk[p] = 0;
                    if ((e >> p) & 1u) rk[p] = atomicAdd(&s_hist[key[p][0] >> 56], 1u);
                }
            }
            if (CENSUS) continue;   // counted; s_hist is added up at the end
            __syncthreads();
            const uint32_t c = s_hist[tid];
            s_hist[tid] = 0;
            const unsigned long long cur = c ? atomicAdd(&a.bucket_cursor[tid], (unsigned long long)c) : 0ull;
            const uint32_t inc = warp_inclusive(c, lane);
            if (lane == 31) s_wbk[warp] = inc;
            __syncthreads();
            uint32_t n;
            const uint32_t start = sum_before(s_wbk, warp, n) + inc - c;
            s_start[tid] = start;
            __syncthreads();
#pragma unroll
            for (uint32_t p = 0; p < CH; ++p)
                if ((e >> p) & 1u) {
                    ulonglong2 *d = reinterpret_cast<ulonglong2 *>(s.stage + N * (s_start[key[p][0] >> 56] + rk[p]));
#pragma unroll
                    for (uint32_t w = 0; w < N; w += 2) d[w / 2] = make_ulonglong2(key[p][w], key[p][w + 1]);
                }
            if (c) {
                const unsigned long long at = a.bucket_base[tid] + cur;
                const unsigned long long end = a.bucket_end[tid] < a.list_cap ? a.bucket_end[tid] : a.list_cap;
                s_ptr[tid] = a.list + N * at - N * (unsigned long long)start;
                s_lim[tid] = start + (uint32_t)(at >= end ? 0ull : (end - at < c ? end - at : c));
                if (at + c > end) s_over = 1;
            }
            __syncthreads();
            const bool over = s_over != 0;
            for (uint32_t i = tid; i < n; i += PT_THREADS) {
                const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(s.stage + N * i);
                const ulonglong2 v = q[0];
                const uint32_t b = (uint32_t)(v.x >> 56);
                if (over && i >= s_lim[b]) continue;
                ulonglong2 *d = reinterpret_cast<ulonglong2 *>(s_ptr[b] + N * (unsigned long long)i);
                d[0] = v;
#pragma unroll
                for (uint32_t w = 1; w < N / 2; ++w) d[w] = q[w];
            }
            if (r0 + PT_THREADS < n_ch) __syncthreads();   // another round: its ranks and stage follow
        }
        if (CENSUS) __syncthreads();   // the chunk list is read before the next tile's
    }
    if (CENSUS) {
        for (int o = 16; o > 0; o >>= 1) n_occ += __shfl_down_sync(FULLW, n_occ, o);
        if (lane == 0 && n_occ) atomicAdd(a.occ, n_occ);
        if (s_hist[tid]) atomicAdd(&a.bucket_hist[tid], (unsigned long long)s_hist[tid]);
    }
}

int part_sms()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

template <int BY, bool W>
cudaError_t launch_part_t(const ExtractArgs &a, cudaStream_t st)
{
    auto kern = k_part<BY, W>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PartSmem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PT_THREADS, sizeof(PartSmem));
    if (e != cudaSuccess) return e;
    const uint64_t grid = std::min<uint64_t>(a.n_tiles, (uint64_t)part_sms() * std::max(per_sm, 1));
    note_kernel_launch();
    kern<<<(unsigned)grid, PT_THREADS, sizeof(PartSmem), st>>>(a);
    return cudaGetLastError();
}

template <uint32_t N, uint32_t LAST, bool CENSUS>
cudaError_t launch_part_wide_t(const ExtractArgs &a, cudaStream_t st)
{
    auto kern = k_part_wide<N, LAST, CENSUS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WidePartSmem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PT_THREADS, sizeof(WidePartSmem));
    if (e != cudaSuccess) return e;
    const uint64_t step = CENSUS ? a.bucket_sample_mask + 1 : 1;
    const uint64_t grid = std::min<uint64_t>((a.n_tiles + step - 1) / step, (uint64_t)part_sms() * std::max(per_sm, 1));
    note_kernel_launch();
    kern<<<(unsigned)grid, PT_THREADS, sizeof(WidePartSmem), st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_part(PartBy by, uint32_t k, const ExtractArgs &a, cudaStream_t st)
{
    if (!a.n_tiles) return cudaSuccess;
    if (by == PART_BY_SAMPLE) return launch_part_t<PART_BY_SAMPLE, true>(a, st);
    if (k > 16)
        return by == PART_BY_STRING ? launch_part_t<PART_BY_STRING, true>(a, st) : launch_part_t<PART_BY_ROOT, true>(a, st);
    return by == PART_BY_STRING ? launch_part_t<PART_BY_STRING, false>(a, st) : launch_part_t<PART_BY_ROOT, false>(a, st);
}

cudaError_t launch_part_wide(bool census, uint32_t k, const ExtractArgs &a, cudaStream_t st)
{
    if (!a.n_tiles) return cudaSuccess;
    if (k <= 32 || k > 128) return cudaErrorInvalidValue;
    if (k <= 64) return census ? launch_part_wide_t<2, 1, true>(a, st) : launch_part_wide_t<2, 1, false>(a, st);
    if (k <= 96) return census ? launch_part_wide_t<4, 2, true>(a, st) : launch_part_wide_t<4, 2, false>(a, st);
    return census ? launch_part_wide_t<4, 3, true>(a, st) : launch_part_wide_t<4, 3, false>(a, st);
}

}  // namespace kc
