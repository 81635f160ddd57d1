// B = Aᵀ on the device (declared in include/casgemm.h).  Part of the
// cas_api.cu translation unit.
//
// The reference makes B on the host and reads it from disk: trpl_transpose
// (src/mm/mm_utils.c:742-754) swaps each triple's row and column and sorts
// the triples by (row, column), txt_transpose (:851-862) writes them as
// <dataset>.trs.mtx, and every driver reads that file as its second input.
// Here B comes from A on the device, as a stable counting sort of A's
// entries by column, so each row of B lists A's rows in increasing order and
// duplicate (row, column) entries keep A's order: entry for entry the result
// of the host's counting-sort transpose (cas_csr_transpose_host).
//
//   k_tr_count     checks A; entries per column, and each entry's place among
//                  those of its column
//   scan           B's row pointers
//   k_tr_scatter   a key for each entry, its row in A above its position, to
//                  its place in its row of B
//   k_tr_rows      rows of B of at most kTrWarpRow entries: a warp sorts a row's
//                  keys in registers and writes its columns and values
//   k_tr_rank      longer rows, where A has at most kRankCols rows: the place of
//                  a key is the rank of its row in a bitmap in shared memory;
//                  rows with a (row, column) pair twice are left to
//   k_tr_sort_block, k_tr_gather
//                  a block's stable LSD radix sort of a row's keys (8-bit
//                  digits of the positions, only the bits the row spans), then
//                  the columns and values; also where A has more rows
//
// A graph of 262144 vertices and 7.9e6 entries, cold caches: count 119 us
// (8-byte atomics on 262144 counters), scatter 150 (scattered 8-byte writes),
// rows 168, rank 150 (7.9e6 scattered reads of values between them).  Before,
// 1240 us: a check 111, count 115, scatter with its own atomics 150, a block
// sort of every row of more than 32 entries 590, and a search in A's row
// pointers for every entry 267.
namespace {

constexpr int kTrBlock = 256;
// Rows a warp sorts: 8 keys a lane, 64 registers.  With 16 (rows of up to 512,
// 128 registers) the rows took 253 us instead of 168 and k_tr_rank no less.
constexpr int kTrWarpRow = 256;

// Entries per column, each entry's place among its column's (in the order the
// atomics come), and the input check: row pointers non-decreasing and within
// [0, nnz], columns in [0, n).  Entries of a warp that hit the same column are
// added up first where that can happen: lanes whose column does not exceed the
// lane's before begin a row, and within a row columns differ as a rule.
__global__ void __launch_bounds__(kTrBlock)
k_tr_count(int64_t nnz, int64_t m, int64_t n, const int64_t* __restrict__ arp, const int32_t* __restrict__ col,
           unsigned long long* __restrict__ cnt, unsigned long long* __restrict__ place,
           unsigned long long* __restrict__ flag) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool bad = false;
  for (int64_t r = first; r < m; r += stride) {
    const int64_t s = arp[r], e = arp[r + 1];
    bad |= s < 0 || e < s || e > nnz;
  }
  for (int64_t e0 = first; e0 - lane < nnz; e0 += U * stride) {
    int32_t c[U];
    unsigned long long at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = e0 + u * stride < nnz ? col[e0 + u * stride] : -1;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = e0 + u * stride < nnz, ok = (uint64_t)(int64_t)c[u] < (uint64_t)n;
      bad |= in && !ok;
      const unsigned begins = __ballot_sync(cas::kFull, __shfl_up_sync(cas::kFull, c[u], 1) >= c[u]);
      if (__popc(begins) <= 2) {  // lane 0 is one of them
        at[u] = ok ? atomicAdd(&cnt[c[u]], 1ull) : 0;
      } else {
        const unsigned peers = __match_any_sync(cas::kFull, c[u]);
        const int leader = __ffs(peers) - 1;
        unsigned long long b = 0;
        if (ok && lane == leader) b = atomicAdd(&cnt[c[u]], (unsigned long long)__popc(peers));
        at[u] = __shfl_sync(cas::kFull, b, leader) + __popc(peers & cas::lanemask_lt());
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e0 + u * stride < nnz) place[e0 + u * stride] = at[u];
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1ull);
}

// Keys to their columns' slots.  Each warp takes a run of consecutive entries
// and carries the row along: the lanes look at the next 32 row pointers and
// each finds the last one at or before its entry among them.
__global__ void __launch_bounds__(kTrBlock)
k_tr_scatter(int64_t nnz, int64_t m, int shift, const int64_t* __restrict__ arp, const int32_t* __restrict__ col,
             const int64_t* __restrict__ brp, const unsigned long long* __restrict__ place,
             unsigned long long* __restrict__ key) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (kTrBlock / 32), w = ((int64_t)blockIdx.x * kTrBlock + threadIdx.x) >> 5;
  const int64_t groups = (nnz + 31) >> 5;
  int64_t base = (groups * w / warps) << 5;
  const int64_t end = (groups * (w + 1) / warps) << 5;
  if (base >= end) return;
  int64_t row = 0;  // the last row that starts at or before base
  for (int64_t h = m; h - row > 1;) {
    const int64_t mid = (row + h) >> 1;
    if (arp[mid] <= base) row = mid; else h = mid;
  }
  int32_t c = base + lane < nnz ? col[base + lane] : -1;
  unsigned long long p = base + lane < nnz ? place[base + lane] : 0ull;
  for (; base < end; base += 32) {
    const int64_t e = base + lane;
    const int64_t at = c >= 0 ? brp[c] + (int64_t)p : 0;
    const bool more = e + 32 < nnz;  // the next entries, on their way during this step
    c = more ? col[e + 32] : -1;
    p = more ? place[e + 32] : 0ull;
    int64_t my = row;
    for (int look = 0;; ++look) {  // rows r0 + 1 .. r0 + 32
      const int64_t r0 = row + 32 * look, i = r0 + 1 + lane;
      const int64_t next = i < m ? arp[i] - base : 0x7FFFFFFF;
      const int d = next > 0x7FFFFFFF ? 0x7FFFFFFF : (int)next;  // their starts, ascending
      int k = 0;  // of the 32, those at or before this entry
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(cas::kFull, d, k + step - 1) <= lane) k += step;
      const int last = __shfl_sync(cas::kFull, d, 31);
      if (k == 31 && last <= lane) k = 32;
      if (k > 0) my = r0 + k;
      if (last > 31) break;
      if (look == 3) {  // a long stretch of empty rows
        for (int64_t h = m; h - my > 1;) {
          const int64_t mid = (my + h) >> 1;
          if (arp[mid] <= e) my = mid; else h = mid;
        }
        break;
      }
    }
    if (e < nnz) key[at] = ((unsigned long long)my << shift) | (unsigned long long)e;
    row = __shfl_sync(cas::kFull, my, 31);
  }
}

// Bitonic sort of 32 * N keys of a warp, key i = lane * N + k in v[k].
template <int N>
__device__ __forceinline__ void tr_sort(unsigned long long (&v)[N], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * N; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= N) {
        const bool up = ((lane * N) & size) == 0, lower = (lane & (stride / N)) == 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const unsigned long long o = __shfl_xor_sync(cas::kFull, v[k], stride / N);
          v[k] = (lower == up) ? (v[k] < o ? v[k] : o) : (v[k] < o ? o : v[k]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < N; ++k) {
          if (k & stride) continue;
          const bool up = ((lane * N + k) & size) == 0;
          const unsigned long long a = v[k], b = v[k + stride];
          const bool swap = (a > b) == up;
          v[k] = swap ? b : a;
          v[k + stride] = swap ? a : b;
        }
      }
    }
  }
}

template <int N, typename V>
__device__ __forceinline__ void tr_row(int64_t s, int len, int shift, const unsigned long long* __restrict__ key,
                                       const V* __restrict__ aval, int32_t* __restrict__ bcol, V* __restrict__ bval,
                                       unsigned long long* __restrict__ tile, int lane) {
  unsigned long long v[N];
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = lane + 32 * k < len ? key[s + lane + 32 * k] : ~0ull;
  tr_sort<N>(v, lane);
  const unsigned long long mask = (1ull << shift) - 1ull;
  if (N > 1) {  // from N consecutive keys a lane to consecutive lanes
#pragma unroll
    for (int k = 0; k < N; ++k) tile[lane * (N + 1) + k] = v[k];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = tile[lane + 32 * k + (lane + 32 * k) / N];
    __syncwarp();
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int i = lane + 32 * k;
    if (i < len) {
      bcol[s + i] = (int32_t)(v[k] >> shift);
      bval[s + i] = aval[v[k] & mask];
    }
  }
}

// A warp per row of at most kTrWarpRow entries; longer rows are listed.
template <typename V>
__global__ void __launch_bounds__(kTrBlock)
k_tr_rows(int64_t n, int shift, const int64_t* __restrict__ rp, const unsigned long long* __restrict__ key,
          const V* __restrict__ aval, int32_t* __restrict__ bcol, V* __restrict__ bval, int32_t* __restrict__ big,
          unsigned long long* __restrict__ nbig) {
  __shared__ unsigned long long tiles[kTrBlock / 32][kTrWarpRow + 32];
  const int lane = threadIdx.x & 31;
  unsigned long long* tile = tiles[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < n; j += warps) {
    const int64_t s = rp[j], len = rp[j + 1] - s;
    if (len == 0) continue;
    if (len > kTrWarpRow) {
      if (lane == 0) big[atomicAdd(nbig, 1ull)] = (int32_t)j;
    } else if (len <= 32) {
      tr_row<1, V>(s, (int)len, shift, key, aval, bcol, bval, tile, lane);
    } else if (len <= 64) {
      tr_row<2, V>(s, (int)len, shift, key, aval, bcol, bval, tile, lane);
    } else if (len <= 128) {
      tr_row<4, V>(s, (int)len, shift, key, aval, bcol, bval, tile, lane);
    } else {
      tr_row<kTrWarpRow / 32, V>(s, (int)len, shift, key, aval, bcol, bval, tile, lane);
    }
  }
}

// A block per longer row: marks the rows of A that its keys name in a bitmap,
// ranks the words, and every key goes to the rank of its row.  No two keys of
// a row may name the same row of A: such rows are listed again.
template <int BLOCK, typename V>
__global__ void __launch_bounds__(BLOCK)
k_tr_rank(int64_t m, int shift, int words, const int64_t* __restrict__ rp, const int32_t* __restrict__ rows,
          const unsigned long long* __restrict__ key, const V* __restrict__ aval, int32_t* __restrict__ bcol,
          V* __restrict__ bval, int32_t* __restrict__ again, unsigned long long* __restrict__ nagain) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ long long tmp[BLOCK / 32 + 1];
  uint32_t* bm = reinterpret_cast<uint32_t*>(smem);
  uint32_t* gbase = bm + words;
  uint8_t* wrank = reinterpret_cast<uint8_t*>(gbase + words / 8);
  const int64_t j = rows[blockIdx.x];
  const int64_t s = rp[j], len = rp[j + 1] - s;
  for (int i = threadIdx.x; i < words; i += BLOCK) bm[i] = 0u;
  __syncthreads();
  bool twice = false;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < len; i += BLOCK) {
    const uint32_t r = (uint32_t)(key[s + i] >> shift);
    const uint32_t bit = 1u << (r & 31);
    twice |= (atomicOr(&bm[r >> 5], bit) & bit) != 0;
  }
  if (__syncthreads_or(twice)) {
    if (threadIdx.x == 0) again[atomicAdd(nagain, 1ull)] = (int32_t)j;
    return;
  }
  cas::slice_ranks<BLOCK>(bm, words, gbase, wrank, tmp);
  const unsigned long long mask = (1ull << shift) - 1ull;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < len; i += BLOCK) {
    const unsigned long long k = key[s + i];
    const uint32_t r = (uint32_t)(k >> shift), w = r >> 5;
    const int64_t at = s + gbase[w >> 3] + wrank[w] + __popc(bm[w] & ((1u << (r & 31)) - 1u));
    bcol[at] = (int32_t)r;
    bval[at] = aval[k & mask];
  }
}

// A block per listed row, a stable LSD radix sort of (position - the row's
// smallest position) by 8-bit digits over only the bits the row spans.
// Each pass runs over the row in tiles of kTrBlock entries in order; within a
// tile an entry's place is its digit's running offset, plus the counts of
// that digit in earlier warps of the tile, plus its rank among the lanes of
// its warp with the same digit, so equal digits keep their order.  The passes
// alternate between `key` and `aux` (the same offsets); an odd number of
// passes ends with a copy back.
__global__ void __launch_bounds__(kTrBlock) k_tr_sort_block(int shift, const int64_t* __restrict__ rp,
                                                            const int32_t* __restrict__ big,
                                                            unsigned long long* __restrict__ key,
                                                            unsigned long long* __restrict__ aux) {
  constexpr int NW = kTrBlock / 32;
  __shared__ unsigned int hist[256];
  __shared__ unsigned int run[256];
  __shared__ unsigned int wcnt[NW][257];
  __shared__ unsigned long long s_min, s_max;
  const unsigned long long mask = (1ull << shift) - 1ull;  // the position in a key
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j = big[blockIdx.x];
  const int64_t s = rp[j], len = rp[j + 1] - s;
  if (threadIdx.x == 0) {
    s_min = ~0ull;
    s_max = 0ull;
  }
  __syncthreads();
  unsigned long long mn = ~0ull, mx = 0ull;
  for (int64_t i = threadIdx.x; i < len; i += kTrBlock) {
    const unsigned long long v = key[s + i] & mask;
    mn = v < mn ? v : mn;
    mx = v > mx ? v : mx;
  }
  atomicMin(&s_min, mn);
  atomicMax(&s_max, mx);
  __syncthreads();
  const unsigned long long kmin = s_min, span = s_max - s_min;
  const int bits = span ? 64 - __clzll((long long)span) : 0;
  const int passes = (bits + 7) / 8;
  unsigned long long* src = key;
  unsigned long long* dst = aux;
  for (int pass = 0; pass < passes; ++pass) {
    const int sh = pass * 8;
    for (int d = threadIdx.x; d < 256; d += kTrBlock) hist[d] = 0u;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < len; i += kTrBlock) atomicAdd(&hist[(((src[s + i] & mask) - kmin) >> sh) & 0xFF], 1u);
    __syncthreads();
    if (warp == 0) {  // exclusive scan of the 256 digit counts: 8 per lane
      unsigned int c[8], t = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        c[q] = hist[lane * 8 + q];
        t += c[q];
      }
      unsigned int ex = cas::warp_inclusive_sum(t) - t;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        run[lane * 8 + q] = ex;
        ex += c[q];
      }
    }
    for (int i = threadIdx.x; i < NW * 257; i += kTrBlock) (&wcnt[0][0])[i] = 0u;
    __syncthreads();
    for (int64_t t0 = 0; t0 < len; t0 += kTrBlock) {
      const int64_t i = t0 + threadIdx.x;
      const bool ok = i < len;
      const unsigned long long v = ok ? src[s + i] : 0ull;
      const int d = ok ? (int)((((v & mask) - kmin) >> sh) & 0xFF) : 256;
      const unsigned peers = __match_any_sync(cas::kFull, d);
      const int rank = __popc(peers & cas::lanemask_lt());
      if (lane == __ffs(peers) - 1) wcnt[warp][d] = (unsigned int)__popc(peers);
      __syncthreads();
      if (threadIdx.x < 256) {  // per digit: offsets of the warps' runs, in warp order
        const int dd = threadIdx.x;
        unsigned int r = run[dd];
        for (int w = 0; w < NW; ++w) {
          const unsigned int c = wcnt[w][dd];
          wcnt[w][dd] = r;
          r += c;
        }
        run[dd] = r;
      }
      __syncthreads();
      if (ok) dst[s + wcnt[warp][d] + rank] = v;
      __syncthreads();
      for (int q = threadIdx.x; q < NW * 257; q += kTrBlock) (&wcnt[0][0])[q] = 0u;
      __syncthreads();
    }
    unsigned long long* t = src;
    src = dst;
    dst = t;
  }
  if (passes & 1)
    for (int64_t i = threadIdx.x; i < len; i += kTrBlock) key[s + i] = aux[s + i];
}

// The columns and values of the listed rows, a block each, from sorted keys.
template <typename V>
__global__ void k_tr_gather(int shift, const int64_t* __restrict__ rp, const int32_t* __restrict__ rows,
                            const unsigned long long* __restrict__ key, const V* __restrict__ aval,
                            int32_t* __restrict__ bcol, V* __restrict__ bval) {
  const int64_t j = rows[blockIdx.x];
  const unsigned long long mask = (1ull << shift) - 1ull;
  for (int64_t p = rp[j] + threadIdx.x; p < rp[j + 1]; p += blockDim.x) {
    bcol[p] = (int32_t)(key[p] >> shift);
    bval[p] = aval[key[p] & mask];
  }
}

// The rows of B from the keys: short rows by warps, long ones by rank, the
// rest (*again of them listed behind the long ones) by sorting.
template <typename V>
cas_status transpose_rows(cas_ctx* ctx, const DevMat& A, int shift, const int64_t* brp, unsigned long long* key,
                          unsigned long long* aux, int32_t* big, int32_t* bcol, V* bval) {
  const int64_t m = A.csr.nrow, n = A.csr.ncol;
  const V* aval = static_cast<const V*>(A.csr.val);
  unsigned long long* nbig = ctx->d_counts + kSlotOvf;       // cleared by the caller, as the next
  unsigned long long* nagain = ctx->d_counts + kSlotNnz;
  k_tr_rows<V><<<grid_for(n * 32, kTrBlock, ctx->sm_count * 16), kTrBlock, 0, ctx->stream>>>(n, shift, brp, key, aval,
                                                                                              bcol, bval, big, nbig);
  CAS_TRY(check_launch(ctx, "k_tr_rows"));
  CAS_TRY(fetch_counts(ctx));
  int64_t rest = (int64_t)ctx->h_counts[kSlotOvf];
  if (rest == 0) return CAS_OK;
  const int32_t* list = big;
  if (m <= cas::kRankCols) {
    const int words = dense_words(m);
    const size_t smem = cas::DenseSmem<double>::ranks(words);
    k_tr_rank<512, V><<<(unsigned)rest, 512, smem, ctx->stream>>>(m, shift, words, brp, big, key, aval, bcol, bval,
                                                                  big + rest, nagain);
    CAS_TRY(check_launch(ctx, "k_tr_rank"));
    CAS_TRY(fetch_counts(ctx));
    list = big + rest;
    rest = (int64_t)ctx->h_counts[kSlotNnz];
    if (rest == 0) return CAS_OK;
  }
  k_tr_sort_block<<<(unsigned)rest, kTrBlock, 0, ctx->stream>>>(shift, brp, list, key, aux);
  CAS_TRY(check_launch(ctx, "k_tr_sort_block"));
  k_tr_gather<V><<<(unsigned)rest, kTrBlock, 0, ctx->stream>>>(shift, brp, list, key, aval, bcol, bval);
  return check_launch(ctx, "k_tr_gather");
}

// The limit is the kernel's on the device, for all contexts and threads: set
// once to the most a call may take, not to what each call does (a narrower
// matrix on another thread would take it from a wide one's launch).
cas_status setup_transpose(cas_ctx* ctx) {
  const size_t smem = cas::DenseSmem<double>::ranks(cas::kRankCols / 32);
  CAS_TRY(allow_smem(ctx, k_tr_rank<512, double>, smem));
  return allow_smem(ctx, k_tr_rank<512, int32_t>, smem);
}

cas_status transpose_device(cas_ctx* ctx, const DevMat& A, int vt, cas_csr* B, bool to_host, double& d2h) {
  const int64_t m = A.csr.nrow, n = A.csr.ncol, nnz = A.nnz;
  const size_t vbytes = vt == CAS_VAL_F64 ? 8 : 4;
  int64_t *brp = nullptr, *cnt = nullptr, *partial = nullptr;
  int32_t *bcol = nullptr, *big = nullptr;
  void* bval = nullptr;
  unsigned long long *key = nullptr, *aux = nullptr;
  int shift = 1;  // bits of a position in a key; the row of A is above
  while ((int64_t(1) << shift) < nnz) ++shift;
  int row_bits = 0;
  while ((int64_t(1) << row_bits) < m) ++row_bits;
  if (shift + row_bits > 64)  // more entries than a device holds twice
    return set_err(ctx, CAS_ERR_OOM, "the transpose of %lld entries does not fit", (long long)nnz);
  std::vector<void*> tmp;
  auto release = [&]() {
    for (void* p : tmp) cudaFreeAsync(p, ctx->stream);
  };
  // all from the results' pool: B comes first, so the scratch cuts up none of
  // its holes
  cas_status rc = [&]() -> cas_status {
    CAS_TRY(out_alloc(ctx, (void**)&brp, sizeof(int64_t) * (size_t)(n + 1)));
    CAS_TRY(out_alloc(ctx, (void**)&bcol, sizeof(int32_t) * (size_t)(nnz > 0 ? nnz : 1)));
    CAS_TRY(out_alloc(ctx, &bval, vbytes * (size_t)(nnz > 0 ? nnz : 1)));
    CAS_TRY(out_alloc(ctx, (void**)&cnt, sizeof(int64_t) * (size_t)(n + 1)));
    tmp.push_back(cnt);
    CAS_TRY(out_alloc(ctx, (void**)&partial, sizeof(int64_t) * (size_t)((n + 1 + cas::kScanTile - 1) / cas::kScanTile + 1)));
    tmp.push_back(partial);
    CAS_TRY(out_alloc(ctx, (void**)&key, sizeof(unsigned long long) * (size_t)(nnz > 0 ? nnz : 1)));
    tmp.push_back(key);
    CAS_TRY(out_alloc(ctx, (void**)&aux, sizeof(unsigned long long) * (size_t)(nnz > 0 ? nnz : 1)));
    tmp.push_back(aux);
    CAS_TRY(out_alloc(ctx, (void**)&big, sizeof(int32_t) * 2 * (size_t)(n > 0 ? n : 1)));
    tmp.push_back(big);
    CAS_CUDA(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (size_t)(n + 1), ctx->stream));
    CAS_TRY(clear_counts(ctx));
    if (m > 0 || nnz > 0) {
      k_tr_count<<<grid_for(std::max(m, nnz), kTrBlock, ctx->sm_count * 8), kTrBlock, 0, ctx->stream>>>(
          nnz, m, n, A.csr.rp, A.csr.col, reinterpret_cast<unsigned long long*>(cnt), aux, ctx->d_counts + kSlotCheck);
      CAS_TRY(check_launch(ctx, "k_tr_count"));
      CAS_TRY(fetch_counts(ctx));
      if (ctx->h_counts[kSlotCheck])
        return set_err(ctx, CAS_ERR_BAD_INPUT, "A's row pointers or columns are out of range");
    }
    CAS_TRY(launch_scan(ctx, brp, cnt, n + 1, partial, nullptr));
    if (nnz > 0) {
      k_tr_scatter<<<ctx->sm_count * 8, kTrBlock, 0, ctx->stream>>>(nnz, m, shift, A.csr.rp, A.csr.col, brp, aux, key);
      CAS_TRY(check_launch(ctx, "k_tr_scatter"));
      if (vt == CAS_VAL_F64)
        CAS_TRY(transpose_rows<double>(ctx, A, shift, brp, key, aux, big, bcol, static_cast<double*>(bval)));
      else
        CAS_TRY(transpose_rows<int32_t>(ctx, A, shift, brp, key, aux, big, bcol, static_cast<int32_t*>(bval)));
    }
    memset(B, 0, sizeof(*B));
    B->num_row = n;
    B->num_col = m;
    B->num_nnz = nnz;
    B->col_bytes = 4;
    B->val_type = vt;
    B->owned = 1;
    if (!to_host) {
      B->on_device = 1;
      B->row_ptrs = brp;
      B->cols = bcol;
      B->rats = bval;
      brp = nullptr;
      bcol = nullptr;
      bval = nullptr;
      return CAS_OK;
    }
    B->on_device = 0;
    B->row_ptrs = static_cast<int64_t*>(malloc(sizeof(int64_t) * (size_t)(n + 1)));
    B->cols = malloc(sizeof(int32_t) * (size_t)(nnz > 0 ? nnz : 1));
    B->rats = malloc(vbytes * (size_t)(nnz > 0 ? nnz : 1));
    if (!B->row_ptrs || !B->cols || !B->rats) {
      free(B->row_ptrs);
      free(B->cols);
      free(B->rats);
      memset(B, 0, sizeof(*B));
      return set_err(ctx, CAS_ERR_OOM, "host allocation of the transpose failed");
    }
    CAS_CUDA(ctx, cudaMemcpyAsync(B->row_ptrs, brp, sizeof(int64_t) * (size_t)(n + 1), cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CAS_CUDA(ctx, cudaMemcpyAsync(B->cols, bcol, sizeof(int32_t) * (size_t)nnz, cudaMemcpyDeviceToHost, ctx->stream));
    CAS_CUDA(ctx, cudaMemcpyAsync(B->rats, bval, vbytes * (size_t)nnz, cudaMemcpyDeviceToHost, ctx->stream));
    d2h += sizeof(int64_t) * (double)(n + 1) + (4.0 + (double)vbytes) * (double)nnz;
    return CAS_OK;
  }();
  if (brp) tmp.push_back(brp);
  if (bcol) tmp.push_back(bcol);
  if (bval) tmp.push_back(bval);
  release();
  cudaStreamSynchronize(ctx->stream);
  return rc;
}

}  // namespace

extern "C" cas_status cas_csr_transpose(cas_ctx* ctx, const cas_csr* A, cas_csr* B) {
  if (!ctx || !B) return CAS_ERR_BAD_INPUT;
  CAS_TRY(basic_checks(ctx, A, "A"));
  CAS_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaGetLastError();
  const bool to_host = B->on_device == 0;
  DevMat dA;
  double h2d = 0, d2h = 0;
  cas_status rc = to_device(ctx, A, dA, h2d);
  if (rc == CAS_OK) rc = transpose_device(ctx, dA, A->val_type, B, to_host, d2h);
  free_owned(ctx, dA);
  cudaStreamSynchronize(ctx->stream);
  ctx->stats.h2d_bytes = h2d;
  ctx->stats.d2h_bytes = d2h;
  return rc;
}
