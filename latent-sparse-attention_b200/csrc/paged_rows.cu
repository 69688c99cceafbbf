// Rows of a paged table: a request's logical row i lies at row i % page_rows of its page i / page_rows. Up to three tables of 32-bit
// words, into the pages or out of them, in one launch. (The same as index arithmetic and one gather or scatter a table took nine
// launches for a request's new buckets and seven for its centroids, 2 to 5 us each for a few hundred rows.)
#include "common.cuh"

namespace lsa {

constexpr int kPagedTables = 3;
constexpr int kPagedThreads = 256;

struct PagedRows {
  const int32_t *pages;  // [max_pages] the request's
  uint32_t *tables[kPagedTables], *dense[kPagedTables];  // [rows, words], [n, words]
  int words[kPagedTables];
  int64_t n, first, rows;  // logical rows first .. first + n - 1; rows of the tables
  int max_pages, page_rows, row_words;
};

template <bool INTO>
__global__ void __launch_bounds__(kPagedThreads) paged_rows_kernel(PagedRows p) {
  const int64_t total = p.n * p.row_words;
  for (int64_t e = (int64_t)blockIdx.x * kPagedThreads + threadIdx.x; e < total; e += (int64_t)gridDim.x * kPagedThreads) {
    const int64_t i = e / p.row_words, logical = p.first + i;
    int word = (int)(e - i * p.row_words), t = 0;
    while (word >= p.words[t]) word -= p.words[t++];
    const int64_t page = logical / p.page_rows;
    const int32_t held = page < p.max_pages ? p.pages[page] : -1;
    const int64_t row = held >= 0 ? (int64_t)held * p.page_rows + logical % p.page_rows : p.rows;
    uint32_t *dense = p.dense[t] + i * p.words[t] + word, *table = p.tables[t] + row * p.words[t] + word;
    if (INTO) {
      if (row < p.rows) *table = *dense;
    } else {
      *dense = row < p.rows ? *table : 0u;
    }
  }
}

}  // namespace lsa

LSA_API int lsa_paged_rows(const int32_t *pages, int max_pages, int page_rows, int64_t first, int64_t n, int64_t rows, void *table0,
                           void *dense0, int words0, void *table1, void *dense1, int words1, void *table2, void *dense2, int words2,
                           int into_pages, void *stream) {
  LSA_REQUIRE(max_pages >= 1 && page_rows >= 1 && first >= 0 && n >= 0 && rows >= 0 && words0 >= 1 && words1 >= 0 && words2 >= 0 &&
                  (int64_t)words0 + words1 + words2 <= INT32_MAX,
              LSA_ERR_ARGUMENT);
  if (n == 0) return LSA_OK;
  LSA_REQUIRE(pages && table0 && dense0 && (words1 == 0 || (table1 && dense1)) && (words2 == 0 || (table2 && dense2)), LSA_ERR_NULL);
  lsa::PagedRows p = {};
  p.pages = pages, p.n = n, p.first = first, p.rows = rows, p.max_pages = max_pages, p.page_rows = page_rows;
  p.tables[0] = (uint32_t *)table0, p.tables[1] = (uint32_t *)table1, p.tables[2] = (uint32_t *)table2;
  p.dense[0] = (uint32_t *)dense0, p.dense[1] = (uint32_t *)dense1, p.dense[2] = (uint32_t *)dense2;
  p.words[0] = words0, p.words[1] = words1, p.words[2] = words2;
  p.row_words = words0 + words1 + words2;
  const int64_t blocks = (n * p.row_words + lsa::kPagedThreads - 1) / lsa::kPagedThreads, most = 16 * (int64_t)lsa::sm_count();
  const auto kernel = into_pages ? lsa::paged_rows_kernel<true> : lsa::paged_rows_kernel<false>;
  kernel<<<(unsigned)(blocks < most ? blocks : most), lsa::kPagedThreads, 0, (cudaStream_t)stream>>>(p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}
