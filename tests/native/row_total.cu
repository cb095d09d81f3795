// row_total.cu -- one row of table_block_row whose hits number more than 2^32.
//
// A real row of so many needs 2^32 edges.  Here the row's f members share one
// list, which holds every member `rounds` times: the kernel's sums are over
// list elements, so the row has f * f * rounds hits, each member f * rounds as
// the list's owner and as many as what is found.
//
// Usage: row_total f rounds; prints the row's credit and total for the
// per-vertex and the global form, and whether every member's credit is right.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../gputrianglecounting_b200/csrc/gtc_count.cuh"

using namespace gtc;

template <bool PV>
__global__ void __launch_bounds__(kThreads) row_kernel(const Data w, VInfo vi, unsigned long long *out)
{
    __shared__ TableBlockSmem sm;
    unsigned long long tri = 0;
    table_block_row<PV, false, unsigned int>(w, 0, vi, w.recs, sm, tri);
    if (threadIdx.x == 0) *out = tri;
}

#define OK(call)                                                              \
    if ((call) != cudaSuccess) {                                              \
        std::printf("CUDA error in %s\n", #call);                             \
        return 1;                                                             \
    }

template <bool PV>
int run(int f, int rounds)
{
    const size_t list = (size_t)f * rounds;
    std::vector<int> ind;
    for (int m = 1; m <= f; ++m) ind.push_back(m);               // the row
    for (size_t i = 0; i < list; ++i) ind.push_back(1 + (int)(i % f));
    std::vector<VInfo> vinfo((size_t)f + 1, VInfo{f, (int)list, 0});
    GraphRec rec;
    rec.nv = f + 1;
    rec.uniform = 1;                                             // lists are in ind
    Data w{};
    unsigned long long *acc = nullptr, *out = nullptr;
    OK(cudaMalloc((void **)&w.ind, 4 * ind.size()));
    OK(cudaMalloc((void **)&w.vinfo, sizeof(VInfo) * vinfo.size()));
    OK(cudaMalloc((void **)&w.recs, sizeof(GraphRec)));
    OK(cudaMalloc((void **)&acc, 8 * vinfo.size()));
    OK(cudaMalloc((void **)&out, 8));
    OK(cudaMemcpy((void *)w.ind, ind.data(), 4 * ind.size(), cudaMemcpyHostToDevice));
    OK(cudaMemcpy(w.vinfo, vinfo.data(), sizeof(VInfo) * vinfo.size(), cudaMemcpyHostToDevice));
    OK(cudaMemcpy(w.recs, &rec, sizeof(rec), cudaMemcpyHostToDevice));
    OK(cudaMemset(acc, 0, 8 * vinfo.size()));
    w.tacc = acc;
    w.n = f + 1;
    row_kernel<PV><<<1, kThreads>>>(w, VInfo{0, f, kWideRow}, out);
    OK(cudaDeviceSynchronize());
    std::vector<unsigned long long> credit(vinfo.size());
    unsigned long long total = 0;
    OK(cudaMemcpy(credit.data(), acc, 8 * credit.size(), cudaMemcpyDeviceToHost));
    OK(cudaMemcpy(&total, out, 8, cudaMemcpyDeviceToHost));
    bool even = true;
    for (int m = 1; m <= f; ++m) even &= credit[m] == (PV ? 2ull * f * rounds : 0ull);
    std::printf("%llu %llu %d\n", credit[0], total, even);
    return 0;
}

int main(int argc, char **argv)
{
    if (argc != 3) return 2;
    const int f = std::atoi(argv[1]), rounds = std::atoi(argv[2]);
    return run<true>(f, rounds) || run<false>(f, rounds);
}
