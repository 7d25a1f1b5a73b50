// Rows of the shared types (throats) of both propagations, made on the device: ids by rank, rows by
// ascending id with the pore lists one after the other, as the table holds them. What bounds it is the
// copy into the table; the sort by key and the lists' gather are a fraction of a millisecond. On one
// host thread (a sort of pairs, then a row after the other from the copied lists) the 270 thousand
// types of a 512^3 random field's watershed took 27.5 ms, here 0.4 ms; its initial propagation's 82
// thousand took 7.9 ms, here 0.3 ms.
#pragma once

#include "devutil.cuh"

namespace pma {
namespace {

__global__ void type_iota(uint32_t* __restrict__ a, size_t n) {
    PMA_GRID_STRIDE(i, n) a[i] = static_cast<uint32_t>(i);
}

// Types in ascending order of their keys count down from UINT32_MAX - 1, so row q, by ascending
// id, is the type of the (n - 1 - q)-th key.
template <class Lists>
__global__ void type_row_lengths(Lists lists, const uint32_t* __restrict__ order, size_t n, unsigned long long* __restrict__ len,
                                 uint32_t* __restrict__ id_of_type) {
    PMA_GRID_STRIDE(q, n) {
        const uint32_t k = static_cast<uint32_t>(n - 1 - q), g = order[k];
        len[q] = lists.length(g);
        id_of_type[g] = 0xFFFFFFFFu - 1u - k;
    }
}

// A warp per row: lists are a few pores long on average, thousands at most.
template <class Lists>
__global__ void type_rows_write(Lists lists, const uint32_t* __restrict__ order, size_t n, const unsigned long long* __restrict__ off,
                                const uint32_t* __restrict__ id_of_type, const unsigned long long* __restrict__ volume,
                                pma_throat* __restrict__ rows, uint32_t* __restrict__ pool) {
    const unsigned lane = threadIdx.x & 31;
    const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
    for (size_t q = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) / 32; q < n; q += warps) {
        const uint32_t g = order[n - 1 - q], m = lists.length(g);
        const unsigned long long at = off[q];
        if (lane == 0) rows[q] = pma_throat{id_of_type[g], m, volume[g], at};
        for (uint32_t j = lane; j < m; j += 32) pool[at + j] = lists.pore(g, j);
    }
}

// Fills t's rows of n > 0 types and id_of_type. keys: distinct, in the order of creation. Lists gives each
// type's length(type) and pore(type, position).
template <class Lists>
void type_rows(pma_ctx* ctx, const unsigned long long* keys, int64_t n, Lists lists, const unsigned long long* volume,
               uint32_t* id_of_type, pma_table* t) {
    cudaStream_t s = ctx->stream;
    auto* sorted = static_cast<unsigned long long*>(ctx->scratch("types.sorted", n * 8));
    auto* iota = static_cast<uint32_t*>(ctx->scratch("types.iota", n * 4));
    auto* order = static_cast<uint32_t*>(ctx->scratch("types.order", n * 4));
    auto* len = static_cast<unsigned long long*>(ctx->scratch("types.len", n * 8));
    auto* off = static_cast<unsigned long long*>(ctx->scratch("types.off", n * 8));
    auto* rows = static_cast<pma_throat*>(ctx->scratch("types.rows", n * sizeof(pma_throat)));
    type_iota<<<grid_for(ctx, n), 256, 0, s>>>(iota, n);
    ctx->check_launch("type_iota");
    sort_pairs(ctx, keys, sorted, iota, order, n);
    type_row_lengths<<<grid_for(ctx, n), 256, 0, s>>>(lists, order, n, len, id_of_type);
    ctx->check_launch("type_row_lengths");
    exclusive_sum(ctx, len, off, n);
    auto* h = static_cast<unsigned long long*>(ctx->host_staging(64));
    ReadBack rb;
    rb.add(&h[0], off + n - 1, 8);
    rb.add(&h[1], len + n - 1, 8);
    read_back(ctx, rb);
    const size_t total = h[0] + h[1];
    auto* pool = static_cast<uint32_t*>(ctx->scratch("types.pool", total * 4));
    type_rows_write<<<grid_for(ctx, static_cast<size_t>(n) * 32), 256, 0, s>>>(lists, order, n, off, id_of_type, volume, rows, pool);
    ctx->check_launch("type_rows_write");
    t->throats.resize(n);
    t->pool.resize(total);
    PMA_CUDA(cudaMemcpyAsync(t->throats.data(), rows, n * sizeof(pma_throat), cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(t->pool.data(), pool, total * 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
}

}  // namespace
}  // namespace pma
