// The attenuator lists of the pair tables (csrc/scatter.cu) against lists sized one entry short: a
// row of crystals, each pair's path crossing the ones between.  Counts the entries that differ from
// the full lists' first ones, that lie past a list's end, or that a record claims beyond it.  The
// buffer holds the full lists besides, so that every store is inside it.  Prints that count, the
// number of chords of the full lists and the CUDA error.
#include <cstdio>
#include <vector>

#include "scatter.cu"

using namespace sysmat;

constexpr int kCrystals = 6, kPairs = kCrystals * kCrystals;

template <class T>
static T* upload(const std::vector<T>& h)
{
    T* d = nullptr;
    cudaMalloc(&d, sizeof(T) * h.size());
    cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
    return d;
}

template <class T>
static std::vector<T> download(const T* d, size_t n)
{
    std::vector<T> h(n);
    cudaMemcpy(h.data(), d, sizeof(T) * n, cudaMemcpyDeviceToHost);
    return h;
}

int main()
{
    std::vector<float4> pos, size, mu, trig;
    for (int i = 0; i < kCrystals; ++i) {
        pos.push_back(make_float4(2.0f * i, 0.1f * i, -0.2f * i, 0.0f));
        size.push_back(make_float4(1.5f, 4.0f, 4.0f, 5.8523f));
        mu.push_back(make_float4(0.2f, 0.1f + 0.01f * i, 0.1f - 0.01f * i, 0.1f));
        trig.push_back(make_float4(1.0f, 0.0f, 1.0f, 0.0f));
    }
    DevGeom g{};
    g.n_det = kCrystals;
    g.cry.pos = upload(pos);
    g.cry.size = upload(size);
    g.cry.mu = upload(mu);
    g.cry.trig = upload(trig);
    const uint32_t* bitmap = upload(std::vector<uint32_t>(bitmap_crystal_words(kCrystals), 0xffffffffu));
    long long* counts = upload(std::vector<long long>(kPairs, 0));
    pair_count_kernel<false><<<kPairs, 32 * kPairWarps>>>(g, 1, bitmap, nullptr, counts);
    const std::vector<long long> full = download(counts, kPairs);

    std::vector<PairRec> rec[2];
    std::vector<AttEntry> att[2];
    std::vector<long long> off[2];
    long long chords = 0;
    for (long long c : full) chords += c;
    for (int shorter = 0; shorter < 2; ++shorter) {
        off[shorter].assign(1, 0);
        for (long long c : full) off[shorter].push_back(off[shorter].back() + (c > 0 ? c - shorter : 0));
        AttEntry* list = upload(std::vector<AttEntry>(chords + 64, AttEntry{-1.0f, -1.0f, -1.0f}));
        PairRec* pairs = upload(std::vector<PairRec>(kPairs));
        pair_fill_kernel<false><<<kPairs, 32 * kPairWarps>>>(g, 1, bitmap, nullptr, upload(off[shorter]), pairs, list);
        rec[shorter] = download(pairs, kPairs);
        att[shorter] = download(list, chords + 64);
    }
    long long bad = 0;
    for (int p = 0; p < kPairs; ++p) {
        const long long room = off[1][p + 1] - off[1][p];
        bad += rec[0][p].att_count != full[p] || rec[1][p].att_count != room;
        for (long long k = 0; k < room; ++k) {
            const AttEntry a = att[0][off[0][p] + k], b = att[1][off[1][p] + k];
            bad += !(a.len > 0.0f) || a.len != b.len || a.mu_pe != b.mu_pe || a.mu_c != b.mu_c;
        }
    }
    for (int which = 0; which < 2; ++which)
        for (size_t k = off[which].back(); k < att[which].size(); ++k) bad += att[which][k].len != -1.0f;
    std::printf("%lld %lld %d\n", bad, chords, (int)cudaGetLastError());
    return 0;
}
