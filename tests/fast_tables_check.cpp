// Walks the tables that the fast and scores builds read as their kernels do,
// for every channel that the firing pass can take from its blocks of four.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "tl_internal.h"

// N species, M channels, order 2S for the first two_s channels, columns of up
// to `most` entries.
static tl_model* network(int N, int M, int two_s, int most, unsigned seed) {
    srand(seed);
    std::vector<int64_t> x0((size_t)N, 100);
    std::vector<double> rate((size_t)M, 0.5);
    std::vector<int32_t> cp(1, 0), row;
    std::vector<int8_t> v;
    for (int j = 0; j < M; ++j) {
        const int s = j % N;
        row.push_back(s);
        v.push_back((int8_t)(j < two_s ? -2 : -1));
        const int products = j == 0 ? most - 1 : rand() % most;
        for (int q = 1; q <= products && q < N; ++q) {
            row.push_back((s + q) % N);
            v.push_back((int8_t)(1 + rand() % 3));
        }
        cp.push_back((int32_t)row.size());
    }
    tl_model_desc d{};
    d.n_species = N;
    d.n_channels = M;
    d.nnz = cp.back();
    d.pop_bits = 32;
    d.x0 = x0.data();
    d.rate = rate.data();
    d.col_ptr = cp.data();
    d.row_ind = row.data();
    d.stoich = v.data();
    tl_model* m = nullptr;
    if (tl_model_create(&d, &m) != TL_OK) {
        printf("model: %s\n", tl_last_error());
        exit(2);
    }
    return m;
}

static int check(int N, int M, int two_s, int most) {
    tl_model* m = network(N, M, two_s, most, (unsigned)(31 * N + M));
    tl::DevModel d;
    std::vector<unsigned char> out;
    tl::fast_tables(m->h, d, out);
    int bad = 0;
    const auto word = [&](int section, size_t i) -> uint32_t {
        const size_t at = (size_t)section + 4 * i;
        if (at + 4 > out.size()) {
            ++bad;
            return 0;
        }
        return *reinterpret_cast<const uint32_t*>(out.data() + at);
    };
    for (int j = 0; j < (M + 3) / 4 * 4 && d.fast_ok; ++j) {
        size_t c0 = (size_t)j, n = 1;
        if (d.t_cp >= 0) {
            c0 = word(d.t_cp, (size_t)j);
            n = word(d.t_cp, (size_t)j + 1) - c0;
        }
        if (n > out.size() || 16 * (c0 + n) > out.size()) {
            ++bad;
            continue;
        }
        std::map<int, int> got, want;
        for (size_t q = 4 * c0; q < 4 * (c0 + n); ++q) {
            const uint32_t e = word(d.t_col, q);
            if (e & 0xfffu) got[(int)(e >> 14)] += (int)(e << 20) >> 20;
        }
        if (j < M)
            for (int q = m->h.net_cp[(size_t)j]; q < m->h.net_cp[(size_t)j + 1]; ++q)
                want[m->h.net_rv[(size_t)q] >> 3] += (m->h.net_rv[(size_t)q] & 7) - 2;
        bad += got != want;
    }
    if (bad || !d.fast_ok) printf("%d species, %d channels, %d of 2S, up to %d entries: %d wrong\n", N, M, two_s, most, bad);
    tl_model_destroy(m);
    return bad || !d.fast_ok;
}

int main() {
    int wrong = 0;
    for (int N : {8, 33, 300})
        for (int M : {N + 1, N + 2, N + 3, N + 4, 2 * N + 1})
            for (int two_s : {0, N})
                for (int most : {3, 4, 5}) wrong += check(N, M, two_s, most);
    return wrong ? 1 : 0;
}
