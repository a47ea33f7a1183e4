// The decode tables of the JPEG path on the host: every 16-bit window of a
// table against its code lengths (csrc/at_jpeg.cu, whose decode compiles for
// the host too).
//
//   jpeg_tables places          tables made until their second levels pass
//                               2^22 entries, and the most a job keeps
//   jpeg_tables shared A B      scans of two files in turn: one set of
//                               tables each
//   jpeg_tables scans A         the tables of each scan of a file, DC and AC,
//                               as its scan header chooses them
#include "../apriltags_fast_b200/csrc/at_jpeg.cu"

extern "C" image_u8_t *image_u8_create(unsigned int, unsigned int) { return nullptr; }

// The code of a window by the code lengths (ITU-T T.81 annex C: codes of a
// length in order, after those of the lengths below); length 0: none.
struct Code {
    int len, sym;
};
static std::vector<Code> codes_of(const uint8_t cnt[17], const uint8_t *vals) {
    std::vector<Code> w(65536, Code{0, 0});
    uint32_t pos = 0;
    for (int l = 1, k = 0; l <= 16; l++)
        for (int i = 0; i < cnt[l]; i++, k++, pos += 1u << (16 - l))
            for (uint32_t p = 0; p < 1u << (16 - l); p++) w[pos + p] = Code{l, vals[k]};
    return w;
}

static int wrong(const JJob &J, const JTab *t, const std::vector<Code> &w, bool ac) {
    int bad = 0;
    for (uint32_t p = 0; p < 65536; p++) {
        const uint32_t e = jdecode(J, t, p << 16 | 0x5a5a);
        const Code c = w[p];
        const int step = !ac ? 1 : c.sym == 0 ? 64 : (c.sym >> 4) + 1;
        bad += jent_len(e) != c.len || jent_size(e) != (c.sym & 15) || jent_bits(e) != c.len + (c.sym & 15) ||
               jent_step(e) != step;
    }
    return bad;
}

static int places() {
    std::vector<uint8_t> pool;
    std::vector<uint32_t> lut2;
    std::vector<JTab> tabs;
    std::vector<std::vector<uint8_t>> vals;
    uint8_t cnt[17] = {};
    cnt[2] = 1, cnt[10] = 160;  // 80 prefixes of 9 bits with two codes each
    int k = 0, same = 0;
    for (; same < 3 && k < 4096; k++) {
        std::vector<uint8_t> v(161);
        for (int i = 0; i < 161; i++) v[i] = (uint8_t)(i * 7 + k * 13 + (k >> 5));
        HTab t;
        if (!htab_define(t, cnt, v.data())) return 2;
        const size_t before = lut2.size();
        tabs.push_back(make_tab(t, k & 1, pool, lut2));
        vals.push_back(v);
        same += lut2.size() == before;
    }
    if (lut2.size() <= (size_t)1 << 22 || k == 4096) {
        printf("second level of %zu entries after %d tables\n", lut2.size(), k);
        return 1;
    }
    JJob J = {};
    J.lut2 = lut2.data();
    J.syms = pool.data();
    int bad = 0;
    for (int i = 0; i < k; i++) {
        const bool edge = (i >= 508 && i <= 518) || i >= k - 6;  // 8192 entries a table: 2^22 at table 512
        if (!edge && i % 37) continue;
        const int n = wrong(J, &tabs[i], codes_of(cnt, vals[i].data()), i & 1);
        if (n) printf("table %d: %d windows\n", i, n);
        bad += n;
    }
    return bad != 0;
}

static HImage parsed(const char *path) {
    FILE *f = fopen(path, "rb");
    std::vector<uint8_t> b(1 << 20);
    b.resize(f ? fread(b.data(), 1, b.size(), f) : 0);
    if (f) fclose(f);
    static std::vector<uint8_t> out(1 << 21);
    HImage im;
    JSink sk;
    sk.p = out.data();
    sk.cap = (int64_t)out.size();
    const int e = parse_image(b.data(), (int64_t)b.size(), 0, im, &sk);
    if (e || im.scans.empty()) {
        printf("%s: error %d\n", path, e);
        exit(3);
    }
    return im;
}

static void add(HJob &J, const HImage &im) {
    add_image(J, im, 0, 0, 256, 1u, [](int, JPlaneDev &) -> size_t { return 0; });
}

static int shared(const char *a, const char *b) {
    const HImage x = parsed(a), y = parsed(b);
    HJob one, J;
    add(one, x);
    add(one, y);
    for (int i = 0; i < 50; i++) {
        add(J, x);
        add(J, y);
    }
    printf("%zu tables, %zu entries; of the two files %zu, %zu\n", J.tabs.size(), J.lut2.size(), one.tabs.size(),
           one.lut2.size());
    return J.tabs.size() != one.tabs.size() || J.lut2.size() != one.lut2.size();
}

static int scans(const char *a) {
    const HImage im = parsed(a);
    HJob H;
    add(H, im);
    JJob J = {};
    J.lut2 = H.lut2.data();
    J.syms = H.syms.data();
    int bad = 0;
    for (size_t s = 0; s < im.scans.size(); s++)
        for (int i = 0; i < im.scans[s].ns; i++)
            for (int ac = 0; ac < 2; ac++) {
                const HTab &t = im.scans[s].tab[ac ? 2 + (im.scans[s].tda[i] & 15) : im.scans[s].tda[i] >> 4];
                std::vector<Code> w(65536, Code{0, 0});
                for (const HRun &r : t.runs)
                    for (uint32_t p = r.start; p < r.end; p++) w[p] = Code{r.len, t.syms[r.sym0 + ((p - r.origin) >> (16 - r.len))]};
                const JScanDev &D = H.scans[s];
                const int n = wrong(J, &H.tabs[D.tab0 + (ac ? D.ac[i] : D.dc[i])], w, ac);
                if (n) printf("scan %zu component %d %s: %d windows\n", s, i, ac ? "AC" : "DC", n);
                bad += n;
            }
    return bad != 0;
}

int main(int argc, char **argv) {
    const std::string m = argc > 1 ? argv[1] : "";
    if (m == "places") return places();
    if (m == "shared" && argc > 3) return shared(argv[2], argv[3]);
    if (m == "scans" && argc > 2) return scans(argv[2]);
    return 9;
}
