// Host side of the linear-MTP path: error state, .almtp parser, alpha-table compiler.
#include "mtp_program.cuh"

#include <algorithm>
#include <cstring>
#include <fstream>
#include <sstream>
#include <string>
#include <vector>

namespace ai2b {

static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int sm_count()
{
    static std::mutex mu;
    static int counts[MAX_DEVICES] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    const bool cached = dev >= 0 && dev < MAX_DEVICES;
    std::lock_guard<std::mutex> guard(mu);
    if (cached && counts[dev] > 0) return counts[dev];
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    if (cached) counts[dev] = n;
    return n;
}

}  // namespace ai2b

using namespace ai2b;

extern "C" const char *ai2b_last_error_string(void) { return ai2b::g_err; }
extern "C" int ai2b_version(void) { return 100; }

// ---------------------------------------------------------------------------------------------
// .almtp parser. Same fields, in the same order, as source/descriptor/mtpr/src/mtpParam.cc:80-200
// reads them; located here by key name rather than by skipping a fixed number of header lines.
// ---------------------------------------------------------------------------------------------
static bool find_key(const std::string &txt, const char *key, size_t &pos)
{
    size_t p = 0;
    const size_t klen = strlen(key);
    while ((p = txt.find(key, p)) != std::string::npos) {
        bool word_start = (p == 0) || !(isalnum((unsigned char)txt[p - 1]) || txt[p - 1] == '_');
        size_t q = p + klen;
        while (q < txt.size() && (txt[q] == ' ' || txt[q] == '\t')) ++q;
        if (word_start && q < txt.size() && txt[q] == '=') {
            pos = q + 1;
            return true;
        }
        p += klen;
    }
    return false;
}

static bool read_int(const std::string &txt, const char *key, int &v)
{
    size_t pos;
    if (!find_key(txt, key, pos)) return false;
    v = (int)strtol(txt.c_str() + pos, nullptr, 10);
    return true;
}

static bool read_list(const std::string &txt, const char *key, std::vector<int> &out)
{
    size_t pos;
    if (!find_key(txt, key, pos)) return false;
    size_t end = txt.find('\n', pos);
    if (end == std::string::npos) end = txt.size();
    out.clear();
    const char *s = txt.c_str() + pos, *e = txt.c_str() + end;
    while (s < e) {
        if (isdigit((unsigned char)*s) || (*s == '-' && s + 1 < e && isdigit((unsigned char)s[1]))) {
            char *nx;
            out.push_back((int)strtol(s, &nx, 10));
            s = nx;
        } else {
            ++s;
        }
    }
    return true;
}

extern "C" int ai2b_mtp_parse_almtp(const char *filename, int *counts, int *basic, int *times, int *mapping)
{
    AI2B_REQUIRE(filename && counts, AI2B_ERR_INVALID, "ai2b_mtp_parse_almtp: NULL argument");
    std::ifstream in(filename);
    AI2B_REQUIRE(in.good(), AI2B_ERR_INVALID, "cannot open MTP template '%s'", filename);
    std::stringstream ss;
    ss << in.rdbuf();
    const std::string txt = ss.str();
    int nm, nb, nt, ns;
    std::vector<int> vb, vt, vm;
    bool ok = read_int(txt, "alpha_moments_count", nm) && read_int(txt, "alpha_index_basic_count", nb) &&
              read_list(txt, "alpha_index_basic", vb) && read_int(txt, "alpha_index_times_count", nt) &&
              read_list(txt, "alpha_index_times", vt) && read_int(txt, "alpha_scalar_moments", ns) &&
              read_list(txt, "alpha_moment_mapping", vm);
    AI2B_REQUIRE(ok, AI2B_ERR_INVALID, "'%s' is not an MTP template (missing alpha_* field)", filename);
    AI2B_REQUIRE((int)vb.size() == 4 * nb && (int)vt.size() == 4 * nt && (int)vm.size() == ns, AI2B_ERR_INVALID,
                 "'%s': table sizes do not match their counts", filename);
    int nmus = 0;
    for (int i = 0; i < nb; i++) nmus = std::max(nmus, vb[4 * i] + 1);   // mtpParam.cc:549-556
    counts[0] = nm; counts[1] = nb; counts[2] = nt; counts[3] = ns; counts[4] = nmus;
    if (basic) memcpy(basic, vb.data(), sizeof(int) * vb.size());
    if (times) memcpy(times, vt.data(), sizeof(int) * vt.size());
    if (mapping) memcpy(mapping, vm.data(), sizeof(int) * vm.size());
    return AI2B_OK;
}

// ---------------------------------------------------------------------------------------------
// Table compiler
// ---------------------------------------------------------------------------------------------
namespace {
struct Blob {
    std::vector<unsigned char> bytes;
    template <typename V>
    size_t add(const std::vector<V> &v)
    {
        size_t off = (bytes.size() + 255) & ~size_t(255);
        bytes.resize(off + std::max<size_t>(sizeof(V) * v.size(), 16));
        if (!v.empty()) memcpy(bytes.data() + off, v.data(), sizeof(V) * v.size());
        return off;
    }
};

// Deals the moments of a phase (by decreasing row count) to `warps` warps of `groups` groups of lanes each: the first
// nwide of them to whole warps, the others to groups, each to the least loaded place, the lowest of equals, completing a
// moment taken as a row. choose() takes the nwide of the least cost; candidates are looked at by a lower bound of their cost,
// so that most are never dealt.
class RowDeal {
public:
    RowDeal(int warps, int groups) : warps(warps), groups(groups), wide_rows(warps), group_rows(warps * groups), load(warps * groups) {}
    int nwide = 0;
    std::vector<int> place;      // warp (of a wide moment) or group

    void choose(const int4 *q, int nq)
    {
        n.resize(nq);
        place.resize(nq);
        for (int i = 0; i < nq; i++) n[i] = q[i].z - q[i].y;
        cand.clear();
        long rest = 0, wide = 0;
        for (int v : n) rest += v;
        for (int i = 0; i < nq; i++) {
            if (i == 0 || n[i] != n[i - 1]) {      // all moments of one row count are dealt alike
                const long sum = wide + (rest + groups - 1) / groups;
                const long longest = std::max<long>({(sum + warps - 1) / warps, n[i], i ? (n[0] + groups - 1) / groups : 0});
                cand.push_back({cost(longest, sum), i});
            }
            wide += (n[i] + groups - 1) / groups;
            rest -= n[i];
        }
        std::stable_sort(cand.begin(), cand.end(), [](const Candidate &x, const Candidate &y) { return x.bound < y.bound; });
        long best = -1;
        int dealt = nwide = 0;
        for (const Candidate &c : cand) {
            if (best >= 0 && (c.bound > best || (c.bound == best && c.wide > nwide))) continue;
            const long v = deal(dealt = c.wide);
            if (best < 0 || v < best || (v == best && c.wide < nwide)) { best = v; nwide = c.wide; }
        }
        if (nq == 0 || dealt != nwide) deal(nwide);
    }
    int length(int w) const { return wide_rows[w] + *std::max_element(group_rows.begin() + w * groups, group_rows.begin() + (w + 1) * groups); }

private:
    struct Candidate { long bound; int wide; };
    const int warps, groups;
    std::vector<Candidate> cand;
    std::vector<int> n, wide_rows, group_rows, load;
    std::vector<unsigned> at_load;      // [load][words]: which places have it

    static long cost(long longest, long sum) { return 60 * longest + 5 * sum; }

    // moments i0 .. i1 to `places` places with the loads load[]; a moment adds size(i) rows and one
    template <typename Size>
    void spread(int i0, int i1, int places, std::vector<int> &rows, Size size)
    {
        if (i0 == i1) return;
        const int words = (places + 31) / 32;
        int most = 0, low = load[0], highest = 0;
        long total = 0;
        for (int p = 0; p < places; p++) { low = std::min(low, load[p]); highest = std::max(highest, load[p]); total += load[p]; }
        for (int i = i0; i < i1; i++) { most = std::max(most, size(i) + 1); total += size(i) + 1; }
        // the least loaded place is never above the mean
        at_load.assign((size_t)words * (std::max<long>(highest, total / places) + most + 1), 0u);
        for (int p = 0; p < places; p++) at_load[(size_t)words * load[p] + p / 32] |= 1u << (p % 32);
        for (int i = i0; i < i1; i++) {
            int w = 0;
            while (at_load[(size_t)words * low + w] == 0)
                if (++w == words) { w = 0; low++; }
            unsigned &set = at_load[(size_t)words * low + w];
            const int p = 32 * w + __builtin_ctz(set);
            set &= set - 1;
            const int to = low + size(i) + 1;
            at_load[(size_t)words * to + p / 32] |= 1u << (p % 32);
            load[p] = to;
            rows[p] += size(i);
            place[i] = p;
        }
    }

    long deal(int nw)
    {
        std::fill(wide_rows.begin(), wide_rows.end(), 0);
        std::fill(group_rows.begin(), group_rows.end(), 0);
        std::fill(load.begin(), load.end(), 0);
        spread(0, nw, warps, wide_rows, [&](int i) { return (n[i] + groups - 1) / groups; });
        for (int p = warps * groups - 1; p >= 0; p--) load[p] = load[p / groups];
        spread(nw, (int)n.size(), warps * groups, group_rows, [&](int i) { return n[i]; });
        long longest = 0, sum = 0;
        for (int w = 0; w < warps; w++) { longest = std::max<long>(longest, length(w)); sum += length(w); }
        return cost(longest, sum);
    }
};
}  // namespace

extern "C" int ai2b_mtp_program_create(int nm, int nb, const int *basic, int nt, const int *times, int ns,
                                       const int *mapping, int nmus, ai2b_mtp_program **out)
{
    AI2B_REQUIRE(out && basic && mapping && (times || nt == 0), AI2B_ERR_INVALID, "ai2b_mtp_program_create: NULL argument");
    AI2B_REQUIRE(nm > 0 && nb > 0 && nt >= 0 && ns > 0 && nb <= nm, AI2B_ERR_INVALID, "ai2b_mtp_program_create: bad counts");
    AI2B_REQUIRE(nm <= 65535, AI2B_ERR_UNSUPPORTED, "alpha_moments_count %d > 65535 (template level > 28?)", nm);
    AI2B_REQUIRE(nmus >= 1 && nmus <= MTP_MAX_MU, AI2B_ERR_UNSUPPORTED, "nmus %d outside 1..%d", nmus, MTP_MAX_MU);

    MtpProgramDev P;
    memset(&P, 0, sizeof(P));
    P.nm = nm; P.nb = nb; P.nt = nt; P.ns = ns; P.nmus = nmus;
    for (int m = 0; m < MTP_MAX_MU; m++) P.kmu[m] = -1;
    for (int i = 0; i < nb; i++) {
        const int *r = basic + 4 * i;
        AI2B_REQUIRE(r[0] >= 0 && r[0] < nmus && r[1] >= 0 && r[2] >= 0 && r[3] >= 0, AI2B_ERR_INVALID,
                     "alpha_index_basic row %d out of range", i);
        int k = r[1] + r[2] + r[3];
        AI2B_REQUIRE(k <= MTP_MAX_DEG, AI2B_ERR_UNSUPPORTED,
                     "basic moment %d has degree %d > %d (template levels above 20 are not supported)", i, k, MTP_MAX_DEG);
        P.kmu[r[0]] = std::max(P.kmu[r[0]], k);
        P.kmax = std::max(P.kmax, k);
    }
    P.doff[0] = 0;
    for (int m = 0; m < nmus; m++) P.doff[m + 1] = P.doff[m] + ncan(P.kmu[m]);
    for (int m = nmus; m < MTP_MAX_MU; m++) P.doff[m + 1] = P.doff[nmus];
    P.ndense = P.doff[nmus];

    // dense numbering and the gather table that turns adjoints of the basic moments into
    // polynomial coefficients {value, d/dux, d/duy, d/duz} per canonical monomial
    std::vector<int> basic_dense(nb);
    std::vector<int4> e4g(P.ndense, make_int4(-1, -1, -1, -1));
    std::vector<int> e4m(P.ndense, 0);
    for (int i = 0; i < nb; i++) {
        const int *r = basic + 4 * i;
        int d = P.doff[r[0]] + canon_index(r[1], r[2], r[3]);
        basic_dense[i] = d;
        AI2B_REQUIRE(e4g[d].x == -1, AI2B_ERR_UNSUPPORTED, "alpha_index_basic row %d duplicates an earlier row", i);
        e4g[d].x = i;
    }
    for (int m = 0; m < nmus; m++)
        for (int k = 0; k <= P.kmu[m]; k++)
            for (int q = 0; q < ndeg(k); q++) {
                Exp3 e = deg_exp(k, q);
                int d = P.doff[m] + ncan(k - 1) + q;
                e4m[d] = (e.x + 1) | ((e.y + 1) << 8) | ((e.z + 1) << 16);
                if (k < P.kmu[m]) {
                    e4g[d].y = e4g[P.doff[m] + canon_index(e.x + 1, e.y, e.z)].x;
                    e4g[d].z = e4g[P.doff[m] + canon_index(e.x, e.y + 1, e.z)].x;
                    e4g[d].w = e4g[P.doff[m] + canon_index(e.x, e.y, e.z + 1)].x;
                }
            }

    std::vector<int> dense_basic(P.ndense, -1);
    std::vector<int4> e4d(P.ndense, make_int4(-1, -1, -1, -1));
    for (int i = 0; i < nb; i++) dense_basic[basic_dense[i]] = i;
    for (int d = 0; d < P.ndense; d++) {
        auto dn = [&](int bi) { return bi >= 0 ? basic_dense[bi] : -1; };
        e4d[d] = make_int4(dn(e4g[d].x), dn(e4g[d].y), dn(e4g[d].z), dn(e4g[d].w));
    }

    // product rows: dependency depth, and the requirement that sources are final before use
    std::vector<int> depth(nm, 0), last_write(nm, -1);
    for (int t = 0; t < nt; t++) {
        const int *r = times + 4 * t;
        AI2B_REQUIRE(r[0] >= 0 && r[0] < nm && r[1] >= 0 && r[1] < nm && r[3] >= 0 && r[3] < nm, AI2B_ERR_INVALID,
                     "alpha_index_times row %d out of range", t);
        last_write[r[3]] = t;
    }
    for (int t = 0; t < nt; t++) {
        const int *r = times + 4 * t;
        AI2B_REQUIRE(last_write[r[0]] < t && last_write[r[1]] < t, AI2B_ERR_UNSUPPORTED,
                     "alpha_index_times row %d reads a moment that a later row still accumulates into", t);
        depth[r[3]] = std::max(depth[r[3]], 1 + std::max(depth[r[0]], depth[r[1]]));
    }
    for (int t = 0; t < nt; t++)
        AI2B_REQUIRE(depth[times[4 * t + 3]] > std::max(depth[times[4 * t]], depth[times[4 * t + 1]]), AI2B_ERR_UNSUPPORTED,
                     "alpha_index_times row %d: inconsistent dependency order", t);
    for (int m = 0; m < nm; m++) P.nlev = std::max(P.nlev, depth[m]);
    AI2B_REQUIRE(P.nlev <= MTP_MAX_LEV, AI2B_ERR_UNSUPPORTED, "product depth %d > %d", P.nlev, MTP_MAX_LEV);

    // The rows of each destination, and the places where each moment is an operand (2 t: as `a` of row t, 2 t + 1: as `b`),
    // one moment behind another. (Everything from here on is made once per set of tables, but a user pays for it with every
    // new model: flat arrays, no allocation per moment. Level 16: 0.25 ms with the upload, 1.06 with lists per moment, heaps
    // and a trial of every split point.)
    auto by_moment = [&](int entries, auto moment_of) {
        std::pair<std::vector<int>, std::vector<int>> r{std::vector<int>(nm + 1, 0), std::vector<int>(entries)};
        for (int i = 0; i < entries; i++) r.first[moment_of(i) + 1]++;
        for (int m = 0; m < nm; m++) r.first[m + 1] += r.first[m];
        std::vector<int> at(r.first.begin(), r.first.end() - 1);
        for (int i = 0; i < entries; i++) r.second[at[moment_of(i)]++] = i;
        return r;
    };
    const auto [row_at, rows_of] = by_moment(nt, [&](int t) { return times[4 * t + 3]; });
    const auto [occ_at, occ_of] = by_moment(2 * nt, [&](int o) { return times[4 * (o >> 1) + (o & 1)]; });
    // The square of a moment: both of its places as an operand (they follow one another) are one adjoint row.
    auto both_places = [&](const int *r) { return r[0] == r[1] && r[2] <= 127; };
    std::vector<int> fwd_count(nm), rev_count(nm);      // rows of each moment
    for (int m = 0; m < nm; m++) { fwd_count[m] = row_at[m + 1] - row_at[m]; rev_count[m] = occ_at[m + 1] - occ_at[m]; }
    for (int t = 0; t < nt; t++) rev_count[times[4 * t]] -= both_places(times + 4 * t);
    // moments of one depth, those with the most rows first
    std::vector<int> members;
    auto moments_of_depth = [&](int lev, const std::vector<int> &count) -> const std::vector<int> & {
        members.clear();
        for (int m = 0; m < nm; m++)
            if (depth[m] == lev && count[m] > 0) members.push_back(m);
        std::stable_sort(members.begin(), members.end(), [&](int x, int y) { return count[x] > count[y]; });
        return members;
    };
    auto bits_f = [](int mult) { const float f = (float)mult; int b; memcpy(&b, &f, 4); return b; };
    auto bits_d = [](int mult) { const double d = mult; long long b; memcpy(&b, &d, 8); return (int)(b >> 32); };
    // forward: destinations by depth, rows contiguous per destination. The flat streams hold the same rows with the
    // multiplier, the moment and a flag on its last row in one word.
    std::vector<int4> fwd_dst, rev_mom;
    std::vector<int2> fwd_rows, rev_ents, fwd_flat, rev_flat;
    fwd_dst.reserve(nm); rev_mom.reserve(nm);
    fwd_rows.reserve(nt); fwd_flat.reserve(nt); rev_ents.reserve(2 * nt); rev_flat.reserve(2 * nt);
    auto add_row = [&](std::vector<int2> &rows, std::vector<int2> &flat, int xy, int mult, int m, bool last) {
        rows.push_back(make_int2(xy, bits_f(mult)));
        flat.push_back(make_int2(xy, (mult & 0xff) | (last ? 0x100 : 0) | (m << 16)));
    };
    P.fwd_lev_off[0] = P.fwd_lev_row[0] = 0;
    for (int lev = 1; lev <= MTP_MAX_LEV; lev++) {
        if (lev <= P.nlev)
            for (int m : moments_of_depth(lev, fwd_count)) {
                const int rb = (int)fwd_rows.size(), re = rb + fwd_count[m];
                for (int i = row_at[m]; i < row_at[m + 1]; i++) {
                    const int *r = times + 4 * rows_of[i];
                    add_row(fwd_rows, fwd_flat, r[0] | (r[1] << 16), r[2], m, i + 1 == row_at[m + 1]);
                }
                fwd_dst.push_back(make_int4(m, rb, re, 0));
            }
        P.fwd_lev_off[lev] = (int)fwd_dst.size();
        P.fwd_lev_row[lev] = (int)fwd_rows.size();
    }
    // reverse: sources by depth, deepest first; adjoint[m] += sum adjoint[dst] * mult * M[other]
    P.rev_lev_off[0] = P.rev_lev_row[0] = 0;
    for (int k = 0; k < MTP_MAX_LEV; k++) {
        if (k < P.nlev)
            for (int m : moments_of_depth(P.nlev - 1 - k, rev_count)) {
                const int rb = (int)rev_ents.size();
                for (int i = occ_at[m]; i < occ_at[m + 1]; i++) {
                    const int o = occ_of[i], *r = times + 4 * (o >> 1);
                    const bool both = !(o & 1) && both_places(r);
                    if (both) i++;
                    add_row(rev_ents, rev_flat, r[1 - (o & 1)] | (r[3] << 16), both ? 2 * r[2] : r[2], m, i + 1 == occ_at[m + 1]);
                }
                rev_mom.push_back(make_int4(m, rb, (int)rev_ents.size(), 0));
            }
        P.rev_lev_off[k + 1] = (int)rev_mom.size();
        P.rev_lev_row[k + 1] = (int)rev_ents.size();
    }
    for (int t = 0; t < nt; t++) {
        AI2B_REQUIRE(times[4 * t + 2] <= 255, AI2B_ERR_UNSUPPORTED, "product multiplier %d > 255", times[4 * t + 2]);
        AI2B_REQUIRE(times[4 * t + 2] >= 0, AI2B_ERR_UNSUPPORTED, "negative product multiplier in row %d", t);
    }
    std::vector<int> map(mapping, mapping + ns);
    for (int s = 0; s < ns; s++)
        AI2B_REQUIRE(map[s] >= 0 && map[s] < nm, AI2B_ERR_INVALID, "alpha_moment_mapping[%d] out of range", s);

    // row streams (see mtp_program.cuh)
    std::vector<int2> stream_d[4], stream_f[4], stream_warp[4];
    std::vector<int> constant;
    {
        std::vector<char> is_source(nm, 0);
        for (int t = 0; t < nt; t++) { is_source[times[4 * t]] = 1; is_source[times[4 * t + 1]] = 1; }
        // moments whose adjoint is just their seed (0 where no scalar is mapped to them, as for products that nothing uses);
        // every other adjoint is written by a gather phase
        for (int m = 0; m < nm; m++)
            if (!is_source[m]) constant.push_back(m);
        P.n_adj_const = (int)constant.size();
        for (int m = nb; m < nm; m++)
            if (fwd_count[m] == 0) constant.push_back(m);
        P.n_constant = (int)constant.size();
    }
    for (int k = 0; k < 4; k++) {
        const int groups = k % 2 == 0 ? 2 : 4, warps = k < 2 ? MTP_PAIR_WARPS : MTP_PAIR_FEW;
        P.stream[k].nrows = 0;
        if (nm > 2046 || nt == 0 || (k >= 2 && nt > MTP_PAIR_FEW_ROWS)) continue;      // the completed moment has 11 bits
        RowDeal deal(warps, groups);
        std::vector<int> row0(warps), next(warps * groups);      // rows that the next records of a warp, a group go to
        stream_warp[k].reserve(2 * P.nlev * warps);
        stream_d[k].reserve(4 * nt + 64 * P.nlev);
        stream_f[k].reserve(4 * nt + 64 * P.nlev);
        for (int phase = 0; phase < 2 * P.nlev; phase++) {
            // A phase lasts as long as its longest warp, and a few moments have many times the rows of the others (69
            // against 13 on average in the last phase of level 16). The moments with the most rows are therefore split
            // over all groups of a warp; the others go to single groups. How many are split is chosen per phase by a cost: a row
            // of the longest warp waits for about 60 cycles, a row of any warp takes about 5 of its scheduler's issue slots.
            const bool fwd = phase < P.nlev;
            const int4 *q = fwd ? fwd_dst.data() + P.fwd_lev_off[phase] : rev_mom.data() + P.rev_lev_off[phase - P.nlev];
            const int nq = fwd ? P.fwd_lev_off[phase + 1] - P.fwd_lev_off[phase] : P.rev_lev_off[phase - P.nlev + 1] - P.rev_lev_off[phase - P.nlev];
            const std::vector<int2> &flat = fwd ? fwd_flat : rev_flat;
            deal.choose(q, nq);
            size_t first = stream_d[k].size();
            for (int w = 0; w < warps; w++) {
                row0[w] = (int)(first / groups);
                stream_warp[k].push_back(make_int2(row0[w], deal.length(w)));
                first += (size_t)deal.length(w) * groups;
            }
            stream_d[k].resize(first, make_int2(0, 0));
            stream_f[k].resize(first, make_int2(0, 0));
            auto put = [&](int row, int g, int at, bool empty, int done) {      // record `at` of the flat stream
                const int mult = empty ? 0 : flat[at].y & 0xff, x = flat[at].x & 0xffff, y = (flat[at].x >> 16) & 0xffff;
                const int xy = fwd ? x | (y << 16) : y | (x << 16);             // (flat adjoint rows hold {other, dst})
                stream_d[k][(size_t)row * groups + g] = make_int2(xy, bits_d(mult) | done);
                stream_f[k][(size_t)row * groups + g] = make_int2(xy, bits_f(mult) | done);
            };
            for (int g = 0; g < warps * groups; g++) next[g] = row0[g / groups];
            for (int i = 0; i < nq; i++) {
                const int n = q[i].z - q[i].y, place = deal.place[i];
                if (i < deal.nwide) {
                    const int rows = (n + groups - 1) / groups;
                    for (int r = 0; r < rows; r++)
                        for (int g = 0; g < groups; g++) {
                            const int at = r * groups + g;      // (empty records: operands that are written by then)
                            put(next[place * groups + g]++, g, at < n ? q[i].y + at : q[i].y, at >= n, r + 1 == rows ? (q[i].x + 1) | MTP_PAIR_WIDE : 0);
                        }
                } else {
                    for (int r = 0; r < n; r++) put(next[place]++, place % groups, q[i].y + r, false, r + 1 == n ? q[i].x + 1 : 0);
                }
            }
        }
        for (int g = 0; g < 2 * groups; g++) { stream_d[k].push_back(make_int2(0, 0)); stream_f[k].push_back(make_int2(0, 0)); }   // read ahead
        P.stream[k].nrows = (int)(stream_d[k].size() / groups);
    }

    Blob blob;
    blob.bytes.reserve(64 * 1024 + 128 * (size_t)(nm + nt) + 16 * (stream_d[0].size() + stream_d[1].size()));
    size_t o_c = blob.add(constant), o_sd[4], o_sf[4], o_sw[4];
    for (int k = 0; k < 4; k++) { o_sd[k] = blob.add(stream_d[k]); o_sf[k] = blob.add(stream_f[k]); o_sw[k] = blob.add(stream_warp[k]); }
    size_t o_bd = blob.add(basic_dense), o_db = blob.add(dense_basic), o_e4d = blob.add(e4d), o_g = blob.add(e4g), o_m = blob.add(e4m), o_fd = blob.add(fwd_dst),
           o_rm = blob.add(rev_mom), o_map = blob.add(map);
    size_t o_frow = blob.add(fwd_rows), o_rent = blob.add(rev_ents), o_ff = blob.add(fwd_flat), o_rf = blob.add(rev_flat);
    ai2b_mtp_program *prog = new ai2b_mtp_program;
    prog->blob_bytes = blob.bytes.size();
    prog->d_blob = nullptr;
    cudaError_t e = cudaGetDevice(&prog->device);
    if (e == cudaSuccess) e = cudaMalloc(&prog->d_blob, prog->blob_bytes);
    if (e == cudaSuccess) e = cudaMemcpy(prog->d_blob, blob.bytes.data(), prog->blob_bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        set_error("ai2b_mtp_program_create: %s", cudaGetErrorString(e));
        if (prog->d_blob) cudaFree(prog->d_blob);
        delete prog;
        return AI2B_ERR_CUDA;
    }
    unsigned char *b = (unsigned char *)prog->d_blob;
    P.basic_dense = (const int *)(b + o_bd);
    P.dense_basic = (const int *)(b + o_db);
    P.e4d = (const int4 *)(b + o_e4d);
    P.e4g = (const int4 *)(b + o_g);
    P.e4m = (const int *)(b + o_m);
    P.fwd_dst = (const int4 *)(b + o_fd);
    P.rev_mom = (const int4 *)(b + o_rm);
    P.map = (const int *)(b + o_map);
    P.fwd_rows = (const int2 *)(b + o_frow);
    P.rev_ents = (const int2 *)(b + o_rent);
    P.fwd_flat = (const int2 *)(b + o_ff);
    P.rev_flat = (const int2 *)(b + o_rf);
    P.constant = (const int *)(b + o_c);
    for (int k = 0; k < 4; k++) {
        P.stream[k].row_d = (const int2 *)(b + o_sd[k]);
        P.stream[k].row_f = (const int2 *)(b + o_sf[k]);
        P.stream[k].warp = (const int2 *)(b + o_sw[k]);
    }
    prog->dev = P;
    *out = prog;
    return AI2B_OK;
}

extern "C" void ai2b_mtp_program_destroy(ai2b_mtp_program *prog)
{
    if (!prog) return;
    if (prog->d_blob) cudaFree(prog->d_blob);
    delete prog;
}
