// td_cert.cu -- certificate records: the reference's on-disk byte format, a
// batched file sink, and a device replay of symbol witnesses with the
// checker's rules.
//
// Format (emitter/src/main/java/br/unb/cic/tdp/base/CertificateCodec.java:22-147):
//   key   = omega in one-line notation, 5 bits per symbol, most significant
//           bit first, zero padding to a whole byte
//   value = the witness as consecutive 15-bit fields (a, b, c), same bit order
// Replay (CertificateValidator.java:14-50): 1 <= moves <= maxMoves; each move
// holds three distinct symbols at increasing positions of the current beta
// array; omega <- omega . (a b c)^-1; beta <- block swap; omega . beta stays
// rho; omega ends as the identity.
#include <cuda_runtime.h>

#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <deque>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#define TD_API extern "C" __attribute__((visibility("default")))

#include "td_core.cuh"
#define TD_CERT_MAX_N 17
#define TD_CERT_MAX_MOVES 9

namespace {

inline void put5(uint8_t *buf, int bit, int v) {
    for (int b = 0; b < 5; ++b) {
        const int o = bit + b;
        buf[o >> 3] |= (uint8_t)(((v >> (4 - b)) & 1) << (7 - (o & 7)));
    }
}

inline int get5(const uint8_t *buf, int bit) {
    int v = 0;
    for (int b = 0; b < 5; ++b) {
        const int o = bit + b;
        v = (v << 1) | ((buf[o >> 3] >> (7 - (o & 7))) & 1);
    }
    return v;
}

inline bool padding_zero(const uint8_t *in, int len, int payload_bits) {
    if (len != (payload_bits + 7) / 8) return false;
    const int pad = 8 * len - payload_bits;
    return pad == 0 || (in[len - 1] & ((1 << pad) - 1)) == 0;
}

}  // namespace

// Key bytes for omega over n symbols (1 <= n <= 32, symbols < 32).  Returns
// the length or -1.
TD_API int td_codec_key(const uint8_t *omega, int n, uint8_t *out, int cap) {
    if (n <= 0 || n > 32) return -1;
    const int len = (5 * n + 7) / 8;
    if (cap < len) return -1;
    std::memset(out, 0, (size_t)len);
    for (int x = 0; x < n; ++x) {
        if (omega[x] >= 32) return -1;
        put5(out, 5 * x, omega[x]);
    }
    return len;
}

// Value bytes for `count` symbol triples (abc[3*m..3*m+2]).
TD_API int td_codec_value(const uint8_t *abc, int count, uint8_t *out, int cap) {
    if (count <= 0) return -1;
    const int len = (15 * count + 7) / 8;
    if (cap < len) return -1;
    std::memset(out, 0, (size_t)len);
    for (int m = 0; m < 3 * count; ++m) {
        if (abc[m] >= 32) return -1;
        put5(out, 5 * m, abc[m]);
    }
    return len;
}

TD_API int td_codec_decode_key(const uint8_t *in, int len, int n, uint8_t *omega) {
    if (!in || n <= 0 || n > 32 || !padding_zero(in, len, 5 * n)) return -1;
    for (int x = 0; x < n; ++x) omega[x] = (uint8_t)get5(in, 5 * x);
    return n;
}

// Decodes a value into symbol triples; returns the move count or -1 for a
// truncated value or nonzero padding (CertificateCodec.java:75-97,120-129).
TD_API int td_codec_decode_value(const uint8_t *in, int len, uint8_t *abc, int cap_moves) {
    if (!in || len <= 0) return -1;
    const int count = (8 * len) / 15;
    if (count == 0 || !padding_zero(in, len, 15 * count) || count > cap_moves) return -1;
    for (int m = 0; m < 3 * count; ++m) abc[m] = (uint8_t)get5(in, 5 * m);
    return count;
}

// ---- device replay of symbol witnesses ------------------------------------
//
// One thread per record.  The records' strides (17 and 27 bytes) leave no
// thread an aligned word, so a block first copies its records to shared memory
// with 16-byte loads.  Where beta is a permutation, the thread then keeps the
// position of every symbol, one byte each in five registers: a block swap adds
// to the positions of one block and subtracts from those of the other, four
// symbols per operation, and keeps omega . beta = rho by itself (the three
// symbols that get another predecessor are those whose image the move of omega
// exchanges), so omega is the identity at the end exactly when the array reads
// rho.  A beta that is no permutation takes the rules step by step.
//
// Integer issue bounds it, about 1,100 instructions per record, with memory
// at a fifth of its rate.  The step-by-step form on byte arrays in local memory
// took 611 us for 2^20 records of S_16, this one 70 us.

#define TD_REPLAY_THREADS 128

// Steps through the rules on byte arrays (any beta whose symbols are below n).
__device__ __noinline__ bool td_replay_steps(const uint8_t *beta, const uint8_t *omega, const uint8_t *abc, int n,
                                             int dep) {
    uint8_t b[TD_CERT_MAX_N], o[TD_CERT_MAX_N], rho[TD_CERT_MAX_N], nb[TD_CERT_MAX_N];
    for (int x = 0; x < n; ++x) {
        b[x] = beta[x];
        o[x] = omega[x];
    }
    // rho = omega . beta (beta read as the cycle b0 -> b1 -> ...)
    for (int x = 0; x < n; ++x) rho[b[x]] = o[b[(x + 1) % n]];
    for (int m = 0; m < dep; ++m) {
        const int a = abc[3 * m], c2 = abc[3 * m + 1], c3 = abc[3 * m + 2];
        if (a == c2 || c2 == c3 || a == c3 || a >= n || c2 >= n || c3 >= n) return false;
        int pa = -1, pb = -1, pc = -1;
        for (int x = 0; x < n; ++x) {
            if (b[x] == a) pa = x;
            if (b[x] == c2) pb = x;
            if (b[x] == c3) pc = x;
        }
        if (!(pa >= 0 && pa < pb && pb < pc)) return false;
        // omega <- omega . (a b c)^-1
        const uint8_t oa = o[a], ob = o[c2], oc = o[c3];
        o[a] = oc;
        o[c2] = oa;
        o[c3] = ob;
        int w = 0;
        for (int x = 0; x < pa; ++x) nb[w++] = b[x];
        for (int x = pb; x < pc; ++x) nb[w++] = b[x];
        for (int x = pa; x < pb; ++x) nb[w++] = b[x];
        for (int x = pc; x < n; ++x) nb[w++] = b[x];
        for (int x = 0; x < n; ++x) b[x] = nb[x];
        for (int x = 0; x < n; ++x)
            if (o[b[(x + 1) % n]] != rho[b[x]]) return false;  // target preserved
    }
    for (int x = 0; x < n; ++x)
        if (o[x] != x) return false;
    return true;
}

// Copies `bytes` bytes of a block's records to shared memory: 16 bytes per
// load where the source allows it (a block's records start at a multiple of
// 128 records, 16 bytes for either stride), single bytes otherwise.
__device__ __forceinline__ void td_stage(uint8_t *dst, const uint8_t *__restrict__ src, int bytes) {
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        done = bytes & ~15;
        for (int i = 16 * threadIdx.x; i < done; i += 16 * TD_REPLAY_THREADS)
            *reinterpret_cast<uint4 *>(dst + i) = __ldg(reinterpret_cast<const uint4 *>(src + i));
    }
    for (int i = done + threadIdx.x; i < bytes; i += TD_REPLAY_THREADS) dst[i] = __ldg(src + i);
}

// Byte i (0..16) of five words.
__device__ __forceinline__ uint32_t td_byte_of(const uint32_t (&w)[5], uint32_t i) {
    const uint32_t lo = __byte_perm(w[0], w[1], i & 7u), hi = __byte_perm(w[2], w[3], i & 7u);
    return (i < 8u ? lo : i < 16u ? hi : w[4]) & 0xffu;
}

__global__ void __launch_bounds__(TD_REPLAY_THREADS)
    td_replay_symbols_kernel(const uint8_t *__restrict__ beta, const uint8_t *__restrict__ omega,
                             const uint8_t *__restrict__ n_arr, const uint8_t *__restrict__ maxm,
                             const uint8_t *__restrict__ depth, const uint8_t *__restrict__ abc,
                             uint8_t *__restrict__ ok, int count) {
    __shared__ __align__(16) uint8_t sb[TD_REPLAY_THREADS * TD_CERT_MAX_N];
    __shared__ __align__(16) uint8_t so[TD_REPLAY_THREADS * TD_CERT_MAX_N];
    __shared__ __align__(16) uint8_t sm[TD_REPLAY_THREADS * 3 * TD_CERT_MAX_MOVES];
    const size_t first = (size_t)blockIdx.x * TD_REPLAY_THREADS;
    const int here = (int)min((size_t)TD_REPLAY_THREADS, (size_t)count - first);
    td_stage(sb, beta + first * TD_CERT_MAX_N, here * TD_CERT_MAX_N);
    td_stage(so, omega + first * TD_CERT_MAX_N, here * TD_CERT_MAX_N);
    td_stage(sm, abc + first * 3 * TD_CERT_MAX_MOVES, here * 3 * TD_CERT_MAX_MOVES);
    __syncthreads();
    if ((int)threadIdx.x >= here) return;
    const size_t idx = first + threadIdx.x;
    const uint8_t *b = sb + threadIdx.x * TD_CERT_MAX_N, *o = so + threadIdx.x * TD_CERT_MAX_N,
                  *t = sm + threadIdx.x * 3 * TD_CERT_MAX_MOVES;
    const int n = n_arr[idx], mm = maxm[idx], dep = depth[idx];
    bool good = n >= 3 && n <= TD_CERT_MAX_N && dep >= 1 && dep <= mm && dep <= TD_CERT_MAX_MOVES;
    if (good) {
        uint32_t seen = 0;
        bool canonical = true, below = true;
#pragma unroll
        for (int x = 0; x < TD_CERT_MAX_N; ++x) {
            const uint32_t bx = b[x], ox = o[x];
            if (x < n) {
                below = below && bx < (uint32_t)n && ox < (uint32_t)n;
                canonical = canonical && bx == (uint32_t)x;
                seen |= 1u << (bx & 31u);
            }
        }
        if (!below) {
            good = false;
        } else if (seen != (1u << n) - 1u) {
            good = td_replay_steps(b, o, t, n, dep);
        } else {
            // P: the position of each symbol, one byte each
            uint32_t P[5] = {0x03020100u, 0x07060504u, 0x0b0a0908u, 0x0f0e0d0cu, 0x10u};
            if (!canonical) {
#pragma unroll
                for (int w = 0; w < 5; ++w) P[w] = 0;
#pragma unroll 1
                for (int x = 0; x < n; ++x) {
                    const uint32_t s = b[x], v = (uint32_t)x << (8 * (s & 3u));
#pragma unroll
                    for (int w = 0; w < 5; ++w) P[w] |= (s >> 2) == (uint32_t)w ? v : 0u;
                }
            }
            const uint32_t H = 0x80808080u, ONE = 0x01010101u;
#pragma unroll 1
            for (int m = 0; m < dep; ++m) {
                const uint32_t a = t[3 * m], c2 = t[3 * m + 1], c3 = t[3 * m + 2];
                if (max(a, max(c2, c3)) >= (uint32_t)n) { good = false; break; }
                const uint32_t pa = td_byte_of(P, a), pb = td_byte_of(P, c2), pc = td_byte_of(P, c3);
                if (!(pa < pb && pb < pc)) { good = false; break; }  // equal symbols share a position
#pragma unroll
                for (int w = 0; w < 5; ++w) {
                    // 0x80 in the bytes not below each cut; positions stay below 0x80
                    const uint32_t ga = (P[w] | H) - pa * ONE, gb = (P[w] | H) - pb * ONE, gc = (P[w] | H) - pc * ONE;
                    const uint32_t first_block = (ga & ~gb & H) >> 7, second_block = (gb & ~gc & H) >> 7;
                    P[w] += first_block * (pc - pb) - second_block * (pb - pa);
                }
            }
            if (good) {
                // the array reads rho: rho of the symbol at x, which is omega of
                // the next one in beta, has the next position
                if (canonical) {
#pragma unroll
                    for (int x = 0; x < TD_CERT_MAX_N; ++x) {
                        if (x < n) {
                            const uint32_t at = (P[x >> 2] >> (8 * (x & 3))) & 0xffu;
                            const uint32_t next = at + 1 == (uint32_t)n ? 0u : at + 1;
                            good = good && td_byte_of(P, o[x + 1 == n ? 0 : x + 1]) == next;
                        }
                    }
                } else {
#pragma unroll 1
                    for (int x = 0; x < n && good; ++x) {
                        const uint32_t at = td_byte_of(P, b[x]);
                        const uint32_t next = at + 1 == (uint32_t)n ? 0u : at + 1;
                        good = td_byte_of(P, o[b[x + 1 == n ? 0 : x + 1]]) == next;
                    }
                }
            }
        }
    }
    ok[idx] = good ? 1 : 0;
}

// Replays `count` symbol witnesses on the device (all pointers are device
// pointers): beta/omega stride 17, abc stride 27 (9 triples).  ok[i] = 1
// when witness i is accepted.
TD_API int td_replay_symbols_device(int count, const uint8_t *d_beta, const uint8_t *d_omega, const uint8_t *d_n,
                                    const uint8_t *d_max_moves, const uint8_t *d_depth, const uint8_t *d_abc,
                                    uint8_t *d_ok, void *stream, char *err, size_t errlen) {
    if (count <= 0) return 0;
    td_replay_symbols_kernel<<<(unsigned)(((size_t)count + TD_REPLAY_THREADS - 1) / TD_REPLAY_THREADS),
                               TD_REPLAY_THREADS, 0, (cudaStream_t)stream>>>(d_beta, d_omega, d_n, d_max_moves,
                                                                             d_depth, d_abc, d_ok, count);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        if (err && errlen) std::snprintf(err, errlen, "td_replay_symbols_device: %s", cudaGetErrorString(e));
        return 3;
    }
    return 0;
}

// Loads the replay kernel on the current device (called when the engine sets
// a device up, so that its first launch never waits for loading while the
// per-call server's resident launch runs).  Returns a cudaError_t.
int td_cert_preload(void) {
    cudaFuncAttributes a;
    return (int)cudaFuncGetAttributes(&a, td_replay_symbols_kernel);
}

// ---- batched certificate sink ----------------------------------------------
//
// AsyncCertificateWriter semantics (AsyncCertificateWriter.java:50-116): one
// writer thread drains a queue of (key, value) records in batches and flushes
// on a period; the first write failure is kept and reported to every later
// call.  Without RocksDB the store is a flat file of records
// [u8 key_len][u8 value_len][key][value].

namespace {

struct CertWriter {
    FILE *f = nullptr;
    std::mutex mu;
    std::condition_variable cv;
    std::deque<std::vector<uint8_t>> q;
    std::thread th;
    bool stop = false;
    int failed = 0;
    double flush_s = 5.0;
    uint64_t written = 0;

    void run() {
        auto last = std::chrono::steady_clock::now();
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            cv.wait_for(lk, std::chrono::milliseconds(50), [&] { return stop || !q.empty(); });
            std::deque<std::vector<uint8_t>> batch;
            batch.swap(q);
            const bool done = stop;
            lk.unlock();
            for (auto &r : batch)
                if (!failed && std::fwrite(r.data(), 1, r.size(), f) != r.size()) failed = 1;
            const auto now = std::chrono::steady_clock::now();
            if (done || std::chrono::duration<double>(now - last).count() >= flush_s) {
                if (std::fflush(f) != 0) failed = 1;
                last = now;
            }
            lk.lock();
            written += batch.size();
            if (done && q.empty()) break;
        }
    }
};

}  // namespace

TD_API void *td_cert_writer_open(const char *path, double flush_seconds) {
    FILE *f = std::fopen(path, "ab");
    if (!f) return nullptr;
    auto *w = new CertWriter();
    w->f = f;
    w->flush_s = flush_seconds > 0 ? flush_seconds : 5.0;
    w->th = std::thread([w] { w->run(); });
    return w;
}

// Queues one certificate: omega one-line over n symbols and `count` symbol
// triples.  Returns 0, -1 for an unencodable record, -2 after a write failure.
TD_API int td_cert_writer_enqueue(void *handle, const uint8_t *omega, int n, const uint8_t *abc, int count) {
    auto *w = static_cast<CertWriter *>(handle);
    if (!w) return -1;
    uint8_t key[32], val[64];
    const int kl = td_codec_key(omega, n, key, sizeof key);
    const int vl = td_codec_value(abc, count, val, sizeof val);
    if (kl < 0 || vl < 0) return -1;
    std::vector<uint8_t> rec(2 + kl + vl);
    rec[0] = (uint8_t)kl;
    rec[1] = (uint8_t)vl;
    std::memcpy(&rec[2], key, kl);
    std::memcpy(&rec[2 + kl], val, vl);
    std::lock_guard<std::mutex> g(w->mu);
    if (w->failed) return -2;
    w->q.push_back(std::move(rec));
    w->cv.notify_one();
    return 0;
}

// Drains, flushes and closes; returns the number of records written or -2.
TD_API long long td_cert_writer_close(void *handle) {
    auto *w = static_cast<CertWriter *>(handle);
    if (!w) return -1;
    {
        std::lock_guard<std::mutex> g(w->mu);
        w->stop = true;
    }
    w->cv.notify_one();
    w->th.join();
    const int failed = w->failed || std::fclose(w->f) != 0;
    const long long n = (long long)w->written;
    delete w;
    return failed ? -2 : n;
}

// Queues the found witnesses of a batch: omega/beta stride 17 (the caller's
// pair), n symbols each, results as td_result records (caller positions).
// Returns the number queued, -1 for an unencodable record, -2 after a write
// failure.
TD_API long long td_cert_writer_enqueue_batch(void *handle, int count, const uint8_t *beta, const uint8_t *omega,
                                              const uint8_t *n, const td_result *results) {
    auto *w = static_cast<CertWriter *>(handle);
    if (!w) return -1;
    std::deque<std::vector<uint8_t>> recs;
    for (int i = 0; i < count; ++i) {
        const td_result &r = results[i];
        if (r.status != TD_FOUND || r.depth <= 0 || r.depth > TD_CERT_MAX_MOVES) continue;
        const int N = n[i];
        if (N < 3 || N > TD_CERT_MAX_N) return -1;
        uint8_t cur[TD_CERT_MAX_N], nxt[TD_CERT_MAX_N], abc[3 * TD_CERT_MAX_MOVES];
        std::memcpy(cur, beta + (size_t)i * TD_CERT_MAX_N, (size_t)N);
        for (int d = 0; d < r.depth; ++d) {  // GPUSortingSearch.java:229-238
            const int a = r.moves[d] & 31, b = (r.moves[d] >> 5) & 31, c = (r.moves[d] >> 10) & 31;
            if (!(a < b && b < c && c < N)) return -1;
            abc[3 * d] = cur[a];
            abc[3 * d + 1] = cur[b];
            abc[3 * d + 2] = cur[c];
            int k = 0;
            for (int x = 0; x < a; ++x) nxt[k++] = cur[x];
            for (int x = b; x < c; ++x) nxt[k++] = cur[x];
            for (int x = a; x < b; ++x) nxt[k++] = cur[x];
            for (int x = c; x < N; ++x) nxt[k++] = cur[x];
            std::memcpy(cur, nxt, (size_t)N);
        }
        uint8_t key[32], val[64];
        const int kl = td_codec_key(omega + (size_t)i * TD_CERT_MAX_N, N, key, sizeof key);
        const int vl = td_codec_value(abc, r.depth, val, sizeof val);
        if (kl < 0 || vl < 0) return -1;
        std::vector<uint8_t> rec(2 + kl + vl);
        rec[0] = (uint8_t)kl;
        rec[1] = (uint8_t)vl;
        std::memcpy(&rec[2], key, kl);
        std::memcpy(&rec[2 + kl], val, vl);
        recs.push_back(std::move(rec));
    }
    std::lock_guard<std::mutex> g(w->mu);
    if (w->failed) return -2;
    const long long q = (long long)recs.size();
    for (auto &r : recs) w->q.push_back(std::move(r));
    w->cv.notify_one();
    return q;
}

// Reads up to `cap` records of a certificate file written for domains of n
// symbols into omega (stride 17), abc (stride 27) and depth.  Returns the
// number read, or -1 for a malformed record.
TD_API long long td_cert_read_file(const char *path, int n, long long cap, uint8_t *omega, uint8_t *abc,
                                   uint8_t *depth) {
    FILE *f = std::fopen(path, "rb");
    if (!f) return -1;
    long long k = 0;
    uint8_t hdr[2], buf[96];
    while (k < cap && std::fread(hdr, 1, 2, f) == 2) {
        const int kl = hdr[0], vl = hdr[1];
        if (kl + vl > (int)sizeof buf || std::fread(buf, 1, (size_t)(kl + vl), f) != (size_t)(kl + vl)) {
            std::fclose(f);
            return -1;
        }
        if (td_codec_decode_key(buf, kl, n, omega + (size_t)k * TD_CERT_MAX_N) < 0) {
            std::fclose(f);
            return -1;
        }
        const int m = td_codec_decode_value(buf + kl, vl, abc + (size_t)k * 27, TD_CERT_MAX_MOVES);
        if (m < 0) {
            std::fclose(f);
            return -1;
        }
        depth[k] = (uint8_t)m;
        ++k;
    }
    std::fclose(f);
    return k;
}

// Caller pairs of S_n permutations (perms int8 stride 16): beta = (0..n),
// omega one-line over n+1 symbols (stride 17).
TD_API void td_pairs_from_perms(int count, const int8_t *perms, const uint8_t *n, uint8_t *beta, uint8_t *omega) {
    for (int i = 0; i < count; ++i) {
        int init;
        if (n[i] > TD_CERT_MAX_N - 1) continue;
        td_perm_to_pair(perms + (size_t)i * 16, n[i], beta + (size_t)i * TD_CERT_MAX_N,
                        omega + (size_t)i * TD_CERT_MAX_N, &init);
    }
}
