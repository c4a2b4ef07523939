// Device-side JPEG entropy decoding for sm_100a: the Huffman stage of cv::imdecode (src/etl_image.cpp:90).
//
// Huffman decoding of a baseline scan is a serial chain -- every code starts where the previous one ended --
// and on the host it was the end-to-end bottleneck of the record path.  Four kernels take it over:
//
//  * jpeg_entropy_parallel_kernel, one thread block per stream, for scans without restart markers (the
//    common case).  The stream is cut into one segment per thread; every thread decodes its segment from a
//    guessed state, and because Huffman streams re-synchronise, most guesses leave their segment in the
//    true state.  Rounds in which each thread restarts from its left neighbour's exit state settle the rest
//    (details at the kernel).  Coefficients are stored in a last pass once every entry state is known.
//  * jpeg_entropy_spread_kernel, a cluster of up to eight thread blocks per stream, for launches of few such
//    scans: shorter segments, each entered once for every place in the MCU, settle without rounds.
//  * jpeg_entropy_restart_kernel, several thread blocks per stream, for scans with restart markers: the
//    intervals between the markers are independent, so a stream is cut into runs of intervals, and each
//    interval into segments as above (jpeg_restart_index_kernel finds the intervals first).
//  * jpeg_entropy_kernel, one warp per stream, walks the stream serially (lane 0 decodes, all lanes build
//    tables, prefetch the stream into a shared-memory window and flush each block with one 128-byte store).
//    It takes callers that give no work area, and damaged streams with restart markers.
//
// All produce what the host decoder produces (ITU-T T.81 F.2.2; same column-major coefficient planes,
// optionally restricted to a rectangle of MCUs), bit for bit.  Every loop is bounded by the stream length,
// the block count or the segment count; a malformed stream sets the record's status word and the block
// returns, it never spins.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "../../include/aeon_b200.h"
#include "context.hpp"

namespace aeonb
{
    namespace
    {
        constexpr int LOOK   = 10;
        constexpr int WINDOW = 1024; // bytes of the stream kept in shared memory (two halves of 512)

        // Work area of a stream with restart markers: room for the copies of its parts without stuffed bytes, a DC difference per
        // block, and the index of its intervals.
        struct restart_header
        {
            uint32_t doubtful; // not 0: the stream is not what the interval decoder expects; the serial kernel takes it
            uint32_t end;      // offset of the first marker that is no restart marker, or the scan's size
            uint32_t found;    // restart markers seen (also past `end`)
            uint32_t reserved;
        };
        struct restart_layout
        {
            uint8_t*        clean;
            int16_t*        dcdiff;
            restart_header* header;
            uint32_t*       start; // offset of the first byte of every interval; intervals + 1 entries
            uint64_t        bytes; // of the whole area
            uint32_t        intervals;
        };
        constexpr int RST_MAX_INTERVALS = 256; // of a part (= what one thread block decodes)
        __host__ __device__ inline uint32_t restart_most_parts(uint32_t intervals)
        {
            return intervals < 96 ? intervals : intervals / RST_MAX_INTERVALS + 96;
        }
        __host__ __device__ inline restart_layout restart_work(const aeonb_entropy_desc& d)
        {
            restart_layout w;
            uint64_t       bpm = 0;
            for (int c = 0; c < d.ncomp && c < 3; ++c)
                bpm += (uint64_t)d.hs[c] * d.vs[c];
            const uint64_t mcus = (uint64_t)d.mcux * d.mcuy;
            w.intervals         = (uint32_t)((mcus + d.restart_interval - 1) / d.restart_interval);
            uint64_t off        = 0;
            w.clean             = static_cast<uint8_t*>(d.scratch);
            off += ((uint64_t)d.scan_size + 64ull * (restart_most_parts(w.intervals) + 2) + 15) & ~15ull;
            w.dcdiff = reinterpret_cast<int16_t*>(w.clean + off);
            off += (mcus * bpm * 2 + 15) & ~15ull;
            w.header = reinterpret_cast<restart_header*>(w.clean + off);
            off += sizeof(restart_header);
            w.start = reinterpret_cast<uint32_t*>(w.clean + off);
            off += (((uint64_t)w.intervals + 1) * 4 + 15) & ~15ull;
            w.bytes = off;
            return w;
        }

        struct huff_table
        {
            uint16_t lookup[1 << LOOK];  // (length << 8) | symbol for codes up to LOOK bits, else 0
            int16_t  fast_ac[1 << LOOK]; // (value << 8) | (run << 4) | total bits for short AC codes, else 0
            int      maxcode[18];        // exclusive upper bound of the codes of each length, left-justified to 16 bits
            int      valoff[17];
            int      first[17];          // first code of each length
            int      count[17];
            uint8_t  vals[256];
        };

        struct warp_state
        {
            huff_table    dc[2], ac[2];
            alignas(16) uint8_t window[WINDOW];
            alignas(16) int16_t block[64];
        };

        // zig-zag position -> index inside a column-major block
        __constant__ uint8_t k_zz_colmajor[64] = {
            0, 8, 1, 2, 9, 16, 24, 17, 10, 3, 4, 11, 18, 25, 32, 40, 33, 26, 19, 12, 5, 6, 13, 20, 27, 34, 41, 48, 56, 49, 42, 35,
            28, 21, 14, 7, 15, 22, 29, 36, 43, 50, 57, 58, 51, 44, 37, 30, 23, 31, 38, 45, 52, 59, 60, 53, 46, 39, 47, 54, 61, 62,
            55, 63};

        // All 32 lanes build one table from the DHT form (16 counts + up to 256 values).
        __device__ void build_table(huff_table& t, const uint8_t* __restrict__ dht, bool is_ac, int lane, int* bad)
        {
            if (lane == 0)
            {
                int code = 0, k = 0;
                for (int len = 1; len <= 16; ++len)
                {
                    const int n   = dht[len - 1];
                    t.first[len]  = code;
                    t.count[len]  = n;
                    t.valoff[len] = k - code;
                    code += n;
                    k += n;
                    if (code > (1 << len) || k > 256)
                        *bad = 1;
                    t.maxcode[len] = n ? (code << (16 - len)) : -1;
                    code <<= 1;
                }
                t.maxcode[17] = 0x7fffffff;
            }
            for (int i = lane; i < 256; i += 32)
                t.vals[i] = dht[16 + i];
            __syncwarp();
            for (int i = lane; i < (1 << LOOK); i += 32)
            {
                uint16_t e = 0;
                for (int len = 1; len <= LOOK; ++len)
                {
                    const int prefix = i >> (LOOK - len);
                    const int idx    = prefix - t.first[len];
                    if (idx >= 0 && idx < t.count[len])
                    {
                        e = (uint16_t)((len << 8) | t.vals[(prefix + t.valoff[len]) & 255]);
                        break;
                    }
                }
                t.lookup[i] = e;
                int16_t f   = 0;
                if (is_ac && e)
                {
                    const int len = e >> 8, rs = e & 255, run = rs >> 4, mag = rs & 15;
                    if (mag && len + mag <= LOOK)
                    {
                        int v = (i >> (LOOK - len - mag)) & ((1 << mag) - 1);
                        if (v < (1 << (mag - 1)))
                            v -= (1 << mag) - 1;
                        if (v >= -128 && v <= 127)
                            f = (int16_t)((v * 256) | (run << 4) | (len + mag));
                    }
                }
                t.fast_ac[i] = f;
            }
            __syncwarp();
        }

        // Bit reader of lane 0 over the shared-memory window.  `pos` counts bytes of the scan consumed.
        struct bit_reader
        {
            const uint8_t* window;
            uint32_t       pos, size; // next byte to take / scan length
            uint64_t       acc;       // bits are consumed from the top
            int            n;
            bool           at_marker;

            __device__ __forceinline__ uint8_t byte_at(uint32_t p) const { return window[p & (WINDOW - 1)]; }
            // Tops the accumulator up to at least 32 bits, byte by byte: removes stuffed zeros, stops at markers.
            __device__ __forceinline__ void refill(uint32_t limit)
            {
                if (n > 32)
                    return;
                if (pos + 4 <= limit && !at_marker)
                {
                    // four bytes at once when none of them is 0xFF (no stuffing, no marker)
                    const uint32_t* w32 = reinterpret_cast<const uint32_t*>(window);
                    const uint32_t  i   = (pos >> 2) & (WINDOW / 4 - 1);
                    const uint32_t  k   = pos & 3;
                    const uint32_t  be  = __byte_perm(w32[i], w32[(i + 1) & (WINDOW / 4 - 1)],
                                                      (k + 3) | ((k + 2) << 4) | ((k + 1) << 8) | (k << 12));
                    const uint32_t  inv = ~be;
                    if (!((inv - 0x01010101u) & ~inv & 0x80808080u))
                    {
                        acc |= (uint64_t)be << (32 - n);
                        n += 32;
                        pos += 4;
                        return;
                    }
                }
                while (n <= 32)
                {
                    uint64_t b = 0;
                    if (pos < limit && !at_marker)
                    {
                        b = byte_at(pos);
                        if (b == 0xFF)
                        {
                            const uint8_t nx = pos + 1 < size ? byte_at(pos + 1) : 0xD9;
                            if (nx == 0)
                                pos += 2;
                            else
                            {
                                b         = 0;
                                at_marker = true; // a marker: feed zero bits and stay put
                            }
                        }
                        else
                            ++pos;
                    }
                    acc |= b << (56 - n);
                    n += 8;
                }
            }
            __device__ __forceinline__ uint32_t peek(int k) const { return (uint32_t)(acc >> (64 - k)); }
            __device__ __forceinline__ void     skip(int k)
            {
                acc <<= k;
                n -= k;
            }
            __device__ __forceinline__ int receive_extend(int s)
            {
                const uint32_t v = peek(s);
                skip(s);
                return (int)v - (int)(((v >> (s - 1)) ^ 1u)) * ((1 << s) - 1);
            }
            __device__ __forceinline__ int decode(const huff_table& t, int* bad)
            {
                const uint16_t e = t.lookup[peek(LOOK)];
                if (e)
                {
                    skip(e >> 8);
                    return e & 255;
                }
                const int c16 = (int)peek(16);
                int       len = LOOK + 1;
                while (len <= 16 && (t.maxcode[len] < 0 || c16 >= t.maxcode[len]))
                    ++len;
                if (len > 16)
                {
                    *bad = 1;
                    return 0;
                }
                skip(len);
                return t.vals[((c16 >> (16 - len)) + t.valoff[len]) & 255];
            }
        };

        __global__ void __launch_bounds__(32) jpeg_entropy_kernel(const __grid_constant__ launch_data data)
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            warp_state&              S    = *reinterpret_cast<warp_state*>(smem_raw);
            const int                lane = threadIdx.x;
            __shared__ aeonb_entropy_desc d; // in shared memory: its arrays are indexed by loop variables
            __shared__ int           pred[3];
            __shared__ int           bad;
            __shared__ uint32_t      fetched; // bytes of the scan loaded into the window so far
            static_assert(sizeof(aeonb_entropy_desc) % 4 == 0, "descriptor is copied word by word");
            data.fetch(d, (int)(blockIdx.x), (int)lane, (int)32);
            if (lane == 0)
            {
                bad     = 0;
                fetched = 0;
                pred[0] = pred[1] = pred[2] = 0;
            }
            __syncwarp();
            if (d.scratch && d.restart_interval == 0)
                return; // the block-parallel kernel's stream
            if (d.scratch && restart_work(d).header->doubtful == 0)
            {
                if (lane == 0 && d.status)
                    *d.status = 0; // decoded interval by interval
                return;
            }
            const bool shape_ok = d.ncomp >= 1 && d.ncomp <= 3 && d.mcux > 0 && d.mcuy > 0 && d.scan && d.tables;
            if (!shape_ok)
            {
                if (lane == 0 && d.status)
                    *d.status = 1;
                return;
            }
            build_table(S.dc[0], d.tables + 0 * 272, false, lane, &bad);
            build_table(S.dc[1], d.tables + 1 * 272, false, lane, &bad);
            build_table(S.ac[0], d.tables + 2 * 272, true, lane, &bad);
            build_table(S.ac[1], d.tables + 3 * 272, true, lane, &bad);
            for (int i = lane; i < 64; i += 32)
                S.block[i] = 0;

            // window loader: all lanes copy the next half window (512 bytes) with 16-byte loads where aligned
            auto load_half = [&](uint32_t from) {
                for (uint32_t i = lane; i < WINDOW / 2; i += 32)
                {
                    const uint32_t p = from + i;
                    S.window[p & (WINDOW - 1)] = p < d.scan_size ? __ldg(d.scan + p) : 0;
                }
                __syncwarp();
            };
            load_half(0);
            load_half(WINDOW / 2);
            if (lane == 0)
                fetched = WINDOW;
            __syncwarp();

            bit_reader br;
            br.window    = S.window;
            br.pos       = 0;
            br.size      = d.scan_size;
            br.acc       = 0;
            br.n         = 0;
            br.at_marker = false;
            int until_restart  = d.restart_interval ? d.restart_interval : -1;
            const int mx0 = max(d.roi[0], 0), my0 = max(d.roi[1], 0), mx1 = min(d.roi[2], d.mcux), my1 = min(d.roi[3], d.mcuy);

            for (int my = 0; my < my1; ++my)
            {
                for (int mx = 0; mx < d.mcux; ++mx)
                {
                    const bool keep = my >= my0 && mx >= mx0 && mx < mx1;
                    if (lane == 0)
                    {
                        if (until_restart == 0)
                        {
                            // restart marker: drop the remaining bits, step over FF Dx, reset the predictors
                            br.acc = 0;
                            br.n   = 0;
                            uint32_t guard = 0;
                            while (br.pos + 1 < br.size && guard < 64 &&
                                   !(br.byte_at(br.pos) == 0xFF && br.byte_at(br.pos + 1) >= 0xD0 && br.byte_at(br.pos + 1) <= 0xD7))
                            {
                                ++br.pos;
                                ++guard;
                            }
                            if (br.pos + 1 < br.size && guard < 64)
                                br.pos += 2;
                            else
                                bad = 1;
                            br.at_marker = false;
                            pred[0] = pred[1] = pred[2] = 0;
                            until_restart               = d.restart_interval;
                        }
                        if (until_restart > 0)
                            --until_restart;
                    }
                    for (int c = 0; c < d.ncomp; ++c)
                    {
                        const int nblk = d.hs[c] * d.vs[c];
                        for (int b = 0; b < nblk; ++b)
                        {
                            // ---- lane 0 decodes one block into shared memory
                            if (lane == 0 && !bad)
                            {
                                const huff_table& dt = S.dc[d.dc_table[c] & 1];
                                const huff_table& at = S.ac[d.ac_table[c] & 1];
                                const uint32_t    limit = min(fetched, br.size);
                                br.refill(limit);
                                const int t = br.decode(dt, &bad);
                                if (t > 15)
                                    bad = 1;
                                else if (t)
                                {
                                    br.refill(limit);
                                    pred[c] += br.receive_extend(t);
                                }
                                S.block[0] = (int16_t)pred[c];
                                int k      = 1;
                                while (k < 64 && !bad)
                                {
                                    br.refill(limit);
                                    const int16_t fa = at.fast_ac[br.peek(LOOK)];
                                    if (fa)
                                    {
                                        k += (fa >> 4) & 15;
                                        if (k > 63)
                                        {
                                            bad = 1;
                                            break;
                                        }
                                        br.skip(fa & 15);
                                        S.block[k_zz_colmajor[k++]] = (int16_t)(fa >> 8);
                                        continue;
                                    }
                                    const int rs = br.decode(at, &bad);
                                    const int r = rs >> 4, s = rs & 15;
                                    if (s == 0)
                                    {
                                        if (r != 15)
                                            break;
                                        k += 16;
                                        continue;
                                    }
                                    k += r;
                                    if (k > 63)
                                    {
                                        bad = 1;
                                        break;
                                    }
                                    S.block[k_zz_colmajor[k++]] = (int16_t)br.receive_extend(s);
                                }
                            }
                            __syncwarp();
                            // ---- all lanes: flush the block (one 128-byte store), clear it, keep the window ahead of the reader
                            if (keep)
                            {
                                const int by = b / d.hs[c], bx = b - by * d.hs[c];
                                int16_t*  out = d.coef[c] + ((size_t)((my - my0) * d.vs[c] + by) * ((mx1 - mx0) * d.hs[c]) +
                                                            ((mx - mx0) * d.hs[c] + bx)) * 64;
                                reinterpret_cast<uint32_t*>(out)[lane] = reinterpret_cast<const uint32_t*>(S.block)[lane];
                            }
                            __syncwarp();
                            reinterpret_cast<uint32_t*>(S.block)[lane] = 0;
                            // the reader may touch at most one block's worth of bytes (< 256) before the next check:
                            // refill the half of the window it has left behind
                            const uint32_t pos = __shfl_sync(0xffffffffu, br.pos, 0);
                            if (fetched < d.scan_size && pos + WINDOW / 2 >= fetched)
                            {
                                load_half(fetched);
                                if (lane == 0)
                                    fetched += WINDOW / 2;
                            }
                            __syncwarp();
                        }
                    }
                    if (bad) // uniform: `bad` lives in shared memory and every lane reads it after the barrier above
                    {
                        if (lane == 0 && d.status)
                            *d.status = 1;
                        return;
                    }
                }
            }
            if (lane == 0 && d.status)
                *d.status = 0;
        }
    

        // ------------------------------------------------------------------------------------------------
        // Block-parallel decoder for streams without restart markers.
        //
        // One thread block per stream.  The stream is first copied without its stuffed zero bytes (so bit
        // positions are plain offsets), then cut into one segment per thread.  Every thread decodes its
        // segment starting from a guessed state (block 0 of an MCU, DC coefficient next) and records the
        // state in which it leaves the segment: the bit position of the first symbol that starts past the
        // segment's end, the block's index inside the MCU and the zig-zag index.  At three evenly spaced
        // checkpoints inside the segment it also notes the state of the first symbol at or past the
        // checkpoint and the blocks completed so far.  Rounds follow in which every thread takes its left
        // neighbour's exit state as its entry state and, if that differs from the entry it used before,
        // decodes again -- but only until it arrives at a checkpoint in the state noted there, because from
        // there on it would repeat the earlier run and leave the segment in the same state.  Segment 0 always
        // starts in the true state, so after round r the first r+1 exits are true, and the rounds stop as
        // soon as nothing changes (at most one round per segment).  A prefix sum over the blocks each
        // segment completed gives every segment its first block number, and a last pass decodes each
        // segment once more from its now true entry state, this time storing the coefficients.  DC values
        // are stored as differences and summed up per component in a final scan.
        //
        // The threads of a warp sit in different segments, so the symbol loop is flat -- every pass of it
        // decodes one symbol in every lane, whatever kind (DC category, AC run/size, end of block, zero run),
        // with the block-end bookkeeping done by selects.  A launch lasts as long as the chain of symbols of its
        // slowest stream, so what counts is how soon the next symbol's lookup can start.  The scan is fetched to
        // shared memory while the tables are being built, cleaned of stuffed bytes in place and decoded from
        // there: in global memory nearly every pass had some lane of the warp waiting for L2.
        //
        // A pass of the loop is one lookup, one byte permute and one addition from position to position, and every other
        // decision (the next table, the window's refill, the end of a block, a code that the window does not hold) is a select or
        // a predicated load beside that chain; with a second, dependent lookup for long codes and a branch for codes in no table a
        // pass took half as long again.
        //
        // Measured on a B200 (kernel times): one stream of about 40 KB 0.183 ms before, 0.133 ms now; 256 streams of up to 55 KB (4:2:0,
        // quality 90, crop regions stored) 0.263 / 0.178 ms; 512 streams of 6 KB 0.232 / 0.123 ms.  Phases of the 256 streams, thousand
        // cycles on average: first pass 56 / 36, rounds 149 / 89 (five of them; the stream that takes longest spends 160 there), storing
        // pass 90 / 56, copy and marker scan 23 / 22, DC 8, set-up 24 / 20.  Of one 43 KB stream that has an SM to itself the
        // storing pass takes 101, 65 without its stores: one of 2 bytes per coefficient, each to a line of its own.
        // A wrong guess falls into step with the true decoder after about 10 blocks on average (the block's
        // position inside the MCU has to match too), and not at all inside flat regions, where every block looks
        // the same: there a chain of segments is settled one round per segment, which is what the slowest streams
        // of a batch spend their time on (5 rounds on average, 11 at most).  Tried and no faster: warming up on the
        // tail of the left neighbour's segment before the guess.
        constexpr int AC_BITS = 11; // bits of the lookup window: AC tables (12: 28 us slower for 256 streams, fewer of which then fit shared memory)
        constexpr int DC_BITS = 9;  //                            DC tables (few, short codes)
        // Each of the four tables is a window, indexed by the bits at hand, behind LONG entries indexed by 16 bits from LONG_FROM on:
        // the codes that are longer than the window are nearly always among the last ones, which start with eight ones.
        //
        // An entry of the passes that only look for states holds, a byte each, what the state -- bit position in bits 0-23, zig-zag
        // index in bits 24-31 -- advances by: byte 0 bits of the pair that the symbol at the head of the window makes with the one
        // behind it, where the pair fits the window (the second one's value bits may lie outside) and the first one does not end the
        // block, otherwise of the symbol alone; byte 1 bits of the symbol alone; byte 2 its advance of the zig-zag index: run + 1, 16 for
        // ZRL, 64 for end of block, 1 for a DC category, 127 for an invalid code (which still takes bits and ends the block, so that a
        // decoder in a wrong state moves on); byte 3 the advance of the pair.  One byte permute turns an entry into the advance.
        // An entry of the storing pass: bits 0-4 bits of the symbol, 5-8 number of value bits (AC size / DC category, 1 for an
        // invalid code, which then looks like a run that leaves the block), 9-15 advance.
        // 0: look the 16 bits up in front of the window.  k_slow: neither window nor LONG entries hold the code (long_symbol finds it).
        constexpr int      LONG = 256, LONG_FROM = 0x10000 - LONG;
        constexpr int      AC_ENTRIES = LONG + (1 << AC_BITS), DC_ENTRIES = LONG + (1 << DC_BITS), ENTRIES = 2 * (AC_ENTRIES + DC_ENTRIES);
        constexpr uint32_t k_position = 0x00ffffffu, k_block_end = 64u << 24;
        constexpr uint32_t k_pair_first = AC_BITS - 1;  // most bits of the first symbol of a pair
        constexpr uint32_t k_pair_limit = 48u << 24;    // from this zig-zag index on (63 - 15) the first symbol can end the block
        constexpr uint32_t k_take_pair = 0x3440, k_take_one = 0x2441; // byte selectors
        constexpr uint32_t k_slow = 0xffff;
        __device__ __forceinline__ uint32_t store_entry(uint32_t total, uint32_t size, uint32_t advance) { return total | size << 5 | advance << 9; }
        constexpr uint32_t k_invalid = 16 | 1 << 5 | 127 << 9;
        __device__ __forceinline__ uint32_t entry_total(uint32_t e) { return e & 31; }
        __device__ __forceinline__ uint32_t entry_size(uint32_t e) { return e >> 5 & 15; }
        __device__ __forceinline__ uint32_t entry_advance(uint32_t e) { return e >> 9; }
        __device__ __forceinline__ uint32_t scan_entry(uint32_t e) // of a storing pass entry, no pair
        {
            return e == k_slow ? k_slow : entry_total(e) * 0x101u + entry_advance(e) * 0x1010000u;
        }
        __device__ __forceinline__ uint32_t pack_symbol(int len, int sym, bool is_ac)
        {
            const int s = sym & 15, r = sym >> 4;
            if (!is_ac && r)
                return k_invalid;
            return store_entry((uint32_t)(len + s), (uint32_t)s, is_ac ? (s ? r + 1 : (r == 15 ? 16 : 64)) : 1);
        }

        struct code_table
        {
            alignas(16) int limit[16]; // limit[len - 1]: exclusive upper bound of the codes of length <= len, left-justified to 16 bits
            int     valoff[17];
            uint8_t vals[256];
        };

        // A warp fills the canonical-code limits of a table from the DHT form (16 counts); the values are copied by the caller.  With n(l)
        // codes of length l, those of length <= l end at the sum of n(j) << (16 - j) over j <= l, left-justified.
        __device__ __forceinline__ void build_code_table(code_table& T, const uint8_t* dht, int lane, int* bad)
        {
            const int n = lane < 16 ? dht[lane] : 0, codes = lane < 16 ? n << (15 - lane) : 0;
            int       k = n, limit = codes;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1)
            {
                const int up_k = __shfl_up_sync(0xffffffffu, k, o), up_limit = __shfl_up_sync(0xffffffffu, limit, o);
                k += lane >= o ? up_k : 0;
                limit += lane >= o ? up_limit : 0;
            }
            if (lane >= 16)
                return;
            T.valoff[lane + 1] = k - n - ((limit - codes) >> (15 - lane));
            T.limit[lane]      = limit;
            if (limit > 1 << 16 || k > 256)
                *bad = 1;
        }
        // The limits of a table in registers: the length of a code is then a count of comparisons that do not wait for one another.
        struct code_limits
        {
            int of[16];
            __device__ __forceinline__ explicit code_limits(const code_table& T)
            {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    const int4 v = reinterpret_cast<const int4*>(T.limit)[k];
                    of[4 * k] = v.x, of[4 * k + 1] = v.y, of[4 * k + 2] = v.z, of[4 * k + 3] = v.w;
                }
            }
            // Length of the code at the head of the 16 bits c16, or MOST if it is not shorter (or not a code).
            template <int MOST>
            __device__ __forceinline__ int length(int c16) const
            {
                int len = 1;
#pragma unroll
                for (int l = 1; l < MOST; ++l)
                    len += c16 >= of[l - 1];
                return len;
            }
        };
        __device__ __forceinline__ uint32_t code_entry(const code_table& T, int c16, int len, bool is_ac)
        {
            return pack_symbol(len, T.vals[((c16 >> (16 - len)) + T.valoff[len]) & 255], is_ac);
        }
        // The symbol at the head of the 16 bits c16, whatever its length, for codes that are in no table.
        __device__ __noinline__ uint32_t long_symbol(const code_table& T, int c16, bool is_ac)
        {
            return c16 >= T.limit[15] ? k_invalid : code_entry(T, c16, code_limits(T).length<16>(c16), is_ac);
        }
        // Where a table starts among the ENTRIES: DC slot 0, DC slot 1, AC slot 0, AC slot 1.
        __device__ __forceinline__ int table_at(int t) { return t < 2 ? t * DC_ENTRIES : 2 * DC_ENTRIES + (t - 2) * AC_ENTRIES; }
        // Eight neighbouring entries of a window of BITS bits, from i on.  Unless a code of the last three lengths starts among them they
        // hold one symbol, so most often two lengths are worked out per eight entries.
        template <int BITS>
        __device__ __forceinline__ void fill_window(uint16_t* out, const code_table& T, int i, bool is_ac, int* slow)
        {
            const code_limits limits(T);
            const int         first = limits.length<BITS>(i << (16 - BITS)), last = limits.length<BITS>((i + 7) << (16 - BITS));
            const auto        entry = [&](int k, int len) -> uint32_t {
                const int c16 = (i + k) << (16 - BITS);
                if (c16 < T.limit[len - 1])
                    return code_entry(T, c16, len, is_ac);
                if (c16 >= LONG_FROM)
                    return 0;
                if (c16 >= T.limit[15])
                    return k_invalid;
                *slow = 1;
                return k_slow;
            };
            if (first == last && first <= BITS - 3)
            {
                const uint32_t e = entry(0, first) * 0x10001u;
                *reinterpret_cast<uint4*>(out) = make_uint4(e, e, e, e);
                return;
            }
            uint32_t e[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                e[k] = entry(k, limits.length<BITS>((i + k) << (16 - BITS)));
            *reinterpret_cast<uint4*>(out) = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
        }
        // `nth` threads (index `tid`) fill the storing pass's entries of the four tables once limits and values are in place.
        __device__ void build_tables(uint16_t* store, const code_table* codes, int tid, int nth, int* slow)
        {
            constexpr int ac8 = (1 << AC_BITS) / 8, dc8 = (1 << DC_BITS) / 8;
            for (int j = tid; j < 2 * ac8; j += nth)
                fill_window<AC_BITS>(store + table_at(2 + j / ac8) + LONG + 8 * (j % ac8), codes[2 + j / ac8], 8 * (j % ac8), true, slow);
            // the last threads first: they have least to do above
            for (int j = nth - 1 - tid; j < 2 * dc8; j += nth)
                fill_window<DC_BITS>(store + table_at(j / dc8) + LONG + 8 * (j % dc8), codes[j / dc8], 8 * (j % dc8), false, slow);
            for (int j = tid; j < 4 * LONG / 2; j += nth)
            {
                const int         t = j / (LONG / 2), i = 2 * (j % (LONG / 2));
                const code_table& T = codes[t];
                const code_limits limits(T);
                uint32_t          e[2];
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    const int c16 = LONG_FROM + i + k;
                    e[k]          = c16 >= T.limit[15] ? k_invalid : code_entry(T, c16, limits.length<16>(c16), t >= 2);
                }
                *reinterpret_cast<uint32_t*>(store + table_at(t) + i) = e[0] | e[1] << 16;
            }
        }
        // The entries of the other passes from those of the storing pass; eight neighbours per thread and pass so that the lookups of
        // the second symbols overlap.
        __device__ void pair_tables(uint32_t* scan, const uint16_t* store, int tid, int nth)
        {
            constexpr uint32_t mask = (1 << AC_BITS) - 1;
            for (int j = tid; j < ENTRIES / 8; j += nth)
            {
                const uint4    in    = reinterpret_cast<const uint4*>(store)[j];
                const uint32_t raw[4] = {in.x, in.y, in.z, in.w};
                uint32_t       e[8], f[8], out[8];
                // the place in an AC window; the entries in front of it, and DC tables, have no pairs
                int i = 8 * j - 2 * DC_ENTRIES - LONG;
                const uint16_t* window = store + 2 * DC_ENTRIES + LONG;
                if (i >= AC_ENTRIES)
                    i -= AC_ENTRIES, window += AC_ENTRIES;
                const bool is_ac = i >= 0 && i <= (int)mask;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    e[k] = raw[k >> 1] >> (16 * (k & 1)) & 0xffff;
                    f[k] = is_ac ? window[(uint32_t)(i + k) << entry_total(e[k]) & mask] : 0; // the bits behind, zeros after them
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    const uint32_t total = entry_total(e[k]), advance = entry_advance(e[k]);
                    out[k] = scan_entry(e[k]);
                    if (e[k] && e[k] != k_slow && advance < 64 && total <= k_pair_first && f[k] && f[k] != k_slow &&
                        entry_total(f[k]) - entry_size(f[k]) <= AC_BITS - total && entry_advance(f[k]) != 127)
                        out[k] = (out[k] & 0x00ffff00u) | (total + entry_total(f[k])) | (advance + entry_advance(f[k])) << 24;
                }
                reinterpret_cast<uint4*>(scan)[2 * j]     = make_uint4(out[0], out[1], out[2], out[3]);
                reinterpret_cast<uint4*>(scan)[2 * j + 1] = make_uint4(out[4], out[5], out[6], out[7]);
            }
        }

        constexpr int PAR_THREADS = 1024; // most threads (= segments) a stream can have; the launch picks the actual number
        constexpr int NCHECK      = 3;    // checkpoints inside a segment (7 measured the same; 3 leaves room for a third kernel's CTA on the SM)

        // What the symbol loops want to know of a block of an MCU, in 16-byte loads: the shared-memory addresses of its AC window, of the
        // next block's DC window and of the next block's link.
        struct alignas(16) block_link
        {
            uint32_t ac, next_dc, next, block;
        };
        // The storing pass also wants to know whether it is the MCU's last block, and where the blocks of this place go:
        // base + 64 * ((mcu row - first row) * dy + (mcu column - first column) * dx)
        struct alignas(16) block_place
        {
            uint32_t ac, next_dc, next, last;
            int16_t* base;
            int32_t  dy, dx;
        };

        struct par_state
        {
            alignas(16) uint32_t scan[ENTRIES];
            alignas(16) uint16_t store[ENTRIES];
            code_table  codes[4]; // DC slot 0, DC slot 1, AC slot 0, AC slot 1
            alignas(16) uint8_t dht[4 * 272]; // the tables as they came
            uint32_t    warp_sums[3][32];
            uint8_t     zz[16 + 64 + 128];       // from 16 on; around them lies what is read for a symbol without a place and not used
            block_place place[16];               // per block of an MCU
            block_link  link[16];
            uint8_t     comp[16];
            aeonb_entropy_desc d;
            int        bpm;                      // blocks per MCU
            int        bad;
            int        slow;                     // some code is not in the tables (see k_slow)
            uint32_t   marker_at;                // first marker byte in the raw scan (or its size)
            uint32_t   tile_end[2];              // last byte of an even / odd tile of the raw scan
        };

        // Per segment (= thread): the state it was entered in and left in, its blocks, and the checkpoints.
        struct seg_arrays
        {
            uint32_t *ent_p, *ext_p, *cnt, *chk; // chk: 2 x NCHECK rows of T words
            uint16_t *ent_bk, *ext_bk;
            uint32_t rows; // most segments
        };
        constexpr uint32_t SEG_BYTES = 4 * (3 + 2 * NCHECK) + 2 * 2; // of shared memory for each segment

        __device__ __forceinline__ seg_arrays seg_arrays_at(unsigned char* p, uint32_t rows)
        {
            uint32_t* const w = reinterpret_cast<uint32_t*>(p);
            uint16_t* const h = reinterpret_cast<uint16_t*>(w + (3 + 2 * NCHECK) * rows);
            return seg_arrays{w, w + rows, w + 2 * rows, w + 3 * rows, h, h + rows, rows};
        }

        __device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
        __device__ __forceinline__ uint32_t lds_u32(uint32_t addr)
        {
            uint32_t v;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
            return v;
        }
        __device__ __forceinline__ uint32_t lds_u16(uint32_t addr)
        {
            uint16_t v;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
            return v;
        }
        // Predicated loads and stores of the symbol loops.  They work their conditions out from what they are given: a condition handed
        // over as a number costs two instructions more, in loops whose time is the issue of their instructions.
        //
        // Past the end of a block (`to` is the state): link = the link at its `next`, and one more block.
        __device__ __forceinline__ void follow_past(block_link& link, uint32_t to, uint32_t& blocks)
        {
            asm volatile("{\n\t.reg .pred q;\n\tsetp.ge.u32 q, %5, %6;\n\t@q ld.shared.v4.u32 {%0, %1, %2, %3}, [%2];\n\t@q add.u32 %4, %4, 1;\n\t}"
                         : "+r"(link.ac), "+r"(link.next_dc), "+r"(link.next), "+r"(link.block), "+r"(blocks)
                         : "r"(to), "n"(64u << 24));
        }
        __device__ __forceinline__ void follow_past(block_place& at, uint32_t to, uint32_t& blocks)
        {
            const uint64_t was = reinterpret_cast<uint64_t>(at.base);
            uint32_t       lo = (uint32_t)was, hi = (uint32_t)(was >> 32);
            asm volatile("{\n\t.reg .pred q;\n\t.reg .b32 a;\n\tsetp.ge.u32 q, %9, %10;\n\tmov.b32 a, %2;\n\t"
                         "@q ld.shared.v4.u32 {%0, %1, %2, %3}, [a];\n\t@q ld.shared.v4.u32 {%4, %5, %6, %7}, [a + 16];\n\t@q add.u32 %8, %8, 1;\n\t}"
                         : "+r"(at.ac), "+r"(at.next_dc), "+r"(at.next), "+r"(at.last), "+r"(lo), "+r"(hi), "+r"(at.dy), "+r"(at.dx), "+r"(blocks)
                         : "r"(to), "n"(64u << 24));
            at.base = reinterpret_cast<int16_t*>((uint64_t)hi << 32 | lo);
        }
        __device__ __forceinline__ uint32_t lds_u8(uint32_t addr)
        {
            uint16_t v;
            asm volatile("ld.shared.u8 %0, [%1];" : "=h"(v) : "r"(addr));
            return v;
        }
        // *p = value for a DC symbol (the state in front of it has index 0)
        __device__ __forceinline__ void store_dc_symbol(int16_t* p, int value, uint32_t was)
        {
            asm volatile("{\n\t.reg .pred q;\n\tsetp.le.u32 q, %2, %3;\n\t@q st.s16 [%0], %1;\n\t}" ::"l"(p), "h"((int16_t)value), "r"(was), "n"(0x00ffffff) : "memory");
        }
        // *p = value for an AC symbol with value bits whose place kk lies in the block, inside the region (mx < w, my < h)
        __device__ __forceinline__ void store_ac_symbol(int16_t* p, int value, uint32_t was, uint32_t size, uint32_t kk, uint32_t mx, uint32_t w, uint32_t my,
                                                        uint32_t h)
        {
            asm volatile("{\n\t.reg .pred q;\n\tsetp.gt.u32 q, %2, %9;\n\tsetp.ne.and.u32 q, %3, 0, q;\n\tsetp.lt.and.u32 q, %4, 64, q;\n\t"
                         "setp.lt.and.u32 q, %5, %6, q;\n\tsetp.lt.and.u32 q, %7, %8, q;\n\t@q st.global.s16 [%0], %1;\n\t}" ::"l"(
                             __cvta_generic_to_global(p)),
                         "h"((int16_t)value), "r"(was), "r"(size), "r"(kk), "r"(mx), "r"(w), "r"(my), "r"(h), "n"(0x00ffffff)
                         : "memory");
        }

        // Words of the copy of a stream, from shared or from global memory.  `next_if` replaces `value` by the next word where
        // `yes` is not 0: only lanes that used a word ask for one.
        struct shared_words
        {
            uint32_t at;
            __device__ __forceinline__ shared_words(const uint32_t* words, uint32_t i)
                : at((uint32_t)__cvta_generic_to_shared(words) + 4 * i)
            {
            }
            __device__ __forceinline__ uint32_t next()
            {
                uint32_t v;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
                at += 4;
                return v;
            }
            __device__ __forceinline__ void next_if(uint32_t& value, uint32_t yes)
            {
                asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.shared.u32 %0, [%1];\n\t@q add.u32 %1, %1, 4;\n\t}"
                             : "+r"(value), "+r"(at)
                             : "r"(yes));
            }
        };
        struct global_words
        {
            const uint32_t* at;
            __device__ __forceinline__ global_words(const uint32_t* words, uint32_t i)
                : at(words + i)
            {
            }
            __device__ __forceinline__ uint32_t next() { return *at++; }
            __device__ __forceinline__ void     next_if(uint32_t& value, uint32_t yes)
            {
                asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.u32 %0, [%1];\n\t@q add.u64 %1, %1, 4;\n\t}"
                             : "+r"(value), "+l"(at)
                             : "r"(yes));
            }
        };

        // Where block `b` of MCU (mx, my) lives in the compact coefficient planes, or NULL outside the region.
        __device__ __forceinline__ int16_t* block_home(const par_state& S, int mx, int my, int b)
        {
            const aeonb_entropy_desc& d = S.d;
            if (my < d.roi[1] || my >= d.roi[3] || mx < d.roi[0] || mx >= d.roi[2])
                return nullptr;
            const block_place& at = S.place[b];
            return at.base + (int64_t)((my - d.roi[1]) * at.dy + (mx - d.roi[0]) * at.dx) * 64;
        }

        struct seg_result
        {
            uint32_t p;      // exit state: bit position of the first symbol past the segment,
            int      b, k;   //             block inside the MCU, zig-zag index
            uint32_t blocks; // blocks completed
            bool     merged; // the run fell into step with the remembered run: the exit state is that run's (p, b, k unset)
        };

        // Decodes symbols from bit position p in state (b, k) on, without their values.  The copy of the stream holds big-endian words, so
        // the 32 bits under a position are one funnel shift of two words.
        template <bool SLOW, typename Words>
        struct scanner
        {
            block_link link;   // of the block in progress
            uint32_t   base;   // bit positions count from the word that the run starts in
            uint32_t   at;     // the state: position, and zig-zag index in the top byte
            uint32_t   look;   // the table of the symbol under the position
            uint32_t   w0, w1, w2; // the 32 bits under the position lie in w0 and w1; w2 is fetched when w1 comes into use
            uint32_t   h, e;   // those bits (a symbol or a pair takes at most 31), and the entry of the symbol
            uint32_t   blocks; // completed
            Words      ahead;

            __device__ __forceinline__ scanner(const par_state& S, const uint32_t* words, uint32_t p, int b, int k)
                : link(S.link[b]), base(p & ~31u), at((p & 31) | (uint32_t)k << 24), look(k == 0 ? S.link[b ? b - 1 : S.bpm - 1].next_dc : link.ac),
                  blocks(0), ahead(words, p >> 5)
            {
                w0 = ahead.next(), w1 = ahead.next(), w2 = ahead.next();
                h  = __funnelshift_l(w1, w0, at);
                e  = lds_u32(look + ((h >> (k == 0 ? 32 - DC_BITS : 32 - AC_BITS)) << 2));
            }
            __device__ __forceinline__ uint32_t position() const { return base + (at & k_position); }
            // The state at the first symbol at or past `stop` (by at most 30 bits), once the run is there.
            __device__ __forceinline__ uint32_t key(uint32_t stop) const { return (position() - stop) << 10 | link.block << 6 | at >> 24; }

            // Goes on until the first symbol that starts at or past bit `until`.  The entry of the symbol under the position is fetched as
            // soon as the position is known, and what else a step has to do is done while that load is under way.  The next table -- the AC
            // one of this block, or after the block's last symbol the DC one of the next -- is at hand before the symbol is known, so
            // that only a select hangs on it.
            __device__ __forceinline__ void run_to(const par_state& S, uint32_t until)
            {
                const uint32_t stop = until > base ? until - base : 0;
                for (uint32_t pos = at & k_position; pos < stop;)
                {
                    // Two symbols at a time as long as the first one cannot reach `stop`: a run stops at the first symbol at or past
                    // it, however it came there.
                    const uint32_t take = at < k_pair_limit && pos + k_pair_first < stop ? k_take_pair : k_take_one;
                    if (SLOW && e == k_slow)
                    {
                        const bool is_ac = at > k_position;
                        const int  slot1 = look == shared_address(S.scan + table_at(is_ac ? 3 : 1) + LONG);
                        e = scan_entry(long_symbol(S.codes[(is_ac ? 2 : 0) + slot1], (int)(h >> 16), is_ac));
                    }
                    const uint32_t by    = __byte_perm(e, 0, take);
                    const uint32_t to    = at + by;
                    const uint32_t cross = (at ^ to) & 32; // the read position has left w0
                    const bool     end = to >= k_block_end, again = by == 0;
                    w0                   = cross ? w1 : w0;
                    w1                   = cross ? w2 : w1;
                    look                 = again ? look - 4 * LONG - 4 * LONG_FROM : end ? link.next_dc : link.ac;
                    const uint32_t shift = again ? 16 : end ? 32 - DC_BITS : 32 - AC_BITS;
                    at                   = end ? to & k_position : to;
                    h                    = __funnelshift_l(w1, w0, at);
                    e                    = lds_u32(look + ((h >> shift) << 2));
                    pos                  = to & k_position;
                    ahead.next_if(w2, cross);
                    follow_past(link, to, blocks);
                }
            }
        };

        // Decodes symbols from bit position p in state (b, k) until the first symbol that starts at or past pend.
        // The state at the checkpoints (first one at bit check_at, then every check_step bits) goes to chk[0],
        // chk[check_stride], ... and the blocks completed by then NCHECK rows further on; with `compare`, the run stops at the
        // first checkpoint that an earlier run over this segment (old_blocks blocks in all) passed in the same state, and the
        // block counts from there on are renumbered for this run.
        template <bool SLOW, typename Words>
        __device__ __forceinline__ seg_result scan_segment(const par_state& S, const uint32_t* words, uint32_t p, int b, int k, uint32_t pend,
                                                           uint32_t* chk, uint32_t check_stride, uint32_t check_at, uint32_t check_step,
                                                           bool compare, uint32_t old_blocks)
        {
            seg_result R;
            R.merged = false;
            scanner<SLOW, Words> run(S, words, p, b, k);
            // checkpoints: `slot` walks down this thread's column (state; the blocks so far NCHECK rows further on); `old_key` is
            // the state an earlier run noted at the next checkpoint (no state has all bits set)
            const uint32_t rows    = NCHECK * check_stride;
            uint32_t*      slot    = chk;
            uint32_t       old_key = compare ? chk[0] : 0xffffffffu;
            // A checkpoint at or past the segment's end is never taken: a run can step over it with its last symbol or stop short
            // of it, so what is noted there could be left from an older run than the one whose block count goes with it.
            uint32_t stop = check_at >= pend ? pend : check_at;
            for (;;)
            {
                run.run_to(S, stop);
                if (stop == pend)
                    break;
                // a checkpoint
                const uint32_t key = run.key(stop);
                if (key == old_key)
                {
                    // in step with the earlier run: its blocks from here on are this run's too
                    const uint32_t was = slot[rows];
                    for (uint32_t* later = slot; later < chk + rows; later += check_stride)
                        later[rows] += run.blocks - was;
                    run.blocks += old_blocks - was;
                    R.merged = true;
                    break;
                }
                slot[0]    = key;
                slot[rows] = run.blocks;
                slot += check_stride;
                const bool more = slot < chk + rows && stop + check_step < pend;
                old_key         = more && compare ? slot[0] : 0xffffffffu; // fetched now, wanted at the next checkpoint
                stop            = more ? stop + check_step : pend;
            }
            R.p      = run.position();
            R.b      = (int)run.link.block;
            R.k      = (int)(run.at >> 24);
            R.blocks = run.blocks;
            return R;
        }

        // Decodes symbols as above and stores coefficients and DC differences; `g` is the number of the block in progress, block `gend`
        // the first that is not wanted.  There is nothing to branch around: where a block goes is worked out anew for
        // every symbol (three multiply-adds), and what a symbol has no part in is a store that is not made.
        struct store_result
        {
            uint32_t p, blocks; // where the first symbol past the segment starts; blocks completed
            bool     bad;
        };
        template <bool SLOW, typename Words>
        __device__ __forceinline__ store_result store_segment(const par_state& S, const uint32_t* words, uint32_t p, int b, int k, uint32_t pend,
                                                              uint32_t g, uint32_t gend, int16_t* __restrict__ dcdiff)
        {
            store_result R{p, 0, false};
            if (g >= gend)
                return R; // nothing of this segment is wanted
            const uint32_t first = g;
            // the MCU, counted from the region's first column and row (negative in front of it), and the region's size
            const int      mx_first = -S.d.roi[0], mx_end = S.d.mcux - S.d.roi[0];
            const uint32_t roi_w = (uint32_t)(S.d.roi[2] - S.d.roi[0]), roi_h = (uint32_t)(S.d.roi[3] - S.d.roi[1]);
            const uint32_t mcu = g / (uint32_t)S.bpm, row = mcu / (uint32_t)S.d.mcux;
            int            my = (int)row - S.d.roi[1], mx = (int)(mcu - row * (uint32_t)S.d.mcux) - S.d.roi[0];
            block_place    place = S.place[b];
            uint32_t       look = k == 0 ? S.place[b ? b - 1 : S.bpm - 1].next_dc : place.ac;
            const uint32_t base = p & ~31u;
            uint32_t       at   = (p - base) | (uint32_t)k << 24, pos = p - base;
            pend                = pend > base ? pend - base : 0;
            const uint32_t zz   = shared_address(S.zz) + 16;
            Words          ahead(words, p >> 5);
            uint32_t       w0 = ahead.next(), w1 = ahead.next(), w2 = ahead.next();
            uint32_t       h = __funnelshift_l(w1, w0, at);
            uint32_t       e = lds_u16(look + ((h >> (k == 0 ? 32 - DC_BITS : 32 - AC_BITS)) << 1));
            while (pos < pend && g < gend)
            {
                if (SLOW && e == k_slow)
                {
                    const bool is_ac = at > k_position;
                    const int  slot1 = look == shared_address(S.store + table_at(is_ac ? 3 : 1) + LONG);
                    e                = long_symbol(S.codes[(is_ac ? 2 : 0) + slot1], (int)(h >> 16), is_ac);
                }
                const uint32_t total = entry_total(e), size = entry_size(e), advance = entry_advance(e);
                const uint32_t x     = h << (total - size); // the value bits at the top
                const uint32_t was = at, to = at + (total | advance << 24);
                const uint32_t kk   = (was >> 24) + advance - 1; // the coefficient's place
                const uint32_t cross = (at ^ to) & 32;
                const bool     end = to >= k_block_end, again = e == 0;
                w0    = cross ? w1 : w0;
                w1    = cross ? w2 : w1;
                look  = again ? look - 2 * LONG - 2 * LONG_FROM : end ? place.next_dc : place.ac;
                const uint32_t shift = again ? 16 : end ? 32 - DC_BITS : 32 - AC_BITS;
                at    = end ? to & k_position : to;
                h     = __funnelshift_l(w1, w0, at);
                e     = lds_u16(look + ((h >> shift) << 1));
                const uint32_t column = lds_u8(zz + kk);
                ahead.next_if(w2, cross);
                pos   = to & k_position;

                const int v = (int)__funnelshift_l(x, 0u, size) + ((int)x >= 0 ? 1 - (1 << size) : 0);
                // an invalid code, or a run that leaves the block
                R.bad |= size != 0 && (int)kk > 63;
                store_dc_symbol(dcdiff + g, v, was);
                store_ac_symbol(place.base + (int64_t)(my * place.dy + mx * place.dx) * 64 + column, v, was, size, kk, (uint32_t)mx, roi_w,
                                (uint32_t)my, roi_h);
                mx += end ? place.last : 0;
                my += mx == mx_end;
                mx = mx == mx_end ? mx_first : mx;
                follow_past(place, to, g);
            }
            R.p      = base + pos;
            R.blocks = g - first;
            return R;
        }

        // Exclusive prefix sum over the block's threads; `total` receives the sum.  `sums` is 32 words of shared memory.
        __device__ __forceinline__ uint32_t cta_exclusive_scan(uint32_t v, uint32_t* sums, uint32_t& total)
        {
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            uint32_t  incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o)
                    incl += up;
            }
            __syncthreads(); // `sums` may still be read from an earlier scan
            if (lane == 31)
                sums[warp] = incl;
            __syncthreads();
            uint32_t to = lane < (int)(blockDim.x >> 5) ? sums[lane] : 0; // the sums up to warp `lane`
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t up = __shfl_up_sync(0xffffffffu, to, o);
                if (lane >= o)
                    to += up;
            }
            const uint32_t before = __shfl_sync(0xffffffffu, to, max(warp - 1, 0));
            total                 = __shfl_sync(0xffffffffu, to, 31);
            return (warp ? before : 0) + incl - v;
        }

        // The same of three values at once.
        __device__ __forceinline__ void cta_exclusive_scan3(const int (&v)[3], uint32_t (*sums)[32], int (&before)[3])
        {
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            int       incl[3] = {v[0], v[1], v[2]};
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                {
                    const int up = __shfl_up_sync(0xffffffffu, incl[c], o);
                    incl[c] += lane >= o ? up : 0;
                }
            __syncthreads(); // `sums` may still be read from an earlier scan
            if (lane == 31)
                for (int c = 0; c < 3; ++c)
                    sums[c][warp] = (uint32_t)incl[c];
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 3; ++c)
                before[c] = __reduce_add_sync(0xffffffffu, lane < warp ? (int)sums[c][lane] : 0) + incl[c] - v[c];
        }

        // The copy of a stream without stuffed bytes holds big-endian 32-bit words (byte i of the copy is byte i ^ 3 of memory).
        // Resident: the raw scan lies in shared memory, from 16-byte vector 0 on, and the copy takes its place -- a tile's bytes are
        // in registers before any of them is written, and never move up.  Otherwise the copy goes to global memory: a thread's
        // bytes start anywhere, so they are laid out in a tile in shared memory first and leave it as whole words (stored byte by
        // byte to global memory they were 11% of the kernel's time).
        template <bool RESIDENT>
        struct clean_writer
        {
            uint32_t* room; // resident: the scan.  Otherwise the tile: 16 bytes for each thread and 4 more
            uint32_t* out;
            uint32_t  size; // bytes appended so far (the same in every thread)
            uint32_t  rest; // the last, incomplete word (thread 0)

            // Appends the bytes of w (in memory order) whose bits are set in `keep`, `at` being their place among the tile's `total`
            // bytes; every thread has passed a barrier since it read its part of the tile.
            __device__ __forceinline__ void append(const uint32_t (&w)[4], uint32_t keep, uint32_t at, uint32_t total)
            {
                uint8_t* const bytes = reinterpret_cast<uint8_t*>(room);
                const uint32_t carry = RESIDENT ? size : size & 3;
                if (!RESIDENT && threadIdx.x == 0)
                    for (uint32_t c = 0; c < carry; ++c)
                        bytes[c ^ 3] = (uint8_t)(rest >> (24 - 8 * c));
                // big-endian words without the bytes that go (as a rule none or one of the sixteen)
                uint32_t       be[4], n = (uint32_t)__popc(keep);
                const uint32_t o = carry + at, end = o + n;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    be[k] = __byte_perm(w[k], 0, 0x0123);
                for (uint32_t gone = ~keep & 0xFFFF; gone;)
                {
                    const uint32_t g = 31 - __clz(gone), in = 8 * (g & 3); // the last one: what lies behind it moves up a byte
                    gone ^= 1u << g;
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)
                    {
                        const uint32_t up   = __funnelshift_l(k < 3 ? be[k + 1] : 0, be[k], 8);
                        const uint32_t mask = k < g >> 2 ? 0 : k > g >> 2 ? 0xFFFFFFFFu : 0xFFFFFFFFu >> in;
                        be[k]               = (be[k] & ~mask) | (up & mask);
                    }
                }
                // They start anywhere in a word: whole words are stored as such, the ends, which belong to two threads, by bytes.
                const uint32_t shift = 8 * (o & 3), w0 = o >> 2, w1 = end >> 2;
                uint32_t       head = 0, tail = 0;
#pragma unroll
                for (uint32_t k = 0; k < 5; ++k)
                {
                    const uint32_t word = __funnelshift_r(k < 4 ? be[k < 4 ? k : 0] : 0, k > 0 ? be[k - 1] : 0, shift);
                    if ((k > 0 || shift == 0) && w0 + k < w1)
                        room[w0 + k] = word;
                    head = k == 0 ? word : head;
                    tail = w0 + k == w1 ? word : tail;
                }
                if (shift != 0)
                    for (uint32_t b = o; b < min(end, (o | 3) + 1); ++b)
                        bytes[b ^ 3] = (uint8_t)(head >> (24 - 8 * (b & 3)));
                if (w1 > w0 || shift == 0)
                    for (uint32_t b = end & ~3u; b < end; ++b)
                        bytes[b ^ 3] = (uint8_t)(tail >> (24 - 8 * (b & 3)));
                if (!RESIDENT)
                {
                    __syncthreads();
                    const uint32_t whole = (carry + total) >> 2, first = size >> 2;
                    for (uint32_t i = threadIdx.x; i < whole; i += blockDim.x)
                        out[first + i] = room[i];
                    if (threadIdx.x == 0)
                        rest = room[whole];
                }
                size += total;
            }
            // Ends the copy with 32 zero bytes that the readers may run into.
            __device__ __forceinline__ void finish()
            {
                if (RESIDENT)
                {
                    __syncthreads(); // the last tile has been read
                    if (threadIdx.x < 32)
                        reinterpret_cast<uint8_t*>(room)[(size + threadIdx.x) ^ 3] = 0;
                    return;
                }
                const uint32_t first = size >> 2, n = ((size + 31) >> 2) - first + 1, kept = 8 * (size & 3);
                if (threadIdx.x < n)
                    out[first + threadIdx.x] = threadIdx.x == 0 && kept ? rest & ~(0xffffffffu >> kept) : 0;
            }
        };

        // Starts the transfer of 16-byte vectors [i0, i1) of the raw scan to shared memory.
        __device__ __forceinline__ void fetch_raw(uint32_t* room, const uint4* vec, uint32_t i0, uint32_t i1)
        {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(room);
            for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + 16 * (i - i0)), "l"(vec + i) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        }

        // What the blocks of a stream need before its bits are looked at: where every block of an MCU goes, and the lookup tables.
        __device__ __forceinline__ void set_up_stream(par_state& S, int tid, int nth)
        {
            const aeonb_entropy_desc& d = S.d;
            // The tables in DHT form are brought in whole by the last threads, while the first ones see to the blocks of an MCU.
            const int back = nth - 1 - tid;
            if ((reinterpret_cast<uintptr_t>(d.tables) & 15) == 0)
            {
                for (int i = back; i < 4 * 272 / 16; i += nth)
                    reinterpret_cast<uint4*>(S.dht)[i] = __ldg(reinterpret_cast<const uint4*>(d.tables) + i);
            }
            else
                for (int i = back; i < 4 * 272; i += nth)
                    S.dht[i] = __ldg(d.tables + i);
            int bpm = 0;
            for (int c = 0; c < d.ncomp; ++c)
                bpm += d.hs[c] * d.vs[c];
            if (tid < bpm)
            {
                const auto part_of = [&](int b, int& at) -> int { // component of block b of an MCU, and the number of its first block
                    at = 0;
                    for (int c = 0;; at += d.hs[c] * d.vs[c], ++c)
                        if (c + 1 == d.ncomp || b < at + d.hs[c] * d.vs[c])
                            return c;
                };
                int           at, unused;
                const int     c = part_of(tid, at), x = (tid - at) % d.hs[c], y = (tid - at) / d.hs[c], next = tid + 1 < bpm ? tid + 1 : 0;
                const int64_t row_blocks = (int64_t)(d.roi[2] - d.roi[0]) * d.hs[c]; // blocks in a row of the compact plane
                const int     ac = table_at(2 + (d.ac_table[c] & 1)) + LONG, dc = table_at(d.dc_table[part_of(next, unused)] & 1) + LONG;
                S.comp[tid]  = (uint8_t)c;
                S.link[tid]  = block_link{shared_address(S.scan + ac), shared_address(S.scan + dc), shared_address(&S.link[next]), (uint32_t)tid};
                S.place[tid] = block_place{shared_address(S.store + ac), shared_address(S.store + dc), shared_address(&S.place[next]),
                                           (uint32_t)(next == 0), d.coef[c] + (y * row_blocks + x) * 64, (int32_t)(d.vs[c] * row_blocks), d.hs[c]};
            }
            if (tid == 0)
                S.bpm = bpm;
            __syncthreads();
            for (int t = tid >> 5; t < 4; t += nth >> 5)
                build_code_table(S.codes[t], S.dht + t * 272, tid & 31, &S.bad);
            for (int i = tid; i < 4 * 256; i += nth)
                S.codes[i >> 8].vals[i & 255] = S.dht[(i >> 8) * 272 + 16 + (i & 255)];
            __syncthreads();
            build_tables(S.store, S.codes, tid, nth, &S.slow);
            __syncthreads();
            pair_tables(S.scan, S.store, tid, nth);
            __syncthreads();
        }

        // Sums the DC differences of MCUs [m0, m1) up from the predictors in front of them and stores the values.
        __device__ __forceinline__ void store_dc(const par_state& S, const int16_t* dcdiff, uint32_t m0, uint32_t m1, int bpm, int (&pred)[3])
        {
            int my = (int)(m0 / (uint32_t)S.d.mcux), mx = (int)(m0 - (uint32_t)my * S.d.mcux);
            for (uint32_t m = m0; m < m1; ++m)
            {
                for (int b = 0; b < bpm; ++b)
                {
                    const int v = dcdiff[(size_t)m * bpm + b];
                    const int c = S.comp[b];
                    int       now;
                    if (c == 0)
                        now = pred[0] += v;
                    else if (c == 1)
                        now = pred[1] += v;
                    else
                        now = pred[2] += v;
                    int16_t* out = block_home(S, mx, my, b);
                    if (out)
                        out[0] = (int16_t)now;
                }
                if (++mx == S.d.mcux)
                {
                    mx = 0;
                    ++my;
                }
            }
        }

        // Decodes every segment from a guessed state (`known`: the true one) and then, in rounds, from its left neighbour's exit state
        // until nothing changes.  Returns the blocks this thread's segment completes; entry states and checkpoints stay in A.
        template <bool SLOW, typename Words>
        __device__ __forceinline__ uint32_t settle_segments(const par_state& S, const seg_arrays& A, const uint32_t* words, uint32_t nseg,
                                                            bool known, uint32_t pbeg, uint32_t pend, uint32_t step)
        {
            const uint32_t  tid = threadIdx.x, T = A.rows;
            const bool      mine       = tid < nseg;
            uint32_t* const chk        = A.chk + tid;
            uint32_t        run_blocks = 0; // blocks of this thread's latest run
            if (mine)
            {
                const seg_result r = scan_segment<SLOW, Words>(S, words, pbeg, 0, 0, pend, chk, T, pbeg + step, step, false, 0);
                A.ent_p[tid]  = pbeg;
                A.ent_bk[tid] = 0;
                A.ext_p[tid]  = r.p;
                A.ext_bk[tid] = (uint16_t)((r.b << 8) | r.k);
                run_blocks    = r.blocks;
            }
            __syncthreads();
            for (uint32_t round = 1; round < nseg; ++round)
            {
                uint32_t cand_p  = 0;
                uint16_t cand_bk = 0;
                bool     redo    = false;
                if (mine && !known)
                {
                    cand_p  = A.ext_p[tid - 1];
                    cand_bk = A.ext_bk[tid - 1];
                    redo    = cand_p != A.ent_p[tid] || cand_bk != A.ent_bk[tid];
                }
                __syncthreads(); // every candidate has been read before any exit state changes
                if (redo)
                {
                    const seg_result r = scan_segment<SLOW, Words>(S, words, cand_p, cand_bk >> 8, cand_bk & 255, pend, chk, T, pbeg + step, step,
                                                                    true, run_blocks);
                    A.ent_p[tid]  = cand_p;
                    A.ent_bk[tid] = cand_bk;
                    run_blocks    = r.blocks;
                    if (!r.merged)
                    {
                        A.ext_p[tid]  = r.p;
                        A.ext_bk[tid] = (uint16_t)((r.b << 8) | r.k);
                    }
                }
                if (!__syncthreads_or(redo))
                    break;
            }
            return run_blocks;
        }

        // The entry state of piece `piece` of segment t, which starts at bit `at`: position, block and zig-zag index, blocks so far.
        __device__ __forceinline__ void piece_entry(const seg_arrays& A, uint32_t t, uint32_t piece, uint32_t at, uint32_t& p,
                                                    uint32_t& bk, uint32_t& before)
        {
            p = A.ent_p[t], bk = A.ent_bk[t], before = 0;
            if (piece > 0)
            {
                const uint32_t key = A.chk[(piece - 1) * A.rows + t];
                p                  = at + (key >> 10);
                bk                 = (key >> 6 & 15) << 8 | (key & 63);
                before             = A.chk[(NCHECK + piece - 1) * A.rows + t];
            }
        }

        // Of 16 bytes, a bit each: those equal to the bytes of `value`; those from number `n` on, and those below it (n may lie outside).
        __device__ __forceinline__ uint32_t byte_mask(const uint32_t (&w)[4], uint32_t value)
        {
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                m |= ((__vcmpeq4(w[k], value) & 0x08040201u) * 0x01010101u >> 24) << (4 * k);
            return m;
        }
        __device__ __forceinline__ uint32_t bits_below(int n) { return n >= 16 ? 0xFFFFu : n <= 0 ? 0 : (1u << n) - 1; }
        __device__ __forceinline__ uint32_t bits_from(int n) { return 0xFFFFu & ~bits_below(n); }

        // Bit b of `keep`: byte b of vector i is part of the data, which ends at `raw_end`; of `marker`: it is not zero and follows 0xFF.
        // `prev` is the byte in front of the vector; the byte in front of the stream (of n bytes, `lead` into the first vector) is not 0xFF.
        __device__ __forceinline__ void scan_masks(const uint32_t (&w)[4], uint32_t prev, uint32_t i, uint32_t lead, uint32_t n, uint32_t raw_end,
                                                   uint32_t& keep, uint32_t& marker)
        {
            const int      at  = (int)(16 * i) - (int)lead;
            const uint32_t own = bits_from(-at) & bits_below((int)n - at), data = own & bits_below((int)raw_end - at);
            const uint32_t ff = byte_mask(w, 0xFFFFFFFFu), zero = byte_mask(w, 0);
            const uint32_t follows = ((ff & own) << 1 | (prev == 0xFF && at > 0)) & 0xFFFF; // bytes that follow 0xFF
            keep   = data & ~(follows & zero);
            marker = own & follows & ~zero;
        }

        // Copies the scan without stuffed bytes, up to the first marker; returns the bytes of the copy.  RESIDENT: in place in `room`,
        // where the scan's vectors have been brought; otherwise from `vec` to `out` through the tile `room`.
        template <bool RESIDENT>
        __device__ __forceinline__ uint32_t copy_scan(par_state& S, uint32_t* room, uint32_t* out, const uint4* vec, uint32_t nv, uint32_t lead)
        {
            const uint32_t         tid = threadIdx.x, T = blockDim.x, N = S.d.scan_size;
            uint32_t               raw_end = S.marker_at;
            clean_writer<RESIDENT> copy{room, out, 0, 0};
            for (uint32_t tile = 0, odd = 0; tile < nv; tile += T, odd ^= 1)
            {
                // (bit 16 of `marker`: the first byte of the next vector)
                const uint32_t i = tile + tid;
                uint32_t       w[4] = {0, 0, 0, 0}, keep = 0, marker = 0;
                if (i < nv)
                {
                    const uint4 x = RESIDENT ? reinterpret_cast<const uint4*>(room)[i] : __ldg(vec + i);
                    w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
                    uint32_t prev = 0;
                    if (i > 0)
                        prev = !RESIDENT  ? (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(vec) + 16 * i - 1)
                               : tid == 0 ? S.tile_end[odd ^ 1] // its place may have been taken
                                          : (uint32_t) reinterpret_cast<const uint8_t*>(room)[16 * i - 1];
                    scan_masks(w, prev, i, lead, N, raw_end, keep, marker);
                    // The second byte of a marker whose first is the tile's last lies in the next tile, which is too late.
                    if (tid == T - 1 && i + 1 < nv && w[3] >> 24 == 0xFF)
                        marker |= (uint32_t)((RESIDENT ? reinterpret_cast<const uint8_t*>(room)[16 * i + 16]
                                                       : __ldg(reinterpret_cast<const uint8_t*>(vec) + 16 * i + 16)) != 0) << 16;
                }
                if (RESIDENT && tid == T - 1)
                    S.tile_end[odd] = w[3] >> 24;
                uint32_t total, at = cta_exclusive_scan((uint32_t)__popc(keep) | (marker ? 1u << 20 : 0), S.warp_sums[0], total);
                at &= (1u << 20) - 1;
                if (total >> 20)
                {
                    // a marker (0xFF followed by anything but 0x00) ends the entropy-coded data
                    if (marker)
                        atomicMin(&S.marker_at, 16 * i + (uint32_t)__ffs(marker) - 1 - lead - 1); // the 0xFF before it
                    __syncthreads();
                    raw_end             = S.marker_at;
                    const uint32_t left = lead + raw_end > 16 * i ? min(lead + raw_end - 16 * i, 16u) : 0;
                    keep &= (1u << left) - 1;
                    at = cta_exclusive_scan((uint32_t)__popc(keep), S.warp_sums[0], total);
                }
                copy.append(w, keep, at, total);
                if (lead + raw_end <= 16 * (tile + T))
                    break;
            }
            copy.finish();
            return copy.size;
        }

        // Everything between the copy and the DC sums: segments, their true entry states, and the storing pass.
        template <bool SLOW, typename Words>
        __device__ __forceinline__ void decode_scan(par_state& S, const seg_arrays& A, const uint32_t* words, uint32_t clean_size, int min_segment,
                                                    uint32_t needed_blocks, int16_t* dcdiff)
        {
            const uint32_t            tid = threadIdx.x, T = blockDim.x;
            const aeonb_entropy_desc& d = S.d;
            // ---- segments: at most one per thread, a multiple of 4 bytes, at least min_segment bytes
            uint32_t seg = (clean_size + A.rows - 1) / A.rows;
            seg          = max((seg + 3u) & ~3u, (uint32_t)max(min_segment, 64) & ~3u);
            // The storing pass deals its pieces out in rounds of T.  Up to a quarter more than a whole number of rounds is avoided by
            // longer segments: the last round would take as long as the others.
            const uint32_t rounds = max(((NCHECK + 1) * ((clean_size + seg - 1) / seg) * 4 + 3 * T) / (4 * T), 1u);
            seg                   = max(seg, ((NCHECK + 1) * clean_size / (rounds * T) + 4u) & ~3u);
            const uint32_t nseg      = (clean_size + seg - 1) / seg; // <= A.rows <= T
            const uint32_t total_bit = clean_size * 8;
            const uint32_t pbeg = tid * seg * 8, pend = min(total_bit, pbeg + seg * 8);
            // checkpoints of a segment, evenly spaced (at least 64 bits apart; a symbol is shorter, so it passes at most one)
            const uint32_t step = seg * 8 / (NCHECK + 1); // bits between checkpoints (seg is a multiple of 4 bytes)

            // ---- clear the coefficient planes now: the stores drain while the segments are being decoded, and the barriers
            // between here and the storing pass order them before that pass's stores.  Warps without a segment do it, if there
            // are four of them, while the others start decoding.
            const uint32_t busy = (nseg + 31) & ~31u, from = T >= busy + 128 ? busy : 0;
            if (tid >= from)
                for (int c = 0; c < d.ncomp; ++c)
                {
                    const size_t n16 = (size_t)(d.roi[2] - d.roi[0]) * d.hs[c] * (d.roi[3] - d.roi[1]) * d.vs[c] * 8; // 16-byte units
                    uint4*       p   = reinterpret_cast<uint4*>(d.coef[c]);
                    for (size_t i = tid - from; i < n16; i += T - from)
                        p[i] = make_uint4(0, 0, 0, 0);
                }

            const uint32_t run_blocks = settle_segments<SLOW, Words>(S, A, words, nseg, tid == 0, pbeg, pend, step);

            // ---- first block number of every segment
            uint32_t       counted;
            const uint32_t g0 = cta_exclusive_scan(run_blocks, S.warp_sums[0], counted);
            if (tid == 0 && counted < needed_blocks)
                S.bad = 1;

            // ---- decode once more from the true entry states, storing (the planes were cleared above).  The checkpoints now
            // describe every segment's final run, so each segment falls into NCHECK + 1 pieces with known entry states and block
            // numbers, and the pieces -- not the segments -- are dealt out to the threads: streams with fewer segments than
            // threads keep every warp busy, and neighbouring lanes work on neighbouring pieces.
            if (tid < nseg)
                A.cnt[tid] = g0;
            __syncthreads();
            for (uint32_t q = tid; q < nseg * (NCHECK + 1); q += T)
            {
                const uint32_t t = q / (NCHECK + 1), piece = q % (NCHECK + 1);
                const uint32_t seg_beg = t * seg * 8, seg_end = min(total_bit, seg_beg + seg * 8);
                const uint32_t at = seg_beg + piece * step; // the checkpoint this piece starts from
                if (at >= seg_end)
                    continue;
                uint32_t p0, bk, before;
                piece_entry(A, t, piece, at, p0, bk, before);
                const store_result r = store_segment<SLOW, Words>(S, words, p0, bk >> 8, bk & 255, min(seg_end, at + step), A.cnt[t] + before,
                                                                needed_blocks, dcdiff);
                if (r.bad)
                    S.bad = 1;
            }
            __syncthreads();
        }

        __device__ __forceinline__ bool parallel_shape_ok(const aeonb_entropy_desc& d, int& bpm, uint64_t& clean_room)
        {
            bpm = 0;
            for (int c = 0; c < 3; ++c)
                if (c < d.ncomp)
                    bpm += d.hs[c] * d.vs[c];
            const uint64_t total_blocks = (uint64_t)d.mcux * d.mcuy * bpm, dc_room = (total_blocks * 2 + 15) & ~15ull;
            clean_room = ((uint64_t)d.scan_size + 32 + 15) & ~15ull;
            return d.ncomp >= 1 && d.ncomp <= 3 && d.mcux > 0 && d.mcuy > 0 && d.scan && d.tables && bpm <= 16 && d.scan_size < (1u << 27) &&
                   total_blocks < (1ull << 30) && d.scratch_bytes >= clean_room + dc_room && (reinterpret_cast<uintptr_t>(d.scratch) & 3) == 0;
        }

        // Shared memory of a block: par_state, SEG_BYTES for each of `rows` segments, and what is left of `smem_bytes` for the scan and
        // behind it the DC differences, where they fit; otherwise they live in the record's work area.
        __global__ void __launch_bounds__(PAR_THREADS) jpeg_entropy_parallel_kernel(const __grid_constant__ launch_data data, int min_segment,
                                                                                    uint32_t rows, uint32_t smem_bytes)
        {
            const uint32_t T = blockDim.x;
            extern __shared__ __align__(16) unsigned char smem_raw[];
            par_state&       S          = *reinterpret_cast<par_state*>(smem_raw);
            const seg_arrays A          = seg_arrays_at(smem_raw + sizeof(par_state), rows);
            const uint32_t   room_at    = ((uint32_t)sizeof(par_state) + SEG_BYTES * rows + 15) & ~15u;
            uint32_t* const  room       = reinterpret_cast<uint32_t*>(smem_raw + room_at);
            const uint32_t   room_bytes = smem_bytes - room_at;
            const int        tid        = threadIdx.x;
            data.fetch(S.d, (int)(blockIdx.x), (int)tid, (int)T);
            if (tid < 64)
                S.zz[16 + tid] = k_zz_colmajor[tid];
            if (tid == 0)
                S.bad = S.slow = 0;
            __syncthreads();
            const aeonb_entropy_desc& d = S.d;
            if (!d.scratch || d.restart_interval != 0)
                return; // the other kernels' stream
            uint64_t clean_room; // of the work area, for the copy; the DC differences lie behind it
            int      bpm;
            if (!parallel_shape_ok(d, bpm, clean_room))
            {
                if (tid == 0 && d.status)
                    *d.status = 1;
                return;
            }
            // The raw scan is read as 16-byte vectors from the aligned address below it; `lead` bytes precede it there.
            const uint32_t     N    = d.scan_size;
            const uint32_t     lead = (uint32_t)(reinterpret_cast<uintptr_t>(d.scan) & 15);
            const uint4* const vec  = reinterpret_cast<const uint4*>(d.scan - lead);
            const uint32_t     nv   = (lead + N + 15) >> 4;
            const uint32_t     scan_room = 16 * nv + 48; // the zero bytes behind the copy, too
            const bool         resident  = scan_room <= room_bytes;
            if (resident)
                fetch_raw(room, vec, 0, nv); // arrives while the tables are being built
            if (tid == 64) // not a thread that sets anything else up
                S.marker_at = N > 0 && __ldg(d.scan + N - 1) == 0xFF ? N - 1 : N;
            set_up_stream(S, tid, (int)T);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();

            const uint32_t needed_mcus   = (uint32_t)min(d.roi[3], d.mcuy) * d.mcux;
            const uint32_t needed_blocks = needed_mcus * bpm;
            uint8_t* const clean         = static_cast<uint8_t*>(d.scratch);
            int16_t*       dcdiff        = reinterpret_cast<int16_t*>(clean + clean_room);
            if (resident)
            {
                if (2ull * needed_blocks <= room_bytes - scan_room)
                    dcdiff = reinterpret_cast<int16_t*>(reinterpret_cast<uint8_t*>(room) + scan_room);
                const uint32_t clean_size = copy_scan<true>(S, room, nullptr, vec, nv, lead);
                __syncthreads();
                if (S.slow)
                    decode_scan<true, shared_words>(S, A, room, clean_size, min_segment, needed_blocks, dcdiff);
                else
                    decode_scan<false, shared_words>(S, A, room, clean_size, min_segment, needed_blocks, dcdiff);
            }
            else
            {
                uint32_t* const words = reinterpret_cast<uint32_t*>(clean);
                // the checkpoints' room and what follows is not in use yet
                const uint32_t clean_size = copy_scan<false>(S, A.chk, words, vec, nv, lead);
                __syncthreads();
                decode_scan<true, global_words>(S, A, words, clean_size, min_segment, needed_blocks, dcdiff);
            }

            // ---- DC: sum the differences per component in scan order.  Thread t owns MCUs [m0, m1).
            const uint32_t mchunk = (needed_mcus + T - 1) / T;
            const uint32_t m0 = min(needed_mcus, tid * mchunk), m1 = min(needed_mcus, m0 + mchunk);
            int            sum[3] = {0, 0, 0};
            for (uint32_t m = m0; m < m1; ++m)
                for (int b = 0; b < bpm; ++b)
                {
                    const int v = dcdiff[(size_t)m * bpm + b];
                    const int c = S.comp[b];
                    sum[0] += c == 0 ? v : 0;
                    sum[1] += c == 1 ? v : 0;
                    sum[2] += c == 2 ? v : 0;
                }
            int pred[3];
            cta_exclusive_scan3(sum, S.warp_sums, pred);
            store_dc(S, dcdiff, m0, m1, bpm, pred);
            __syncthreads();
            if (tid == 0 && d.status)
                *d.status = S.bad ? 1 : 0;
        }

        // ------------------------------------------------------------------------------------------------
        // Few streams without restart markers: a cluster of thread blocks per stream.
        //
        // With fewer streams than SMs the kernel above leaves most of the chip idle, and more threads would not help it: its time
        // is the chain of symbols that a wrong guess takes to fall into step, 820 bits on average and 5000 at the worst place of a
        // 40 KB stream (4:2:0), and most of that is waiting for the block's place in the MCU to match; codes alone are in step after 80
        // bits, 1100 at worst.  So here every segment (128 bytes) is entered once for each place in the MCU; one of these runs
        // is in step after half a segment nearly always.  A run that leaves its segment goes on into the next ones until it is at one
        // of their checkpoints in the state of one of their runs.  That makes a graph -- from each run to the run
        // it falls into step with, and the blocks in between -- in which the stream is the path from the first segment's
        // run 0.  Following the path takes no decoding; it is shortened by following it from the first segment of every group of
        // segments, and of every block, at the same time.  The storing pass is dealt out in the pieces between the known states.
        // The tables are built in every block of the cluster, each cleans an equal part of the scan; what crosses blocks are the clean
        // scan (through the work area), the states at the checkpoints, the graph and sums of DC differences.
        //
        // Measured on a B200 (kernel times), one block per stream / this: one stream of 43 KB (eight blocks) 133 us / 56 us, 4 of them
        // 153 / 54, 32 (four blocks) 170 / 84; the work is about 2.5 times that of the rounds, so it is for SMs that would be idle.
        // Phases of the one stream, thousand cycles: set-up 13, copy 11, first pass 25, going on 11 on average and 16 at worst,
        // path 8, storing pass 16, DC 4.  The first pass is bound by the issue of integer instructions; so short
        // segments do not pay, and more checkpoints (eight) cost it more than the shorter pieces of the storing pass give.
        constexpr int SPREAD_MOST   = 8;    // blocks in a cluster
        constexpr int SPREAD_PLACES = 6;    // places in an MCU, at most
        constexpr int SPREAD_CHECKS = 4;    // checkpoints of a segment, the last one at its end
        constexpr int SPREAD_SEG    = 128;  // bytes of a segment, at least (64 with two checkpoints: 4 us more for 32 streams)
        constexpr int SPREAD_GROUP  = 16;   // segments
        constexpr int SPREAD_EXTRA  = 256;  // states noted between a run's exit and where it falls into step
        constexpr uint32_t k_none = 0xffffffffu;

        // A place on a path: checkpoint of a run (segment << 6 | place in the MCU << 3 | checkpoint), k_none behind the stream's
        // end; `blocks`: how many more blocks are complete there than the run itself counts (at the end: how many in all).
        struct spread_hop
        {
            uint32_t to, blocks;
        };
        struct spread_extra
        {
            uint32_t node, p, bk, blocks, end; // the run; state, blocks since the run's start; where the next known state is
        };
        struct spread_state
        {
            par_state    S;
            spread_extra extra[SPREAD_EXTRA];
            // What the blocks of the cluster tell one another: each writes its own entry in all blocks (a block that fetched the others'
            // would wait for one after the other).
            struct
            {
                uint32_t   bytes, marker;          // of its part of the scan: bytes without stuffed ones, first marker
                uint32_t   kept;                   // its bytes in front of the stream's first marker
                int32_t    dc[3];                  // sums of its DC differences
                uint32_t   bad;
                spread_hop through[SPREAD_PLACES]; // from its first segment's runs to the first run outside the block
            } all[SPREAD_MOST];
            uint32_t extras, bytes, marker;
            int32_t  dc[3];
        };
        // Of each run, states as scanner::key gives them at the checkpoints (k_none: the stream ended in front of it), blocks by then,
        // the run it falls into step with, and where the next known state behind its exit is.
        struct spread_nodes
        {
            uint32_t*   key; // SPREAD_CHECKS rows of `cap`
            uint16_t*   cnt; // as many
            spread_hop* next;
            uint32_t*   end;
            spread_hop* group;  // from the runs of each group's first segment to the first run outside the group
            spread_hop* inside; // per group: where the path comes in
            spread_hop* truth;  // per segment: the path's run and checkpoint there
        };
        __host__ __device__ inline uint32_t spread_bytes(uint32_t cap)
        {
            return cap * (8 + SPREAD_CHECKS * 6 + 4) + (cap / SPREAD_GROUP + 2 * SPREAD_PLACES) * 16 + (cap + 2) * 8;
        }
        __device__ __forceinline__ spread_nodes spread_nodes_at(unsigned char* p, uint32_t cap)
        {
            spread_nodes N;
            N.next   = reinterpret_cast<spread_hop*>(p);
            N.group  = N.next + cap;
            N.inside = N.group + cap / SPREAD_GROUP + 2 * SPREAD_PLACES;
            N.truth  = N.inside + cap / SPREAD_GROUP + 2 * SPREAD_PLACES;
            N.key    = reinterpret_cast<uint32_t*>(N.truth + cap + 2);
            N.end    = N.key + SPREAD_CHECKS * cap;
            N.cnt    = reinterpret_cast<uint16_t*>(N.end + cap);
            return N;
        }

        template <typename T>
        __device__ __forceinline__ T* in_block(T* p, uint32_t rank)
        {
            return cooperative_groups::this_cluster().map_shared_rank(p, rank);
        }

        // Copies the scan without stuffed bytes, up to the first marker: each block the vectors [v0, v1), which have been brought to
        // `room`, to the work area, and from there every block all of it to `room`.  Returns the bytes of the copy.  Takes the wait that
        // belongs to the arrival at the cluster's barrier at the kernel's beginning.
        __device__ __forceinline__ uint32_t copy_spread(spread_state& D, uint32_t* room, uint32_t* work, const uint4* vec, uint32_t v0, uint32_t v1,
                                                        uint32_t lead)
        {
            cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
            par_state&     S = D.S;
            const uint32_t tid = threadIdx.x, T = blockDim.x, C = cluster.num_blocks(), rank = cluster.block_rank();
            const uint32_t n = S.d.scan_size;
            auto look = [&](uint32_t i, uint32_t prev, uint32_t raw_end, uint32_t (&w)[4], uint32_t& keep, uint32_t& marker) {
                const uint4 x = reinterpret_cast<const uint4*>(room)[i - v0];
                w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
                scan_masks(w, prev, i, lead, n, raw_end, keep, marker);
            };
            const uint32_t first_prev = v0 > 0 && v0 < v1 ? (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(vec) + 16 * v0 - 1) : 0;
            // once as if no part in front held a marker, for the markers and the counts
            uint32_t kept = 0;
            for (uint32_t i = v0 + tid; i < v1; i += T)
            {
                uint32_t w[4], keep, marker;
                look(i, i == v0 ? first_prev : reinterpret_cast<const uint8_t*>(room)[16 * (i - v0) - 1], S.marker_at, w, keep, marker);
                kept += __popc(keep);
                if (marker)
                    atomicMin(&D.marker, 16 * i + (uint32_t)__ffs(marker) - 1 - lead - 1); // the 0xFF before it
            }
            uint32_t all;
            cta_exclusive_scan(kept, S.warp_sums[0], all);
            cluster.barrier_wait(); // every block of the cluster has started (it arrived on entry): its memory may be written from now on
            if (tid < C)
            {
                in_block(D.all, tid)[rank].bytes  = all;
                in_block(D.all, tid)[rank].marker = D.marker;
            }
            cluster.sync();
            uint32_t before = 0, raw_end = S.marker_at;
            for (uint32_t r = 0; r < C; ++r)
            {
                raw_end = min(raw_end, D.all[r].marker);
                before += r < rank ? D.all[r].bytes : 0;
            }
            // the copy of this part, in place; what lies behind the marker goes
            clean_writer<true> copy{room, nullptr, 0, 0};
            for (uint32_t tile = v0, odd = 0; tile < v1; tile += T, odd ^= 1)
            {
                const uint32_t i = tile + tid;
                uint32_t       w[4] = {0, 0, 0, 0}, keep = 0, marker;
                if (i < v1)
                    look(i, i == v0 ? first_prev : tid == 0 ? S.tile_end[odd ^ 1] : reinterpret_cast<const uint8_t*>(room)[16 * (i - v0) - 1],
                         raw_end, w, keep, marker);
                if (tid == T - 1)
                    S.tile_end[odd] = w[3] >> 24; // the next tile finds its place taken
                uint32_t       total;
                const uint32_t at = cta_exclusive_scan((uint32_t)__popc(keep), S.warp_sums[0], total);
                copy.append(w, keep, at, total);
            }
            __syncthreads();
            // to its place in the work area: whole words, and bytes where two parts share a word
            if (tid < C)
                in_block(D.all, tid)[rank].kept = copy.size;
            uint8_t* const bytes = reinterpret_cast<uint8_t*>(work);
            const uint32_t end = before + copy.size, shift = 8 * (before & 3);
            for (uint32_t i = (before >> 2) + tid; 4 * i < end; i += T)
            {
                const uint32_t k    = i - (before >> 2); // the word of the part that begins in it
                const uint32_t word = __funnelshift_r(room[k], k ? room[k - 1] : 0, shift);
                if (4 * i >= before && 4 * i + 4 <= end)
                    work[i] = word;
                else
                    for (uint32_t b = max(4 * i, before); b < min(4 * i + 4, end); ++b)
                        bytes[b ^ 3] = (uint8_t)(word >> (24 - 8 * (b & 3)));
            }
            cluster.sync();
            uint32_t size = 0;
            for (uint32_t r = 0; r < C; ++r)
                size += D.all[r].kept;
            // (the last vector brings what lies behind the copy too; the readers want 32 zero bytes there)
            fetch_raw(room, reinterpret_cast<const uint4*>(work), 0, (size + 15) >> 4);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (tid < 32)
                reinterpret_cast<uint8_t*>(room)[(size + tid) ^ 3] = 0;
            __syncthreads();
            return size;
        }

        template <bool SLOW>
        __device__ __forceinline__ void decode_spread(spread_state& D, const spread_nodes& N, const uint32_t* words, uint32_t clean_size, uint32_t cap,
                                                      uint32_t needed_blocks, int16_t* dcdiff)
        {
            using run = scanner<SLOW, shared_words>;
            cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
            par_state&     S = D.S;
            const uint32_t tid = threadIdx.x, T = blockDim.x, C = cluster.num_blocks(), rank = cluster.block_rank();
            const uint32_t H = (uint32_t)S.bpm, total = clean_size * 8;
            // segments: a multiple of SPREAD_CHECKS bytes; a block's runs fit `cap` nodes
            const uint32_t most = C * (cap / H - 2);
            const uint32_t seg  = max((uint32_t)SPREAD_SEG, ((clean_size + most - 1) / most + SPREAD_CHECKS - 1) & ~(SPREAD_CHECKS - 1u));
            const uint32_t bits = seg * 8, step = bits / SPREAD_CHECKS; // at least 128: a symbol passes one checkpoint at most
            const uint32_t nseg = (clean_size + seg - 1) / seg, per = max((nseg + C - 1) / C, 1u);
            const uint32_t s0 = rank * per, mine = s0 < nseg ? min(per, nseg - s0) : 0, nodes = mine * H;

            // ---- clear this block's share of the planes: warps without a run, if there are four of them, while the others decode.  The
            // cluster's barriers stand between here and the storing pass.
            const uint32_t busy = (nodes + 31) & ~31u, from = T >= busy + 128 ? busy : 0;
            if (tid >= from)
                for (int c = 0; c < S.d.ncomp; ++c)
                {
                    const size_t n16 = (size_t)(S.d.roi[2] - S.d.roi[0]) * S.d.hs[c] * (S.d.roi[3] - S.d.roi[1]) * S.d.vs[c] * 8; // 16-byte units
                    uint4*       p   = reinterpret_cast<uint4*>(S.d.coef[c]);
                    for (size_t i = n16 * rank / C + tid - from, last = n16 * (rank + 1) / C; i < last; i += T - from)
                        p[i] = make_uint4(0, 0, 0, 0);
                }

            // ---- every segment from every place in the MCU.  Neighbouring threads have the same segment.
            for (uint32_t t = tid; t < nodes; t += T)
            {
                const uint32_t ls = t / H, beg = (s0 + ls) * bits;
                run            r(S, words, beg, (int)(t - ls * H), 0);
                uint32_t       j = 0;
                for (uint32_t stop = beg + step; j < SPREAD_CHECKS && stop < total; ++j, stop += step)
                {
                    r.run_to(S, stop);
                    N.key[j * cap + t] = r.key(stop);
                    N.cnt[j * cap + t] = (uint16_t)r.blocks;
                }
                if (j < SPREAD_CHECKS)
                {
                    r.run_to(S, total);
                    for (; j < SPREAD_CHECKS; ++j)
                    {
                        N.key[j * cap + t] = k_none;
                        N.cnt[j * cap + t] = (uint16_t)r.blocks;
                    }
                }
            }
            cluster.sync();

            // ---- from every exit on until the run falls into step with another one
            for (uint32_t t = tid; t < nodes; t += T)
            {
                const uint32_t key = N.key[(SPREAD_CHECKS - 1) * cap + t], had = N.cnt[(SPREAD_CHECKS - 1) * cap + t];
                spread_hop     hop{k_none, had};
                if (key != k_none)
                {
                    uint32_t  q = s0 + t / H + 1, j = 0, stop = q * bits;
                    run       r(S, words, stop + (key >> 10), (int)(key >> 6 & 15), (int)(key & 63));
                    uint32_t* end = N.end + t; // the end of the piece under way
                    for (;;)
                    {
                        stop += step;
                        if (stop >= total)
                        {
                            r.run_to(S, total);
                            *end = total;
                            hop  = spread_hop{k_none, had + r.blocks};
                            break;
                        }
                        r.run_to(S, stop);
                        const uint32_t        at = r.key(stop), owner = q / per, first = j * cap + (q - owner * per) * H;
                        const uint32_t* const there = (owner == rank ? N.key : in_block(N.key, owner)) + first;
                        uint32_t              h     = H;
#pragma unroll
                        for (uint32_t k = 0; k < SPREAD_PLACES; ++k) // the loads do not wait for one another
                            h = k < H && there[k] == at ? k : h;
                        if (h < H)
                        {
                            *end = r.position();
                            hop  = spread_hop{q << 6 | h << 3 | j, had + r.blocks - (owner == rank ? N.cnt : in_block(N.cnt, owner))[first + h]};
                            break;
                        }
                        const uint32_t x = atomicAdd(&D.extras, 1);
                        if (x < SPREAD_EXTRA)
                        {
                            *end       = r.position();
                            D.extra[x] = spread_extra{t, r.position(), at & 1023, had + r.blocks, 0};
                            end        = &D.extra[x].end;
                        }
                        j = (j + 1) % SPREAD_CHECKS;
                        q += j == 0;
                    }
                }
                N.next[t] = hop;
            }
            for (uint32_t i = tid; i < mine; i += T)
                N.truth[i] = spread_hop{k_none, 0};
            const uint32_t groups = (mine + SPREAD_GROUP - 1) / SPREAD_GROUP;
            for (uint32_t i = tid; i < groups; i += T)
                N.inside[i] = spread_hop{k_none, 0};
            __syncthreads();

            // ---- the path.  From the runs of each group's first segment to the first run outside the group
            auto segment = [](uint32_t to) { return to >> 6; };
            auto place   = [](uint32_t to) { return to >> 3 & 7; };
            auto local   = [&](const spread_hop& a) { return a.to != k_none && segment(a.to) - s0 < mine; };
            auto through_group = [&](spread_hop a, uint32_t g, auto visit) {
                for (const uint32_t last = min((g + 1) * SPREAD_GROUP, mine); a.to != k_none && segment(a.to) - s0 < last;)
                {
                    const uint32_t   ls = segment(a.to) - s0;
                    const spread_hop b  = N.next[ls * H + place(a.to)];
                    visit(ls, a);
                    a = spread_hop{b.to, a.blocks + b.blocks};
                }
                return a;
            };
            for (uint32_t i = tid; i < groups * H; i += T)
            {
                const uint32_t g = i / H;
                N.group[i]       = through_group(spread_hop{(s0 + g * SPREAD_GROUP) << 6 | (i - g * H) << 3, 0}, g, [](uint32_t, const spread_hop&) {});
            }
            __syncthreads();
            // one hop from a run of a block whose first segment is `base`: through its group where the run is of the group's first segment
            auto hop = [&](const spread_hop& a, const spread_hop* next, const spread_hop* group, uint32_t base) {
                const uint32_t   ls = segment(a.to) - base;
                const spread_hop b  = ls % SPREAD_GROUP == 0 ? group[ls / SPREAD_GROUP * H + place(a.to)] : next[ls * H + place(a.to)];
                return spread_hop{b.to, a.blocks + b.blocks};
            };
            if (tid < H && nodes)
            {
                spread_hop a{s0 << 6 | tid << 3, 0};
                while (local(a))
                    a = hop(a, N.next, N.group, s0);
                for (uint32_t r = rank + 1; r < C; ++r)
                    in_block(D.all, r)[rank].through[tid] = a;
            }
            cluster.sync();
            if (tid == 0)
            {
                spread_hop a{nseg ? 0u : k_none, 0};
                while (a.to != k_none && segment(a.to) < s0) // in a block in front of this one
                {
                    const uint32_t owner = segment(a.to) / per;
                    if (segment(a.to) == owner * per)
                    {
                        const spread_hop b = D.all[owner].through[place(a.to)];
                        a                  = spread_hop{b.to, a.blocks + b.blocks};
                    }
                    else
                        a = hop(a, in_block(N.next, owner), in_block(N.group, owner), owner * per);
                }
                // and through this one, noting where each group is entered
                const bool comes = local(a) || (nseg == 0 && rank == 0);
                while (local(a))
                {
                    const uint32_t g = (segment(a.to) - s0) / SPREAD_GROUP;
                    if (N.inside[g].to == k_none)
                        N.inside[g] = a;
                    a = hop(a, N.next, N.group, s0);
                }
                // the block in which the path ends knows how many blocks the stream holds
                if (comes && a.to == k_none && a.blocks < needed_blocks)
                    S.bad = 1;
            }
            __syncthreads();
            for (uint32_t g = tid; g < groups; g += T)
                through_group(N.inside[g], g, [&](uint32_t ls, const spread_hop& a) { N.truth[ls] = a; });
            __syncthreads();

            // ---- store.  Pieces: from each checkpoint of the path's runs to the next one, from their exits to the next known state, from
            // the states noted on the way, and the stream's beginning.
            const uint32_t extras = min(D.extras, (uint32_t)SPREAD_EXTRA), checks = SPREAD_CHECKS * mine;
            const uint32_t pieces = checks + extras + (rank == 0 && mine > 0);
            bool           bad    = false;
            for (uint32_t i = tid; i < pieces; i += T)
            {
                uint32_t p, bk, g, end;
                if (i < checks)
                {
                    const uint32_t   ls = i / SPREAD_CHECKS, j = i % SPREAD_CHECKS, t = ls * H, beg = (s0 + ls) * bits;
                    const spread_hop a = N.truth[ls];
                    if (a.to == k_none || j < (a.to & 7))
                        continue; // the path does not come here, or comes in further on
                    const uint32_t row = j * cap + t + place(a.to), key = N.key[row];
                    if (key == k_none)
                        continue; // the stream ended in front of it
                    p   = beg + (j + 1) * step + (key >> 10);
                    bk  = key & 1023;
                    g   = a.blocks + N.cnt[row];
                    end = j < SPREAD_CHECKS - 1 ? min(beg + (j + 2) * step, total) : N.end[t + place(a.to)];
                }
                else if (i < checks + extras)
                {
                    const spread_extra x = D.extra[i - checks];
                    const spread_hop   a = N.truth[x.node / H];
                    if (a.to == k_none || place(a.to) != x.node % H)
                        continue;
                    p = x.p, bk = x.bk, g = a.blocks + x.blocks, end = x.end;
                }
                else
                    p = bk = g = 0, end = min(step, total);
                const store_result r = store_segment<SLOW, shared_words>(S, words, p, (int)(bk >> 6), (int)(bk & 63), end, g, needed_blocks, dcdiff);
                bad |= r.bad;
            }
            if (bad)
                S.bad = 1;
        }

        __global__ void __launch_bounds__(PAR_THREADS) jpeg_entropy_spread_kernel(const __grid_constant__ launch_data data, uint32_t cap)
        {
            cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
            const uint32_t T = blockDim.x, C = cluster.num_blocks(), rank = cluster.block_rank(), tid = threadIdx.x;
            extern __shared__ __align__(16) unsigned char smem_raw[];
            spread_state&      D    = *reinterpret_cast<spread_state*>(smem_raw);
            par_state&         S    = D.S;
            const spread_nodes N    = spread_nodes_at(smem_raw + sizeof(spread_state), cap);
            uint32_t* const    room = reinterpret_cast<uint32_t*>(smem_raw + ((sizeof(spread_state) + spread_bytes(cap) + 15) & ~15u));
            data.fetch(S.d, (int)(blockIdx.x / C), (int)tid, (int)T);
            if (tid < 64)
                S.zz[16 + tid] = k_zz_colmajor[tid];
            if (tid == 0)
                S.bad = S.slow = 0, D.extras = 0, D.marker = k_none;
            __syncthreads();
            const aeonb_entropy_desc& d = S.d;
            if (!d.scratch || d.restart_interval != 0)
                return; // the other kernels' stream; all blocks of the cluster leave here
            uint64_t clean_room;
            int      bpm;
            if (!parallel_shape_ok(d, bpm, clean_room))
            {
                if (tid == 0 && rank == 0 && d.status)
                    *d.status = 1;
                return;
            }
            // Nothing else promises that the other blocks have started by the time this one first writes to their memory; copy_spread
            // waits for all of them there, behind the tables, so that the wait costs nothing.
            cluster.barrier_arrive();
            const uint32_t     n = d.scan_size;
            const uint32_t     lead = (uint32_t)(reinterpret_cast<uintptr_t>(d.scan) & 15);
            const uint4* const vec  = reinterpret_cast<const uint4*>(d.scan - lead);
            const uint32_t     nv   = (lead + n + 15) >> 4;
            // this block's share of the scan, which arrives while the tables are being built
            const uint32_t part = (nv + C - 1) / C, v0 = min(nv, rank * part), v1 = min(nv, v0 + part);
            fetch_raw(room, vec, v0, v1);
            if (tid == 64) // not a thread that sets anything else up
                S.marker_at = n > 0 && __ldg(d.scan + n - 1) == 0xFF ? n - 1 : n;
            set_up_stream(S, (int)tid, (int)T);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            const uint32_t needed_mcus = (uint32_t)min(d.roi[3], d.mcuy) * d.mcux;
            int16_t* const dcdiff      = reinterpret_cast<int16_t*>(static_cast<uint8_t*>(d.scratch) + clean_room);
            const uint32_t clean_size  = copy_spread(D, room, reinterpret_cast<uint32_t*>(d.scratch), vec, v0, v1, lead);
            if (S.slow)
                decode_spread<true>(D, N, room, clean_size, cap, needed_mcus * bpm, dcdiff);
            else
                decode_spread<false>(D, N, room, clean_size, cap, needed_mcus * bpm, dcdiff);
            cluster.sync(); // the differences are there

            // ---- DC: sum the differences per component in scan order; block r of the cluster owns the r-th run of MCUs, its thread t
            // MCUs [m0, m1).  The differences of an MCU are fetched together.
            const uint32_t share = (needed_mcus + C - 1) / C, b0 = min(needed_mcus, rank * share), b1 = min(needed_mcus, b0 + share);
            const uint32_t mchunk = (share + T - 1) / T, m0 = min(b1, b0 + tid * mchunk), m1 = min(b1, m0 + mchunk);
            int            sum[3] = {0, 0, 0}, pred[3], diff[SPREAD_PLACES];
            for (uint32_t m = m0; m < m1; ++m)
            {
#pragma unroll
                for (int b = 0; b < SPREAD_PLACES; ++b)
                    diff[b] = b < bpm ? dcdiff[(size_t)m * bpm + b] : 0;
#pragma unroll
                for (int b = 0; b < SPREAD_PLACES; ++b)
                {
                    const int c = b < bpm ? S.comp[b] : 0;
                    sum[0] += c == 0 ? diff[b] : 0;
                    sum[1] += c == 1 ? diff[b] : 0;
                    sum[2] += c == 2 ? diff[b] : 0;
                }
            }
            cta_exclusive_scan3(sum, S.warp_sums, pred);
            if (tid == T - 1)
                for (int c = 0; c < 3; ++c)
                    D.dc[c] = pred[c] + sum[c];
            __syncthreads();
            if (tid < C)
            {
                auto& mine = in_block(D.all, tid)[rank];
                mine.dc[0] = D.dc[0], mine.dc[1] = D.dc[1], mine.dc[2] = D.dc[2];
                mine.bad   = (uint32_t)S.bad;
            }
            cluster.sync(); // nothing touches another block's memory afterwards
            for (uint32_t r = 0; r < rank; ++r)
                for (int c = 0; c < 3; ++c)
                    pred[c] += D.all[r].dc[c];
            if (m1 == m0 + 1)
            {
                const int my = (int)(m0 / (uint32_t)d.mcux), mx = (int)(m0 - (uint32_t)my * d.mcux);
#pragma unroll
                for (int b = 0; b < SPREAD_PLACES; ++b)
                    if (b < bpm)
                    {
                        const int c   = S.comp[b];
                        const int now = (c == 0 ? pred[0] : c == 1 ? pred[1] : pred[2]) + diff[b];
                        pred[0] = c == 0 ? now : pred[0];
                        pred[1] = c == 1 ? now : pred[1];
                        pred[2] = c == 2 ? now : pred[2];
                        if (int16_t* const out = block_home(S, mx, my, b))
                            out[0] = (int16_t)now;
                    }
            }
            else
                store_dc(S, dcdiff, m0, m1, bpm, pred);
            if (tid == 0 && rank == 0 && d.status)
            {
                uint32_t bad = 0;
                for (uint32_t r = 0; r < C; ++r)
                    bad |= D.all[r].bad;
                *d.status = bad ? 1 : 0;
            }
        }

        // ------------------------------------------------------------------------------------------------
        // Streams with restart markers.
        //
        // Behind every restart marker a decoder starts afresh -- byte aligned, first block of an MCU, DC predictors zero -- so the
        // intervals between them are independent and their first block numbers known.  An index kernel (a cluster of blocks per stream)
        // notes where the intervals start; the stream is then cut into parts of up to RST_MAX_INTERVALS whole intervals, one thread
        // block each, and inside a part the intervals into segments as in the kernel above, except that the first segment of
        // every interval starts in the true state and block numbers are counted from there: a wrong guess travels to the end of
        // its interval at most.  DC differences are summed by a warp per interval.
        // What the serial kernel makes of a damaged stream (missing or foreign markers, fill bytes, intervals with too little or
        // too much in them) is a matter of its resynchronisation rules, so nothing is decided about such a stream here: it is
        // marked doubtful and the serial kernel, launched behind, decodes it anew.
        //
        // Measured on a B200, 32 pictures of 900-1400 pixels a side (4:2:2, quality 92, a marker after every MCU row, 0.3 MB
        // each): 88 ms with the serial kernel (one warp per stream), 0.21 ms with these two.  Two blocks of 512 threads fit an SM by
        // their tables; five of 128 threads with parts of at most 10 KB took 0.09 ms more, most of it spent on building tables.
        constexpr int RST_THREADS       = 512;
        constexpr int RST_INDEX_THREADS = 1024;
        constexpr int RST_ROOM          = 46 * 1024; // shared memory for a part's bytes (see jpeg_restart_parts): 2 blocks fit an SM

        struct rst_state
        {
            par_state S;
            uint32_t  raw[RST_MAX_INTERVALS + 1];   // offset of the first byte of every interval; behind the last: of its end + 2
            uint32_t  clean[RST_MAX_INTERVALS + 1]; // the same in the copy
            uint32_t  seg[RST_MAX_INTERVALS + 1];   // first segment
        };

        __device__ __forceinline__ bool restart_shape_ok(const aeonb_entropy_desc& d, const restart_layout& w, int& bpm)
        {
            bpm = 0;
            for (int c = 0; c < 3; ++c)
                if (c < d.ncomp)
                    bpm += d.hs[c] * d.vs[c];
            return d.ncomp >= 1 && d.ncomp <= 3 && d.mcux > 0 && d.mcuy > 0 && d.scan && d.tables && bpm <= 16 && d.scan_size < (1u << 26) &&
                   (uint64_t)d.mcux * d.mcuy * bpm < (1ull << 30) && d.scratch_bytes >= w.bytes && (reinterpret_cast<uintptr_t>(d.scratch) & 15) == 0;
        }

        // Finds the intervals of a stream: the blocks of a cluster per stream, every warp a run of 16-byte vectors, which
        // it goes through twice, counting markers and then numbering them from the counts of the warps in front.  What bounds
        // it is the latency of those passes: 16 streams of 0.6 MB took 82 us with one block each, about 20 with four.
        __global__ void __launch_bounds__(RST_INDEX_THREADS) jpeg_restart_index_kernel(const __grid_constant__ launch_data data)
        {
            namespace cg = cooperative_groups;
            constexpr uint32_t            warps = RST_INDEX_THREADS / 32;
            __shared__ aeonb_entropy_desc d;
            __shared__ uint32_t           counts[warps], other, total;
            cg::cluster_group             cluster = cg::this_cluster();
            const uint32_t                tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = cluster.num_blocks(), rank = cluster.block_rank();
            data.fetch(d, (int)(blockIdx.x / C), (int)tid, (int)RST_INDEX_THREADS);
            __syncthreads();
            if (!d.scratch || d.restart_interval == 0)
                return; // as all blocks of the cluster
            const restart_layout w = restart_work(d);
            int                  bpm;
            if (!restart_shape_ok(d, w, bpm))
            {
                if (tid == 0 && rank == 0 && d.scratch_bytes >= w.bytes)
                    w.header->doubtful = 1;
                return;
            }
            const uint32_t     N    = d.scan_size;
            const uint32_t     lead = (uint32_t)(reinterpret_cast<uintptr_t>(d.scan) & 15);
            const uint4* const vec  = reinterpret_cast<const uint4*>(d.scan - lead);
            const uint32_t     nv   = (lead + N + 15) >> 4;
            if (tid == 0)
                other = N > 0 && __ldg(d.scan + N - 1) == 0xFF ? N - 1 : N;
            __syncthreads();
            // bit b of the result = byte b of vector i is the second byte of a restart marker; of `foreign`, of another marker
            auto markers = [&](uint32_t i, uint32_t& foreign) -> uint32_t {
                const uint4    x    = i < nv ? __ldg(vec + i) : make_uint4(0, 0, 0, 0);
                const uint32_t up   = __shfl_up_sync(0xffffffffu, x.w, 1) >> 24;
                const uint32_t prev = lane > 0 ? up : i > 0 && i < nv ? (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(vec) + 16 * i - 1) : 0;
                const uint32_t v[4] = {x.x, x.y, x.z, x.w}, f8[4] = {x.x & 0xF8F8F8F8u, x.y & 0xF8F8F8F8u, x.z & 0xF8F8F8F8u, x.w & 0xF8F8F8F8u};
                const uint32_t own  = bits_from((int)lead - (int)(16 * i)) & bits_below((int)(lead + N) - (int)(16 * i));
                const uint32_t follows = ((byte_mask(v, 0xFFFFFFFFu) & own) << 1 | (prev == 0xFF && 16 * i > lead)) & own & ~byte_mask(v, 0);
                const uint32_t restart = byte_mask(f8, 0xD0D0D0D0u);
                foreign                = follows & ~restart;
                return follows & restart;
            };
            // a warp owns a run of vectors, so that markers are numbered by warp, then by pass, then by lane
            const uint32_t per = (nv + warps * C - 1) / (warps * C);
            const uint32_t v0 = (rank * warps + warp) * per, v1 = min(nv, v0 + per);
            uint32_t       count = 0;
            for (uint32_t base = v0; base < v1; base += 32)
            {
                const uint32_t i = base + lane;
                uint32_t       foreign;
                const uint32_t mask = markers(i, foreign);
                if (i < v1)
                {
                    count += __popc(mask);
                    if (foreign)
                        atomicMin(&other, 16 * i + (uint32_t)__ffs(foreign) - 1 - lead - 1); // the 0xFF before it
                }
            }
            count = __reduce_add_sync(0xffffffffu, count);
            if (lane == 0)
                counts[warp] = count;
            __syncthreads();
            const uint32_t here   = counts[lane], mine = __reduce_add_sync(0xffffffffu, here);
            uint32_t       before = __reduce_add_sync(0xffffffffu, lane < warp ? here : 0);
            if (tid == 0)
                total = mine;
            cluster.sync();
            uint32_t all = 0, end = other;
            for (uint32_t r = 0; r < C; ++r)
            {
                const uint32_t theirs = *cluster.map_shared_rank(&total, r);
                before += r < rank ? theirs : 0;
                all += theirs;
                end = min(end, *cluster.map_shared_rank(&other, r));
            }
            cluster.sync(); // nothing touches another block's memory afterwards
            if (tid == 0 && rank == 0)
            {
                w.header->doubtful = 0;
                w.header->end      = end;
                w.header->found    = all;
                w.start[0]         = 0;
            }
            if (count == 0)
                return;
            for (uint32_t base = v0; base < v1; base += 32)
            {
                uint32_t       foreign;
                const uint32_t i    = base + lane;
                uint32_t       mask = markers(i, foreign);
                mask                = i < v1 ? mask : 0;
                if (!__any_sync(0xffffffffu, mask != 0))
                    continue;
                uint32_t incl = __popc(mask);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o)
                        incl += up;
                }
                uint32_t at = before + incl - __popc(mask); // markers in front of this lane's
                before += __shfl_sync(0xffffffffu, incl, 31);
                for (; mask; mask &= mask - 1)
                    if (++at <= w.intervals)
                        w.start[at] = 16 * i + (uint32_t)__ffs(mask) - lead;
            }
        }

        // Copies intervals R.raw[0..I) without stuffed bytes and markers and notes in R.clean where each starts; returns the bytes of
        // the copy.  RESIDENT as in copy_scan, vector i0 being the first in `room`.
        template <bool RESIDENT>
        __device__ __forceinline__ uint32_t copy_intervals(rst_state& R, uint32_t I, uint32_t* room, uint32_t* out, const uint4* vec, uint32_t lead)
        {
            constexpr uint32_t     T   = RST_THREADS;
            const uint32_t         tid = threadIdx.x;
            const uint32_t         r0 = R.raw[0], r1 = R.raw[I] - 2;
            const uint32_t         i0 = (lead + r0) >> 4, i1 = (lead + r1 + 15) >> 4;
            const uint8_t* const   base = reinterpret_cast<const uint8_t*>(vec);
            clean_writer<RESIDENT> copy{room, out, 0, 0};
            for (uint32_t tile = i0, odd = 0; tile < i1; tile += T, odd ^= 1)
            {
                const uint32_t i = tile + tid;
                uint32_t       words[4] = {0, 0, 0, 0}, keep = 0, starts = 0;
                if (i < i1)
                {
                    const uint4 x = RESIDENT ? reinterpret_cast<const uint4*>(room)[i - i0] : __ldg(vec + i);
                    words[0] = x.x, words[1] = x.y, words[2] = x.z, words[3] = x.w;
                    uint32_t prev = 0;
                    if (i > i0)
                        prev = !RESIDENT  ? (uint32_t)__ldg(base + 16 * i - 1)
                               : tid == 0 ? R.S.tile_end[odd ^ 1] // its place may have been taken
                                          : (uint32_t) reinterpret_cast<const uint8_t*>(room)[16 * (i - i0) - 1];
                    const int      o = (int)(16 * i) - (int)lead; // where the vector starts in the scan
                    const uint32_t own = bits_from((int)r0 - o) & bits_below((int)r1 - o), ff = byte_mask(words, 0xFFFFFFFFu), zero = byte_mask(words, 0);
                    // bytes that follow 0xFF (a stuffed zero, or a marker's second byte; the byte in front of the part is a marker's)
                    const uint32_t follows = own & ((ff & bits_from((int)r0 - o)) << 1 | (prev == 0xFF && o > (int)r0));
                    // first bytes of markers: 0xFF in front of anything but zero, inside the part
                    uint32_t       last = 0;
                    if ((ff & own) >> 15 && o + 16 < (int)r1)
                        last = (uint32_t)(__ldg(base + 16 * i + 16) != 0) << 15;
                    const uint32_t head = ff & own & ((~zero & bits_below((int)r1 - o)) >> 1 | last);
                    keep                = own & ~follows & ~head;
                    starts              = follows & ~zero;
                }
                if (RESIDENT && tid == T - 1)
                    R.S.tile_end[odd] = words[3] >> 24;
                uint32_t       total;
                const uint32_t at = cta_exclusive_scan((uint32_t)__popc(keep), R.S.warp_sums[0], total);
                for (uint32_t m = starts; m; m &= m - 1)
                {
                    const uint32_t b = (uint32_t)__ffs(m) - 1, pos = 16 * i + b - lead + 1; // offset of the interval behind the marker
                    uint32_t       lo = 0, hi = I; // the last interval that starts at or before it
                    while (hi - lo > 1)
                    {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (R.raw[mid] <= pos)
                            lo = mid;
                        else
                            hi = mid;
                    }
                    R.clean[lo] = copy.size + at + (uint32_t)__popc(keep & ((1u << b) - 1));
                }
                copy.append(words, keep, at, total);
            }
            copy.finish();
            if (tid == 0)
                R.clean[0] = 0, R.clean[I] = copy.size;
            return copy.size;
        }

        // Clears the coefficients of the MCUs [m0, m1) inside the region: row by row, runs of blocks that follow one another.
        __device__ __forceinline__ void clear_mcus(const aeonb_entropy_desc& d, uint32_t m0, uint32_t m1, uint32_t tid, uint32_t nth)
        {
            const int mcux = d.mcux;
            for (int my = max((int)(m0 / (uint32_t)mcux), d.roi[1]); my < d.mcuy; ++my)
            {
                const int64_t row = (int64_t)my * mcux;
                if (row >= (int64_t)m1)
                    break;
                const int x0 = (int)max((int64_t)d.roi[0], (int64_t)m0 - row), x1 = (int)min((int64_t)min(d.roi[2], mcux), (int64_t)m1 - row);
                for (int c = 0; c < d.ncomp && x0 < x1; ++c)
                    for (int y = 0; y < d.vs[c]; ++y)
                    {
                        const int64_t block = ((int64_t)(my - d.roi[1]) * d.vs[c] + y) * ((d.roi[2] - d.roi[0]) * d.hs[c]) + (x0 - d.roi[0]) * d.hs[c];
                        uint4* const  p     = reinterpret_cast<uint4*>(d.coef[c] + block * 64);
                        for (uint32_t i = tid; i < (uint32_t)((x1 - x0) * d.hs[c] * 8); i += nth)
                            p[i] = make_uint4(0, 0, 0, 0);
                    }
            }
        }

        // Segments of a part's intervals, their true entry states, and the storing pass.
        template <bool SLOW, typename Words>
        __device__ __forceinline__ void decode_intervals(rst_state& R, const seg_arrays& A, const uint32_t* words, uint32_t first, uint32_t I,
                                                         uint32_t clean_size, int min_segment, int bpm, uint32_t needed_mcus, int16_t* dcdiff)
        {
            constexpr uint32_t T   = RST_THREADS;
            par_state&         S   = R.S;
            const uint32_t     tid = threadIdx.x, ri = (uint32_t)S.d.restart_interval;
            auto first_block = [&](uint32_t i) { return (uint32_t)min((uint64_t)needed_mcus, (uint64_t)(first + i) * ri) * (uint32_t)bpm; };
            // interval i goes on below the region
            auto cut = [&](uint32_t i) { return needed_mcus < min((uint64_t)S.d.mcux * S.d.mcuy, (uint64_t)(first + i + 1) * ri); };
            // an interval has ceil(its bytes / seg) segments; I < T of them are shorter than seg, so this many fit
            uint32_t seg = (clean_size + (T - I) - 1) / (T - I);
            seg          = max((seg + 3u) & ~3u, (uint32_t)max(min_segment, 64) & ~3u);
            uint32_t       nseg; // <= T
            const uint32_t mine_of = tid < I ? (R.clean[tid + 1] - R.clean[tid] + seg - 1) / seg : 0;
            const uint32_t seg0    = cta_exclusive_scan(mine_of, S.warp_sums[0], nseg);
            if (tid < I)
                R.seg[tid] = seg0;
            if (tid == 0)
                R.seg[I] = nseg;
            __syncthreads();
            const bool mine = tid < nseg;
            uint32_t   iv   = 0; // this thread's interval: the last one whose first segment is not behind it
            for (uint32_t hi = I; hi - iv > 1;)
            {
                const uint32_t mid = (iv + hi) >> 1;
                if (R.seg[mid] <= tid)
                    iv = mid;
                else
                    hi = mid;
            }
            const uint32_t pbeg = (R.clean[iv] + (tid - R.seg[iv]) * seg) * 8, pend = min(R.clean[iv + 1] * 8, pbeg + seg * 8);
            const uint32_t step = seg * 8 / (NCHECK + 1);
            // ---- clear the coefficients of these intervals' MCUs: warps without a segment, if there are four of them, while the others
            // decode; the barriers between here and the storing pass order the two
            const uint32_t busy = (nseg + 31) & ~31u, from = T >= busy + 128 ? busy : 0;
            if (tid >= from)
                clear_mcus(S.d, (uint32_t)min((uint64_t)needed_mcus, (uint64_t)first * ri),
                           (uint32_t)min((uint64_t)needed_mcus, (uint64_t)(first + I) * ri), tid - from, T - from);
            const uint32_t run_blocks = settle_segments<SLOW, Words>(S, A, words, nseg, R.seg[iv] == tid, pbeg, pend, step);

            // ---- first block number of every segment, counted from its interval's first block
            uint32_t counted;
            A.cnt[tid] = cta_exclusive_scan(run_blocks, S.warp_sums[0], counted);
            if (mine)
                A.ext_bk[tid] = (uint16_t)iv; // the exit states have served
            __syncthreads();
            if (mine)
                A.ext_p[tid] = first_block(iv) + A.cnt[tid] - A.cnt[R.seg[iv]];
            if (tid < I)
            {
                const uint32_t a = R.seg[tid], b = R.seg[tid + 1];
                const uint32_t has = a == b ? 0 : (b < nseg ? A.cnt[b] : counted) - A.cnt[a];
                if (has < first_block(tid + 1) - first_block(tid))
                    S.bad = 1;
            }
            __syncthreads();

            // ---- decode once more, storing; the pieces between checkpoints are dealt out to the threads
            for (uint32_t q = tid; q < nseg * (NCHECK + 1); q += T)
            {
                const uint32_t t = q / (NCHECK + 1), piece = q % (NCHECK + 1), i = A.ext_bk[t];
                const uint32_t all_end = R.clean[i + 1] * 8;
                const uint32_t seg_beg = (R.clean[i] + (t - R.seg[i]) * seg) * 8, seg_end = min(all_end, seg_beg + seg * 8);
                const uint32_t at = seg_beg + piece * step; // the checkpoint this piece starts from
                if (at >= seg_end)
                    continue;
                uint32_t p0, bk, before;
                piece_entry(A, t, piece, at, p0, bk, before);
                const uint32_t     g = A.ext_p[t] + before, gend = first_block(i + 1);
                const store_result r = store_segment<SLOW, Words>(S, words, p0, bk >> 8, bk & 255, min(seg_end, at + step), g, gend, dcdiff);
                // the interval's last block leaves less than a byte, unless the region ends in front of that block
                if (r.bad || (r.blocks > 0 && g + r.blocks == gend && (r.p > all_end || (all_end - r.p > 7 && !cut(i)))))
                    S.bad = 1;
            }
            __syncthreads();
        }

        // Part blockIdx.x = {record, first interval, intervals, number of the part within its stream}.  Shared memory: rst_state,
        // SEG_BYTES per thread, and what is left of `smem_bytes` for the part's bytes, where they fit.
        __global__ void __launch_bounds__(RST_THREADS, 2) jpeg_entropy_restart_kernel(const __grid_constant__ launch_data data,
                                                                                   const int4* __restrict__ parts, int min_segment,
                                                                                   uint32_t smem_bytes)
        {
            constexpr uint32_t T = RST_THREADS;
            extern __shared__ __align__(16) unsigned char smem_raw[];
            rst_state&       R       = *reinterpret_cast<rst_state*>(smem_raw);
            par_state&       S       = R.S;
            const seg_arrays A       = seg_arrays_at(smem_raw + sizeof(rst_state), T);
            const uint32_t   room_at = ((uint32_t)sizeof(rst_state) + SEG_BYTES * T + 15) & ~15u;
            uint32_t* const  room    = reinterpret_cast<uint32_t*>(smem_raw + room_at);
            const uint32_t   tid     = threadIdx.x;
            const int4       part    = __ldg(parts + blockIdx.x);
            data.fetch(S.d, (int)(part.x), (int)tid, (int)T);
            if (tid < 64)
                S.zz[16 + tid] = k_zz_colmajor[tid];
            if (tid == 0)
                S.bad = S.slow = 0;
            __syncthreads();
            const aeonb_entropy_desc& d = S.d;
            const restart_layout      w = restart_work(d);
            int                       bpm;
            if (!restart_shape_ok(d, w, bpm))
                return; // the index kernel has said so
            const uint32_t first = (uint32_t)part.y, I = (uint32_t)part.z;
            const uint32_t found = w.header->found, end = w.header->end;
            // a part whose intervals are not all there, in order, in front of the stream's end is not looked at
            bool odd = first + I > found + 1;
            for (uint32_t i = tid; i <= I && !odd; i += T)
            {
                const uint32_t k = first + i;
                // behind the stream's last interval, and behind the last one of all: the end of the entropy-coded data
                const uint32_t at = k <= found && k <= w.intervals && !(i == I && w.start[k] > end) ? w.start[k] : end + 2;
                R.raw[i]          = at;
                odd               = at > end + (i == I ? 2 : 0);
            }
            if (__syncthreads_or(odd))
            {
                if (tid == 0)
                    w.header->doubtful = 1;
                return;
            }
            const uint32_t     lead = (uint32_t)(reinterpret_cast<uintptr_t>(d.scan) & 15);
            const uint4* const vec  = reinterpret_cast<const uint4*>(d.scan - lead);
            const uint32_t     r0 = R.raw[0], i0 = (lead + r0) >> 4, i1 = (lead + R.raw[I] - 2 + 15) >> 4;
            const bool         resident = 16 * (i1 - i0) + 48 <= smem_bytes - room_at;
            if (resident)
                fetch_raw(room, vec, i0, i1); // arrives while the tables are being built
            set_up_stream(S, (int)tid, (int)T);

            const uint32_t needed_mcus = (uint32_t)min(d.roi[3], d.mcuy) * d.mcux;
            const uint32_t ri          = (uint32_t)d.restart_interval;
            const uint32_t lane = tid & 31, warp = tid >> 5;
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            int16_t* const dcdiff = w.dcdiff;
            if (resident)
            {
                const uint32_t clean_size = copy_intervals<true>(R, I, room, nullptr, vec, lead);
                __syncthreads();
                if (S.slow)
                    decode_intervals<true, shared_words>(R, A, room, first, I, clean_size, min_segment, bpm, needed_mcus, dcdiff);
                else
                    decode_intervals<false, shared_words>(R, A, room, first, I, clean_size, min_segment, bpm, needed_mcus, dcdiff);
            }
            else
            {
                // the parts' copies follow one another with 64 bytes between them; the checkpoints' room is not in use yet
                uint32_t* const clean      = reinterpret_cast<uint32_t*>(w.clean + (r0 & ~15u) + 64u * (uint32_t)part.w);
                const uint32_t  clean_size = copy_intervals<false>(R, I, A.chk, clean, vec, lead);
                __syncthreads();
                decode_intervals<true, global_words>(R, A, clean, first, I, clean_size, min_segment, bpm, needed_mcus, dcdiff);
            }
            if (S.bad)
            {
                if (tid == 0)
                    w.header->doubtful = 1;
                return;
            }

            // ---- DC: a warp per interval sums the differences in scan order, lane l the l-th run of MCUs
            for (uint32_t i = warp; i < I; i += T / 32)
            {
                const uint32_t b0 = (uint32_t)min((uint64_t)needed_mcus, (uint64_t)(first + i) * ri);
                const uint32_t b1 = (uint32_t)min((uint64_t)needed_mcus, (uint64_t)(first + i + 1) * ri), chunk = (b1 - b0 + 31) / 32;
                const uint32_t m0 = min(b1, b0 + lane * chunk), m1 = min(b1, m0 + chunk);
                int            sum[3] = {0, 0, 0};
                for (uint32_t m = m0; m < m1; ++m)
                    for (int b = 0; b < bpm; ++b)
                    {
                        const int v = dcdiff[(size_t)m * bpm + b];
                        const int c = S.comp[b];
                        sum[0] += c == 0 ? v : 0;
                        sum[1] += c == 1 ? v : 0;
                        sum[2] += c == 2 ? v : 0;
                    }
                int pred[3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                {
                    int incl = sum[c];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const int up = __shfl_up_sync(0xffffffffu, incl, o);
                        if ((int)lane >= o)
                            incl += up;
                    }
                    pred[c] = incl - sum[c];
                }
                store_dc(S, dcdiff, m0, m1, bpm, pred);
            }
        }
    }

    int jpeg_entropy_min_segment()
    {
        static const int value = [] {
            int v = 160;
            if (const char* e = std::getenv("AEONB_ENTROPY_SEGMENT"))
                v = std::atoi(e);
            return v < 64 ? 64 : v > (1 << 20) ? (1 << 20) : v;
        }();
        return value;
    }

    int jpeg_entropy_threads(int n)
    {
        static const int value = [] {
            int v = 0;
            if (const char* e = std::getenv("AEONB_ENTROPY_THREADS"))
                v = std::max(128, std::min(std::atoi(e), PAR_THREADS)) & ~31;
            return v;
        }();
        return value ? value : n <= 148 ? PAR_THREADS : 512;
    }

    int jpeg_entropy_block(int n, uint32_t longest)
    {
        // A stream that has an SM to itself gets a thread for each piece of the storing pass; of more streams than SMs two share one,
        // and a thread per segment has to do.
        const int segments = (int)((longest + (uint32_t)jpeg_entropy_min_segment() - 1) / (uint32_t)jpeg_entropy_min_segment());
        const int wanted   = n <= 148 ? segments * (NCHECK + 1) : segments;
        int       threads  = jpeg_entropy_threads(n);
        while (threads > 256 && wanted <= threads / 2)
            threads /= 2;
        return threads & ~31;
    }

    int64_t jpeg_entropy_scratch_bytes(const aeonb_entropy_desc& d)
    {
        if (d.restart_interval > 0)
            return (int64_t)restart_work(d).bytes;
        int64_t bpm = 0;
        for (int c = 0; c < d.ncomp && c < 3; ++c)
            bpm += (int64_t)d.hs[c] * d.vs[c];
        const int64_t blocks = (int64_t)d.mcux * d.mcuy * bpm;
        return (((int64_t)d.scan_size + 32 + 15) & ~15ll) + ((blocks * 2 + 15) & ~15ll);
    }

    void jpeg_restart_parts(const aeonb_entropy_desc* descs, int n, std::vector<int4>& parts)
    {
        // A stream of no bytes gets its parts too: the serial kernel reads the header that the index kernel writes.
        uint64_t total = 0;
        for (int i = 0; i < n; ++i)
            if (descs[i].scratch && descs[i].restart_interval > 0)
                total += descs[i].scan_size;
        // Two blocks of a part fit an SM, and all parts should run at once; parts of less than 4 KB are mostly set-up, parts of more than
        // 46 KB do not fit a block's shared memory.
        const uint64_t target = std::min<uint64_t>(std::max<uint64_t>(total / (148 * 2), 4096), 36 * 1024);
        for (int i = 0; i < n; ++i)
        {
            const aeonb_entropy_desc& d = descs[i];
            if (!d.scratch || d.restart_interval <= 0)
                continue;
            const uint32_t all    = restart_work(d).intervals;
            const uint64_t mcus   = (uint64_t)std::min(d.roi[3], d.mcuy) * d.mcux;
            const uint32_t needed = (uint32_t)((mcus + d.restart_interval - 1) / d.restart_interval);
            const uint64_t split  = std::max<uint64_t>(1, (d.scan_size + target / 2) / target);
            uint64_t       per    = std::max<uint64_t>(1, (all + split - 1) / split);
            per = std::max<uint64_t>(per, (needed + restart_most_parts(all) - 1) / restart_most_parts(all));
            per = std::min<uint64_t>(per, RST_MAX_INTERVALS);
            for (uint32_t first = 0, k = 0; first < needed; first += (uint32_t)per, ++k)
                parts.push_back(make_int4(i, (int)first, (int)std::min<uint64_t>(per, needed - first), (int)k));
        }
    }

    // Shared memory of a block of the block-parallel kernel: room for the launch's longest stream and its DC differences.  More
    // streams than SMs: as much as lets as many blocks share an SM as there are streams for it (four at most), the longest
    // streams falling back on global memory -- unless fewer and longer segments (`rows` of them at most), which take less room, let
    // them stay: 256 streams of up to 61 KB 488 us with the longest in global memory, 407 with 260 segments instead of 382.
    static size_t jpeg_entropy_smem(int n, int threads, int& rows, uint32_t longest, uint64_t most_blocks)
    {
        const int     share = std::min({(n + 147) / 148, 4, std::max(1, 1280 / threads)}); // the kernel's registers allow 1280 threads
        const int64_t most  = std::min((228 * 1024) / share - 1024, 227 * 1024), fixed = sizeof(par_state) + 16, scan = (int64_t)longest + 16 + 64;
        const int64_t fit   = (most - fixed - scan) / (int64_t)SEG_BYTES;
        if (fit >= 128)
            rows = (int)std::min<int64_t>(rows, fit);
        const int64_t want = fixed + (int64_t)SEG_BYTES * rows + scan + (int64_t)most_blocks * 2;
        // (a copy in global memory leaves through a tile of 16 bytes per thread, laid over the checkpoints and what follows)
        const int64_t least = fixed + std::max((int64_t)SEG_BYTES * rows, (int64_t)12 * rows + 16 * threads + 16);
        return (size_t)std::max(least, std::min(want, most));
    }

    // Blocks of the cluster of each of n streams: as many as all clusters find room for at once, one block to an SM: 15 clusters of eight, 33
    // of four, 66 of two (what cudaOccupancyMaxActiveClusters says for a B200 and blocks that have an SM to themselves).
    static int jpeg_entropy_cluster(int n) { return n <= 15 ? 8 : n <= 33 ? 4 : n <= 66 ? 2 : 1; }

    // How a launch of few streams is spread: blocks in the cluster of each stream (0: not spread), and runs a block has room for.
    struct spread_plan
    {
        int      blocks = 0, threads = 0;
        uint32_t cap    = 0;
        size_t   smem   = 0;
    };
    static spread_plan jpeg_entropy_spread(int n, uint32_t longest, int most_places)
    {
        spread_plan p;
        if (jpeg_entropy_cluster(n) == 1 || most_places < 1 || most_places > SPREAD_PLACES)
            return p;
        // A block has less than a warp for each of its schedulers to decode with if it has fewer than 128 runs.
        const uint32_t segments = longest / SPREAD_SEG + 1;
        int            blocks   = jpeg_entropy_cluster(n);
        while (blocks > 1 && segments * (uint32_t)most_places <= (uint32_t)blocks / 2 * 128)
            blocks /= 2;
        p.threads = 512;
        p.cap     = std::min<uint32_t>(1200, ((segments + blocks - 1) / blocks + 3) * most_places);
        p.smem    = ((sizeof(spread_state) + spread_bytes(p.cap) + 15) & ~(size_t)15) + longest + 16 + 64;
        p.blocks  = p.smem <= 227 * 1024 ? blocks : 0;
        return p;
    }

    cudaError_t launch_jpeg_entropy(const launch_data& descs, int n, bool any_parallel, bool any_serial, int min_segment,
                                    uint32_t longest, uint64_t most_blocks, int most_places, const int4* parts_dev, int n_parts,
                                    cudaStream_t stream)
    {
        if (n <= 0)
            return cudaSuccess;
        const spread_plan spread = any_parallel ? jpeg_entropy_spread(n, longest, most_places) : spread_plan();
        if (spread.blocks > 0)
        {
            cudaError_t err = cudaFuncSetAttribute(jpeg_entropy_spread_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (err != cudaSuccess)
                return err;
            cudaLaunchConfig_t  cfg  = {};
            cudaLaunchAttribute attr = {};
            cfg.gridDim              = dim3(n * spread.blocks);
            cfg.blockDim             = dim3(spread.threads);
            cfg.dynamicSmemBytes     = spread.smem;
            cfg.stream               = stream;
            attr.id                  = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x    = spread.blocks;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs    = &attr;
            cfg.numAttrs = 1;
            err          = cudaLaunchKernelEx(&cfg, jpeg_entropy_spread_kernel, descs, spread.cap);
            if (err != cudaSuccess)
                return err;
        }
        else if (any_parallel)
        {
            const int    threads = jpeg_entropy_block(n, longest);
            int          rows = std::min(threads, (int)(longest / (uint32_t)min_segment) + 1);
            const size_t smem = jpeg_entropy_smem(n, threads, rows, longest, most_blocks);
            // always the most a block can have: the setting is the kernel's, and another thread may launch it with another size between
            // this call and the launch
            cudaError_t  err  = cudaFuncSetAttribute(jpeg_entropy_parallel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (err != cudaSuccess)
                return err;
            jpeg_entropy_parallel_kernel<<<n, threads, smem, stream>>>(descs, min_segment, (uint32_t)rows, (uint32_t)smem);
            err = cudaGetLastError();
            if (err != cudaSuccess)
                return err;
        }
        if (n_parts > 0)
        {
            const size_t smem = sizeof(rst_state) + 16 + (size_t)SEG_BYTES * RST_THREADS + RST_ROOM;
            cudaError_t  err  = cudaFuncSetAttribute(jpeg_entropy_restart_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (err != cudaSuccess)
                return err;
            // Both kernels, us, with one / two / four / eight blocks per stream: 256 streams of 1.6 KB 60 / 69 / 92 / 153, 64 of 42 KB
            // 145 / 143 / 147 / 167, 16 of 0.6 MB 336 / 297 / 273 / 277, one of 0.6 MB 163 / 124 / 102 / 92.
            const int           blocks = jpeg_entropy_cluster(n);
            cudaLaunchConfig_t  cfg    = {};
            cudaLaunchAttribute attr   = {};
            cfg.gridDim                = dim3(n * blocks);
            cfg.blockDim               = dim3(RST_INDEX_THREADS);
            cfg.stream                 = stream;
            attr.id                    = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x      = blocks;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs    = &attr;
            cfg.numAttrs = 1;
            err          = cudaLaunchKernelEx(&cfg, jpeg_restart_index_kernel, descs);
            if (err != cudaSuccess)
                return err;
            jpeg_entropy_restart_kernel<<<n_parts, RST_THREADS, smem, stream>>>(descs, parts_dev, min_segment, (uint32_t)smem);
            err = cudaGetLastError();
            if (err != cudaSuccess)
                return err;
        }
        if (any_serial)
        {
            const size_t smem = sizeof(warp_state);
            cudaError_t  err  = cudaFuncSetAttribute(jpeg_entropy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (err != cudaSuccess)
                return err;
            jpeg_entropy_kernel<<<n, 32, smem, stream>>>(descs);
            return cudaGetLastError();
        }
        return cudaSuccess;
    }
}
