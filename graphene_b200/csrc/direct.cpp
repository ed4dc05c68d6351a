// Host side of the direct sweep kernels (kernels_direct.cu): row records in
// execution order and the step table of every tile. See HostDirect in
// device.hpp for the layout.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "device.hpp"

namespace gr {

namespace {

// Entries of tile-order row p (tile-local index il) in the order the sweep
// subtracts them: lower ascending (ilu/Solver.cpp:391-403), upper descending
// without halo (:424-436), or all in tile-local order
// (gauss-seidel/Solver.cpp:76-79).
template <class F>
void eachEntry(const HostMatrix& H, RingKind kind, bool upper, i64 p, i64 il, i64 nRows, F&& f) {
  const i64 b = H.rowPtr[p], e = H.rowPtr[p + 1];
  if (kind == RingKind::GaussSeidel) {
    for (i64 k = b; k < e; ++k) f(k);
  } else if (upper) {
    for (i64 k = e - 1; k >= b && H.colLocal[k] >= il; --k)
      if (H.colLocal[k] < nRows) f(k);
  } else {
    for (i64 k = b; k < e && H.colLocal[k] <= il && H.colLocal[k] < nRows; ++k) f(k);
  }
}

// CRS entry (row p, tile-local column j), -1 when the pattern has none.
i32 entryAt(const HostMatrix& H, i64 p, i64 j) {
  for (i64 k = H.rowPtr[p]; k < H.rowPtr[p + 1]; ++k)
    if (H.colLocal[k] == j) return static_cast<i32>(k);
  return -1;
}

// Whether no tile has three rows that are pairwise coupled (a grid, a mesh of
// hexahedra): ILU(0) then changes an entry only by its own division, and the
// diagonal.
bool triangleFree(const HostMatrix& H) {
  std::atomic<bool> ok{true};
  parallelFor(H.P, [&](i64 T) {
    const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
    for (i64 r = 0; r < nRows && ok.load(std::memory_order_relaxed); ++r) {
      const i64 b = H.rowPtr[base + r], e = H.rowPtr[base + r + 1];
      for (i64 k = b; k < e && H.colLocal[k] < r; ++k)
        for (i64 j = k + 1; j < e && H.colLocal[j] < nRows; ++j)
          if (entryAt(H, base + H.colLocal[k], H.colLocal[j]) >= 0) {
            ok = false;
            return;
          }
    }
  });
  return ok;
}

i64 blockBytes(int valueBytes, uint32_t word) {
  const bool diag = (word & kDirectDiag) != 0;
  return valueBytes == 4 ? DirectBlock<4>(word, diag).bytes : DirectBlock<8>(word, diag).bytes;
}

// Whether every in-tile entry above the diagonal lies in a later level than
// its row, so that a sweep can overwrite the start values in place.
bool sweepsInPlace(const HostMatrix& H) {
  std::atomic<bool> ok{true};
  parallelFor(H.P, [&](i64 T) {
    const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
    for (i64 r = 0; r < nRows && ok.load(std::memory_order_relaxed); ++r)
      for (i64 k = H.rowPtr[base + r]; k < H.rowPtr[base + r + 1]; ++k) {
        const i64 lc = H.colLocal[k];
        if (lc > r && lc < nRows && H.lowerLevel[base + lc] <= H.lowerLevel[base + r]) {
          ok = false;
          break;
        }
      }
  });
  return ok;
}

i64 xSlotsOf(const HostMatrix& H, RingKind kind, bool inPlace, i64 T) {
  const i64 nRows = H.tileStart[T + 1] - H.tileStart[T];
  return kind == RingKind::GaussSeidel ? (inPlace ? 1 : 2) * nRows + H.tiles[T].nHalo + 1 : nRows + 1;
}

}  // namespace

bool directFits(const HostMatrix& H, RingKind kind) {
  for (i32 T = 0; T < H.P; ++T)
    if (xSlotsOf(H, kind, false, T) > kDirectMaxSlots) return false;
  std::atomic<bool> ok{true};
  parallelChunks(H.P, [&](i64 t0, i64 t1) {
    for (i64 T = t0; T < t1 && ok.load(std::memory_order_relaxed); ++T) {
      const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
      for (i64 r = 0; r < nRows; ++r) {
        int c[2] = {0, 0};
        for (int up = 0; up < (kind == RingKind::Ilu ? 2 : 1); ++up)
          eachEntry(H, kind, up != 0, base + r, r, nRows, [&](i64) { ++c[up]; });
        if (c[0] > 6 || c[1] > 6) ok = false;
      }
    }
  }, 16);
  return ok;
}

HostDirect buildDirect(const HostMatrix& H, RingKind kind, bool dilu, i32 warps, DType vt) {
  const int threads = 32 * warps;
  if (warps < 1 || warps == 3 || warps > 4) fail(GR_EINVAL, "direct sweeps run 1, 2 or 4 warps a tile");
  if (!directFits(H, kind)) fail(GR_EUNSUPPORTED, "rows or tiles too large for the direct sweep");
  const bool gs = kind != RingKind::Ilu;
  HostDirect D;
  D.kind = kind;
  D.dilu = dilu;
  D.warps = warps;
  D.valueBytes = static_cast<int>(dtypeSize(vt));
  D.gsInPlace = gs && (kind == RingKind::GaussSeidelLower || sweepsInPlace(H));
  std::vector<std::vector<uint32_t>> tileSteps(H.P);
  std::vector<std::vector<i32>> order(H.P);  // record -> tile-local row, -1: padding
  std::vector<i64> nForward(H.P, 0);         // records of the forward sweep
  std::vector<i64> tileUnits(H.P, 0);        // 16-byte units of a tile's blocks
  std::atomic<bool> second{false}, longForward{false};
  parallelFor(H.P, [&](i64 T) {
    const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
    std::vector<uint32_t>& st = tileSteps[T];
    std::vector<i32>& ord = order[T];
    bool tileSecond = false, tileLongForward = false;
    st.assign(kDirectHead, 0u);
    for (int sweep = 0; sweep < (gs ? 1 : 2); ++sweep) {
      const bool upper = sweep == 1;
      const std::vector<i32>& lev = upper ? H.upperLevel : H.lowerLevel;
      const i32 nL = upper ? H.nUpperLevels[T] : H.nLowerLevels[T];
      std::vector<i64> count(nL, 0), longs(nL, 0), next(nL, -1);
      std::vector<char> isLong(nRows, 0);
      for (i64 r = 0; r < nRows; ++r) {
        const i32 l = lev[base + r];
        ++count[l];
        int c = 0;
        eachEntry(H, kind, upper, base + r, r, nRows, [&](i64) { ++c; });
        if (c > 3) {
          tileSecond = true;
          if (!upper) tileLongForward = true;
          isLong[r] = 1;
          ++longs[l];
        }
      }
      // Forward rows without entries keep their right-hand side: level 0 is
      // left out.
      i64 size = static_cast<i64>(ord.size());
      for (i32 l = !gs && !upper && !dilu ? 1 : 0; l < nL; ++l) {
        next[l] = size;
        size += (count[l] + kDirectAlign - 1) / kDirectAlign * kDirectAlign;
        for (i64 s = 0; s < count[l]; s += threads) {
          const i64 k = std::min<i64>(threads, count[l] - s);
          st.push_back(static_cast<uint32_t>(k) | (s + k == count[l] ? kDirectEnd : 0u) |
                       (gs || upper || dilu ? kDirectDiag : 0u) |
                       static_cast<uint32_t>(std::clamp<i64>(longs[l] - s, 0, k)) << kDirectLongShift);
        }
      }
      while ((st.size() - kDirectHead) % kDirectUnroll != 0) st.push_back(0u);
      st[upper || gs ? 2 : 1] = static_cast<uint32_t>(st.size() - kDirectHead);
      ord.resize(size, -1);
      for (const char want : {char(1), char(0)})  // long rows first
        for (i64 r = 0; r < nRows; ++r)
          if (i64& q = next[lev[base + r]]; q >= 0 && isLong[r] == want) ord[q++] = static_cast<i32>(r);
      if (!upper) nForward[T] = size;
    }
    for (size_t i = kDirectHead; i < st.size(); ++i) tileUnits[T] += blockBytes(D.valueBytes, st[i]) / 16;
    st.resize(st.size() + kDirectAhead, 0u);
    if (tileSecond) second = true;
    if (tileLongForward) longForward = true;
  });
  D.second = second;
  D.longForward = longForward;
  D.stepStart.assign(H.P + 1, 0);
  std::vector<i64> recStart(H.P + 1, 0);
  for (i32 T = 0; T < H.P; ++T) {
    recStart[T + 1] = recStart[T] + static_cast<i64>(order[T].size());
    D.stepStart[T + 1] = D.stepStart[T] + static_cast<i32>(tileSteps[T].size());
    D.maxSteps = std::max<i32>(D.maxSteps, static_cast<i32>(tileSteps[T].size()));
    D.maxRows = std::max<i64>(D.maxRows, H.tileStart[T + 1] - H.tileStart[T]);
    D.maxXSlots = std::max(D.maxXSlots, xSlotsOf(H, kind, D.gsInPlace, T));
  }
  std::vector<i64> unitStart(H.P + 1, 0);
  for (i32 T = 0; T < H.P; ++T) unitStart[T + 1] = unitStart[T] + tileUnits[T];
  D.records = recStart[H.P];
  D.units = unitStart[H.P];
  if (D.records >= (i64(1) << 31) || D.units >= (i64(1) << 32))
    fail(GR_EUNSUPPORTED, "direct sweep exceeds 2^31 records");
  D.steps.resize(D.stepStart[H.P]);
  D.stepRecord.resize(D.stepStart[H.P]);
  D.stepUnit.resize(D.stepStart[H.P]);
  const int4 none = make_int4(-1, -1, -1, 0);
  D.src.resize(D.records);
  D.tail.resize(D.records);
  if (D.second) {
    D.src2.resize(D.records);
    D.tail2.resize(D.records);
  }
  parallelFor(H.P, [&](i64 T) {
    const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
    const i64 start = gs && !D.gsInPlace ? nRows : 0;  // where sweep-start values live
    const uint32_t zero = static_cast<uint32_t>(4 * (xSlotsOf(H, kind, D.gsInPlace, T) - 1));
    i64 at = D.stepStart[T], firstRecord = recStart[T], firstUnit = unitStart[T];
    for (size_t i = 0; i < tileSteps[T].size(); ++i, ++at) {
      const uint32_t w = tileSteps[T][i];
      const bool step = i >= static_cast<size_t>(kDirectHead);
      const i64 units = step ? blockBytes(D.valueBytes, w) / 16 : 0;
      D.steps[at] = step ? w | static_cast<uint32_t>(units) << kDirectUnitShift : w;
      D.stepRecord[at] = static_cast<uint32_t>(firstRecord);
      D.stepUnit[at] = static_cast<uint32_t>(firstUnit);
      if (step) firstRecord += (static_cast<i64>(w & 0xFFu) + kDirectAlign - 1) / kDirectAlign * kDirectAlign;
      firstUnit += units;
    }
    for (i64 q = 0; q < static_cast<i64>(order[T].size()); ++q) {
      const i64 r = order[T][q], rec = recStart[T] + q;
      if (r < 0) {
        D.src[rec] = none;
        D.tail[rec] = 0;
        if (D.second) {
          D.src2[rec] = none;
          D.tail2[rec] = 0;
        }
        continue;
      }
      i32 e[6] = {-1, -1, -1, -1, -1, -1};
      uint32_t c[6] = {zero, zero, zero, zero, zero, zero};
      int m = 0;
      eachEntry(H, kind, q >= nForward[T], base + r, r, nRows, [&](i64 k) {
        const i64 lc = H.colLocal[k];
        e[m] = static_cast<i32>(k);
        c[m++] = static_cast<uint32_t>(4 * (gs && lc >= r ? start + lc : lc));
      });
      D.src[rec] = make_int4(e[0], e[1], e[2], static_cast<int>(c[0] | c[1] << 16));
      D.tail[rec] = c[2] | static_cast<uint32_t>(4 * r) << 16;
      if (D.second) {
        D.src2[rec] = make_int4(e[3], e[4], e[5], static_cast<int>(c[3] | c[4] << 16));
        D.tail2[rec] = c[5];
      }
    }
  });
  // The factorisation (DILU never changes an entry).
  D.factors = !gs && (dilu || triangleFree(H));
  if (D.factors) {
    D.levelStart.assign(H.P + 1, 0);
    std::vector<i64> forward(H.P + 1, 0);  // forward records before each tile
    for (i32 T = 0; T < H.P; ++T) {
      forward[T + 1] = forward[T] + nForward[T];
      D.levelStart[T + 1] = D.levelStart[T] + H.nLowerLevels[T] - (dilu || H.nLowerLevels[T] == 0 ? 0 : 1);
    }
    D.levels.resize(D.levelStart[H.P]);
    D.transposed.resize(forward[H.P]);
    if (D.longForward) D.transposed2.resize(forward[H.P]);
    parallelFor(H.P, [&](i64 T) {
      const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
      i64 l = D.levelStart[T];
      int4 level = make_int4(-1, 0, 0, 0);
      for (uint32_t i = 0; i < D.steps[D.stepStart[T] + 1]; ++i) {
        const i64 at = D.stepStart[T] + kDirectHead + i;
        const uint32_t w = D.steps[at];
        if ((w & 0xFFu) == 0) continue;
        if (level.x < 0)
          level = make_int4(static_cast<int>(D.stepRecord[at]), 0, static_cast<int>(at),
                            static_cast<int>(forward[T] + D.stepRecord[at] - recStart[T]));
        level.y += static_cast<int>((w & 0xFFu) | ((w >> kDirectLongShift) & 0xFFu) << 16);
        if (w & kDirectEnd) {
          D.levels[l++] = level;
          level.x = -1;
        }
      }
      for (i64 q = 0; q < nForward[T]; ++q) {
        const i64 r = order[T][q];
        if (r < 0) {
          D.transposed[forward[T] + q] = none;
          if (D.longForward) D.transposed2[forward[T] + q] = none;
          continue;
        }
        i32 t[6] = {-1, -1, -1, -1, -1, -1};
        int m = 0;
        eachEntry(H, kind, false, base + r, r, nRows, [&](i64 k) { t[m++] = entryAt(H, base + H.colLocal[k], r); });
        D.transposed[forward[T] + q] = make_int4(t[0], t[1], t[2], 0);
        if (D.longForward) D.transposed2[forward[T] + q] = make_int4(t[3], t[4], t[5], 0);
      }
    });
  }
  if (gs) D.haloStart.assign(H.P + 1, 0);  // sweeps from x = 0 read no halo
  if (kind == RingKind::GaussSeidel) {
    for (i32 T = 0; T < H.P; ++T) D.haloStart[T + 1] = D.haloStart[T] + static_cast<i32>(H.tiles[T].nHalo);
    D.haloSrc.assign(D.haloStart[H.P], -1);
    parallelFor(H.P, [&](i64 T) {
      const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
      for (i64 k = H.rowPtr[base]; k < H.rowPtr[base + nRows]; ++k)
        if (H.colLocal[k] >= nRows) D.haloSrc[D.haloStart[T] + H.colLocal[k] - nRows] = H.colPerm[k];
    });
    for (i32 v : D.haloSrc)
      if (v < 0) fail(GR_EINVAL, "direct sweep: a halo cell no entry reads");
  }
  return D;
}

void checkDirect(const HostMatrix& H, const HostDirect& D) {
  const bool gs = D.kind != RingKind::Ilu;
  const i64 threads = 32 * D.warps;
  auto bad = [](i64 T, const std::string& what) {
    fail(GR_EINVAL, "direct sweep check: tile " + std::to_string(T) + ": " + what);
  };
  if (static_cast<i64>(D.src.size()) != D.records || static_cast<i64>(D.tail.size()) != D.records ||
      static_cast<i32>(D.stepStart.size()) != H.P + 1 || static_cast<i64>(D.steps.size()) != D.stepStart[H.P] ||
      D.stepRecord.size() != D.steps.size() || D.stepUnit.size() != D.steps.size() ||
      (D.second && (static_cast<i64>(D.src2.size()) != D.records || static_cast<i64>(D.tail2.size()) != D.records)))
    fail(GR_EINVAL, "direct sweep check: table sizes");
  parallelFor(H.P, [&](i64 T) {
    const i64 base = H.tileStart[T], nRows = H.tileStart[T + 1] - base;
    const i64 nHalo = D.kind == RingKind::GaussSeidel ? H.tiles[T].nHalo : 0;
    const i64 start = gs && !D.gsInPlace ? nRows : 0;
    const i64 slots = start + nRows + nHalo + 1;
    if (gs && D.haloStart[T + 1] - D.haloStart[T] != nHalo) bad(T, "halo cells");
    if (slots > D.maxXSlots || slots > kDirectMaxSlots || nRows > D.maxRows) bad(T, "slots");
    const uint32_t* head = D.steps.data() + D.stepStart[T];
    const i64 nS = D.stepStart[T + 1] - D.stepStart[T] - kDirectHead - kDirectAhead;
    if (nS < 0 || nS + kDirectHead + kDirectAhead > D.maxSteps || head[2] != static_cast<uint32_t>(nS) ||
        head[1] > head[2] || head[1] % kDirectUnroll != 0 || head[2] % kDirectUnroll != 0 || (gs && head[1] != 0))
      bad(T, "steps");
    const uint32_t* steps = head + kDirectHead;
    for (i64 s = nS; s < nS + kDirectAhead; ++s)
      if (steps[s] != 0) bad(T, "steps after the last");
    if (gs) {
      for (i64 h = 0; h < nHalo; ++h) {
        const i32 src = D.haloSrc[D.haloStart[T] + h];
        if (src < 0 || src >= H.n || (src >= base && src < base + nRows)) bad(T, "halo source");
      }
    }
    // The level phase (barrier count) in which a row of the sweep was
    // written, -1 before.
    std::vector<i64> wroteLo(nRows, -1), wroteUp(nRows, -1);
    // The kernel takes a tile's first block and adds up the steps' sizes.
    i64 unit = D.stepUnit[D.stepStart[T]];
    i64 phase = 0;
    bool ended = true;
    for (i64 s = 0; s < nS; ++s) {
      const uint32_t w = steps[s];
      const i64 k = w & 0xFFu;
      const bool upper = !gs && s >= head[1];
      if (!gs && s == head[1] && !ended) bad(T, "sweep order");
      const i64 rows = (k + kDirectAlign - 1) / kDirectAlign * kDirectAlign;
      const i64 nLong = (w >> kDirectLongShift) & 0xFFu, units = blockBytes(D.valueBytes, w) / 16;
      i64 rec = D.stepRecord[D.stepStart[T] + kDirectHead + s];
      if (k > threads || rec + rows > D.records || nLong > k || (nLong > 0 && !D.second) || (!gs && !upper && nLong > 0 && !D.longForward) ||
          (w >> kDirectUnitShift) != units || unit + units > D.units ||
          unit != D.stepUnit[D.stepStart[T] + kDirectHead + s])
        bad(T, "step range");
      unit += units;
      if (k == 0 ? (!ended || w != 0) : ((w & kDirectDiag) != 0) != (gs || upper || D.dilu)) bad(T, "step flags");
      if (k > 0) ended = false;
      std::vector<i64>& wrote = upper ? wroteUp : wroteLo;
      for (i64 q = 0; q < k; ++q, ++rec) {
        const uint32_t tail = D.tail[rec];
        const i64 r = (tail >> 16) / 4;
        if (r >= nRows || wrote[r] >= 0 || (tail >> 16) % 4 != 0) bad(T, "row");
        std::vector<i64> want, wantC;
        eachEntry(H, D.kind, upper, base + r, r, nRows, [&](i64 e) {
          want.push_back(e);
          const i64 lc = H.colLocal[e];
          wantC.push_back(4 * (gs && lc >= r ? start + lc : lc));
        });
        const int4 a = D.src[rec], b = D.second ? D.src2[rec] : make_int4(-1, -1, -1, 0);
        const i64 e[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
        const uint32_t ca = static_cast<uint32_t>(a.w), cb = static_cast<uint32_t>(b.w);
        const i64 c[6] = {ca & 0xFFFFu, ca >> 16, tail & 0xFFFFu, cb & 0xFFFFu, cb >> 16,
                          D.second ? D.tail2[rec] : 0};
        const size_t read = q < nLong ? 6 : 3;
        if (want.size() > read) bad(T, "entries");
        for (size_t j = 0; j < read; ++j) {
          if (j >= want.size()) {
            if (e[j] != -1 || c[j] != 4 * (slots - 1)) bad(T, "padding");
            continue;
          }
          if (e[j] != want[j] || c[j] != wantC[j] || c[j] < 0 || c[j] >= 4 * (slots - 1)) bad(T, "entry");
          const i64 lc = H.colLocal[want[j]];
          if (lc >= nRows) continue;  // halo
          if (gs && lc > r) {
            if (D.gsInPlace && wroteLo[lc] >= 0) bad(T, "start value overwritten");
            if (D.gsInPlace && H.lowerLevel[base + lc] <= H.lowerLevel[base + r]) bad(T, "start value in its level");
          } else {
            const i64 when = (upper ? wroteUp : wroteLo)[lc];
            const bool leftOut = !upper && !gs && !D.dilu && H.lowerLevel[base + lc] == 0;
            if (when >= phase || (when < 0 && !leftOut)) bad(T, "dependency order");
          }
        }
        wrote[r] = phase;
      }
      if (w & kDirectEnd) {
        ended = true;
        ++phase;
      }
    }
    if (!ended) bad(T, "after the last step");
    if (D.factors) {
      // The levels cover the forward steps in order; an entry's transpose is
      // the entry of its column's row, and no other entry of the two rows
      // shares a column (not checked for DILU, which changes no entry).
      i64 l = D.levelStart[T], at = D.stepStart[T] + kDirectHead;
      const i64 stop = at + head[1];
      for (; l < D.levelStart[T + 1]; ++l) {
        const int4 v = D.levels[l];
        if (at >= stop || v.z != at || v.x != static_cast<i64>(D.stepRecord[at])) bad(T, "level start");
        i64 k = 0, nl = 0;
        for (bool more = true; more; ++at) {
          if (at >= stop || (k > 0 && k % threads != 0)) bad(T, "level steps");
          if (static_cast<i64>(D.stepRecord[at]) != v.x + k) bad(T, "level records");
          k += D.steps[at] & 0xFFu;
          nl += (D.steps[at] >> kDirectLongShift) & 0xFFu;
          more = (D.steps[at] & kDirectEnd) == 0;
        }
        if ((v.y & 0xFFFF) != k || (v.y >> 16) != nl) bad(T, "level rows");
        for (i64 q = 0; q < k; ++q) {
          const i64 r = (D.tail[v.x + q] >> 16) / 4;
          const int4 a = D.transposed.at(v.w + q), b = D.longForward ? D.transposed2.at(v.w + q) : make_int4(-1, -1, -1, 0);
          const i32 t[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
          int m = 0;
          eachEntry(H, D.kind, false, base + r, r, nRows, [&](i64 e) {
            const i64 c = H.colLocal[e];
            const i64 p0 = H.rowPtr[base + c], p1 = H.rowPtr[base + c + 1];
            if (t[m] < 0 ? entryAt(H, base + c, r) >= 0 : (t[m] < p0 || t[m] >= p1 || H.colLocal[t[m]] != r))
              bad(T, "transpose");
            for (i64 j = e + 1; !D.dilu && j < H.rowPtr[base + r + 1] && H.colLocal[j] < nRows; ++j)
              if (entryAt(H, base + c, H.colLocal[j]) >= 0) bad(T, "fill-in");
            ++m;
          });
          for (; m < 6; ++m)
            if (t[m] != -1) bad(T, "transpose padding");
        }
      }
      while (at < stop && D.steps[at] == 0) ++at;
      if (at != stop) bad(T, "levels end");
    }
    for (i64 r = 0; r < nRows; ++r) {
      if (wroteLo[r] < 0 && (gs || D.dilu || H.lowerLevel[base + r] != 0)) bad(T, "row not covered");
      if (!gs && wroteUp[r] < 0) bad(T, "row not covered");
    }
  });
}

size_t directSmem(const DirectPlan& P, DType coefficients, DType W, i32 depth) {
  const size_t rec = coefficients == DType::F32 ? (P.second ? 44 : 24) : (P.second ? 72 : 40);
  const i64 rhs = P.kind == RingKind::Ilu ? 0 : (P.maxRows + 3) / 4 * 4;
  return rec * static_cast<size_t>(depth) * 32 * static_cast<size_t>(P.warps) +
         static_cast<size_t>((P.maxXSlots + 3) / 4 * 4 + rhs) * dtypeSize(W) + 4 * static_cast<size_t>(P.maxSteps);
}

double rowsPerLevel(const HostMatrix& H) {
  i64 levels = 1;
  for (i32 l : H.nLowerLevels) levels += l;
  return static_cast<double>(H.n) / static_cast<double>(levels);
}

// What counts is how many tiles share an SM (t), how many rows a level has,
// how many tiles are resident at once, and whether the sweep's data stay in
// L2; results do not depend on the shape. All figures: us on B200, level ring
// -> direct, back-to-back applications; e/P: e^3 grid in P tiles, m: the
// permuted hexahedral mesh.
//
// ILU, float vectors. Warps: with t <= 1 a wide level needs four (64/64, 89
// rows a level: 37.0 -> 18.6, two 20.7), a narrow one two (32/64, 23 rows:
// 16.5 -> 8.4). Up to two tiles an SM, four from 80 rows a level on (128/296:
// 65.6 -> 43.2, two 47.4; below, 96/300: 39.6 -> 28.0, four 31.9). Then two
// while a level fills them (128/512, 89 rows: 46.3 -> 39.1; 160/600, 119 rows:
// 118.9 -> 100.1, one 108.7), else one (64/512: 18.6 -> 10.4; 128/1024: 41.2 ->
// 35.0, two 41.0); tiles of several waves with levels beyond 80 rows, two
// (192/1184: 125.9 -> 125.5, one 148). Depth: 8, or 4 where that saves a wave
// (160/1370: 91.7 -> 80.0, with 8 103.7; 176/4096, 1.5 waves for 2.3: 99.3,
// with 8 104.9; in as many waves, 192/2368: 109.4, with 8 104.8, ring 104.9).
// Direct in several waves ran at 0.84 to 1.10 of the ring's time over 60
// grids, with no line between them, and its set-up takes half as long, so it
// is kept (176x160x172/2595: 104.2 -> 88; 176/2000: 98.8 -> 108). Ring for
// wide levels on five to seven tiles an SM with data beyond L2, if its blocks
// then all fit beside a ring of 16 KB (144/800: 59.5, 69.7; 140/850: 57.2, 64;
// 150/1000: 67.7, 78; not where it needs a second wave, 150/900: 95.0 -> 81,
// nor in L2, m100/700: 30.8 -> 22.7).
// Narrow levels cost the ring its hand-overs (2048^2 in 2368 tiles, 20 rows:
// 150.2 -> 91.5, a chain of 2^20 rows in 1024: 1154 -> 207).
//
// ILU, double vectors. A step costs twice the cycles, so that few resident
// warps no longer hide DRAM. Float coefficients: ring beyond about 165 MB
// with up to ten tiles an SM and more than 40 rows a level (160/600: 151.6,
// direct 160.7; 160/1370: 138.3, 154; 144/1300: 89.9, 110; more tiles,
// 160/2048: 110 -> 102; below, 128/1024: 66.4 -> 46.9); beyond half of L2 for
// wide levels on up to 2.5 tiles an SM (128/148: 107.5, 125; 112/300: 73.5,
// 89; 96/148: 51.4 -> 43) and on little more than four (130x107x112/609: 51.2,
// 59.5; 112/750: 45.1, 45.3). Double coefficients: ring for more than one and a
// quarter waves, for up to four tiles an SM (wide levels: five) beyond L2
// (128/148: 105.5, 125; 112/300: 73.9, 95; 112/450: 47.3, 52.1; 120/640: 53.4,
// 59.9; 128/512: 57.4, 56.3; below, 96/148: 49.3 -> 43.3) or up to five whose
// rings all fit (101x122x116/599: 49.2, 57.5; not 130x107x112/609: 71.4 ->
// 61.6) and from three on already in L2 (96/560: 32.9, 35.0; m100/700: 32.8, 37.0); else direct
// (128/1024: 67.0 -> 49.2, 96/1200: 47.3 -> 33.5).
//
// Gauss-Seidel (two sweeps; a row costs a division and up to six entries).
// Float coefficients: direct always; four warps with t <= 2, two from 45 rows
// a level on (128/1024: 78.0 -> 65.9, 160/1370: 264.5 -> 153.6, m100/1024:
// 49.4 -> 40.8, 192/1184 with double vectors: 1591 -> 1145). Double
// coefficients, whose divisions keep the ring's warps as busy: direct with
// t > 4 in one wave (one warp; m100/1024: 86.2 -> 62, 64/1000: 49.3 -> 33.0;
// 109x80x107/931, 1.05 waves: 82, 107) and on few tiles of very wide levels
// (four warps; m100/256, 202 rows: 97 -> 64, m80/148: 49.3 -> 45.2). Between,
// the ring: 96/432: 61.4, direct 82; 112/450: 127, 242; m80/400: 37.1, 53;
// 80/256: 49.9, 57.
DirectShape directShape(const HostMatrix& H, RingKind kind, DType coefficients, DType vec, i32 numSMs,
                        i64 smemPerSM) {
  const bool gs = kind != RingKind::Ilu, f32 = coefficients == DType::F32;
  i64 halo = 0;
  for (const HostMatrix::Tile& tile : H.tiles) halo = std::max(halo, tile.nHalo);
  const double t = static_cast<double>(H.P) / numSMs, rows = rowsPerLevel(H);
  // Waves of blocks with room for second triples, copying d steps ahead.
  const i64 vs = static_cast<i64>(dtypeSize(vec)), rec = f32 ? 44 : 72;
  auto waves = [&](i32 warps, i32 d, i64 vs) {
    i64 steps = 0;  // of the longest tile, at most
    for (i32 T = 0; T < H.P; ++T) {
      const i64 nRows = H.tileStart[T + 1] - H.tileStart[T];
      steps = std::max(steps, H.nLowerLevels[T] + (gs ? 0 : H.nUpperLevels[T]) + (gs ? 1 : 2) * (nRows / (32 * warps)));
    }
    const i64 block = vs * (gs ? 2 * H.maxTileRows + halo : H.maxTileRows) + rec * d * 32 * warps +
                      4 * (steps + kDirectHead + kDirectAhead) + 1024;
    const i64 slots = smemPerSM / block * numSMs;
    return slots > 0 ? static_cast<double>(H.P) / static_cast<double>(slots) : 1e9;
  };
  if (gs) {
    i32 warps = t <= 2 ? 4 : rows > 45 ? 2 : 1;
    if (!f32) {
      warps = t <= 2 && rows > 150 ? 4 : t > 4 ? 1 : 0;
      if (warps == 0 || waves(warps, kDirectGsDepth, vs) > 1) return {};
    }
    return {warps, kDirectGsDepth};
  }
  const i32 warps = t <= 1                               ? (rows > 40 ? 4 : 2)
                    : t <= 2                             ? (rows > 80 ? 4 : 2)
                    : t <= 4                             ? (rows > 40 ? 2 : 1)
                    : t <= 6                             ? (rows > 64 ? 2 : 1)
                    : rows > 80 && waves(1, 8, 4) > 1.3 ? 2
                                                         : 1;
  const double w8 = waves(warps, 8, vs), w4 = waves(warps, 4, vs);
  const i32 depth = w8 > 1 && std::ceil(w4) < std::ceil(w8) ? 4 : 8;
  // A seven-point grid's coefficients and two vectors.
  const double mb = static_cast<double>(H.n) * (f32 ? 50 + 2 * vs : 116) * 1e-6;
  // What a level ring's block may use beside its x when all tiles are resident
  // at once. Rings take 16 KB (float) or twice their widest level (double),
  // and 1.5 KB of barriers and level table.
  const double room = static_cast<double>(smemPerSM) / std::ceil(t) -
                      static_cast<double>(vs) * static_cast<double>(H.maxTileRows) - 1024;
  bool ring;
  if (!f32) {
    ring = (depth == 4 ? w4 : w8) > 1.25 || (rows > 40 && t <= (rows > 64 ? 5 : 4) && (mb > 120 || t > 3)) ||
           (rows > 40 && t <= 5 && mb > 120 && room > 23.3e3);
  } else if (vec == DType::F64) {
    ring = (mb > 165 && rows > 40 && t <= 10) ||
           (mb > 66 && ((rows > 80 && t <= 2.5) || (rows > 55 && t > 4 && t <= 5)));
  } else {
    ring = mb > 100 && rows > 64 && t > 4.5 && room > 17.5e3;
  }
  if (ring) return {};
  return {warps, depth};
}

const DirectShape& DeviceMatrix::directShapeFor(RingKind kind, DType vec) {
  const auto [at, made] = directShapes.try_emplace({static_cast<int>(kind), static_cast<int>(vec)});
  if (made) {
    int perSM = 0;
    GR_CUDA(cudaDeviceGetAttribute(&perSM, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
    at->second = directShape(*host, kind, vt, vec, numSMs, perSM);
  }
  return at->second;
}

DirectPlan* DeviceMatrix::directPlan(RingKind kind, bool dilu, i32 warps, i32 depth, size_t smemMax) {
  std::unique_ptr<DirectPlan>& slot = directPlans[std::make_tuple(static_cast<int>(kind), dilu, warps)];
  auto usable = [&](const DirectPlan& R) { return R.accepted && directSmem(R, vt, DType::F64, depth) <= smemMax; };
  if (slot && (slot->resident || !usable(*slot))) return usable(*slot) ? slot.get() : nullptr;
  auto R = std::make_unique<DirectPlan>();
  R->accepted = directFits(*host, kind);
  if (R->accepted) {
    const HostDirect D = buildDirect(*host, kind, dilu, warps, vt);
    R->kind = kind;
    R->dilu = dilu;
    R->second = D.second;
    R->longForward = D.longForward;
    R->gsInPlace = D.gsInPlace;
    R->warps = warps;
    R->maxSteps = D.maxSteps;
    R->records = D.records;
    R->units = D.units;
    R->maxRows = D.maxRows;
    R->maxXSlots = D.maxXSlots;
    if (usable(*R)) {
      R->src.upload(D.src);
      R->tail.upload(D.tail);
      if (D.second) {
        R->src2.upload(D.src2);
        R->tail2.upload(D.tail2);
      }
      // Chains, whose levels are single rows, on more than a tile an SM
      // factorise apart: the many streams of the fused factorisation cost more
      // than its launches save (2^20 rows in 1024 tiles: 2.8 ms, with separate
      // kernels 1.5; in 256 tiles 5.5 and 4.9; 65,536 rows in 64 tiles, one an
      // SM: 0.9 and 1.2).
      R->factors = D.factors && (P <= numSMs || rowsPerLevel(*host) >= 2);
      if (R->factors) {
        R->levelStart.upload(D.levelStart);
        R->levels.upload(D.levels);
        R->transposed.upload(D.transposed);
        if (D.longForward) R->transposed2.upload(D.transposed2);
      }
      R->steps.upload(D.steps);
      R->stepStart.upload(D.stepStart);
      R->stepRecord.upload(D.stepRecord);
      R->stepUnit.upload(D.stepUnit);
      if (kind != RingKind::Ilu) {
        R->haloStart.upload(D.haloStart);
        if (!D.haloSrc.empty()) R->haloSrc.upload(D.haloSrc);
      }
      R->resident = true;
    }
  }
  slot = std::move(R);
  return usable(*slot) ? slot.get() : nullptr;
}

}  // namespace gr
