// Checks bhsrc::tile_pixel on the host: "W H" frames on the command line, in full
// up to 2^22 pixels, else runs of pixels at the ends, in the middle and spread out.
// Every pixel must lie in the frame and no two may be the same.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "tile_order.h"

int main(int argc, char** argv) {
  int bad = 0;
  for (int k = 1; k + 1 < argc; k += 2) {
    const long long W = std::atoll(argv[k]), H = std::atoll(argv[k + 1]), n = W * H;
    std::vector<long long> ws, ps;
    if (n <= 1 << 22) {
      for (long long w = 0; w < n; ++w) ws.push_back(w);
    } else {
      for (long long at : {0LL, n / 3, n / 2, n - 5000})
        for (long long w = at; w < at + 5000; ++w) ws.push_back(w);
      for (long long i = 0; i < 50000; ++i) ws.push_back((long long)((double)i / 50000.0 * (double)(n - 1)));
      std::sort(ws.begin(), ws.end());
      ws.erase(std::unique(ws.begin(), ws.end()), ws.end());
    }
    long long out = 0;
    for (long long w : ws) {
      const long long p = bhsrc::tile_pixel(w, (int)W, n);
      if (p < 0 || p >= n) ++out;
      ps.push_back(p);
    }
    std::sort(ps.begin(), ps.end());
    const long long twice = (long long)(ps.end() - std::unique(ps.begin(), ps.end()));
    if (out || twice) {
      std::printf("%lld x %lld: %lld of %zu pixels outside the frame, %lld taken twice\n", W, H, out, ws.size(), twice);
      bad = 1;
    }
  }
  return bad;
}
