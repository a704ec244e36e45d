// Reading whitespace-separated words and integers from a spec text (host).
#pragma once
#include <climits>
#include <cstdlib>
#include <string>

namespace cz {

// A cursor over [p, end). The specs are long lists of small integers (a rus-spec holds 370,000), so integers are read in
// place; a string is made only for what the short path does not cover.
struct TextCursor {
  const char *p, *end;

  static bool space(char c) { return c == ' ' || (c >= '\t' && c <= '\r'); }   // isspace in the "C" locale
  void skip() { while (p < end && space(*p)) p++; }

  // the next word; false at the end
  bool word(std::string &out) {
    skip();
    if (p >= end) return false;
    const char *b = p;
    while (p < end && !space(*p)) p++;
    out.assign(b, p);
    return true;
  }
  // the value of the next word's leading integer (the rest of the word is passed over); false at the end or when the
  // word starts with none. As strtoll reads it: values out of range saturate.
  bool word_number(long long &v) {
    skip();
    if (p >= end) return false;
    const char *b = p, *q = p;
    const bool neg = *q == '-';
    if (*q == '-' || *q == '+') q++;
    const char *d = q;
    long long x = 0;
    while (q < end && *q >= '0' && *q <= '9' && q - d < 18) x = 10 * x + (*q++ - '0');
    const bool whole = q > d && (q >= end || space(*q));
    if (whole) {
      p = q;
      v = neg ? -x : x;
      return true;
    }
    while (p < end && !space(*p)) p++;                // more than 18 digits, or something else: through strtoll
    const std::string s(b, p);
    char *e;
    v = std::strtoll(s.c_str(), &e, 10);
    return e != s.c_str();
  }
  // the next int as a formatted stream reads it: sign and digits, stopping at the first other character; false when
  // there are no digits or the value does not fit
  bool stream_int(int &v) {
    skip();
    const bool neg = p < end && *p == '-';
    if (p < end && (*p == '-' || *p == '+')) p++;
    const char *d = p;
    long long x = 0;
    bool over = false;
    for (; p < end && *p >= '0' && *p <= '9'; p++) {
      if (x > INT_MAX) over = true;
      else x = 10 * x + (*p - '0');
    }
    if (neg) x = -x;
    if (p == d || over || x > INT_MAX || x < INT_MIN) return false;
    v = (int)x;
    return true;
  }
};

}  // namespace cz
