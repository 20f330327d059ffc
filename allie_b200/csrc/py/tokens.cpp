// Token ids of many games in one call, straight from the Python objects (loaded with ctypes.PyDLL, so
// the interpreter lock is held throughout).  The Python statement of the same rules is
// UCITokenizer.token_ids: 12 to 14 us per game of 150 plies (strings hashed before or not) against 2 here, in a batch of
// 256, which is what a batch of a few hundred prompts waits for before its first kernel.
//
// Ids are the tokenizer's dictionary's as it is at the call.  Moves of the usual form (two squares, an optional promotion
// piece) come from a table by their squares, laid out again whenever the dictionary has changed; any other string is
// looked up.  (All of them looked up, a batch of 30 games waits 30 us longer: the dictionary is not in the caches.)  A game
// that is not plain (other types than the usual ones, anything the Python rules would refuse) is
// left to the Python statement: its entry of `lens` is -1 and it adds nothing to the ids.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <vector>

namespace {

struct Ref {                               // one owned reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

// index of a move in the table: from square, to square, promotion (none, q, r, b, n); -1 for other strings
inline int move_index(const Py_UCS1* s, Py_ssize_t n) {
  if (n != 4 && n != 5) return -1;
  const unsigned a = s[0] - 'a', b = s[1] - '1', c = s[2] - 'a', d = s[3] - '1';
  if ((a | b | c | d) > 7) return -1;
  int promo = 0;
  if (n == 5) {
    promo = s[4] == 'q' ? 1 : s[4] == 'r' ? 2 : s[4] == 'b' ? 3 : s[4] == 'n' ? 4 : -1;
    if (promo < 0) return -1;
  }
  return promo * 4096 + static_cast<int>((a * 8 + b) * 64 + c * 8 + d);
}

// A number that no other dictionary of this process and no other state of this one has; 0 where the interpreter keeps none
inline uint64_t dict_version(PyObject* d) {
#if PY_VERSION_HEX < 0x030D0000
#pragma GCC diagnostic push
#pragma GCC diagnostic ignored "-Wdeprecated-declarations"
  return reinterpret_cast<PyDictObject*>(d)->ma_version_tag;
#pragma GCC diagnostic pop
#else
  return 0;
#endif
}

// Kept by the tokenizer between calls, all zero at first.
struct MoveTable {
  uint64_t version;                        // dict_version that the ids are of
  int32_t id[5 * 4096];                    // by move_index; -1: ask the dictionary
};

struct Tokens {
  PyObject *ids, *outcomes;                // dictionaries: token -> id, outcome -> mask
  long unk, vocab, resigned, eos;
  MoveTable* table;

  // 20 us
  void lay_out(uint64_t version) const {
    table->version = version;
    for (int32_t& x : table->id) x = -1;
    PyObject *k, *v;
    Py_ssize_t at = 0;
    while (PyDict_Next(ids, &at, &k, &v)) {
      if (!PyUnicode_CheckExact(k) || !PyUnicode_IS_COMPACT_ASCII(k) || !PyLong_CheckExact(v)) continue;
      const int m = move_index(PyUnicode_1BYTE_DATA(k), PyUnicode_GET_LENGTH(k));
      int overflow = 0;
      const long x = PyLong_AsLongAndOverflow(v, &overflow);
      if (m >= 0 && !overflow && x >= 0 && x <= 0x7fffffff) table->id[m] = static_cast<int32_t>(x);
    }
  }

  // id of a token in the dictionary, `unk` without one; false when Python raised or the id is no small int
  bool lookup(PyObject* token, uint32_t* out) const {
    PyObject* v = PyDict_GetItemWithError(ids, token);
    if (!v) {
      if (PyErr_Occurred()) return false;
      *out = static_cast<uint32_t>(unk);
      return true;
    }
    const long x = PyLong_CheckExact(v) ? PyLong_AsLong(v) : -1;
    if (x < 0 || x > 0x7fffffff) return false;
    *out = static_cast<uint32_t>(x);
    return true;
  }

  bool rating(PyObject* game, const char* name, std::vector<uint32_t>& row) const {
    Ref r(PyObject_GetAttrString(game, name));
    if (!r.p || !PyLong_CheckExact(r.p)) return false;
    int overflow = 0;
    const long long v = PyLong_AsLongLongAndOverflow(r.p, &overflow);
    if (overflow || v < -0x40000000LL || v > 0x40000000LL || v + vocab < 0) return false;
    row.push_back(static_cast<uint32_t>(v + vocab));
    return true;
  }

  // appends the ids of a plain game; false (and possibly a pending exception) for any other
  bool game(PyObject* g, std::vector<uint32_t>& row) const {
    if (!rating(g, "white_elo", row) || !rating(g, "black_elo", row)) return false;
    Ref tc(PyObject_GetAttrString(g, "time_control"));
    uint32_t id;
    if (!tc.p || !PyUnicode_CheckExact(tc.p) || !lookup(tc.p, &id)) return false;
    row.push_back(id);
    Ref moves(PyObject_GetAttrString(g, "moves")), secs(PyObject_GetAttrString(g, "moves_seconds"));
    if (!moves.p || !secs.p || !PyList_CheckExact(moves.p) || !PyList_CheckExact(secs.p) ||
        PyList_GET_SIZE(moves.p) != PyList_GET_SIZE(secs.p))
      return false;
    const uint64_t version = dict_version(ids);
    if (version && version != table->version) lay_out(version);
    // exact strings and ints only from here on: no Python code runs that could change the lists
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(moves.p); ++i) {
      PyObject *m = PyList_GET_ITEM(moves.p, i), *t = PyList_GET_ITEM(secs.p, i);
      if (!PyUnicode_CheckExact(m) || !PyLong_CheckExact(t)) return false;
      int overflow = 0;
      const long long sec = PyLong_AsLongLongAndOverflow(t, &overflow);
      if (overflow > 0 || (overflow == 0 && sec >= 0xFFFF)) return false;
      const int k = version && PyUnicode_IS_COMPACT_ASCII(m)
                        ? move_index(PyUnicode_1BYTE_DATA(m), PyUnicode_GET_LENGTH(m)) : -1;
      if (k >= 0 && table->id[k] >= 0) id = static_cast<uint32_t>(table->id[k]);
      else if (!lookup(m, &id)) return false;
      row.push_back(id);
    }
    Ref normal(PyObject_GetAttrString(g, "normal_termination")), outcome(PyObject_GetAttrString(g, "outcome"));
    if (!normal.p || !outcome.p) return false;
    const int yes = PyObject_IsTrue(normal.p);
    if (yes < 0) return false;
    if (yes) row.push_back(static_cast<uint32_t>(resigned));
    if (outcome.p != Py_None) {
      if (!PyUnicode_CheckExact(outcome.p) || PyDict_Contains(outcomes, outcome.p) != 1) return false;
      row.push_back(static_cast<uint32_t>(eos));
    }
    return true;
  }
};

}  // namespace

// games: list; table: a MoveTable.  Returns (ids, lens): the ids & 0x3fff of all plain games behind one another, each cut to
// max_length, as bytes of uint32; and a count per game as bytes of int32 (-1: not plain).  Null with an
// exception set when memory runs out.
extern "C" PyObject* allie_token_rows(PyObject* games, PyObject* ids, PyObject* outcomes, void* table,
                                      long unk, long vocab, long resigned, long eos, long max_length) {
  if (!PyList_CheckExact(games) || !PyDict_CheckExact(ids) || !PyDict_CheckExact(outcomes) || max_length < 0) {
    PyErr_SetString(PyExc_TypeError, "a list of games and two dictionaries expected");
    return nullptr;
  }
  try {
    const Tokens tok{ids, outcomes, unk, vocab, resigned, eos, static_cast<MoveTable*>(table)};
    std::vector<uint32_t> all, row;
    std::vector<int32_t> lens;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(games); ++i) {      // attribute access may run Python code
      Ref g(Py_NewRef(PyList_GET_ITEM(games, i)));
      row.clear();
      if (!tok.game(g.p, row)) {
        PyErr_Clear();                     // raised again by the Python statement of the rules
        lens.push_back(-1);
        continue;
      }
      if (row.size() > static_cast<size_t>(max_length)) row.resize(max_length);
      for (uint32_t v : row) all.push_back(v & 0x3FFFu);
      lens.push_back(static_cast<int32_t>(row.size()));
    }
    Ref a(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(all.data()), all.size() * 4));
    Ref b(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(lens.data()), lens.size() * 4));
    if (!a.p || !b.p) return nullptr;
    return PyTuple_Pack(2, a.p, b.p);
  } catch (...) {                          // std::bad_alloc must not leave through a C entry
    return PyErr_NoMemory();
  }
}
