#include "speculable.hpp"

#include <cctype>
#include <map>
#include <set>
#include <string_view>
#include <unordered_map>
#include <vector>

namespace sodecl_b200 {

namespace {

enum class Kind { Ident, Number, Punct };

// The scan runs on every compilation and gradient call, so a word is looked up
// once, when it is read.
enum Class : unsigned char { kPlain = 0, kIntType = 1, kRefusedWord = 2, kKeyword = 4 };

struct Tok {
    Kind kind;
    std::string_view text;
    unsigned char cls = kPlain;
};

using Toks = std::vector<Tok>;
using Names = std::set<std::string_view>;

bool ident_start(char c) { return std::isalpha(static_cast<unsigned char>(c)) || c == '_'; }
bool ident_char(char c) { return std::isalnum(static_cast<unsigned char>(c)) || c == '_'; }

const std::string_view kIntTypes[] = {"int",   "unsigned", "signed", "long",   "short",    "char",      "size_t",   "ptrdiff_t",
                         "uint",  "ulong",    "ushort", "uchar",  "intptr_t", "uintptr_t", "int8_t",   "int16_t",
                         "int32_t", "int64_t", "uint8_t", "uint16_t", "uint32_t", "uint64_t", "wchar_t"};

const std::string_view kRefused[] = {"while",    "do",      "goto",  "switch",   "asm",       "__asm",    "__asm__",  "printf",
                        "template", "union",   "enum",  "typedef",  "using",     "namespace", "class",   "struct",
                        "auto",     "decltype", "typeof", "__typeof__", "operator", "new",    "delete",   "malloc",
                        "free",     "try",     "throw", "volatile", "reinterpret_cast", "const_cast", "__builtin_assume",
                        "sizeof",   "alignof", "extern", "__trap", "__syncthreads", "__syncwarp"};

bool vector_of_ints(std::string_view w)  // int2, uchar4, longlong2, ...
{
    if (w.size() < 4 || !std::isdigit(static_cast<unsigned char>(w.back()))) return false;
    size_t n = w.size();
    while (n > 0 && std::isdigit(static_cast<unsigned char>(w[n - 1]))) --n;
    std::string_view base = w.substr(0, n);
    if (!base.empty() && base[0] == 'u') base.remove_prefix(1);
    return base == "int" || base == "long" || base == "longlong" || base == "short" || base == "char";
}

unsigned char class_of(std::string_view w)
{
    static const std::unordered_map<std::string_view, unsigned char> words = [] {
        std::unordered_map<std::string_view, unsigned char> m;
        for (const auto t : kIntTypes) m[t] = kIntType;
        for (const auto t : kRefused) m[t] = kRefusedWord;
        for (const std::string_view t : {"double", "float", "if", "for", "const", "return"}) m[t] = kKeyword;
        return m;
    }();
    const auto it = words.find(w);
    if (it != words.end()) return it->second;
    return w.substr(0, 6) == "atomic" || vector_of_ints(w) ? kRefusedWord : kPlain;
}

// One logical line or the whole text into tokens; literals become one number
// token "0" or, for strings, an identifier nothing accepts.
void tokenize(std::string_view s, size_t i, size_t end, Toks &out)
{
    static const std::string_view three[] = {"<<=", ">>=", "..."};
    static const std::string_view two[] = {"++", "--", "+=", "-=", "*=", "/=", "%=", "&=", "|=", "^=", "==", "!=", "<=",
                                ">=", "&&", "||", "<<", ">>", "->", "##", "::"};
    while (i < end) {
        const char c = s[i];
        if (std::isspace(static_cast<unsigned char>(c)) || (c == '\\' && i + 1 < end && s[i + 1] == '\n')) {
            ++i;
        } else if (ident_start(c)) {
            size_t j = i + 1;
            while (j < end && ident_char(s[j])) ++j;
            out.push_back({Kind::Ident, s.substr(i, j - i), class_of(s.substr(i, j - i))});
            i = j;
        } else if (std::isdigit(static_cast<unsigned char>(c)) ||
                   (c == '.' && i + 1 < end && std::isdigit(static_cast<unsigned char>(s[i + 1])))) {
            size_t j = i + 1;
            while (j < end && (ident_char(s[j]) || s[j] == '.' ||
                               ((s[j] == '+' || s[j] == '-') && std::string_view("eEpP").find(s[j - 1]) != std::string_view::npos)))
                ++j;
            out.push_back({Kind::Number, s.substr(i, j - i)});
            i = j;
        } else if (c == '"' || c == '\'') {
            size_t j = i + 1;
            while (j < end && s[j] != c) j += (s[j] == '\\') ? 2 : 1;
            out.push_back({Kind::Ident, "\"literal\"", kRefusedWord});
            i = j + 1;
        } else {
            size_t n = 1;
            if (i + 1 < end && std::string_view("=+-&|<>:#.").find(s[i + 1]) != std::string_view::npos) {
                for (const std::string_view t : three)
                    if (s.substr(i, 3) == t) n = 3;
                for (const std::string_view t : two)
                    if (n == 1 && s.substr(i, 2) == t) n = 2;
            }
            const std::string_view p = s.substr(i, n);
            out.push_back({Kind::Punct, p});
            i += p.size();
        }
    }
}

bool int_literal(std::string_view w)
{
    const bool hex = w.size() > 2 && w[0] == '0' && (w[1] == 'x' || w[1] == 'X');
    for (const char c : w)
        if (c == '.' || (!hex && (c == 'e' || c == 'E' || c == 'f' || c == 'F')) || (hex && (c == 'p' || c == 'P')))
            return false;
    return true;
}

class Scan {
public:
    explicit Scan(std::string_view code)
    {
        split(code);
        if (!hazard_.empty()) return;
        collect();
        if (hazard_.empty()) check();
    }
    std::string hazard_;

private:
    struct Macro {
        std::string_view name;
        Toks body;
    };
    struct Function {
        size_t begin, end;          // its name's position, one past its body
        std::vector<bool> is_int;   // per parameter
        Names pointers;             // pointer and array parameters, local arrays
    };

    Toks t_;                  // the file without its directives, then every macro's body
    std::vector<Macro> macros_;
    Names index_ = {"_numeq_", "_numpar_", "_numnoi_", "_numsteps_", "_listsize_"};
    Names flags_;             // ints that hold a comparison
    Names tables_;            // arrays at file scope
    std::map<std::string_view, Function> functions_;
    std::vector<char> allowed_;  // positions whose assignment a for header or a declaration makes

    bool refuse(const std::string &why)
    {
        if (hazard_.empty()) hazard_ = why;
        return false;
    }
    bool is(size_t i, std::string_view s) const { return i < t_.size() && t_[i].text == s; }
    bool ident(size_t i) const { return i < t_.size() && t_[i].kind == Kind::Ident; }
    bool int_name(size_t i) const { return ident(i) && (index_.count(t_[i].text) || flags_.count(t_[i].text)); }

    // the matching closer of the opener at i, or npos
    size_t match(size_t i) const
    {
        const std::string_view open = t_[i].text, close = open == "(" ? ")" : open == "[" ? "]" : "}";
        int depth = 0;
        for (size_t k = i; k < t_.size(); ++k) {
            if (t_[k].text == open) ++depth;
            else if (t_[k].text == close && --depth == 0) return k;
        }
        return std::string::npos;
    }

    // tokens [a, b) make an int of literals, sizes and index names
    bool index_expr(size_t a, size_t b) const
    {
        if (a >= b) return false;
        for (size_t k = a; k < b; ++k) {
            const Tok &w = t_[k];
            if (w.kind == Kind::Number ? !int_literal(w.text)
                : w.kind == Kind::Ident
                    ? !index_.count(w.text)
                    : w.text != "+" && w.text != "-" && w.text != "*" && w.text != "/" && w.text != "%" && w.text != "(" &&
                          w.text != ")")
                return false;
        }
        return true;
    }

    // tokens [a, b) make a comparison or a logical expression: 0 or 1
    bool truth_expr(size_t a, size_t b) const
    {
        while (a < b && t_[a].text == "(" && match(a) == b - 1) ++a, --b;
        bool found = false;
        int depth = 0;
        for (size_t k = a; k < b; ++k) {
            const std::string_view w = t_[k].text;
            if (w == "(" || w == "[") ++depth;
            else if (w == ")" || w == "]") --depth;
            else if (depth == 0) {
                if (w == "<" || w == ">" || w == "<=" || w == ">=" || w == "==" || w == "!=" || w == "&&" || w == "||")
                    found = true;
                else if (w == "?" || w == "=" || w == "," || w == "&" || w == "|" || w == "^" || w == "{" || w == "<<" ||
                         w == ">>")
                    return false;
            }
        }
        return found;
    }

    // [a, b) at depth-0 commas
    std::vector<std::pair<size_t, size_t>> pieces(size_t a, size_t b, std::string_view sep) const
    {
        std::vector<std::pair<size_t, size_t>> out;
        int depth = 0;
        size_t from = a;
        for (size_t k = a; k < b; ++k) {
            const std::string_view w = t_[k].text;
            if (w == "(" || w == "[" || w == "{") ++depth;
            else if (w == ")" || w == "]" || w == "}") --depth;
            else if (depth == 0 && w == sep) {
                out.push_back({from, k});
                from = k + 1;
            }
        }
        out.push_back({from, b});
        return out;
    }

    // directives out of the text; macro bodies behind it, each closed by ';'
    void split(std::string_view s)
    {
        const size_t n = s.size();
        size_t i = 0;
        while (i < n) {
            size_t e = i;  // the logical line's end
            while (e < n && !(s[e] == '\n' && (e == 0 || s[e - 1] != '\\'))) ++e;
            size_t k = i;
            while (k < e && std::isspace(static_cast<unsigned char>(s[k]))) ++k;
            if (k < e && s[k] == '#') {
                Toks d;
                tokenize(s, k + 1, e, d);
                const std::string_view what = d.empty() ? std::string_view() : d[0].text;
                if (what == "define") {
                    if (d.size() < 2 || d[1].kind != Kind::Ident) { refuse("#define"); return; }
                    const std::string_view name = d[1].text;
                    if (d[1].cls == kIntType || d[1].cls == kKeyword) {
                        refuse("#define " + std::string(name));
                        return;
                    }
                    const size_t at = s.find(name, s.find("define", k) + 6) + name.size();
                    const bool function = at < e && s[at] == '(';
                    size_t from = 2;
                    Names arguments;
                    if (function) {
                        for (; from < d.size() && d[from].text != ")"; ++from)
                            if (d[from].kind == Kind::Ident) arguments.insert(d[from].text);
                        ++from;
                    }
                    Macro m{name, {}};
                    for (size_t q = from; q < d.size(); ++q) {
                        if (d[q].text == "##" || d[q].text == "#") { refuse("#" + std::string(name)); return; }
                        m.body.push_back(d[q]);
                        // whatever it stands for, it is no int of the file's
                        if (arguments.count(d[q].text)) m.body.back().text = "macro argument";
                    }
                    if (function) m.name = {};  // never an index by itself
                    macros_.push_back(m);
                } else if (what == "include" || what == "import" || what == "include_next") {
                    refuse("#include");
                    return;
                }
            } else {
                tokenize(s, i, e, t_);
            }
            i = e + 1;
        }
        t_.push_back({Kind::Punct, ";"});
        for (const Macro &m : macros_) {
            for (const Tok &w : m.body) t_.push_back(w);
            t_.push_back({Kind::Punct, ";"});
        }
        allowed_.assign(t_.size(), 0);
    }

    bool starts_statement(size_t i) const  // token i is the first of a statement
    {
        if (i == 0) return true;
        const std::string_view w = t_[i - 1].text;
        return w == ";" || w == "{" || w == "}" || w == ")" || w == "else" || w == ":" || w == "static" || w == "inline";
    }

    // int declarations, parameters, functions and macros: fills the name sets
    void collect()
    {
        // function definitions at file scope
        int brace = 0;
        for (size_t i = 0; i < t_.size(); ++i) {
            if (t_[i].text == "{") ++brace;
            else if (t_[i].text == "}") --brace;
            else if (brace == 0 && t_[i].text == "(" && i > 0 && t_[i - 1].kind == Kind::Ident) {
                const size_t close = match(i);
                if (close == std::string::npos) { refuse("unbalanced parentheses"); return; }
                if (is(close + 1, "{")) {
                    const size_t end = match(close + 1);
                    if (end == std::string::npos) { refuse("unbalanced braces"); return; }
                    Function f{i - 1, end + 1, {}, {}};
                    for (const auto &p : pieces(i + 1, close, ",")) {
                        bool whole = false;
                        for (size_t k = p.first; k < p.second; ++k) {
                            if ((t_[k].cls == kIntType)) whole = true;
                            if ((t_[k].text == "*" || t_[k].text == "&") && ident(k + 1)) f.pointers.insert(t_[k + 1].text);
                            if (t_[k].text == "[" && k > p.first && ident(k - 1)) f.pointers.insert(t_[k - 1].text);
                        }
                        f.is_int.push_back(whole);
                    }
                    for (size_t k = close; k + 2 < end; ++k)
                        if ((is(k, "double") || is(k, "float") || is(k, ",")) && ident(k + 1) && is(k + 2, "["))
                            f.pointers.insert(t_[k + 1].text);
                    if (functions_.count(t_[i - 1].text)) { refuse("two functions of one name"); return; }
                    functions_[t_[i - 1].text] = f;
                }
                i = close;
            } else if (brace == 0 && t_[i].text == "[" && i > 0 && ident(i - 1)) {
                tables_.insert(t_[i - 1].text);
            }
        }
        // object-like macros that are int expressions, in any order
        bool grown = true;
        for (int q = 0; grown && q < 8; ++q) {
            grown = false;
            size_t at = t_.size();
            for (size_t m = macros_.size(); m-- > 0;) {
                at -= macros_[m].body.size() + 1;
                if (!macros_[m].name.empty() && !index_.count(macros_[m].name) &&
                    index_expr(at, at + macros_[m].body.size())) {
                    index_.insert(macros_[m].name);
                    grown = true;
                }
            }
            for (size_t i = 0; i < t_.size(); ++i) {
                if (!(t_[i].cls == kIntType)) continue;
                size_t first = i;
                while (first > 0 && is(first - 1, "const")) --first;
                size_t j = i;
                while (j < t_.size() && ((t_[j].cls == kIntType) || is(j, "const"))) ++j;
                if (!declare(first, j)) return;
                i = j - 1;
            }
        }
        // a name that is an index in one place and a flag in another is no index
        for (const auto &f : flags_) index_.erase(f);
        // a macro defined twice counts as an index only if every body is one
        size_t at = t_.size();
        for (size_t m = macros_.size(); m-- > 0;) {
            at -= macros_[m].body.size() + 1;
            if (index_.count(macros_[m].name) && !index_expr(at, at + macros_[m].body.size())) index_.erase(macros_[m].name);
        }
    }

    // the declaration whose type starts at `first` and whose names start at j
    bool declare(size_t first, size_t j)
    {
        const bool in_for = first >= 2 && is(first - 1, "(") && is(first - 2, "for");
        const bool in_list = !in_for && first >= 1 && (is(first - 1, "(") || is(first - 1, ","));
        if (in_list) {
            if (!ident(j) || !(is(j + 1, ",") || is(j + 1, ")"))) return refuse("conversion to an integer type");
            index_.insert(t_[j].text);
            return true;
        }
        if (!in_for && !starts_statement(first)) return refuse("conversion to an integer type");
        for (size_t k = j;;) {
            if (!ident(k)) return refuse("integer declaration");
            const std::string_view name = t_[k].text;
            size_t e = k + 1;
            if (is(e, "=")) {
                int depth = 0;
                size_t q = e + 1;
                for (; q < t_.size(); ++q) {
                    const std::string_view w = t_[q].text;
                    if (w == "(" || w == "[") ++depth;
                    else if (w == ")" || w == "]") --depth;
                    else if (depth == 0 && (w == "," || w == ";")) break;
                }
                if (!flags_.count(name) && index_expr(e + 1, q)) index_.insert(name);
                else if (truth_expr(e + 1, q)) flags_.insert(name), index_.erase(name);
                else if (!unresolved(e + 1, q)) return refuse("integer " + std::string(name) + " from a value");
                allowed_[k] = 1;
                e = q;
            } else if (!flags_.count(name)) {
                index_.insert(name);
            }
            if (is(e, ";")) return true;
            if (!is(e, ",")) return refuse("integer declaration");
            k = e + 1;
        }
    }

    // an int expression but for names that a later round of collect may
    // resolve (a macro or an int declared further down); check() judges it
    bool unresolved(size_t a, size_t b) const
    {
        for (size_t k = a; k < b; ++k)
            if (t_[k].kind == Kind::Ident && !index_.count(t_[k].text)) return pending(t_[k].text);
        return false;
    }
    bool pending(std::string_view name) const
    {
        for (const Macro &m : macros_)
            if (m.name == name) return true;
        return false;
    }

    void check()
    {
        int brace = 0;
        for (size_t i = 0; i < t_.size() && hazard_.empty(); ++i) {
            const std::string_view w = t_[i].text;
            if (w == "{") ++brace;
            if (w == "}") --brace;
            if (t_[i].kind == Kind::Ident) {
                if (t_[i].cls == kRefusedWord) { refuse(w == "\"literal\"" ? "literal" : std::string(w)); return; }
                if (w == "static" && brace > 0) { refuse("static"); return; }
                if (w == "for") header(i);
                // an int's name with another type elsewhere (the sets have no scopes)
                if (i > 0 && ident(i - 1) && int_name(i) && !(t_[i - 1].cls == kIntType) && !is(i - 1, "const") &&
                    !is(i - 1, "return") && !is(i - 1, "else"))
                    refuse(std::string(w) + " of two types");
                if ((w == "double" || w == "float") && is(i + 1, "*") && brace > 0) { refuse("pointer"); return; }
                const auto f = functions_.find(w);
                if (f != functions_.end() && i != f->second.begin) {
                    if (is(i + 1, "(")) call(i, f->second);
                    else refuse("function " + std::string(w) + " as a value");
                }
            }
            if (w == "[") {
                const size_t close = match(i);
                if (close == std::string::npos) { refuse("unbalanced brackets"); return; }
                if (close > i + 1 && !index_expr(i + 1, close)) { refuse("subscript"); return; }
            }
            if (w == "&" && int_name(i + 1) && i > 0 && t_[i - 1].kind == Kind::Punct && !is(i - 1, ")") && !is(i - 1, "]"))
                refuse("address of an integer");
            // values: initialisers left open in collect
            if (allowed_[i] && is(i + 1, "=") && index_.count(w) == 0 && flags_.count(w) == 0) refuse("integer " + std::string(w) + " from a value");
        }
        for (size_t i = 0; i < t_.size() && hazard_.empty(); ++i) {
            const bool moved = assigned(i);
            if (moved && int_name(i) && !allowed_[i]) refuse("assignment to integer " + std::string(t_[i].text));
        }
        for (const auto &f : functions_)
            for (size_t i = f.second.begin; i < f.second.end && hazard_.empty(); ++i)
                if (ident(i) && (f.second.pointers.count(t_[i].text) || tables_.count(t_[i].text)) && pointer_moved(i))
                    refuse("pointer arithmetic on " + std::string(t_[i].text));
    }

    // an address other than an array's element is formed or assigned
    bool pointer_moved(size_t i) const
    {
        if (is(i + 1, "[")) return i > 0 && (is(i - 1, "++") || is(i - 1, "--"));
        const bool through = i > 0 && is(i - 1, "*");  // *c = ...
        if (assigned(i)) return !(through && is(i + 1, "="));
        return is(i + 1, "+") || is(i + 1, "-") || (i > 0 && (is(i - 1, "+") || is(i - 1, "-")));
    }

    bool assigned(size_t i) const
    {
        if (!ident(i)) return false;
        static const Names ops = {"=", "+=", "-=", "*=", "/=", "%=", "<<=", ">>=", "&=", "|=", "^=", "++", "--"};
        return (i + 1 < t_.size() && ops.count(t_[i + 1].text)) || (i > 0 && (is(i - 1, "++") || is(i - 1, "--")));
    }

    // for (int i = E; i < E; i++)
    bool header(size_t i)
    {
        if (!is(i + 1, "(")) return refuse("for");
        const size_t close = match(i + 1);
        if (close == std::string::npos) return refuse("for");
        const auto part = pieces(i + 2, close, ";");
        if (part.size() != 3) return refuse("for");
        size_t a = part[0].first;
        while (a < part[0].second && ((t_[a].cls == kIntType) || is(a, "const"))) ++a;
        for (const auto &p : pieces(a, part[0].second, ",")) {
            if (!ident(p.first) || !index_.count(t_[p.first].text) || !is(p.first + 1, "=") || !index_expr(p.first + 2, p.second))
                return refuse("for");
            allowed_[p.first] = 1;
        }
        a = part[1].first;
        if (!ident(a) || !index_.count(t_[a].text) || !(is(a + 1, "<") || is(a + 1, "<=") || is(a + 1, ">") || is(a + 1, ">=")) ||
            !index_expr(a + 2, part[1].second))
            return refuse("for");
        for (const auto &p : pieces(part[2].first, part[2].second, ",")) {
            const size_t n = p.second - p.first;
            size_t name = p.first;
            if (n == 2 && (is(p.first, "++") || is(p.first, "--"))) name = p.first + 1;
            else if (n == 2 && (is(p.first + 1, "++") || is(p.first + 1, "--"))) name = p.first;
            else if (n > 2 && (is(p.first + 1, "+=") || is(p.first + 1, "-=") || is(p.first + 1, "=")) &&
                     index_expr(p.first + 2, p.second))
                name = p.first;
            else return refuse("for");
            if (!ident(name) || !index_.count(t_[name].text)) return refuse("for");
            allowed_[name] = 1;
        }
        return true;
    }

    // a call of one of the file's functions: not its own, and ints for ints
    bool call(size_t i, const Function &f)
    {
        const size_t close = match(i + 1);
        if (close == std::string::npos) return refuse("call");
        if (is(close + 1, ";") && i > 0 && t_[i - 1].kind == Kind::Ident && !is(i - 1, "return") && !is(i - 1, "else"))
            return true;  // a prototype: a type stands before the name
        if (i < f.end) return refuse("recursion");
        const auto args = pieces(i + 2, close, ",");
        for (size_t k = 0; k < args.size() && k < f.is_int.size(); ++k)
            if (f.is_int[k] && !index_expr(args[k].first, args[k].second)) return refuse("integer argument");
        return true;
    }
};

}  // namespace

std::string speculation_hazard(const std::string &code) { return Scan(code).hazard_; }

}  // namespace sodecl_b200
